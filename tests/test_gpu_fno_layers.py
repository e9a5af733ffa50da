"""The warm-start network's fused layer kernels (pfc_b200/csrc/fno.cu) where they
can go wrong: the smallest and larger tiles, one tile, more tiles than a mixing
block's sixteen rows, and input tensors that start off a 16-byte boundary, against
the CPU oracle; and the GELU over its whole range through a network whose output
is the GELU of its input.

Tolerances as in test_gpu_fno: outputs to 1e-4 of the largest value, gradients to
2e-3 in relative L2 norm per parameter block (FP32 sums with BF16 weights against
float64)."""
import numpy as np
import pytest

from oracle import fno_oracle as O
from pfc_b200 import fno

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _params(seed):
    p = fno.init_params(seed, out_scale=1.0)
    rng = np.random.default_rng(seed)
    for k, (o, s) in fno.layout().items():
        n = int(np.prod(s))
        if k[:2] in ("Rr", "Ri"):
            p[o:o + n] = rng.uniform(-1, 1, n) * 0.02
        if k in ("p", "q") or k[0] == "b":
            p[o:o + n] = rng.uniform(-0.1, 0.1, n)
    return p


def _off(a, shift):
    """a on the device, starting `shift` floats after a 512-byte boundary."""
    buf = torch.empty(a.size + shift, dtype=torch.float32, device="cuda")
    v = buf[shift:].view(*a.shape)
    v.copy_(torch.tensor(a))
    return v


@pytest.mark.parametrize("T,B,shift", [(32, 17, 0), (32, 1, 1), (128, 2, 3), (256, 1, 0)])
def test_layers_match_oracle(T, B, shift):
    rng = np.random.default_rng(T + B)
    p = _params(T)
    x = rng.normal(scale=0.5, size=(B, 2, T, T)).astype(np.float32)
    t = (x + rng.normal(scale=0.1, size=x.shape)).astype(np.float32)
    with fno.Network(T, B) as net:
        net.set_params(p)
        dx, dt = _off(x, shift), _off(t, shift)
        dy, dy0 = torch.empty(x.shape, device="cuda"), torch.empty(x.shape, device="cuda")
        torch.cuda.synchronize()
        net.forward(_off(x, 0).data_ptr(), dy0.data_ptr(), B)
        net.forward(dx.data_ptr(), dy.data_ptr(), B)
        loss, g = net.loss_grad(dx.data_ptr(), dt.data_ptr(), B, want_grad=True)
    assert torch.equal(dy, dy0)
    loss_o, g_o, y_o = O.loss_and_grad(fno.bf16_round(p).astype(np.float64), x, t)
    assert np.abs(dy.cpu().numpy() - y_o).max() < 1e-4 * np.abs(y_o).max()
    assert abs(loss - loss_o) < 1e-4 * loss_o
    for k, (o, s) in fno.layout().items():
        n = int(np.prod(s))
        err = np.linalg.norm(g[o:o + n] - g_o[o:o + n]) / max(np.linalg.norm(g_o[o:o + n]), 1e-30)
        assert err < 2e-3, (k, err)


def test_gelu_over_its_range():
    """W0 = I on channel 0, the other layers pass it on far in GELU's linear range:
    the output less the input is GELU(x0) to FP32 rounding of the added offset."""
    T = 32
    p = np.zeros(fno.NPARAM, dtype=np.float32)
    lay = fno.layout()

    def put(name, idx, v):
        o, s = lay[name]
        p[o + np.ravel_multi_index(idx, s)] = v

    put("P", (0, 0), 1.0)
    for l in range(fno.LAYERS):
        put("W%d" % l, (0, 0), 1.0)
    for l in (1, 2):
        put("b%d" % l, (0,), 16.0)  # GELU(z + 16) = z + 16 to FP32
    put("b3", (0,), -32.0)
    put("Q", (1, 0), 1.0)
    z = np.linspace(-12, 12, T * T, dtype=np.float32).reshape(T, T)
    x = np.stack([z, np.zeros_like(z)])[None]
    with fno.Network(T, 1) as net:
        net.set_params(p)
        dx = torch.tensor(x, device="cuda")
        dy = torch.empty_like(dx)
        torch.cuda.synchronize()
        net.forward(dx.data_ptr(), dy.data_ptr(), 1)
    got = dy.cpu().numpy()[0, 1].astype(np.float64)
    want = torch.nn.functional.gelu(torch.tensor(z, dtype=torch.float64)).numpy()
    # offsets of 16 and 32 on values up to 12: four roundings at 2^-19, and the products'
    # BF16 splits, 2^-16 of the largest operand (44) each in four layers
    assert np.abs(got - want).max() < 4 * 2.0 ** -19 + 4 * 44 * 2.0 ** -16
    assert np.all(np.isfinite(got))


def test_lifted_modes_are_fp32_sums():
    """The modes of the lifted input are FP32 sums, which all channels share: of a wave
    above the retained modes they are zero but for rounding. With W0 = 0 and one
    channel's K0 = 1 the first layer's z is the field of those errors. A row's sum of 64
    products in FP32 is off by about 2^-25 of its partial sums, 40 of them in rms, which
    makes 128 modes of 64 rows 5e-8 of the field in rms; sums of BF16 pairs (2^-18 a
    product) make 4.7e-7. Three GELUs near zero halve it each."""
    T = 64
    p = np.zeros(fno.NPARAM, dtype=np.float32)
    lay = fno.layout()

    def put(name, idx, v):
        o, s = lay[name]
        p[o + np.ravel_multi_index(idx, s)] = v

    put("P", (0, 0), 1.0)
    for ky in range(16):
        for kx in range(8):
            put("Rr0", (0, 0, ky, kx), 1.0)
    for l in (1, 2, 3):
        put("W%d" % l, (0, 0), 1.0)
    put("Q", (1, 0), 1.0)
    x = np.zeros((1, 2, T, T), dtype=np.float32)
    i = np.arange(T)
    x[0, 0] = np.cos(2 * np.pi * (20 * i[None, :] + 9 * i[:, None]) / T + 0.3)
    with fno.Network(T, 1) as net:
        net.set_params(p)
        dx = torch.tensor(x, device="cuda")
        dy = torch.empty_like(dx)
        torch.cuda.synchronize()
        net.forward(dx.data_ptr(), dy.data_ptr(), 1)
    want = O.loss_and_grad(fno.bf16_round(p).astype(np.float64), x, x)[2][0, 1]
    err = np.abs(dy.cpu().numpy()[0, 1] - want).max() * 8
    assert err < 1.5e-7, err


@pytest.mark.parametrize("T", [32, 128])
def test_transform_and_bias_round_once(T):
    """A layer's inverse transform is a sum of its own, added to the bias in FP32: with
    W3 = 0, b3 = 1 and a transform of a few 2^-13 the last layer's z = 1 + s is off by
    half a unit in the last place, 2^-24, and by s's own error, 2^-16 of 2^-12 (products
    of values split into BF16 pairs). Sums that carry the bias through the tensor
    core, which does not round to nearest, are off by several times as much."""
    p = np.zeros(fno.NPARAM, dtype=np.float32)
    lay = fno.layout()

    def put(name, idx, v):
        o, s = lay[name]
        p[o + np.ravel_multi_index(idx, s)] = v

    put("P", (0, 0), 1.0)
    for l in range(3):
        put("W%d" % l, (0, 0), 1.0)
    put("b3", (0,), 1.0)
    for k in range(1, 7):
        put("Rr3", (0, 0, k, k), 2.0 ** -11)
        put("Ri3", (0, 0, k, 7 - k), -2.0 ** -11)
    put("Q", (1, 0), 1.0)
    x = np.zeros((1, 2, T, T), dtype=np.float32)
    x[0, 0] = np.random.default_rng(T).normal(scale=1.0, size=(T, T))
    with fno.Network(T, 1) as net:
        net.set_params(p)
        dx = torch.tensor(x, device="cuda")
        dy = torch.empty_like(dx)
        torch.cuda.synchronize()
        net.forward(dx.data_ptr(), dy.data_ptr(), 1)
    want = O.loss_and_grad(fno.bf16_round(p).astype(np.float64), x, x)[2][0, 1]
    s = np.abs(want - 1).max()
    assert 2.0 ** -16 < s < 2.0 ** -12, s
    assert np.abs(dy.cpu().numpy()[0, 1] - want).max() < 2.0 ** -24 + 2.0 ** -26
