"""The network's fitted GELU and its derivative (pfc_b200/csrc/fno_gelu.cuh) by
themselves, on a dense grid and at the special values, against FP64; and a network
whose hidden layer overflows.

Bounds. The tail Phi(-u) = t Q(t) exp(-u^2 / 2) has a relative error of a few units
of 2^-23: 1 from the reciprocal, twice that through Q, 2 from the exponential, 3
half units times u^2 / 2 from its argument, 4 from the polynomial and the products:
1.4e-6 at worst where u phi and phi are large. GELU is max(z, 0) less u phi <= 0.17 of it, 2.4e-7,
and half a unit in the last place, 2^-24 |z|. The derivative takes phi <= 0.5, whose
error is smallest at u = 0, and a product below 0.25: 5e-7."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from pfc_b200 import fno

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc is not installed")
    d = tmp_path_factory.mktemp("gelu")
    subprocess.run([NVCC, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(d / "gelu_check"),
                    os.path.join(HERE, "cuda", "gelu_check.cu")], check=True, capture_output=True, timeout=300)

    def run(z):
        np.asarray(z, dtype=np.float32).tofile(d / "z")
        subprocess.run([str(d / "gelu_check"), str(d / "z"), str(d / "out")], check=True, timeout=120)
        return np.fromfile(d / "out", dtype=np.float32).reshape(-1, 2).T

    return run


def exact(z):
    z = torch.tensor(np.asarray(z, dtype=np.float32), dtype=torch.float64)
    cdf = 0.5 * torch.special.erfc(-z / 2 ** 0.5)
    return (z * cdf).numpy(), (cdf + z * torch.exp(-0.5 * z * z) / (2 * np.pi) ** 0.5).numpy()


def test_gelu_and_derivative(evaluate):
    z = np.concatenate([np.linspace(-14, 14, 2 ** 20), np.linspace(-1e-3, 1e-3, 2001), [0.0, -0.0]]).astype(np.float32)
    g, d = evaluate(z)
    eg, ed = exact(z)
    assert (np.abs(g - eg) - 2.0 ** -24 * np.abs(z)).max() < 2.4e-7
    assert np.abs(d - ed).max() < 5e-7
    # rms errors, which a slip in one coefficient of the fit would show first
    m = np.abs(z) < 9
    assert np.sqrt(((g - eg)[m] ** 2).mean()) < 6e-8


def test_gelu_far_out(evaluate):
    big = np.array([20, 100, 1e4, 1e19, 1e30, 3e38, 3.4028235e38], dtype=np.float32)
    g, d = evaluate(np.concatenate([big, -big]))
    n = len(big)
    np.testing.assert_array_equal(g[:n], big)
    np.testing.assert_array_equal(np.abs(g[n:]), 0.0)
    np.testing.assert_array_equal(d[:n], 1.0)
    np.testing.assert_array_equal(np.abs(d[n:]), 0.0)
    g, d = evaluate([np.nan, -np.inf, np.inf])  # as 0.5 z (1 + erf) has them
    assert np.isnan(g[:2]).all() and g[2] == np.inf and np.isnan(d).all()


@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_overflowing_network_is_not_finite(sign):
    """A first layer whose pre-activation overflows, to one side: the output is not a
    number, as with GELU from the error function, where a GELU of 0 at -inf would hide it."""
    T = 32
    p = np.zeros(fno.NPARAM, dtype=np.float32)
    lay = fno.layout()

    def put(name, idx, v):
        o, s = lay[name]
        p[o + np.ravel_multi_index(idx, s)] = v

    put("P", (0, 0), 2.0 ** 100)
    put("W0", (0, 0), sign * 2.0 ** 100)
    for l in (1, 2, 3):
        put("W%d" % l, (0, 0), 1.0)
    put("Q", (1, 0), 1.0)
    x = torch.zeros((1, 2, T, T), device="cuda")
    x[0, 0] = 1.0
    y = torch.empty_like(x)
    with fno.Network(T, 1) as net:
        net.set_params(p)
        torch.cuda.synchronize()
        net.forward(x.data_ptr(), y.data_ptr(), 1)
    assert not torch.isfinite(y).all()
