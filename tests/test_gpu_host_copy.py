"""Fields that come from and go to ordinary host memory, against the same through
device memory: equal to the bit (the copies change no value). Sizes on both sides of
4 MB, from where several threads copy through pinned chunks of 1 MB: whole
chunks, a remainder, fewer chunks than slots and many more; and two handles on two
threads at once, of which one finds the chunks taken."""
import threading

import numpy as np
import pytest

from pfc_b200 import lib
from pfc_b200 import params as P
from pfc_b200 import synth

pytestmark = pytest.mark.gpu


def _round(Nx, Ny, U, prec, seed, out):
    import torch

    p = P.make_params(P.honeycomb_1c(-0.25), 1.0, 1.0) if U == 1 else P.make_params(P.hetero_2c(0.04), 1.0, 0.25)
    f0 = np.array([synth.noise_state(Nx, Ny, 0.25, 0.05, seed, stream=u) for u in range(U)])
    with lib.Relaxation(p, Nx, Ny, 0.7, 0.7, prec) as r:
        d = torch.from_numpy(f0).cuda()
        torch.cuda.synchronize()
        r.upload_device(d.data_ptr())
        r.download_device(d.data_ptr())
        ref = d.cpu().numpy()
        nave = r.evaluate(want_f=True)
        r.upload(f0)
        again = r.evaluate(want_f=True)
        out.append((ref, r.download(), nave, again))


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("Nx,Ny,U", [(1024, 504, 1), (1024, 512, 1), (1050, 500, 1), (1000, 900, 2), (2048, 2048, 1)])
def test_host_copies_equal_device_copies(Nx, Ny, U, prec):
    out = []
    _round(Nx, Ny, U, prec, 5, out)
    ref, got, a, b = out[0]
    np.testing.assert_array_equal(got, ref)
    np.testing.assert_array_equal(b[2], a[2])
    assert a[0] == b[0]


def test_two_threads_at_once():
    outs = [[], []]
    ts = [threading.Thread(target=lambda i=i: [_round(1024, 1024, 2, "fp64", 7 + i, outs[i]) for _ in range(4)]) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for out in outs:
        assert len(out) == 4
        for ref, got, a, b in out:
            np.testing.assert_array_equal(got, ref)
            np.testing.assert_array_equal(b[2], a[2])


@pytest.mark.parametrize("prec,U", [("fp32", 1), ("fp32", 3), ("fp64", 2), ("fp64", 4)])
def test_device_arrays_of_any_alignment(prec, U):
    """The kernels read and write a device array in place where it is aligned to 16
    bytes, and a copy of it at 8: equal to the bit, and nothing beside it is touched."""
    import torch

    from test_gpu_rt import MEANS, _params

    Nx, Ny = 120, 90
    n = U * Nx * Ny
    f0 = np.array([synth.noise_state(Nx, Ny, MEANS[u] if U > 1 else 0.25, 0.05, 3, stream=u) for u in range(U)])
    got = []
    with lib.Relaxation(_params(U), Nx, Ny, 0.7, 0.7, prec) as r:
        for shift in (0, 1, 2):
            d = torch.full((n + 4,), 7.5, dtype=torch.float64, device="cuda")
            d[shift:shift + n] = torch.from_numpy(f0.reshape(-1)).cuda()
            torch.cuda.synchronize()
            r.upload_device(d.data_ptr() + 8 * shift)
            r.step(3)
            r.download_device(d.data_ptr() + 8 * shift)
            out = d.cpu().numpy()
            assert (out[:shift] == 7.5).all() and (out[shift + n:] == 7.5).all()
            got.append(out[shift:shift + n])
    np.testing.assert_array_equal(got[1], got[0])
    np.testing.assert_array_equal(got[2], got[0])
