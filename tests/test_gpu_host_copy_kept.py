"""Copies through the pinned chunks, which a handle makes once it has moved 64 MB: fields
in and out of ordinary host memory on a kept handle, before and after, and on another one
beside it whose first copy uses them, against device memory: equal to the bit. Sizes on both sides of
4 MB up and 16 MB down, whole chunks and remainders; and two handles on two threads."""
import threading

import numpy as np
import pytest

from pfc_b200 import lib
from pfc_b200 import params as P
from pfc_b200 import synth

pytestmark = pytest.mark.gpu

P1 = P.make_params(P.honeycomb_1c(-0.25), 1.0, 1.0)


def _through_device(r, f):
    import torch

    d = torch.from_numpy(f).cuda()
    torch.cuda.synchronize()
    r.upload_device(d.data_ptr())
    r.download_device(d.data_ptr())
    return d.cpu().numpy()


def _round(r, f, ref):
    r.upload(f)
    np.testing.assert_array_equal(r.download(), ref)


@pytest.mark.parametrize("Nx,Ny", [(1024, 504), (1050, 500), (1024, 2048), (1000, 2100), (2048, 2048)])
def test_kept_handle_and_another(Nx, Ny):
    big = np.array([synth.noise_state(2048, 1050, 0.25, 0.05, 9)])
    f = np.array([synth.noise_state(Nx, Ny, 0.25, 0.05, 11)])
    with lib.Relaxation(P1, 2048, 1050, 0.7, 0.7, "fp64") as a, lib.Relaxation(P1, Nx, Ny, 0.7, 0.7, "fp64") as b:
        ref, want = _through_device(a, big), _through_device(b, f)
        for _ in range(4):  # 17.2 MB each way: the chunks are there from the second round on
            _round(a, big, ref)
        for _ in range(2):
            _round(b, f, want)


def test_two_threads_on_kept_handles():
    def work(seed, bad):
        f = np.array([synth.noise_state(2048, 1050, 0.25, 0.05, seed)])
        with lib.Relaxation(P1, 2048, 1050, 0.7, 0.7, "fp32") as r:
            ref = _through_device(r, f)
            for _ in range(8):
                r.upload(f)
                bad.append(not np.array_equal(r.download(), ref))

    bad = [[], []]
    ts = [threading.Thread(target=work, args=(21 + i, bad[i])) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert [len(b) for b in bad] == [8, 8] and not any(bad[0] + bad[1])
