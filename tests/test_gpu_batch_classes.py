"""Batch classes on the kernels of run-time lengths: their launch shapes, which follow
from all the class's blocks, against the same problems one at a time.

Fields agree as in test_gpu_batch.py (1e-12 in FP64, 1e-6 in FP32) and, for three and
four FP32 fields, to the parity suite's 2e-5."""
import time

import numpy as np
import pytest

from pfc_b200 import lib
from pfc_b200 import synth
from test_gpu_rt import MEANS, _params

pytestmark = pytest.mark.gpu


def _state(U, Nx, Ny, seed):
    return np.array([synth.noise_state(Nx, Ny, MEANS[u] if U > 1 else 0.25, 0.05, seed, stream=u) for u in range(U)])


# few blocks, with more threads than their passes need; many, with no more; a chip's worth of
# blocks, at 64 threads, and one problem beyond; lengths, fields and both in one class
CLASSES = [[(1, 128, 128)] * 2, [(1, 128, 128)] * 40, [(1, 256, 256)] * 9, [(1, 256, 256)] * 10, [(2, 96, 96)] * 3,
           [(2, 128, 100)] * 24, [(1, 90, 98), (1, 1000, 36), (1, 64, 210)], [(2, 720, 90), (2, 8, 10), (2, 64, 256)] * 4,
           [(3, 96, 70), (4, 60, 84)], [(1, 120, 90), (2, 300, 50), (3, 90, 294), (4, 32, 48)]]


@pytest.mark.parametrize("k", range(len(CLASSES)))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_class_matches_single_problems(k, precision, monkeypatch):
    monkeypatch.setenv("PFCG_GENERIC_KERNELS", "1")
    probs = CLASSES[k]
    tol = 1e-12 if precision == "fp64" else 2e-5 if max(p[0] for p in probs) > 2 else 1e-6
    with lib.Batch([(_params(U), Nx, Ny, 0.7, 0.65) for U, Nx, Ny in probs], precision, autotune=False) as b:
        for i, (q, (U, Nx, Ny)) in enumerate(zip(b.problems, probs)):
            q.upload(_state(U, Nx, Ny, 30 + i))
        b.step(5)
        got = [q.download() for q in b.problems]
    for i in sorted({0, 1, len(probs) // 2, len(probs) - 1}):
        U, Nx, Ny = probs[i]
        with lib.Relaxation(_params(U), Nx, Ny, 0.7, 0.65, precision) as r:
            r.upload(_state(U, Nx, Ny, 30 + i))
            r.step(5)
            assert np.abs(got[i] - r.download()).max() < tol, i


def test_many_small_problems_fill_the_chip():
    """64 problems of 512^2 have the points of one of 4096^2 and shorter transforms: a
    step of them takes less (0.88 of it; 1.37 with threads chosen for one problem's grid,
    which keep half of the blocks off the chip)."""
    took = []
    for probs in ([(1, 512, 512)] * 64, [(1, 4096, 4096)]):
        with lib.Batch([(_params(U), Nx, Ny, 0.7, 0.7) for U, Nx, Ny in probs], "fp64", autotune=False) as b:
            for q, (U, Nx, Ny) in zip(b.problems, probs):
                q.upload(np.full((U, Ny, Nx), 0.25))
            best = 1e9
            for _ in range(4):  # the first captures the graph
                t = time.perf_counter()
                b.step(50)
                best = min(best, time.perf_counter() - t)
            took.append(best)
    assert took[0] < 1.1 * took[1], took
