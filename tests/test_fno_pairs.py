"""make_pairs orders its device buffer between torch's stream, which copies out of
it, and the problems' own streams, which write the next state into it. On the CPU:
torch's copies are held back until something waits for them, as a busy stream would,
and the problems' downloads write at once."""
import ctypes

import numpy as np
import pytest

from pfc_b200 import fno

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,chunk", [(5, 2), (3, 3), (1, 4)])
def test_pairs_wait_for_copies(monkeypatch, n, chunk):
    N, held, base = 4, [], [0]
    real_copy, real_empty = torch.Tensor.copy_, torch.empty

    def wait(*_):
        for dst, src in held:
            real_copy(dst, src)
        held.clear()

    def write(ptr, value):
        np.ctypeslib.as_array(ctypes.cast(ptr, ctypes.POINTER(ctypes.c_double)), (2, N, N))[:] = value

    class Problem:
        def __init__(self, batch, index):
            self.batch, self.index = batch, index

        def upload_device(self, ptr):
            pass

        def download_device(self, ptr):
            write(ptr, 1000 * self.batch.done + self.index)

    class Batch:
        def __init__(self, problems, precision, autotune):
            self.done = 0
            self.problems = [Problem(self, base[0] + i) for i in range(len(problems))]
            base[0] += len(problems)

        def step(self, k):
            self.done += k

        def __enter__(self):
            return self

        def __exit__(self, *exc):
            pass

    def init_hetero(ptr, Nx, Ny, dx, dy, spec):  # on torch's stream, and waits for it
        wait()
        write(ptr, -1 - spec)

    monkeypatch.setattr(fno.lib, "Batch", Batch)
    monkeypatch.setattr(fno.lib, "init_hetero", init_hetero)
    monkeypatch.setattr(fno, "state_spec", lambda i, seed0, N: i)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: real_empty(*a, **{q: v for q, v in k.items() if q != "device"}))
    monkeypatch.setattr(torch.Tensor, "copy_", lambda dst, src: held.append((dst, src)) or dst)
    monkeypatch.setattr(torch.cuda, "synchronize", wait)
    X, Ys = fno.make_pairs(n, N, (3, 7), chunk=chunk, log=lambda *_: None)
    assert not held
    for i in range(n):
        assert (X[i] == -1 - i).all()
        for s in (3, 7):
            assert (Ys[s][i] == 1000 * s + i).all()
