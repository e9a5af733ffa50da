"""The kernels of run-time lengths (and, for three and four FP32 fields, those of
kernels_wide.cuh) against the CPU oracle at the shapes where
they can go wrong: plans with each radix (2 to 10, 12, 14, 15, 16), with and
without padding, one to four fields with rows or fields paired, a single row per
tile (4096 points of two or three fields in FP64), tiles and column groups that
do not fill a warp, and f(r), which takes the weighted spectra through the
one-field kernels.

Bounds: FP64 fields and energies agree with the oracle to rounding (1e-12, as in
test_gpu_parity); FP32 fields to 2e-5 and energies to 1e-6 relative after five
steps, the parity suite's bounds for its FP32 kernels."""
import os
import sys

import numpy as np
import pytest

import pyoracle
from pfc_b200 import lib
from pfc_b200 import params as P
from pfc_b200 import synth

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_golden as G  # noqa: E402

pytestmark = pytest.mark.gpu

MEANS = (0.3, -0.3, -0.32, -0.28)


def _params(U):
    if U == 1:
        return P.make_params(P.honeycomb_1c(-0.25), 1.0, 1.0)
    if U == 2:
        return P.make_params(P.hetero_2c(0.04), 1.0, 0.25)
    d = G.hetero_3c()
    if U == 4:  # a fourth field like the third, uncoupled from it
        for k in ("alpha", "beta", "gamma", "epsilon", "inv_mu"):
            d[k] = [row + [0.0] for row in d[k]] + [[0.0] * 4]
        d["alpha"][3][3], d["beta"][3][3], d["epsilon"][0][3] = -0.3, 1.0, -0.4
        for k, v in (("lambda", 0.0), ("delta", 1.0), ("inv_nu", [1.018]), ("omega", [1.0]), ("phi", [0.0])):
            d[k] = d[k] + [v]
    return P.make_params(d, 1.0, 0.25)


@pytest.mark.parametrize("U,Nx,Ny", [(1, 8, 10), (1, 90, 98), (2, 126, 150), (2, 210, 48), (3, 96, 70), (4, 60, 84),
                                     (1, 640, 36), (2, 1440, 90), (4, 1000, 12), (2, 4096, 8), (3, 4096, 8),
                                     (2, 16, 2744)])
def test_run_time_lengths_match_oracle(U, Nx, Ny, monkeypatch):
    monkeypatch.setenv("PFCG_GENERIC_KERNELS", "1")
    p, dx, dy = _params(U), 0.7, 0.65
    f0 = np.array([synth.noise_state(Nx, Ny, MEANS[u] if U > 1 else 0.25, 0.05, 41, stream=u) for u in range(U)])
    o = pyoracle.Oracle(p, Nx, Ny, dx, dy)
    o.upload(f0)
    o.step(5)
    ref = o.download()
    fo, no, fr = o.evaluate(want_f=True)
    o.close()
    for prec, tol, etol in (("fp64", 1e-12, 1e-12), ("fp32", 2e-5, 1e-6)):
        with lib.Relaxation(p, Nx, Ny, dx, dy, prec) as r:
            r.upload(f0)
            r.step(5)
            got = r.download()
            fg, ng, frg = r.evaluate(want_f=True)
        assert np.abs(got - ref).max() < tol, (prec, np.abs(got - ref).max())
        assert abs(fg - fo) < etol * abs(fo), (prec, fg, fo)
        assert np.abs(ng - no).max() < 1e-12
        # f(r) is a polynomial of degree four in fields of order one with coefficients below 3
        assert np.abs(frg - fr).max() < 20 * tol, (prec, np.abs(frg - fr).max())


@pytest.mark.parametrize("U,Nx,Ny", [(1, 128, 128), (2, 256, 150), (1, 300, 640), (1, 360, 500), (2, 64, 256), (3, 90, 294),
                                     (4, 60, 150)])
def test_work_before_the_wait_matches_oracle(U, Nx, Ny, monkeypatch):
    """A small problem by itself takes its state and coefficients, and turns a
    transform, before the wait for the previous pass: one CTA of a pass per SM, one
    CTA more than SMs, two, and grids just too large for it. Bounds as above."""
    test_run_time_lengths_match_oracle(U, Nx, Ny, monkeypatch)
