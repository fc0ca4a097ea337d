"""3D Gaussian per-step sweeps (csrc/gauss.cuh) against the FP64 oracle where their
branches change: a single 64-row tile, a full and a partial last 128-row item, row tiles
too wide for the expanded exponent (kernel width small against the tile) and compact ones,
widths at which most 32-point blocks lie beyond the cut-off, momenta that vanish on most
of the shape (the cut-off then moves outwards), and a NaN momentum, which must reach the
objective.  Tolerance 1e-5, that of every FP32 sum of the library."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _problem(n, width, seed):
    from lddmm_b200 import problem, shapes

    v, f = shapes.decimated_star(n, 6, 0.05, seed)
    tv, tf = shapes.decimated_star(200, 6, 0.05, seed + 1)
    cen, dr, vol = shapes.varifold_of(tv, tf)
    return problem.Problem(v, f, cen, dr, vol, knl_order=-1, knl_width=width, time_num=4,
                           time_stp=1 / 3, cen_width=0.3)


@pytest.mark.parametrize("n,width", [(40, 0.3), (64, 2.5), (65, 2.5), (128, 0.8), (642, 0.3),
                                     (642, 3.0), (1500, 0.08), (1500, 1.2)])
@pytest.mark.parametrize("patch", [False, True])
def test_gauss_sweeps_against_the_oracle(oracle, n, width, patch):
    from lddmm_b200 import api

    P = _problem(n, width, n)
    a = np.random.default_rng(n).normal(size=(P.T, n, 3)) * 0.02
    if patch:  # momenta on one side of the shape only
        a[:, P.ini_nde[:, 2] < 0.5] = 0.0
    with api.Context(P, persistent=-1) as ctx:
        f, g = ctx.objgrd(a.reshape(-1))
    fo, go = oracle.objgrd(P, a.reshape(-1))
    assert abs(f[0] - fo) <= TOL * abs(fo)
    assert rel(g, go) < TOL


def test_gauss_sweeps_keep_nan():
    from lddmm_b200 import api

    P = _problem(1500, 0.08, 3)
    a = np.zeros(P.var_num)
    a[7] = np.nan
    with api.Context(P, persistent=-1) as ctx:
        f, g = ctx.objgrd(a)
    assert np.isnan(f[0]) and np.isnan(g).any()
