"""The three launch forms of the time loops give the same objective and gradient:
per-step sweeps (persistent=-1), the persistent sweeps whose split row groups meet in
L2 (persistent=1), and the cluster form (persistent=2), where each thread-block
cluster owns whole row groups and combines their parts in distributed shared memory.
Checked on the full sphere -> cube workload (2562 landmarks, Matern nu = 3/2, T = 20)
and on the 2D circle -> square workload against the FP64 oracle, for run-to-run
bitwise determinism, and through a short L-BFGS run."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _objgrd(P, alp, persistent):
    from lddmm_b200 import api

    with api.Context(P, persistent=persistent) as ctx:
        shape = ctx.launch_shape()
        f, g = ctx.objgrd(alp)
        f2, g2 = ctx.objgrd(alp)
    assert f2[0] == f[0] and np.array_equal(g, g2)  # bit-reproducible
    return f[0], g, shape


@pytest.mark.parametrize("which", ["sphere2cube", "circle2square"])
def test_forms_agree_with_the_oracle(oracle, which):
    from lddmm_b200 import problem

    P = problem.sphere_to_cube() if which == "sphere2cube" else problem.circle_to_square()
    alp = np.random.default_rng(3).normal(size=P.var_num) * 0.02
    fo, go = oracle.objgrd(P, alp)
    out = {}
    for form in (-1, 1, 2):
        f, g, shape = _objgrd(P, alp, form)
        assert shape["persistent"] == max(form, 0), (form, shape)
        assert abs(f - fo) / abs(fo) < TOL, (form, f, fo)
        assert rel(g, go) < TOL, (form, rel(g, go))
        out[form] = (f, g)
    # the forms cut the rows' j ranges at different points, so their FP32 partial sums
    # differ at the FP32 rounding level only
    for form in (1, 2):
        assert abs(out[form][0] - out[-1][0]) <= 1e-7 * abs(out[-1][0])
        assert rel(out[form][1], out[-1][1]) < 1e-6


def test_cluster_form_lbfgs_follows_the_l2_form():
    """The first 8 iterations of the two persistent forms' L-BFGS runs agree."""
    from lddmm_b200 import api, problem

    P = problem.sphere_to_cube(subdiv=3, cube_n=12, time_num=11)
    traces = []
    for form in (1, 2):
        with api.Context(P, persistent=form) as ctx:
            x, res = ctx.lbfgs(np.zeros(P.var_num), itr_max=15)
            traces.append(ctx.trace(0))
            assert res[0]["status"] == 0 and res[0]["iters"] == 15
    # the same early path (rounding-level differences grow over the iterations, as
    # between any two launch shapes)
    r = np.abs(traces[0][:9, 0] - traces[1][:9, 0]) / np.abs(traces[0][:9, 0])
    assert r.max() < 1e-5, r.max()


@pytest.mark.parametrize("order,width", [(-1, 0.5), (3, 0.15)])
@pytest.mark.parametrize("sizes", [(5,), (64,), (65, 300), (128,), (129,), (257,), (500, 496),
                                   (512,), (513,)])
def test_small_pairs_against_the_oracle(oracle, sizes, order, width):
    """The small form's edges: pairs that give 4, 8 and 16 CTAs, one row to a full block of
    rows per CTA, two pairs of unequal size, 512 points (its last) and 513 (another form); the
    2D Matern width puts its Bessel arguments on both sides of 2.  Tolerance 1e-5, that of
    every FP32 sum of the library."""
    from lddmm_b200 import api, problem

    Ps = [problem.circle_to_square(n, 40, width) for n in sizes]
    for P in Ps:
        P.knl_order = order
    alp = [np.random.default_rng(P.nde_num).normal(size=P.var_num) * 0.02 for P in Ps]
    with api.Context(Ps, autotune=False) as ctx:
        f, g = ctx.objgrd(np.concatenate(alp))
    g = np.split(g, np.cumsum([P.var_num for P in Ps])[:-1])
    for k, P in enumerate(Ps):
        fo, go = oracle.objgrd(P, alp[k])
        assert abs(f[k] - fo) <= TOL * abs(fo)
        assert rel(g[k], go) < TOL


@pytest.mark.parametrize("n", [64, 65, 1200, 2049, 3000])
def test_row_tiles_against_the_oracle(oracle, n):
    """The L2 form's 64-row tiles: one tile, a second of one row, tiles cut into more than 8
    parts (1200), CTAs that take the end of one tile and the start of the next (3000)."""
    from lddmm_b200 import api, problem, shapes

    v, f = shapes.decimated_star(n, 6, 0.05, n)
    tv, tf = shapes.icosphere(1)
    P = problem.Problem(v, f, *shapes.varifold_of(tv, tf), knl_order=1, knl_width=0.4, time_num=4,
                        time_stp=1 / 3, cen_width=0.3)
    alp = np.random.default_rng(n).normal(size=P.var_num) * 0.02
    f, g, _ = _objgrd(P, alp, 1)
    fo, go = oracle.objgrd(P, alp)
    assert abs(f - fo) <= TOL * abs(fo)
    assert rel(g, go) < TOL


def test_row_tiles_of_many_pairs(oracle):
    """More tiles than twice the resident CTAs: shares of three and more whole tiles."""
    from lddmm_b200 import api, problem

    Ps = [problem.circle_to_square(200 + 5 * k, 40, time_num=4) for k in range(130)]
    alp = [np.random.default_rng(k).normal(size=P.var_num) * 0.02 for k, P in enumerate(Ps)]
    with api.Context(Ps, persistent=1) as ctx:
        f, g = ctx.objgrd(np.concatenate(alp))
    g = np.split(g, np.cumsum([P.var_num for P in Ps])[:-1])
    for k in (0, 64, 129):
        fo, go = oracle.objgrd(Ps[k], alp[k])
        assert abs(f[k] - fo) <= TOL * abs(fo)
        assert rel(g[k], go) < TOL


@pytest.mark.parametrize("sizes,ctas", [((5,), 4), ((64,), 4), ((65, 250), 8),
                                        ((65, 300), 0), ((128,), 8), ((257,), 16), ((512,), 16),
                                        ((513,), 0)])
def test_the_small_form_runs_where_it_should(sizes, ctas):
    """The rule without tuning: pairs of at most 512 points, as many CTAs as the smallest pair
    has 16-row groups of 64-row padding, at most 16, if the largest pair's rows then fit a CTA
    (32, of 16 threads each)."""
    from lddmm_b200 import api, problem

    with api.Context([problem.circle_to_square(n, 40, 0.5) for n in sizes], autotune=False) as ctx:
        shape = ctx.launch_shape()
    assert shape["persistent"] == 1 and shape["small_ctas"] == ctas


def test_the_small_form_is_not_the_rule_beyond_one_wave():
    """Without tuning, 16 clusters of 16 CTAs would take turns: 16 pairs of 500 points run on
    the 64-row tiles."""
    from lddmm_b200 import api, problem

    with api.Context([problem.circle_to_square(500, 40, 0.5)] * 16, autotune=False) as ctx:
        shape = ctx.launch_shape()
    assert shape["persistent"] == 1 and shape["small_ctas"] == 0


@pytest.mark.parametrize("sizes", [(400,), (500,), (513,), (640,), (500, 17, 497)])
def test_whole_row_groups_against_the_oracle(oracle, sizes):
    """2D Gaussian pairs of a few hundred points, tuned: whole 16-row groups, one per CTA (on one
    pair of 500 points a seventh faster than the next form).  Tolerance 1e-5, that of every FP32
    sum of the library; bit for bit the same on a second call."""
    from lddmm_b200 import api, problem

    Ps = [problem.circle_to_square(n, 40, 0.5) for n in sizes]
    for P in Ps:
        P.knl_order = -1
    alp = [np.random.default_rng(P.nde_num).normal(size=P.var_num) * 0.02 for P in Ps]
    with api.Context(Ps) as ctx:
        shape = ctx.launch_shape()
        f, g = ctx.objgrd(np.concatenate(alp))
        f2, g2 = ctx.objgrd(np.concatenate(alp))
    assert sizes != (500,) or shape["groups"], shape
    assert np.array_equal(f, f2) and np.array_equal(g, g2)
    g = np.split(g, np.cumsum([P.var_num for P in Ps])[:-1])
    for k, P in enumerate(Ps):
        fo, go = oracle.objgrd(P, alp[k])
        assert abs(f[k] - fo) <= TOL * abs(fo)
        assert rel(g[k], go) < TOL
