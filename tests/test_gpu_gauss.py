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


def _grid_problem(n, width, seed):
    P = _problem(n, width, seed)
    P.cen_width = 0.1
    return P


@pytest.mark.parametrize("n", [40000, 40962])
def test_gridded_sums_against_fp64(n):
    """A pair large enough for the gridded kernel sums (csrc/grid.cuh), 40,000 landmarks
    leaving a partial 32-point tile's worth of padding and 40,962 an odd tile count:
    velocities and costate steps of a row sample against FP64 pair sums.  The grid's kernel
    is within 3.4e-11 of the Gaussian and 2.5e-9 of its derivative, far below the FP32
    rounding of the pair sweeps, so 1e-7 of the largest value bounds what the FP32 momenta
    leave."""
    import ctypes as C

    import torch

    from lddmm_b200 import _lib, api

    P = _grid_problem(n, 0.3, 5)
    rng = np.random.default_rng(n)
    a = rng.normal(size=(P.T, n, 3)) * 0.001 + 0.0005 * P.ini_nde
    with api.Context(P) as ctx:
        (q, v), = ctx.shoot(a.reshape(-1))
        d = torch.from_numpy(a.reshape(-1)).cuda()
        f, g, pst = torch.empty(1, dtype=torch.float64, device="cuda"), d.clone(), d.clone()
        args = [C.c_void_p(x.data_ptr()) for x in (d, f, g, pst)]
        _lib.check(_lib.lib.lddmm_objgrd_costate(ctx.handle, *args))
        f2, g2 = ctx.objgrd(a.reshape(-1))
        g, pst = (x.cpu().numpy().reshape(a.shape) for x in (g, pst))
        assert f2[0] == f.item() and np.array_equal(g2.reshape(a.shape), g)
        big, _ = ctx.objgrd(a.reshape(-1) * 4000)  # outgrows its grid: the pair sweeps
        assert np.isfinite(big[0])
        a[1, 3, 0] = np.inf
        assert not np.isfinite(ctx.objgrd(a.reshape(-1))[0][0])
    rows = rng.integers(0, n, 40)
    w2 = P.knl_width ** 2
    a[1, 3, 0] = 0.0
    for t in range(P.T):
        d = q[t][rows][:, None] - q[t][None]
        K = np.exp(-(d ** 2).sum(-1) / w2)
        if t != 1:  # row 3's momentum was replaced at step 1
            assert np.max(np.abs(K @ a[t] - v[t][rows])) < 1e-7 * np.max(np.abs(v[t]))
            u = a[t] - pst[t]
            assert np.max(np.abs(P.time_stp * K @ u - g[t][rows])) < 1e-7 * np.max(np.abs(g[t]))
        if t == 2:
            l = 0.5 * a[t] - pst[t]
            lr = l[rows] @ a[t].T + a[t][rows] @ l.T
            dq = -2 / w2 * ((K * lr)[..., None] * d).sum(1)
            step = pst[t][rows] - pst[t - 1][rows]
            assert np.max(np.abs(P.time_stp * dq - step)) < 1e-7 * np.max(np.abs(pst[t]))


def test_gridded_sums_of_the_large_pair():
    """163,842 landmarks, all steps on the grid: velocities and gradients of a row sample
    against FP64 sums.  Tolerance as above."""
    import ctypes as C

    import torch

    from lddmm_b200 import _lib, api, problem

    P = problem.star_pair(time_num=4)
    a = np.random.default_rng(1).normal(size=(P.T, P.nde_num, 3)) * 2e-4 + 1e-4 * P.ini_nde
    with api.Context(P) as ctx:
        (q, v), = ctx.shoot(a.reshape(-1))
        d = torch.from_numpy(a.reshape(-1)).cuda()
        f, g, pst = torch.empty(1, dtype=torch.float64, device="cuda"), d.clone(), d.clone()
        _lib.check(_lib.lib.lddmm_objgrd_costate(
            ctx.handle, *[C.c_void_p(x.data_ptr()) for x in (d, f, g, pst)]))
    g, pst = (x.cpu().numpy().reshape(a.shape) for x in (g, pst))
    rows = np.random.default_rng(2).integers(0, P.nde_num, 40)
    for t in range(P.T):
        K = np.exp(-((q[t][rows][:, None] - q[t][None]) ** 2).sum(-1) / P.knl_width ** 2)
        u = a[t] - pst[t]
        assert np.max(np.abs(K @ a[t] - v[t][rows])) < 1e-7 * np.max(np.abs(v[t]))
        assert np.max(np.abs(P.time_stp * K @ u - g[t][rows])) < 1e-7 * np.max(np.abs(g[t]))


def test_gridded_sums_of_huge_momenta():
    """Finite momenta whose largest value times N exceeds the largest float: the first step
    still runs on the grid (later ones outgrow it).  Tolerance as above."""
    from lddmm_b200 import api

    P = _grid_problem(40000, 0.3, 5)
    a = np.random.default_rng(3).normal(size=(P.T, 40000, 3)) * 1e34
    assert a.max() < 3e38 < 40000 * a.max()
    with api.Context(P) as ctx:
        (q, v), = ctx.shoot(a.reshape(-1))
    rows = np.random.default_rng(4).integers(0, 40000, 40)
    d2 = ((q[0][rows][:, None] - q[0][None]) ** 2).sum(-1)
    vo = np.exp(-d2 / P.knl_width ** 2) @ a[0]
    assert np.max(np.abs(v[0][rows] - vo)) < 1e-7 * np.max(np.abs(vo))


@pytest.mark.parametrize("n,cw", [(40, 0.1), (66, 0.5), (1500, 1.0), (1500, 0.3), (1500, 0.1),
                                  (1500, 0.02)])
def test_split_varifold_sweep_against_the_oracle(oracle, n, cw):
    """csrc/vfd.cuh: element tiles that are compact against the centre kernel's width, near
    ones and wide ones (double-single differences), one 64-element tile and a partial last
    one; value and gradient."""
    from lddmm_b200 import api

    P = _problem(n, 0.3, n + 1)
    P.cen_width = cw
    v, dq = api.varifold(P, P.ini_nde)
    vo, go = oracle.varifold(P, P.ini_nde)
    assert abs(v - vo) <= TOL * abs(vo)
    assert rel(dq, go) < TOL


@pytest.mark.parametrize("cw", [0.4, 0.15, 0.05])
def test_split_varifold_value_near_convergence(cw):
    """Compact, near and wide element tiles: V between two meshes of one surface, small
    against TT, so that its error is the systematic one of DD and DT.  Of the exponential's
    mean error (3.7e-8 and 4.6e-8 over a kernel's pairs, removed) its variation with the
    distribution of the arguments remains, some 0.5e-8; rounding errors average out over
    3.6e7 pairs.  8e-9 of TT."""
    import torch

    from lddmm_b200 import api, problem, shapes

    v, f = shapes.decimated_star(3000, 6, 0.05, 23)
    tv, tf = shapes.decimated_star(3100, 6, 0.05, 23)
    P = problem.Problem(v, f, *shapes.varifold_of(tv, tf), knl_order=-1, knl_width=0.3,
                        time_num=2, time_stp=1.0, cen_width=cw)
    V, _ = api.varifold(P, P.ini_nde)
    S, T = ([torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in y]
            for y in (shapes.varifold_of(v, f), shapes.varifold_of(tv, tf)))

    def dot(x, y):
        d2 = sum((x[0][:, None, k] - y[0][None, :, k]) ** 2 for k in range(3))
        return float(x[2] @ (torch.exp(-d2 / cw ** 2) * (x[1] @ y[1].T) ** 2) @ y[2])

    tt = dot(T, T)
    v64 = dot(S, S) - 2 * dot(S, T) + tt
    assert v64 < 0.2 * tt
    assert abs(V - v64) < 8e-9 * tt, (V - v64) / tt


def _radial(P, growth):
    """Momenta whose velocities carry the unit sphere's neighbourhood outwards by `growth` in
    each of the T steps: the kernel's mass on a sphere of radius R is N w^2 / (4 R^2)."""
    a, R = np.empty((P.T, P.nde_num, 3)), 1.0
    for t in range(P.T):
        a[t] = P.ini_nde * (growth / P.time_stp * 4 * R * R / (P.nde_num * P.knl_width ** 2))
        R *= 1 + growth
    return a.reshape(-1)


def _shoot_ms(P, a, reps=3):
    from lddmm_b200 import api

    with api.Context(P) as ctx:
        ctx.objgrd(a)
        return min(ctx.time_sweeps(reps)["shoot"] for _ in range(3))


def test_a_larger_target_leaves_the_grid_its_room():
    """163,842 landmarks on the way to a target 1.5 times as large stay on the grid, at twice
    the time of a source that does not move at most (the pair sums take 15 times as long)."""
    from lddmm_b200 import problem, shapes

    P = problem.star_pair()
    tv, tf = shapes.icosphere(4)
    P = problem.Problem(P.ini_nde, P.elm_vtx, *shapes.varifold_of(1.5 * tv, tf), knl_order=-1,
                        knl_width=0.3, time_num=4, time_stp=1 / 3, cen_width=0.1)
    assert _shoot_ms(P, _radial(P, 0.3)) < 2.0 * _shoot_ms(P, np.zeros(P.var_num))


def test_steps_off_the_grid_skip_blocks():
    """Steps that outgrow their grid take the time of pair sums that never had one (a landmark
    far away, without momentum), whose distance test skips most blocks at this width."""
    from lddmm_b200 import problem

    P = problem.star_pair()
    P.time_num, P.time_stp, P.knl_width = 4, 1 / 3, 0.15
    a = _radial(P, 0.7)  # steps 1 and 2 are off the grid
    off = _shoot_ms(P, a)
    P.ini_nde = P.ini_nde.copy()
    P.ini_nde[0] *= 100.0
    a.reshape(P.T, -1, 3)[:, 0] = 0.0
    assert off < 1.2 * _shoot_ms(P, a)


def test_from_grid_to_pairs_against_fp64():
    """Step 0 on the grid, steps 1 and 2 beyond it, alone and in a batch with a pair too small
    for a grid: velocities, gradients and costate steps of a row sample against FP64 sums.
    FP32 sums are accurate against the sum of their terms' absolute values (the costate step's
    terms cancel): 1e-6 of each row's."""
    import ctypes as C

    import torch

    from lddmm_b200 import _lib, api

    P, small = _grid_problem(40000, 0.3, 5), _grid_problem(3000, 0.3, 6)
    P.dis_wgt = small.dis_wgt = 1e-3
    noise = np.random.default_rng(2).normal(size=(P.T, P.nde_num, 3))
    a = _radial(P, 0.7).reshape(P.T, -1, 3)
    a *= 1 + 0.3 * noise
    b = _radial(small, 0.2)
    rows = np.random.default_rng(1).integers(0, P.nde_num, 40)
    ab = lambda x: np.abs(x).sum(1)  # noqa: E731
    for batch in ([P], [P, small]):
        x = np.concatenate([a.reshape(-1), b][:len(batch)])
        with api.Context(batch) as ctx:
            q, v = ctx.shoot(x)[0]
            d = torch.from_numpy(x).cuda()
            f, g = torch.empty(len(batch), dtype=torch.float64, device="cuda"), d.clone()
            pst = d.clone()
            _lib.check(_lib.lib.lddmm_objgrd_costate(
                ctx.handle, *[C.c_void_p(z.data_ptr()) for z in (d, f, g, pst)]))
            f = f.cpu().numpy()
            g, pst = (z.cpu().numpy()[:P.var_num].reshape(a.shape) for z in (g, pst))
        w2 = P.knl_width ** 2
        energy = 0.0
        for t in range(P.T):
            dx = q[t][rows][:, None] - q[t][None]
            K = np.exp(-(dx ** 2).sum(-1) / w2)
            u, l = a[t] - pst[t], 0.5 * a[t] - pst[t]
            assert np.all(ab(K @ a[t] - v[t][rows]) < 1e-6 * ab(K @ np.abs(a[t])))
            assert np.all(ab(K @ u - g[t][rows] / P.time_stp) < 1e-6 * ab(K @ np.abs(u)))
            energy += 0.5 * P.time_stp * np.sum(a[t] * v[t])
            if t:
                lr = l[rows] @ a[t].T + a[t][rows] @ l.T
                dq = -2 / w2 * ((K * lr)[..., None] * dx).sum(1)
                step = (pst[t][rows] - pst[t - 1][rows]) / P.time_stp
                al, ar = np.abs(l), np.abs(a[t])
                tot = 2 / w2 * (K * (al[rows] @ ar.T + ar[rows] @ al.T)
                                * np.sqrt((dx ** 2).sum(-1))).sum(1)
                assert np.all(ab(dq - step) < 1e-6 * tot)
        value, _ = api.varifold(P, q[-1])
        assert abs(f[0] - energy - P.dis_wgt * value) < 1e-6 * abs(f[0])


def test_momenta_on_a_part_of_a_gridded_shape():
    """Momenta on a cap only.  The grid's kernel is wrong by an absolute 3.6e-11 where it is
    near 1, less further out (1e-6 of itself at 4.2 scaled units, 3.5 widths), and the node
    sums are multiples of N max|a| 2^-61: every row, however far from the momenta, is within
    1e-6 of its own sum of absolute values (the FP32 coordinates of pair sums leave as much
    there), or within 1e-12 of the largest."""
    from lddmm_b200 import api

    P = _grid_problem(40000, 0.3, 5)
    rng = np.random.default_rng(8)
    a = (rng.normal(size=(P.T, 40000, 3)) * 0.01).astype(np.float32).astype(np.float64)
    a[:, P.ini_nde[:, 2] < 0.6] = 0.0
    with api.Context(P) as ctx:
        (q, v), = ctx.shoot(a.reshape(-1))
    rows = rng.integers(0, 40000, 400)
    for t in range(P.T):
        K = np.exp(-((q[t][rows][:, None] - q[t][None]) ** 2).sum(-1) / P.knl_width ** 2)
        own, err = (K @ np.abs(a[t])).sum(1), np.abs(K @ a[t] - v[t][rows]).sum(1)
        assert np.all(err < 1e-6 * own + 1e-12 * own.max())


@pytest.mark.parametrize("kind", ["multiply", "dq"])
def test_single_sums_prepare_no_grid(kind):
    """One kernel sum of 60,000 3D Gaussian points on host arrays costs about what the Matern
    sum of the same size does (whose kernel takes longer): no k-d order, no grids."""
    import time

    from lddmm_b200 import api

    rng = np.random.default_rng(4)
    q, a = rng.normal(size=(2, 60000, 3))
    q /= np.linalg.norm(q, axis=1, keepdims=True)

    def ms(order):
        t = []
        for _ in range(6):  # the first one tunes
            t0 = time.perf_counter()
            api.multiplyKernel(q, a, order, 0.3) if kind == "multiply" else \
                api.dqKernel(q, a, a, order, 0.3)
            t.append(time.perf_counter() - t0)
        return min(t)

    assert ms(-1) < 1.5 * ms(1)


@pytest.mark.parametrize("far", [np.inf, -np.inf, 1e30])
def test_a_point_at_infinity_adds_nothing(far):
    """Beyond the persistent forms' sizes: K of a point at infinity is 0, for every other row."""
    from lddmm_b200 import api

    rng = np.random.default_rng(6)
    q, a = rng.normal(size=(2, 10500, 3))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    q = q[np.argsort(q[:, 2])]  # compact tiles
    v0 = api.multiplyKernel(np.delete(q, 7000, 0), np.delete(a, 7000, 0), -1, 1.0)
    q[7000, 1] = far
    v = np.delete(api.multiplyKernel(q, a, -1, 1.0), 7000, 0)
    assert rel(v, v0) < 1e-6
