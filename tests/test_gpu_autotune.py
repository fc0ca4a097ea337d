"""The launch-shape autotuner (lddmm_config.autotune, on by default): it times the
candidate shapes of each sweep on the context's own batch (64-row tiles per work
item, cluster splits, persistent or per-step time loops) and keeps the fastest.
Checked here: the chosen sizes are valid, its trial sweeps leave nothing behind (the
tuned context gives bitwise the same objective and gradient as a fresh context created
with those sizes given explicitly -- every reduction has a fixed order for a given
launch plan, and two-tile items give bitwise the sums of one-tile items), the result
agrees with the default context's within the FP32 tolerance, and the tuned shape is
never slower than the built-in rule's on the sphere -> cube pair and the large pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mrel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(np.max(np.abs(b)), 1e-300))


def test_autotune_valid_and_stateless():
    from lddmm_b200 import api, problem

    P = problem.sphere_to_cube(subdiv=5)  # 10,242 landmarks: per-step sweeps
    x = np.random.default_rng(7).normal(size=P.var_num) * 0.01
    with api.Context(P, autotune=True) as tuned:
        cfg = tuple(int(s) for s in tuned.launch_config())
        f1, g1 = tuned.objgrd(x)
    assert cfg[0] in (1, 2, 4, 8) and cfg[1] in (1, 2, 4, 8) and 1 <= cfg[2] <= 8
    with api.Context(P, cluster=cfg) as same:
        f2, g2 = same.objgrd(x)
    assert f1[0] == f2[0] and np.array_equal(g1, g2)
    with api.Context(P) as default:
        f3, g3 = default.objgrd(x)
    assert abs(f1[0] - f3[0]) <= 1e-6 * abs(f3[0])
    assert mrel(g1, g3) < 1e-5


def _eval_ms(ctx, reps, tries=3):
    """Fastest of `tries` measurements of the average evaluation time."""
    return min(ctx.time_sweeps(reps=reps)["eval"] for _ in range(tries))


@pytest.mark.parametrize("which", ["sphere2cube", "large_pair"])
def test_autotuned_shape_is_never_slower_than_the_rule(which):
    """The default context (autotuned: tiles per work item, cluster splits, persistent
    or per-step time loops) against the built-in rule (autotune off), on the 2562-
    landmark sphere -> cube pair and the 163,842-landmark star pair: the tuned shape's
    objective + gradient evaluation is at most 2 % slower (it is chosen by timing, so
    it should not be slower at all beyond noise)."""
    from lddmm_b200 import api, problem

    P = problem.sphere_to_cube() if which == "sphere2cube" else problem.star_pair()
    reps = 20 if which == "sphere2cube" else 2
    with api.Context(P, autotune=False) as rule:
        shape_rule = rule.launch_shape()
        ms_rule = _eval_ms(rule, reps)
    with api.Context(P) as tuned:
        shape_tuned = tuned.launch_shape()
        ms_tuned = _eval_ms(tuned, reps)
    print(f"{which}: rule {shape_rule} {ms_rule:.3f} ms, tuned {shape_tuned} {ms_tuned:.3f} ms")
    assert ms_tuned <= 1.02 * ms_rule, (shape_rule, ms_rule, shape_tuned, ms_tuned)


def _surface_pair(n, width=0.3):
    from lddmm_b200 import problem, shapes

    v, f = shapes.decimated_star(n, 8, 0.05, n)
    tv, tf = shapes.decimated_star(n, 8, 0.05, n + 1)
    return problem.Problem(v, f, *shapes.varifold_of(tv, tf), knl_order=-1, knl_width=width,
                           time_num=11, time_stp=0.1, cen_width=0.1)


def _loops_ms(ctx, reps, tries=3):
    """The same of a shooting and an adjoint step (the varifold's split is tuned by itself)."""
    t = [ctx.time_sweeps(reps=reps) for _ in range(tries)]
    return min(x["shoot"] + x["adjoint"] for x in t)


@pytest.mark.parametrize("n,width", [(3000, 0.3), (5000, 0.1), (9001, 0.3), (9001, 0.1)])
def test_tuned_time_loops_with_momenta(n, width):
    """The Gaussian per-step sweeps skip blocks according to the momenta and the width: the
    form that the tuner picks (on momenta of one magnitude) is at most 5 % slower, with random
    momenta, than the faster of the two that it chose from."""
    from lddmm_b200 import api

    P = _surface_pair(n, width)
    x = np.random.default_rng(n).normal(size=P.var_num) * 1e-4
    ms = {}
    for form in (0, 1, -1):
        with api.Context(P, persistent=form) as ctx:
            ctx.objgrd(x)
            ms[form] = _loops_ms(ctx, 20)
            shape = ctx.launch_shape()["persistent"] if form == 0 else shape
    print(n, width, shape, ms)
    assert ms[0] <= 1.05 * min(ms[1], ms[-1]), (shape, ms)


def test_contexts_of_other_widths_are_tuned_again():
    """A context of the same sizes takes over the shapes (no trial sweeps), one of another
    kernel width does not: what its sweeps skip differs."""
    import time

    from lddmm_b200 import api

    def seconds(P):
        t0 = time.perf_counter()
        with api.Context(P):
            pass
        return time.perf_counter() - t0

    P, other = _surface_pair(8999, 0.3), _surface_pair(8999, 0.2)
    seconds(P)
    again = min(seconds(P) for _ in range(3))
    assert seconds(other) > 1.5 * again
    assert min(seconds(other) for _ in range(3)) < 1.5 * again


def test_tuned_batch_of_small_gaussian_pairs():
    """30 pairs of 200 to 1,070 landmarks: the tuned form is at most 5 % slower than the
    persistent loops and than per-step launches, and its gradient is theirs to rounding."""
    from lddmm_b200 import api

    Ps = [_surface_pair(200 + 30 * k) for k in range(30)]
    x = np.concatenate([np.random.default_rng(k).normal(size=P.var_num) * 1e-4
                        for k, P in enumerate(Ps)])
    ms, out = {}, {}
    for form in (0, 1, -1):
        with api.Context(Ps, persistent=form) as ctx:
            out[form] = ctx.objgrd(x)
            ms[form] = _loops_ms(ctx, 20)
    assert ms[0] <= 1.05 * min(ms[1], ms[-1]), ms
    for form in (1, -1):
        assert np.allclose(out[form][0], out[0][0], rtol=1e-6)
        assert mrel(out[form][1], out[0][1]) < 1e-5


@pytest.mark.parametrize("kind", ["multiply", "dq"])
def test_single_sums_of_another_width_are_not_tuned_again(kind):
    """One sum per call: the trial sweeps of a size serve every kernel width."""
    import time

    from lddmm_b200 import api

    q, a = np.random.default_rng(3).normal(size=(2, 8900, 3))

    def seconds(width):
        t0 = time.perf_counter()
        api.multiplyKernel(q, a, -1, width) if kind == "multiply" else \
            api.dqKernel(q, a, a, -1, width)
        return time.perf_counter() - t0

    seconds(0.3)
    again = min(seconds(0.3) for _ in range(3))
    assert min(seconds(w) for w in (0.31, 0.32, 0.33)) < 2.0 * again
