"""Timing cases of the library: what a registration program has it do, through its public
entry points, from single kernel sums to the 163,842-landmark pair.

The all-pairs sums are evaluated in FP32 with compensated accumulation and returned in
FP64 buffers (about 1e-7 relative accuracy), so ``run`` hands its results on in float32,
the precision that they carry (as ``warmstart.generate`` does with its labels).

Kinds:
  objgrd    one objective + gradient on device buffers (``lddmm_objgrd_device``): the
            body of every optimiser iteration, for one pair or an uneven batch
  lbfgs     L-BFGS iterations of a resident context (``lddmm_lbfgs_device``)
  register  the whole ``LDDMM`` call on host arrays (``api.LDDMM``)
  ksum      one kernel sum on device buffers (``lddmm_multiply_kernel_noalloc``)
  dq        the two-set ``dqKernel`` on host arrays
  ws_grad   loss and gradient of the warm-start network (one training batch)
  ws_pred   its prediction of momenta for a batch of targets
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from lddmm_b200 import _lib, api, problem, shapes, warmstart
from lddmm_b200._lib import check, lib


def listed():
    return [
        # the 2D circle -> square registration's evaluation: pure latency
        dict(name="curve_200", kind="objgrd", mesh="curve", n=200, m=256, order=-1, width=0.5,
             cen="G", cen_width=0.2, dir="B", steps=20, wgt=1.0),
        # the reference's 2D example: Bessel-form Matern, Cauchy centres
        dict(name="curve_500_matern", kind="objgrd", mesh="curve", n=500, m=1000, order=3,
             width=0.025, cen="C", cen_width=0.1, dir="B", steps=20, wgt=100.0),
        # the headline sphere -> cube evaluation
        dict(name="sphere_2562", kind="objgrd", mesh="cube", n=2562, m=12288, order=1,
             width=0.4, cen="G", cen_width=0.15, dir="B", steps=20, wgt=1.0),
        # an odd-sized decimated mesh, as the population's larger pairs
        dict(name="mesh_9001", kind="objgrd", mesh="decimated", n=9001, m=14998, order=-1,
             width=0.3, cen="G", cen_width=0.1, dir="B", steps=10, wgt=1.0),
        # a dense surface pair: a step fills the GPU
        dict(name="star_40962", kind="objgrd", mesh="star", n=40962, m=20480, order=-1,
             width=0.3, cen="G", cen_width=0.1, dir="B", steps=10, wgt=1.0),
        # the large pair, the biggest single registration
        dict(name="star_163842", kind="objgrd", mesh="star", n=163842, m=81920, order=-1,
             width=0.3, cen="G", cen_width=0.1, dir="B", steps=10, wgt=1.0),
        # a slice of the uneven population: 12 pairs of 500 to 20,000 landmarks
        dict(name="batch_12", kind="objgrd", mesh="population", n=20000, m=40000, pairs=12,
             order=-1, width=0.3, cen="G", cen_width=0.1, dir="B", steps=10, wgt=1.0),
        # the head of the sphere -> cube registration: evaluations, line searches, updates
        dict(name="lbfgs_2562", kind="lbfgs", mesh="cube", n=2562, m=12288, order=1,
             width=0.4, cen="G", cen_width=0.15, dir="B", steps=20, wgt=1.0, iters=6),
        # a small registration called the MATLAB way, host arrays in and out
        dict(name="register_200", kind="register", mesh="curve", n=200, m=256, order=-1,
             width=0.5, cen="G", cen_width=0.2, dir="B", steps=20, wgt=1.0, iters=6),
        # one kernel sum inside somebody else's device program
        dict(name="ksum_10243", kind="ksum", dim=3, n=10243, order=-1, width=0.3),
        # one training batch of the configured warm-start network
        dict(name="ws_grad_64", kind="ws_grad", n=2562, m=5120, pairs=64, steps=10, local=0),
        # momenta for a few new targets, with local target features
        dict(name="ws_pred_8", kind="ws_pred", n=2562, m=5120, pairs=8, steps=10, local=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["curve", "surface", "batch", "lbfgs", "register", "ksum", "dq",
                        "ws_grad", "ws_pred"], [4, 8, 2, 2, 1, 2, 1, 1, 1])[0]
    if kind in ("curve", "register"):
        order = rng.choice([-1, -1, 1, 3, 4])
        c = dict(kind="objgrd", mesh="curve", n=_log_int(rng, 40, 2000),
                 m=4 * _log_int(rng, 12, 600), order=order,
                 width=rng.choice([0.2, 0.3, 0.5]) if order < 0 else rng.choice([0.025, 0.1, 0.3]),
                 cen=rng.choice("GGC"), cen_width=rng.choice([0.1, 0.2]), dir=rng.choice("BBBL"),
                 steps=rng.choice([10, 20]), wgt=rng.choice([1.0, 10.0]))
        if kind == "register":
            c.update(kind="register", n=_log_int(rng, 40, 600), order=-1,
                     width=rng.choice([0.3, 0.5]), cen="G", cen_width=0.2, dir="B", wgt=1.0,
                     iters=rng.randint(3, 6))
        return c
    if kind in ("surface", "lbfgs"):
        order = rng.choice([-1, -1, -1, -1, 1, 1, 1, 2, 3, 4])
        c = dict(kind="objgrd", mesh="decimated", n=_log_int(rng, 300, 40000),
                 m=2 * _log_int(rng, 300, 20000), order=order,
                 width=rng.choice([0.2, 0.3, 0.4] if order < 2 else [0.15, 0.2]),
                 cen=rng.choice("GGGGC"), cen_width=rng.choice([0.1, 0.15, 0.2]),
                 dir=rng.choice("BBBBBLOU"), steps=rng.choice([10, 10, 20]),
                 wgt=rng.choice([1.0, 10.0]))
        if kind == "lbfgs":
            c.update(kind="lbfgs", n=_log_int(rng, 300, 8000), order=rng.choice([-1, 1]),
                     cen="G", dir="B", iters=rng.randint(3, 6), wgt=1.0)
        return c
    if kind == "batch":
        return dict(kind="objgrd", mesh="population", n=_log_int(rng, 1000, 12000),
                    m=_log_int(rng, 2000, 30000), pairs=rng.randint(2, 16),
                    order=rng.choice([-1, -1, 1]), width=0.3, cen="G", cen_width=0.1, dir="B",
                    steps=10, wgt=1.0)
    if kind == "ksum":
        return dict(kind="ksum", dim=rng.choice([2, 3, 3, 3]), n=_log_int(rng, 100, 32768),
                    order=rng.choice([-1, -1, -1, 1, 2, 3]), width=rng.choice([0.2, 0.3, 0.5]))
    if kind == "dq":
        return dict(kind="dq", dim=rng.choice([2, 3, 3]), n=_log_int(rng, 100, 12000),
                    m=_log_int(rng, 100, 12000), order=rng.choice([-1, 1, 2]),
                    width=rng.choice([0.2, 0.3, 0.5]))
    return dict(kind=kind, n=rng.choice([642, 2562]), m=2 * _log_int(rng, 300, 2560),
                pairs=_log_int(rng, 2, 64), steps=10,
                local=0 if kind == "ws_grad" else rng.choice([0, 8, 24]))


# ------------------------------------------------------------------------ inputs

def _curve(n, rng, amp):
    """n points of a closed star-shaped curve, radius 1 + a few small harmonics."""
    th = 2.0 * np.pi * np.arange(n) / n
    r = np.ones(n)
    for k in range(1, 5):
        r += amp / k * (rng.normal() * np.cos(k * th) + rng.normal() * np.sin(k * th))
    e = np.stack([np.arange(n), (np.arange(n) + 1) % n], axis=1).astype(np.int32)
    return np.stack([r * np.cos(th), r * np.sin(th)], axis=1), e


def _mesh(case, k, rng):
    """Source and target meshes of pair k (host arrays)."""
    kind, n, m = case["mesh"], case["n"], case["m"]
    if kind == "population":  # log-spread sizes up to the case's, the same for every seed
        if k:
            u = random.Random(1000 * n + k)
            n = _log_int(u, min(500, n), n)
            m = _log_int(u, 1000, m)
        kind = "decimated"
    if kind == "curve":
        return _curve(n, rng, 0.05), shapes.square_boundary(m, float(rng.uniform(0.7, 1.0)))
    s1, s2 = (int(x) for x in rng.integers(0, 2**31 - 1, 2))
    if kind == "cube":
        v, f = shapes.icosphere(round(math.log((n - 2) / 10, 4)))
        r = shapes.star_radius(v, 4, 0.02, s1)
        return (v * r[:, None], f), shapes.cube_surface(round(math.sqrt(m / 12)), 1.0)
    if kind == "star":
        return (shapes.star_surface(round(math.log((n - 2) / 10, 4)), 8, 0.05, s1),
                shapes.star_surface(round(math.log(m / 20, 4)), 8, 0.05, s2))
    return (shapes.decimated_star(n, 8, 0.05, s1),
            shapes.decimated_star(max(m // 2 + 2, 12), 8, 0.05, s2))


def _momenta(P, rng):
    """Momenta as a registration meets them: a smooth field that varies over time plus
    node noise, scaled so that the flow moves the shape by about a quarter."""
    q, T = P.ini_nde, P.T
    rows = q[rng.integers(0, q.shape[0], 64)]
    d = np.sqrt(((rows[:, None] - q[None]) ** 2).sum(-1)) / P.knl_width
    mass = float((np.exp(-d * d) if P.knl_order < 0 else (1 + d) * np.exp(-d)).sum(1).mean())
    out = np.empty((T, q.shape[0], P.dim))
    base = rng.normal(size=(3, P.dim, 1 + P.dim))
    for t in range(T):
        w = np.array([1.0, t / T, (t / T) ** 2])
        c = np.tensordot(w, base, 1)
        out[t] = c[:, 0] + q @ c[:, 1:].T
    out += 0.5 * rng.normal(size=out.shape)
    return (out * (0.15 / mass)).reshape(-1)


def _problems(case, seed):
    rng = np.random.default_rng(seed)
    probs, alps = [], []
    for k in range(case.get("pairs", 1)):
        (v, f), (tv, tf) = _mesh(case, k, rng)
        cen, dr, vol = shapes.varifold_of(tv, tf)
        P = problem.Problem(v, f, cen, dr, vol, knl_order=case["order"],
                            knl_width=case["width"], time_num=case["steps"] + 1,
                            time_stp=1.0 / case["steps"], cen_type=case["cen"],
                            cen_width=case["cen_width"], dir_type=case["dir"],
                            dir_width=1.0 if case["dir"] in "OU" else 0.0,
                            dis_wgt=case["wgt"])
        probs.append(P)
        alps.append(_momenta(P, rng))
    return probs, alps


def _points(case, seed):
    """Points on a unit sphere's (circle's) neighbourhood and vectors, FP64."""
    rng = np.random.default_rng(seed)

    def pts(n):
        x = rng.normal(size=(n, case["dim"]))
        return x / np.linalg.norm(x, axis=1, keepdims=True) * rng.uniform(0.9, 1.1, (n, 1))

    if case["kind"] == "ksum":
        return pts(case["n"]), rng.normal(size=(case["n"], case["dim"]))
    return (pts(case["n"]), pts(case["m"]), rng.normal(size=(case["n"], case["dim"])),
            rng.normal(size=(case["m"], case["dim"])))


def _ws_dims(case):
    r16 = lambda n: (n + 15) // 16 * 16  # noqa: E731
    t3, pin = 3 * case["steps"], 3 + 64 + 7 * case["local"]
    return [(16, 7, 64, 64), (64, 64, 64, 64), (r16(pin), pin, 256, 256), (256, 256, 256, 256),
            (256, 256, r16(t3), t3)]


def _ws_inputs(case, seed):
    """Source landmarks, target features, labels, network parameters (host arrays)."""
    rng = np.random.default_rng(seed)
    v, _ = shapes.icosphere(round(math.log((case["n"] - 2) / 10, 4)))
    tri = np.empty((case["pairs"], case["m"], 7), dtype=np.float32)
    d = rng.normal(size=(case["m"], 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    for k in range(case["pairs"]):
        tri[k, :, :3] = d * shapes.star_radius(d, 6, 0.08, int(rng.integers(2**31 - 1)))[:, None]
        tri[k, :, 3:6] = d + 0.05 * rng.normal(size=d.shape)
        tri[k, :, 3:6] /= np.linalg.norm(tri[k, :, 3:6], axis=1, keepdims=True)
        tri[k, :, 6] = rng.uniform(0.7, 1.3, case["m"])
    w = rng.normal(size=(case["pairs"], 3, 3 * case["steps"]))
    lab = (np.einsum("nd,pdc->pnc", v, w) + 0.3 * rng.normal(
        size=(case["pairs"], v.shape[0], 3 * case["steps"]))).astype(np.float32)
    flat = []
    for i, ir, o, orr in _ws_dims(case):
        wt, b = np.zeros((o, i), np.float32), np.zeros(o, np.float32)
        wt[:orr, :ir] = rng.uniform(-1, 1, (orr, ir)) / math.sqrt(ir)
        b[:orr] = rng.uniform(-1, 1, orr) / math.sqrt(ir)
        flat += [wt.ravel(), b]
    return v, tri, lab, np.concatenate(flat)


# ----------------------------------------------------------------------- the passes

def _ptr(t):
    return C.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind in ("objgrd", "lbfgs"):
        probs, alps = _problems(case, seed)
        s["stream"] = torch.cuda.Stream()
        s["ctx"] = api.Context(probs, stream=s["stream"].cuda_stream)
        s["alp"] = torch.from_numpy(np.concatenate(alps)).cuda()
    elif kind == "register":
        (P,), (a,) = _problems(case, seed)
        s["args"] = (P.ini_nde.T.copy(), a.reshape(P.T, P.nde_num, P.dim).transpose(2, 1, 0).copy(),
                     dict(dfmElmVtxMat=P.elm_vtx.T + 1, tgtCenPosMat=P.tgt_cen.T,
                          tgtUniDirMat=P.tgt_dir.T, tgtElmVolVec=P.tgt_vol, cenKnlType=P.cen_type,
                          cenKnlWidth=P.cen_width, dirKnlType=P.dir_type,
                          dirKnlWidth=P.dir_width, disWgt=P.dis_wgt),
                     P.knl_order, P.knl_width, 1.0 + 1e-9, P.time_stp,
                     dict(MaxIterations=case["iters"], OptimalityTolerance=1e-9, Columns=5))
    elif kind == "ksum":
        s["q"], s["a"] = (torch.from_numpy(x).cuda() for x in _points(case, seed))
    elif kind == "dq":
        s["args"] = _points(case, seed)
    else:
        v, tri, lab, par = _ws_inputs(case, seed)
        s["ws"] = warmstart.WarmStart(v, case["steps"], case["pairs"], case["m"], 1.0,
                                      local_k=case["local"])
        s["ws"].params = par
        s["tri"], s["lab"] = torch.from_numpy(tri).cuda(), torch.from_numpy(lab).cuda()
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "objgrd":
        ctx = s["ctx"]
        with torch.cuda.stream(s["stream"]):
            f = torch.empty(ctx.P, dtype=torch.float64, device="cuda")
            g = torch.empty_like(s["alp"])
            check(lib.lddmm_objgrd_device(ctx.handle, _ptr(s["alp"]), _ptr(f), _ptr(g), 0))
            return f.float(), g.float()
    if kind == "lbfgs":
        ctx = s["ctx"]
        with torch.cuda.stream(s["stream"]):
            x = s["alp"].clone()
            opt = _lib.Opt(case["iters"], 1e-9, 1e-4, 0.9, 5, 0, 0.0)
            res = (_lib.Result * ctx.P)()
            check(lib.lddmm_lbfgs_device(ctx.handle, C.byref(opt), _ptr(x), res))
            return torch.tensor([r.fcn for r in res]), x.float()
    if kind == "register":
        o = api.LDDMM(*s["args"])
        return [x.astype(np.float32) for x in (o.ndeStk, o.vlcStk, o.alpStk)]
    if kind == "ksum":
        v = torch.empty_like(s["q"])
        check(lib.lddmm_multiply_kernel_noalloc(case["dim"], case["n"], _ptr(s["q"]),
                                                _ptr(s["a"]), case["order"], case["width"],
                                                _ptr(v), None))
        return v.float()
    if kind == "dq":
        qi, qj, l, r = s["args"]
        dqi, dqj = api.dqKernel(qi, qj, l, r, case["order"], case["width"])
        return dqi.astype(np.float32), dqj.astype(np.float32)
    if kind == "ws_grad":
        return s["ws"].grad(s["tri"], s["lab"])
    return s["ws"].predict(s["tri"]).float()


# ------------------------------------------------------------------------- the work

def work(case):
    """Pair interactions times the arithmetic of one (subtractions, squared distance,
    kernel function, accumulations), and inputs and outputs once."""
    kind = case["kind"]
    if kind.startswith("ws"):
        rows, tri = case["pairs"] * case["n"], case["pairs"] * case["m"]
        mac = sum(i * o * (tri if k < 2 else rows) for k, (_, i, _, o) in enumerate(_ws_dims(case)))
        back = 3 if kind == "ws_grad" else 1
        return dict(bytes=4.0 * (tri * 7 + rows * 3 * case["steps"]), flops=2.0 * mac * back)
    n, k = float(case["n"]), 1.0 if case.get("order", -1) < 0 else 4.0
    if kind in ("ksum", "dq"):
        d = case["dim"]
        m = n if kind == "ksum" else 2.0 * case["m"]
        per = (3 * d + k + 2 * d) if kind == "ksum" else (3 * d + k + 4 * d + 1)
        return dict(bytes=8.0 * d * (3 * n + (0 if kind == "ksum" else 3 * case["m"])),
                    flops=n * m * per)
    d, t = 2 if case["mesh"] == "curve" else 3, case["steps"]
    nn, ed, et = [n], [n if d == 2 else 2 * n - 4], [float(case["m"])]
    if case["mesh"] == "population":
        for j in range(1, case["pairs"]):
            u = random.Random(1000 * case["n"] + j)
            nn.append(float(_log_int(u, min(500, case["n"]), case["n"])))
            ed.append(2 * nn[-1] - 4)
            et.append(float(_log_int(u, 1000, case["m"])))
    flops = sum(t * a * a * ((5 * d + k) + (9 * d + 1 + k)) + e * (e + f) * (9 * d + 5)
                for a, e, f in zip(nn, ed, et))
    evals = 1 if kind == "objgrd" else case["iters"] + 1
    nvar = sum(nn) * d * t
    return dict(bytes=evals * (16.0 * nvar + 8.0 * (2 * d + 1) * sum(et) + 8.0 * d * sum(nn)),
                flops=evals * flops)


# ---------------------------------------------------------------- 64-bit references

def _kernel(r2, order, w, dim):
    """K and the factor W of dK/dq_i = W (q_i - q_j), from squared distances."""
    if order < 0:
        k = torch.exp(r2 * (-1.0 / w ** 2))
        return k, k * (-2.0 / w ** 2)
    x = torch.sqrt(r2) / w
    if dim == 2:
        y = x.clamp_min(1e-150)
        p0, p1 = y * y * torch.special.modified_bessel_k0(y), y * torch.special.modified_bessel_k1(y)
        p0, p1, x2 = torch.where(x > 0, p0, 0.0), torch.where(x > 0, p1, 1.0), x * x
        form = [p1, 0.5 * p0 + p1, (4 * p0 + (8 + x2) * p1) / 8,
                ((24 + x2) * p0 + 8 * (6 + x2) * p1) / 48,
                (12 * (16 + x2) * p0 + (384 + x2 * (72 + x2)) * p1) / 384]
        return form[order], (form[order - 1] * (-1.0 / (2 * order * w * w)) if order else 0.0 * x)
    e = torch.exp(-x)
    pk = [1 + 0 * x, 1 + x, 1 + x + x * x / 3, 1 + x + 0.4 * x * x + x ** 3 / 15,
          1 + x + 3 * x * x / 7 + 2 * x ** 3 / 21 + x ** 4 / 105][order]
    pw = [0 * x, 1 + 0 * x, 1 + x, 3 + 3 * x + x * x, 15 + 15 * x + 6 * x * x + x ** 3][order]
    return e * pk, e * pw * (-1.0 / ([1, 1, 3, 15, 105][order] * w * w))


def _rows(n, m):
    step = max(1, (1 << 25) // m)
    return [slice(i, min(i + step, n)) for i in range(0, n, step)]


def _r2(a, b):
    return sum((a[:, None, d] - b[None, :, d]) ** 2 for d in range(a.shape[1]))


def _sums(qi, qj, order, w, u=None, l=None, r=None, li=None, ri=None):
    """sum_j K u_j and sum_j (li.r_j [+ ri.l_j]) dK/dq_i."""
    v, dq = torch.zeros_like(qi), torch.zeros_like(qi)
    for s in _rows(qi.shape[0], qj.shape[0]):
        k, wt = _kernel(_r2(qi[s], qj), order, w, qi.shape[1])
        if u is not None:
            v[s] = k @ u
        if r is not None:
            c = li[s] @ r.T
            if l is not None:
                c += ri[s] @ l.T
            c *= wt
            dq[s] = qi[s] * c.sum(1, keepdim=True) - c @ qj
    return v, dq


def _geometry(q, e):
    if q.shape[1] == 2:
        t = q[e[:, 1]] - q[e[:, 0]]
        a = t.norm(dim=1)
        return 0.5 * (q[e[:, 0]] + q[e[:, 1]]), t / a[:, None], a
    n = torch.linalg.cross(q[e[:, 1]] - q[e[:, 0]], q[e[:, 2]] - q[e[:, 0]])
    a = n.norm(dim=1)
    return (q[e[:, 0]] + q[e[:, 1]] + q[e[:, 2]]) / 3, n / a[:, None], 0.5 * a


def _varifold(P, x, y):
    """sum_ij a_i a_j k(c_i, c_j) b(n_i . n_j) of two element sets (c, n, a)."""
    r2 = _r2(x[0], y[0]) / P.cen_width ** 2
    k = torch.exp(-r2) if P.cen_type == "G" else 1 / (1 + r2)
    g = x[1] @ y[1].T
    w2 = 2 / P.dir_width ** 2 if P.dir_width else 0
    b = {"B": lambda: g * g, "L": lambda: g, "O": lambda: torch.exp((g - 1) * w2),
         "U": lambda: torch.exp((g * g - 1) * w2)}[P.dir_type]()
    return x[2] @ (k * b) @ y[2]


def _objgrd(P, alp):
    cu = lambda x, t=torch.float64: torch.from_numpy(np.ascontiguousarray(x)).to("cuda", t)  # noqa: E731
    q = [cu(P.ini_nde)]
    a = alp.view(P.T, P.nde_num, P.dim)
    dt, o, w = P.time_stp, P.knl_order, P.knl_width
    f = 0.0
    for t in range(P.T):
        v, _ = _sums(q[t], q[t], o, w, u=a[t])
        f = f + 0.5 * dt * (a[t] * v).sum()
        q.append(q[t] + dt * v)
    qT = q[-1].clone().requires_grad_()
    geo = _geometry(qT, cu(P.elm_vtx, torch.int64))
    leaf = [x.detach().requires_grad_() for x in geo]
    tgt = [cu(P.tgt_cen), cu(P.tgt_dir), cu(P.tgt_vol)]
    for other, fac in ((leaf, 1.0), (tgt, -2.0)):
        for s in _rows(leaf[0].shape[0], 2 * other[0].shape[0]):
            val = fac * P.dis_wgt * _varifold(P, [x[s] for x in leaf], other)
            val.backward()
            f = f + val.detach()
    for s in _rows(tgt[0].shape[0], tgt[0].shape[0]):
        f = f + P.dis_wgt * _varifold(P, [x[s] for x in tgt], tgt)
    torch.autograd.backward(geo, [x.grad for x in leaf])
    p, grd = -qT.grad, torch.empty_like(a)
    for t in range(P.T - 1, -1, -1):
        lt = 0.5 * a[t] - p
        v, dq = _sums(q[t], q[t], o, w, u=a[t] - p, l=lt, r=a[t], li=lt, ri=a[t])
        grd[t], p = dt * v, p - dt * dq
    return f, grd.reshape(-1)


def _lbfgs(P, x, iters, w1=1e-4, w2=0.9, mem=5):
    """L-BFGS with the weak-Wolfe bisection line search, two-loop directions."""
    f, g = _objgrd(P, x)
    pairs = []
    for _ in range(iters):
        d, al = -g.clone(), []
        for s, y in reversed(pairs):
            al.append((s @ d) / (s @ y))
            d = d - al[-1] * y
        if pairs:
            s, y = pairs[-1]
            d = d * ((s @ y) / (y @ y))
        for (s, y), c in zip(pairs, reversed(al)):
            d = d + (c - (y @ d) / (s @ y)) * s
        slope, t, lo, hi = float(g @ d), 1.0, 0.0, math.inf
        while True:
            fn, gn = _objgrd(P, x + t * d)
            if float(fn) >= float(f) + w1 * t * slope:
                hi = t
            elif float(gn @ d) <= w2 * slope:
                lo = t
            else:
                break
            t = 2 * t if hi == math.inf else 0.5 * (lo + hi)
        pairs = (pairs + [(t * d, gn - g)])[-mem:]
        x, f, g = x + t * d, fn, gn
    return f, x


def _network(case, seed):
    v, tri, lab, par = _ws_inputs(case, seed)
    v = torch.from_numpy(np.array(v, dtype=np.float32)).cuda()
    tri, lab = torch.from_numpy(tri).cuda(), torch.from_numpy(lab).cuda().double()
    par = torch.from_numpy(par).cuda().double().requires_grad_()
    layers, off = [], 0
    for i, ir, o, orr in _ws_dims(case):
        layers.append((par[off:off + o * i].view(o, i)[:orr, :ir], par[off + o * i:][:orr]))
        off += o * i + o
    gelu = torch.nn.functional.gelu
    lin = torch.nn.functional.linear
    out = []
    for p in range(case["pairs"]):
        h = lin(gelu(lin(tri[p].double(), *layers[0])), *layers[1])
        x = [v.double(), h.max(0).values.expand(v.shape[0], -1)]
        if case["local"]:
            d = tri[p, None, :, :3] - v[:, None]
            t = tri[p][(d * d).sum(-1).topk(case["local"], largest=False).indices].double()
            t[..., :3] = (t[..., :3] - v[:, None].double()) * 10
            x.append(t.flatten(1))
        out.append(lin(gelu(lin(gelu(lin(torch.cat(x, 1), *layers[2])), *layers[3])), *layers[4]))
    y = torch.stack(out)
    if case["kind"] == "ws_pred":
        return y.detach().view(len(out), v.shape[0], -1, 3).transpose(1, 2).reshape(len(out), -1)
    loss = (y - lab).square().mean()
    loss.backward()
    return float(loss.detach()), par.grad


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("ws"):
        return _network(case, seed)
    if kind in ("ksum", "dq"):
        x = [torch.from_numpy(a).cuda() for a in _points(case, seed)]
        if kind == "ksum":
            return _sums(x[0], x[0], case["order"], case["width"], u=x[1])[0]
        qi, qj, l, r = x
        return (_sums(qi, qj, case["order"], case["width"], li=l, r=r)[1].cpu().numpy(),
                _sums(qj, qi, case["order"], case["width"], li=r, r=l)[1].cpu().numpy())
    if case["n"] > 60000:
        return None  # 64-bit all-pairs sums of this size take minutes
    probs, alps = _problems(case, seed)
    alps = [torch.from_numpy(a).cuda() for a in alps]
    if kind == "objgrd":
        got = [_objgrd(P, a) for P, a in zip(probs, alps)]
        return torch.stack([f for f, _ in got]), torch.cat([g for _, g in got])
    P = probs[0]
    f, x = _lbfgs(P, alps[0], case["iters"])
    if kind == "lbfgs":
        return f.reshape(1), x
    a, q, vs = x.view(P.T, P.nde_num, P.dim), [torch.from_numpy(P.ini_nde).cuda()], []
    for t in range(P.T):
        vs.append(_sums(q[t], q[t], P.knl_order, P.knl_width, u=a[t])[0])
        q.append(q[t] + P.time_stp * vs[t])
    return [z.permute(2, 1, 0).cpu().numpy() for z in (torch.stack(q), torch.stack(vs), a)]
