"""The work that a flow solver has this library do, as cases that can be timed and compared.

A case is one velocity (or potential) evaluation of a particle set: the 2D field on device buffers, eagerly or as a
replayed graph, in the plain FP64 and the mixed form; the velocity step and the potential on host buffers; a batch of
independent solves; the 3D treecode on the octree and on the TreeCell. The particle sets are the package's own
workloads (jittered lattices with vortices, a multi-resolution boundary layer, a vortex ring).
"""
import math

import numpy as np
import torch

from lsmps_vpm_v2_b200 import (PREC_FP64, PREC_MIXED, Context, Particle, VelocityCalc, default_params, fmm2D,
                               treecell3d_params, workloads)
from lsmps_vpm_v2_b200._lib import PREC_MIXED_TC

FORMS = {"fp64": PREC_FP64, "mixed": PREC_MIXED, "mixed_tc": PREC_MIXED_TC}

#: A solver runs all its work on one stream: evaluations follow one another.
_stream = None


def stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---- the cases ----------------------------------------------------------------

def field2d(field, size, form, p, caps, graph, inactive=False, **more):
    """`size`: particles ("vortices"), lattice side ("lamb") or 1000 x the spacing factor ("layer")."""
    return dict(more, op="field2d", field=field, size=size, form=form, p=p, max_src=caps[0], max_par=caps[1],
                graph=graph, inactive=inactive)


def listed():
    return [
        # The smallest call: a start-up or near-body field of some thousand particles whose number changes from step
        # to step, so each evaluation is launched eagerly. Reference order and leaf caps.
        field2d("vortices", 2001, "fp64", 10, (50, 75), False, name="field2d_2k_fp64_eager"),
        # A wake after redistribution: odd size, the particles without vorticity marked inactive, eager, mixed form.
        field2d("vortices", 49_993, "mixed", 12, (50, 75), False, True, name="field2d_50k_mixed_eager_inactive"),
        # The 65,536-particle Lamb-Oseen lattice at the reference's parameters, in a loop of fixed particles.
        field2d("lamb", 256, "fp64", 10, (50, 75), True, name="field2d_lamb65k_fp64_graph"),
        # The 778,377-particle boundary layer: the plain form at the reference's parameters ...
        field2d("layer", 660, "fp64", 10, (50, 75), True, name="field2d_layer778k_fp64_graph"),
        # ... and the mixed form at the pair that the selector picks for 1e-4.
        field2d("layer", 660, "mixed", 8, (100, 150), True, name="field2d_layer778k_mixed_graph"),
        # High order: the setting for errors of 1e-6, mixed form.
        field2d("layer", 800, "mixed", 16, (50, 75), True, name="field2d_layer530k_mixed_p16"),
        # The velocity step of a CPU solver: host arrays in and out, literal boundary-layer spacings.
        dict(name="velocity2d_layer340k_host", op="velocity2d", field="layer", size=1000, form="fp64", p=10,
             max_src=50, max_par=75, inactive=False),
        # The pressure solver's potential, host arrays in and out.
        dict(name="potential2d_120k_host", op="potential2d", field="vortices", size=120_011, form="fp64", p=10,
             max_src=50, max_par=75, inactive=True),
        # A parameter study: 64 uneven solves at once.
        dict(name="batch2d_64_mixed", op="batch2d", solves=64, lo=4096, hi=400_000, layout=3, form="mixed", p=12,
             max_src=50, max_par=75),
        # 3D: the 222,688-particle ring by the default octree path, plain form.
        dict(name="ring3d_222k_fp64", op="velocity3d", h=0.02, form="fp64", support=2.0),
        # The same ring by the TreeCell path, plain form, near-body targets flagged.
        dict(name="treecell3d_222k_fp64", op="treecell3d", h=0.02, form="fp64", support=2.0, targets=True),
        # The largest: the 2,009,183-particle ring, mixed form.
        dict(name="ring3d_2m_mixed", op="velocity3d", h=0.0096, form="mixed", support=2.0),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["field2d"] * 5 + ["velocity2d", "potential2d", "batch2d", "velocity3d", "velocity3d",
                                       "treecell3d"])
    form = rng.choice(["fp64", "mixed"])
    caps = rng.choice([(50, 75), (50, 75), (100, 150), (30, 50)])
    p = rng.choice([8, 10, 12, 16])
    if op == "batch2d":
        return dict(op=op, solves=rng.randint(3, 80), lo=rng.randint(1000, 8000), hi=rng.randint(20_000, 300_000),
                    layout=rng.randrange(1 << 20), form=form, p=p, max_src=caps[0], max_par=caps[1])
    if op in ("velocity3d", "treecell3d"):
        support = rng.choice([2.0, 2.0, 3.0])
        # the stricter far test takes about three times as long: no more than 360k particles there
        h = round(_log_uniform(rng, 0.0125 if support == 2.0 else 0.017, 0.07), 5)
        case = dict(op=op, h=h, form=form, support=support)
        if op == "treecell3d":
            case["targets"] = rng.random() < 0.5
        return case
    field = rng.choice(["lamb", "vortices", "layer"])
    if field == "lamb":
        size = int(_log_uniform(rng, 16, 700))
    elif field == "vortices":
        size = int(_log_uniform(rng, 300, 1_200_000))
    else:
        size = int(_log_uniform(rng, 600, 4000))
    if op == "field2d":
        if rng.random() < 0.15:
            form, p = rng.choice([("mixed_tc", 8), ("mixed_tc", 12), ("mixed", 20)])
        return field2d(field, size, form, p, caps, rng.random() < 0.5, rng.random() < 0.3)
    if op == "potential2d":
        form = "fp64"
    return dict(op=op, field=field, size=size, form=form, p=p, max_src=caps[0], max_par=caps[1],
                inactive=rng.random() < 0.3)


# ---- inputs -------------------------------------------------------------------

def _vortices(n, seed):
    """multi_vortex_2d cut to exactly n particles (its last lattice row stays incomplete)."""
    side = math.isqrt(max(n - 1, 0)) + 1
    d = workloads.multi_vortex_2d(side * side, seed)
    return {k: v[:n] if isinstance(v, np.ndarray) else v for k, v in d.items()}


def _particles2d(case, seed):
    if case["field"] == "lamb":
        d = workloads.lamb_oseen_2d(n_side=case["size"], seed=seed)
    elif case["field"] == "layer":
        d = workloads.boundary_layer_2d(scale=case["size"] / 1000, seed=seed)
    else:
        d = _vortices(case["size"], seed)
    if case["inactive"]:
        # The solver's own mark: particles of too little vorticity are inactive, and carry none.
        on = np.abs(d["omega"]) >= 1e-4 * np.abs(d["omega"]).max()
        d = dict(d, active=on.astype(np.uint8), omega=np.where(on, d["omega"], 0.0), q=np.where(on, d["q"], 0.0))
    return d


def _batch_sizes(case):
    rng = np.random.default_rng(case["layout"])
    return np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["solves"])).astype(int)


def _batch(case, seed):
    ds = [_vortices(int(m), seed * 1000 + i) for i, m in enumerate(_batch_sizes(case))]
    offs = np.concatenate([[0], np.cumsum([d["x"].size for d in ds])]).astype(np.int64)
    return offs, {k: np.concatenate([d[k] for d in ds]) for k in ("x", "y", "q", "active")}


def _ring(case, seed):
    return workloads.vortex_ring_3d(h=case["h"], seed=seed)


def _targets3d(d):
    """Near-body targets: the particles of one half of the ring."""
    return (d["x"] >= 0.0).astype(np.uint8)


def _params(case):
    if case["op"] == "treecell3d":
        return treecell3d_params(precision=FORMS[case["form"]], support_3d=case["support"])
    if case["op"] == "velocity3d":
        return default_params(precision=FORMS[case["form"]], support_3d=case["support"])
    return default_params(precision=FORMS[case["form"]], p=case["p"], max_src=case["max_src"],
                          max_par=case["max_par"], binom=0 if case["form"] == "fp64" else 1,
                          use_graph=int(case.get("graph", case["op"] == "batch2d")))


def prepare(case, seed):
    op, prm = case["op"], _params(case)
    ctx = Context(0)
    ctx.set_stream(stream().cuda_stream)
    if op in ("velocity2d", "potential2d"):
        d = _particles2d(case, seed)
        if op == "velocity2d":
            return dict(op=op, calc=VelocityCalc(ctx, prm, u_inf=1.0),
                        par=Particle(d["x"], d["y"], d["s"], d["omega"], d["active"]))
        return dict(op=op, fmm=fmm2D(ctx, prm), pos=np.stack([d["x"], d["y"]], axis=1), active=d["active"], q=d["q"])
    if op == "field2d":
        d, names, outs = _particles2d(case, seed), ("x", "y", "q", "active"), 2
    elif op == "batch2d":
        offs, d = _batch(case, seed)
        names, outs = ("x", "y", "q", "active"), 2
    else:
        d, names, outs = _ring(case, seed), ("x", "y", "z", "ax", "ay", "az", "active"), 3
    dev = [torch.from_numpy(np.ascontiguousarray(d[k])).cuda() for k in names]
    st = dict(op=op, ctx=ctx, prm=prm, n=dev[0].numel(), dev=dev, out=[torch.zeros_like(dev[0]) for _ in range(outs)])
    if op == "batch2d":
        st["offs"] = offs
    if op == "treecell3d":
        st["target"] = torch.from_numpy(_targets3d(d)).cuda() if case["targets"] else None
    stream().wait_stream(torch.cuda.current_stream())
    return st


def run(st):
    op = st["op"]
    if op == "velocity2d":
        st["calc"].get_velocity(st["par"])
        return st["par"].u, st["par"].v
    if op == "potential2d":
        st["fmm"].calcPotential(None, st["pos"], st["active"], st["q"])
        return st["fmm"].get_Potential()
    ctx, prm, dev, out = st["ctx"], st["prm"], st["dev"], st["out"]
    if op == "field2d":
        ctx.field2d_device(*dev, *out, prm)
        return out
    ptr = [t.data_ptr() for t in dev]
    res = [t.data_ptr() for t in out]
    if op == "batch2d":
        ctx.field2d_batched_device(st["offs"], *ptr, *res, prm)
    elif op == "velocity3d":
        ctx.velocity3d_device(st["n"], *ptr, *res, prm)
    else:
        target = st["target"]
        ctx.velocity3d_treecell_device(st["n"], *ptr, None if target is None else target.data_ptr(), *res, prm)
    return out


# ---- what a pass cannot do without ----------------------------------------------

def _count2d(case):
    if case["op"] == "batch2d":
        return int(_batch_sizes(case).sum())
    if case["field"] == "lamb":
        return case["size"] ** 2
    if case["field"] == "vortices":
        return case["size"]
    s = case["size"] / 1000  # the three zones of the boundary layer by area over spacing squared
    return int(0.4 / (0.005 * s) ** 2 + 39.6 / (0.02 * s) ** 2 + 360 / (0.04 * s) ** 2)


def work(case):
    if case["op"] in ("velocity3d", "treecell3d"):
        # the ring's tube of radius 3 sigma; near pairs at 26 flops and far ones at 130, per target as counted on the
        # 222k ring (340 and 480), growing with the far test's sphere
        n = 2 * math.pi * math.pi * 0.3 ** 2 / case["h"] ** 3
        far = (case["support"] / 2) ** 2
        t = n * (0.5 if case.get("targets") else 1.0)
        return {"bytes": n * 49 + t * 24, "flops": t * far * (340 * 26 + 480 * 130)}
    n, p = _count2d(case), case["p"]
    leaf = 0.5 * case["max_src"]  # mean particles of a leaf
    cells = 4 / 3 * n / leaf
    values = 1 if case["op"] == "potential2d" else 2
    inputs = 33 if case["op"] == "velocity2d" else 25
    # near field 9 leaves at 12 flops a pair; 27 translations of 8 (p+1)^2 a cell; P2M and L2P 16 p a particle
    return {"bytes": n * (inputs + 8 * values),
            "flops": n * 9 * leaf * 12 + cells * 27 * 8 * (p + 1) ** 2 + n * 16 * p}


# ---- the same values in 64 bits, by direct summation ------------------------------

def _direct2d(x, y, q, kind, rows=2048, cols=16384):
    """sum_j q_j r / r^2 (both components) or sum_j q_j log r over j != i, in chunks that stay in cache."""
    x, y, q = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y, q))
    n = x.numel()
    res = torch.zeros((n, 3 if kind == "field" else 1), dtype=torch.float64, device="cuda")
    rhs = torch.stack([q, q * x, q * y], dim=1) if kind == "field" else q[:, None]
    for i in range(0, n, rows):
        xi, yi, acc = x[i:i + rows, None], y[i:i + rows, None], res[i:i + rows]
        for j in range(0, n, cols):
            r2 = (xi - x[None, j:j + cols]).square_()
            r2.add_((yi - y[None, j:j + cols]).square_())
            if j < i + rows and i < j + cols:  # the pair (i, i) adds nothing
                at = torch.arange(max(i, j), min(i + rows, j + cols, n), device="cuda")
                r2[at - i, at - j] = math.inf if kind == "field" else 1.0
            w = r2.reciprocal_() if kind == "field" else r2.log_().mul_(0.5)
            acc.addmm_(w, rhs[j:j + cols])
    if kind != "field":
        return res[:, 0].contiguous()
    return x * res[:, 0] - res[:, 1], y * res[:, 0] - res[:, 2]


def _direct3d(d, rows=2048, cols=16384):
    """sum_j alpha_j x (x_i - x_j) / r^3 over j != i."""
    x, y, z, ax, ay, az = (torch.from_numpy(d[k]).cuda() for k in ("x", "y", "z", "ax", "ay", "az"))
    n = x.numel()
    rhs = torch.stack([ax, ay, az, ay * z - az * y, az * x - ax * z, ax * y - ay * x], dim=1)
    res = torch.zeros((n, 6), dtype=torch.float64, device="cuda")
    for i in range(0, n, rows):
        acc = res[i:i + rows]
        for j in range(0, n, cols):
            r2 = (x[i:i + rows, None] - x[None, j:j + cols]).square_()
            r2.add_((y[i:i + rows, None] - y[None, j:j + cols]).square_())
            r2.add_((z[i:i + rows, None] - z[None, j:j + cols]).square_())
            if j < i + rows and i < j + cols:
                at = torch.arange(max(i, j), min(i + rows, j + cols, n), device="cuda")
                r2[at - i, at - j] = math.inf
            r2.rsqrt_()
            acc.addmm_(r2 * r2 * r2, rhs[j:j + cols])
    sx, sy, sz = res[:, 0], res[:, 1], res[:, 2]
    return [sy * z - sz * y - res[:, 3], sz * x - sx * z - res[:, 4], sx * y - sy * x - res[:, 5]]


def exact(case, seed):
    op = case["op"]
    if op in ("velocity3d", "treecell3d"):
        d = _ring(case, seed)
        if d["x"].size > 400_000:
            return None
        out = _direct3d(d)
        if op == "treecell3d" and case["targets"]:
            t = torch.from_numpy(_targets3d(d)).cuda()
            out = [v * t for v in out]
        return out
    if op == "batch2d":
        offs, d = _batch(case, seed)
        sizes = np.diff(offs)
        if float((sizes.astype(float) ** 2).sum()) > 7e11:
            return None
        parts = [_direct2d(*(d[k][a:b] for k in ("x", "y", "q")), "field") for a, b in zip(offs[:-1], offs[1:])]
        return [torch.cat([p[k] for p in parts]) for k in range(2)]
    d = _particles2d(case, seed)
    if d["x"].size > 800_000:
        return None
    if op == "potential2d":
        return _direct2d(d["x"], d["y"], d["q"], "potential").cpu().numpy()
    ex, ey = _direct2d(d["x"], d["y"], d["q"], "field")
    if op == "velocity2d":
        return (ey + 1.0).cpu().numpy(), (-ex).cpu().numpy()
    return [ex, ey]
