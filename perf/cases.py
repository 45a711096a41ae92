"""The calls this framework is used for, as timed cases.

Every case goes through a public entry point: kroupa_gpu on host arrays, Plan
(FP64 and FP32 compensated, line and loopon method), BatchPlan, the learned
displacement, a stretch of network training, and the C-ABI calls on device
arrays (matter step, epilogue, atom lines).  Inputs are lattices with random
loops of the distributions in disco_b200/workloads.py, made from the seed.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program has in hand before the call
    run(state)          one pass, and its outputs
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits by plain torch, where they are
                        computed numbers and that is quick enough
"""
import ctypes
import math

import numpy as np
import torch

from disco_b200 import _capi as C
from disco_b200 import backend as B
from disco_b200 import geometry as G
from disco_b200 import learned as L

BCC_A0, FCC_A0 = 2.855, 3.615
SEGMENTS_PER_LOOP = 28            # mean of the loop distribution below
LINE_FLOP, LOOPON_FLOP = 128, 66  # one closed-form term: a segment, a loopon

_N111 = [(1, 1, 1), (-1, 1, 1), (1, -1, 1), (1, 1, -1)]
_D110 = [(1, -1, 0), (1, 0, -1), (0, 1, -1), (1, 1, 0), (1, 0, 1), (0, 1, 1)]


def listed():
    return [
        # the smallest call a user makes: a test box on host arrays, one kroupa_gpu
        dict(name="call_small", kind="call", lattice="bcc", nx=10, ny=10, nz=10, loops=2, rmin=6.0, rmax=8.0,
             method="line", images=1, precision="fp64", nu=0.35, vacancies=0.0),
        # the quadrupole's size: four loops of about 60 chords in 40^3 BCC cells
        dict(name="quadrupole", kind="plan", lattice="bcc", nx=40, ny=40, nz=40, loops=4, rmin=26.0, rmax=34.0,
             method="line", images=1, precision="fp64", nu=0.29, vacancies=0.0, chords=64),
        # production size: a large FCC box, more image shells than the default
        dict(name="fcc_large", kind="plan", lattice="fcc", nx=100, ny=100, nz=100, loops=16, rmin=10.0, rmax=40.0,
             method="line", images=2, precision="fp64", nu=0.34, vacancies=0.0),
        # an uneven box with vacant sites (odd atom count), three image shells
        dict(name="bcc_ragged", kind="plan", lattice="bcc", nx=61, ny=47, nz=33, loops=9, rmin=8.0, rmax=30.0,
             method="line", images=3, precision="fp64", nu=0.29, vacancies=0.03),
        # the FP32 compensated form on a mid-size box
        dict(name="fcc_fp32c", kind="plan", lattice="fcc", nx=40, ny=40, nz=40, loops=12, rmin=10.0, rmax=40.0,
             method="line", images=2, precision="fp32c", nu=0.34, vacancies=0.0),
        # the loopon method on prismatic loops
        dict(name="bcc_loopons", kind="plan", lattice="bcc", nx=40, ny=40, nz=40, loops=8, rmin=20.0, rmax=50.0,
             method="loopons", images=1, precision="fp64", nu=0.28, vacancies=0.01),
        dict(name="bcc_loopons_fp32c", kind="plan", lattice="bcc", nx=25, ny=24, nz=23, loops=6, rmin=10.0,
             rmax=20.0, method="loopons", images=1, precision="fp32c", nu=0.28, vacancies=0.0),
        # the matter step of 16 prismatic loops on device arrays
        dict(name="matter", kind="matter", lattice="bcc", nx=128, ny=128, nz=128, loops=16, rmin=20.0, rmax=50.0),
        # the epilogue and the atom lines of the output file
        dict(name="output", kind="output", atoms=1000003, copies=6666, lammps=False),
        # many independent samples in one launch
        dict(name="batch", kind="batch", samples=24, edge_min=10, edge_max=30, loops_max=24, images_max=3,
             precision="fp32c"),
        # near images + network + check on a box with its trained-size network
        dict(name="learned", kind="learned", nx=50, ny=50, nz=50, loops=16),
        # a stretch of the network's training: gradient and Adam steps, then the weights
        dict(name="train", kind="train", batch=4096, steps=16),
    ]


def draw(rng):
    """Sizes over the listed ranges (cells over their logarithm), odd ones
    among them; loops cut so that no case costs more than the largest."""
    kind = rng.choice(["plan"] * 6 + ["call", "call", "matter", "output", "batch", "learned", "train"])

    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind in ("plan", "call"):
        method = rng.choice(["line", "line", "line", "loopons"])
        lattice = rng.choice(["bcc", "fcc"]) if method == "line" else "bcc"
        edge = logint(8, {"bcc": 120, "fcc": 95}[lattice] if kind == "plan" else 50)
        nx, ny, nz = (max(6, int(edge * rng.uniform(0.6, 1.4))) for _ in range(3))
        side = min(nx, ny, nz) * (BCC_A0 if lattice == "bcc" else FCC_A0)
        rmax = min(50.0 if method == "loopons" else 40.0, 0.33 * side)
        images = rng.choice([1, 1, 2, 2, 3, 4] if method == "line" else [0, 1, 1, 2])
        c = dict(kind=kind, lattice=lattice, nx=nx, ny=ny, nz=nz, loops=logint(1, 64), rmin=0.3 * rmax, rmax=rmax,
                 method=method, images=images, precision=rng.choice(["fp64", "fp64", "fp32c"]),
                 nu=rng.choice([0.28, 0.29, 0.34, 0.35]), vacancies=rng.choice([0.0, 0.0, 0.01, 0.1]))
        while c["loops"] > 1 and _evals(c) > 1.2e11:
            c["loops"] -= 1
        while _evals(c) > 1.2e11 and c["images"] > 0:
            c["images"] -= 1
        return c
    if kind == "matter":
        e = logint(12, 150)
        return dict(kind=kind, lattice="bcc", nx=max(8, int(e * rng.uniform(0.7, 1.3))),
                    ny=max(8, int(e * rng.uniform(0.7, 1.3))), nz=max(8, int(e * rng.uniform(0.7, 1.3))),
                    loops=rng.randint(1, 24), rmin=6.0, rmax=max(8.0, min(50.0, 0.3 * e * BCC_A0 * 0.7)))
    if kind == "output":
        return dict(kind=kind, atoms=logint(500, 4000000), copies=rng.randint(0, 400), lammps=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, samples=rng.randint(2, 32), edge_min=8, edge_max=rng.randint(12, 32),
                    loops_max=rng.randint(2, 24), images_max=rng.randint(1, 3),
                    precision=rng.choice(["fp64", "fp32c"]))
    if kind == "learned":
        e = logint(24, 64)
        return dict(kind=kind, nx=e, ny=e + rng.randint(0, 5), nz=e, loops=rng.randint(4, 24))
    return dict(kind=kind, batch=rng.choice([1000, 2048, 4096, 8192]), steps=rng.randint(1, 32))


# ---- inputs ----------------------------------------------------------------------------


def _lattice(case):
    fcc = case.get("lattice", "fcc") == "fcc"
    return (G.FCC, FCC_A0, 4) if fcc else (G.BCC, BCC_A0, 2)


def _box(case):
    a0 = _lattice(case)[1]
    return case["nx"] * a0, case["ny"] * a0, case["nz"] * a0


def _sites(case):
    _, _, basis = _lattice(case)
    n = basis * case["nx"] * case["ny"] * case["nz"]
    return n - int(n * case.get("vacancies", 0.0))


def _mean_radius_sq(case):
    lo, hi = case["rmin"], case["rmax"]
    return (lo * lo + lo * hi + hi * hi) / 3.0


def _terms(case):
    """Segments or loopons of all loops, on average."""
    if case.get("method", "line") == "line":
        return case["loops"] * case.get("chords", SEGMENTS_PER_LOOP)
    return case["loops"] * math.pi * _mean_radius_sq(case)


def _evals(case):
    per = 1.0 if case["method"] == "line" else LOOPON_FLOP / LINE_FLOP
    return per * _sites(case) * _terms(case) * (2 * case["images"] + 1) ** 3


def _positions(case, rng):
    kind, a0, _ = _lattice(case)
    x, y, z = G.lattice(kind, case["nx"], case["ny"], case["nz"], a0)
    n = _sites(case)
    if n < len(x):
        keep = np.sort(rng.permutation(len(x))[:n])
        x, y, z = x[keep], y[keep], z[keep]
    return np.stack([x, y, z])


def _glide_loops(case, rng):
    """Half circles, a quarter hexagons, a quarter rectangles on {111} planes
    (FCC) or {110} planes (BCC) with b in the plane, centres snapped."""
    kind, a0, _ = _lattice(case)
    cells = (case["nx"], case["ny"], case["nz"])
    fam_n, fam_b = (_N111, _D110) if kind == G.FCC else (_D110, _N111)
    out = []
    for _ in range(case["loops"]):
        n = fam_n[rng.integers(len(fam_n))]
        ms = [b for b in fam_b if b[0] * n[0] + b[1] * n[1] + b[2] * n[2] == 0]
        m = ms[rng.integers(len(ms))]
        if rng.random() < 0.5:
            m = tuple(-t for t in m)
        c = [rng.uniform(-k * a0 / 2, k * a0 / 2) for k in cells]
        cs, _ = G.snap(c, n, a0, *cells, kind)
        R = rng.uniform(case["rmin"], case["rmax"])
        shape = "circle" if "chords" in case else ("circle", "circle", "hexagon", "rectangle")[rng.integers(4)]
        if shape == "circle":
            lp = G.Loop.circle(1.0, R, cs, m, n, a0)
            P = lp.polyline(G.circle_eps_for_chords(R, case.get("chords", 48)))
        elif shape == "hexagon":
            lp = G.Loop.polygon(1.0, G.regular_polygon(6, R, m, n), 0.0, cs, m, n, a0)
            P = lp.polyline(0.01)
        else:
            lp = G.Loop.rectangle(1.0, R, R * rng.uniform(0.5, 1.0), 0.0, cs, m, n, a0)
            P = lp.polyline(0.01)
        out.append(lp.line_data(vertices=P))
    return out


def _prismatic(case, rng):
    """Prismatic circles on {111}, b along n: (loopon loops, slab loops)."""
    kind, a0, _ = _lattice(case)
    cells = (case["nx"], case["ny"], case["nz"])
    loops, slabs = [], []
    for _ in range(case["loops"]):
        n = _N111[rng.integers(len(_N111))]
        m = n if rng.random() < 0.5 else tuple(-t for t in n)
        c = [rng.uniform(-k * a0 / 2, k * a0 / 2) for k in cells]
        cs, d = G.snap(c, n, a0, *cells, kind)
        lp = G.Loop.circle(1.0, rng.uniform(case["rmin"], case["rmax"]), cs, m, n, a0)
        loops.append(lp)
        slabs.append(lp.slab_loop(d, apply=True, frank=False, a0=a0))
    return loops, slabs


def _loops(case, rng):
    if case.get("method", "line") == "line":
        return _glide_loops(case, rng)
    return [lp.loopon_data() for lp in _prismatic(case, rng)[0]]


def _precision(case):
    return C.DISCO_FP32C if case["precision"] == "fp32c" else C.DISCO_FP64


class _Sample:
    """One sample of a batch, as the batch plan takes it."""

    def __init__(self, n, loops, box, images, nu):
        self.n, self.loops, self.box, self.images, self.nu = n, loops, box, images, nu
        self.image_min = 0


def _batch_samples(case, rng):
    """(positions, loops, box, images) per sample: sizes by the case, loops by rng."""
    sizes, out = np.random.default_rng(case["samples"]), []
    for _ in range(case["samples"]):
        e = sizes.integers(case["edge_min"], case["edge_max"] + 1, size=3)
        sub = dict(lattice="bcc", nx=int(e[0]), ny=int(e[1]), nz=int(e[2]), method="line",
                   loops=int(sizes.integers(1, case["loops_max"] + 1)), rmin=6.0,
                   rmax=max(8.0, 0.3 * float(min(e)) * BCC_A0))
        images = int(sizes.integers(1, case["images_max"] + 1))
        out.append((_positions(sub, rng), _loops(sub, rng), _box(sub), images))
    return out


def _net_params(rng):
    """Weights of the size a trained network has: 14 -> 128 -> 128 -> 128 -> 3,
    padded to 16 inputs and 16 outputs."""
    parts = []
    for rows, cols, rr, cc in ((128, 16, 128, 14), (128, 128, 128, 128), (128, 128, 128, 128), (16, 128, 3, 128)):
        w = np.zeros((rows, cols))
        w[:rr, :cc] = rng.uniform(-1, 1, size=(rr, cc)) * math.sqrt(3.0 / cc)
        b = np.zeros(rows)
        b[:rr] = rng.uniform(-0.1, 0.1, size=rr)
        parts += [w.ravel(), b]
    return np.concatenate(parts).astype(np.float32)


def _far_norm():
    """Standardisation of the learned form's features (order of its header)."""
    mu = np.zeros(16, np.float32)
    isd = np.ones(16, np.float32)
    mu[3], isd[:3], isd[3], isd[14:] = 0.1, 2.0, 20.0, 0.0
    return L.FarNorm(mu, isd, 0.01, 4, 2)


def _slab_args(slabs):
    return (C.DiscoSlabLoop * max(1, len(slabs)))(*slabs), (C.DiscoSlabInfo * max(1, len(slabs)))()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("plan", "call"):
        loops, box = _loops(case, rng), _box(case)
        pos = _positions(case, rng)
        if kind == "call":
            return dict(kind=kind, case=case, loops=loops, box=box, atoms=B.AtomArrays.zeros_like_positions(*pos))
        d = torch.tensor(pos, device="cuda")
        plan = B.Plan(loops, box, precision=_precision(case), images=case["images"], nu=case["nu"],
                      max_atoms=d.shape[1])
        return dict(kind=kind, plan=plan, pos=d, u=torch.zeros_like(d))
    if kind == "matter":
        _, slabs = _prismatic(case, rng)
        d = torch.tensor(_positions(case, rng), device="cuda")
        n = d.shape[1]
        arr, info = _slab_args(slabs)
        cap = 65536
        return dict(kind=kind, pos=d, n=n, slabs=arr, nl=len(slabs), info=info, cap=cap,
                    box=(ctypes.c_double * 3)(*_box(case)), counts=(ctypes.c_int64 * 3)(),
                    out=torch.zeros_like(d), new_index=torch.empty(n, dtype=torch.int32, device="cuda"),
                    atoms=torch.zeros(cap, dtype=torch.int32, device="cuda"),
                    side=torch.zeros(cap, dtype=torch.int8, device="cuda"),
                    copies=torch.zeros((cap, 4), dtype=torch.int64, device="cuda"))
    if kind == "output":
        pos, u, src, shift, box = _output_inputs(case, seed)
        n, nc = case["atoms"], case["copies"]
        cp = torch.zeros((max(1, nc), 4), dtype=torch.float64, device="cuda")
        cp.view(torch.int32)[:nc, 0] = src
        cp[:nc, 1:] = shift
        return dict(kind=kind, pos=pos, u=u, copies=cp, n=n, nc=nc, box=(ctypes.c_double * 3)(*box),
                    final=torch.empty((3, n + nc), dtype=torch.float64, device="cuda"),
                    text=torch.zeros(64 * (n + nc), dtype=torch.uint8, device="cuda"),
                    lammps=1 if case["lammps"] else 0)
    if kind == "batch":
        smp = _batch_samples(case, rng)
        pos = [torch.tensor(s[0], device="cuda") for s in smp]
        u = torch.zeros(3 * sum(p.shape[1] for p in pos), dtype=torch.float64, device="cuda")
        views, at = [], 0
        for p in pos:
            views.append(u[at:at + p.numel()].view(3, -1))
            at += p.numel()
        ptrs = [tuple(t.data_ptr() for t in (*p, *v)) for p, v in zip(pos, views)]
        objs = [_Sample(p.shape[1], s[1], s[2], s[3], 0.29) for p, s in zip(pos, smp)]
        return dict(kind=kind, plan=B.BatchPlan(objs, ptrs, precision=_precision(case)), pos=pos, u=u)
    if kind == "learned":
        full = dict(case, lattice="fcc", rmin=10.0, rmax=40.0)
        d = torch.tensor(_positions(full, rng), device="cuda")
        loops = _glide_loops(full, rng)
        net = L.MLP(seed=1)
        net.set_params(_net_params(np.random.default_rng(seed + 1)))
        return dict(kind=kind, net=net, norm=_far_norm(), pos=d, u=torch.zeros_like(d), loops=loops, box=_box(full))
    X, T, p0 = _train_inputs(case, seed)
    net = L.MLP(seed=1)
    net.set_params(p0)
    return dict(kind=kind, net=net, X=X, T=T, batch=case["batch"], steps=case["steps"])


def _output_inputs(case, seed):
    """Atoms of a box with displacements of up to a few A, some across its faces."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, nc = case["atoms"], case["copies"]
    side = (n / 0.0859) ** (1.0 / 3.0)
    box = (side, side * 1.07, side * 0.93)
    Lb = torch.tensor(box, dtype=torch.float64, device="cuda")[:, None]
    pos = (torch.rand((3, n), dtype=torch.float64, device="cuda", generator=g) - 0.5) * Lb
    u = torch.randn((3, n), dtype=torch.float64, device="cuda", generator=g) * 0.4
    src = torch.randint(0, n, (nc,), dtype=torch.int32, device="cuda", generator=g)
    shift = torch.randn((nc, 3), dtype=torch.float64, device="cuda", generator=g)
    return pos, u, src, shift, box


def _train_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["batch"] * case["steps"]
    X = torch.zeros((n, 16), dtype=torch.float32, device="cuda")
    X[:, :14] = torch.randn((n, 14), device="cuda", generator=g)
    T = torch.stack([torch.sin(2 * X[:, 0]) * X[:, 3], X[:, 1] * X[:, 2], torch.cos(X[:, 4] + X[:, 5])], 1).contiguous()
    return X, T, _net_params(np.random.default_rng(seed))


# ---- one pass --------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "plan":
        state["u"].zero_()
        state["plan"].execute(state["pos"], state["u"])
        return state["u"]
    if kind == "call":
        a, c = state["atoms"], state["case"]
        for v in (a.ux, a.uy, a.uz):
            v.fill(0.0)
        B.kroupa_gpu(a, state["loops"], *state["box"], B.GpuOptions(fp32=c["precision"] == "fp32c"),
                     images=c["images"], nu=c["nu"])
        return [a.ux, a.uy, a.uz]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "matter":
        lib, p, o = C.cuda_lib(), state["pos"], state["out"]
        C.check(lib.disco_b200_prismatic_noalloc(
            p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), state["n"], state["slabs"], state["nl"], state["box"],
            o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), state["new_index"].data_ptr(), state["info"],
            state["atoms"].data_ptr(), state["side"].data_ptr(), state["cap"], state["copies"].data_ptr(),
            state["cap"], state["counts"], s), lib)
        # the buffers as the caller holds them (zero past the counts); sites as their bits
        return dict(sites=o.view(torch.int64), new_index=state["new_index"], atoms=state["atoms"],
                    side=state["side"], copies=state["copies"], counts=[int(v) for v in state["counts"]])
    if kind == "output":
        lib, p, u, f, m = C.cuda_lib(), state["pos"], state["u"], state["final"], state["n"] + state["nc"]
        C.check(lib.disco_b200_finalize_resident(
            *[t.data_ptr() for t in (*p, *u)], state["n"], state["copies"].data_ptr(), state["nc"], state["box"],
            *[t.data_ptr() for t in f], None, None, None, s), lib)
        got = ctypes.c_int64()
        C.check(lib.disco_b200_format_atoms(state["lammps"], b"Fe", *[t.data_ptr() for t in f], m,
                                            state["text"].data_ptr(), state["text"].numel(), ctypes.byref(got), s), lib)
        return dict(final=f, text=state["text"], bytes=int(got.value))
    if kind == "batch":
        state["u"].zero_()
        state["plan"].execute(torch.cuda.current_stream().cuda_stream)
        return state["u"]
    if kind == "learned":
        # tolerances that the untrained network passes, as a trained one passes its own
        state["u"].zero_()
        L.learned_displace(state["net"], state["norm"], state["pos"], state["u"], state["loops"], state["box"], 0.34,
                           tol_loop=10.0, tol_total=100.0)
        return state["u"]
    net, b = state["net"], state["batch"]
    for i in range(state["steps"]):
        loss = net.grad(state["X"][i * b:(i + 1) * b], state["T"][i * b:(i + 1) * b],
                        want_loss=i == state["steps"] - 1)
        net.adam(lr=1e-3)
    return dict(params=net.params(), loss=loss)


# ---- what a pass cannot do without -----------------------------------------------------


def work(case):
    """Bytes: inputs read and outputs written once.  Operations: for a field,
    one closed-form term per atom and loop (the least that still depends on
    both; how many terms the sum takes beyond that is the method's choice)."""
    kind = case["kind"]
    if kind in ("plan", "call"):
        n = _sites(case)
        per = LINE_FLOP if case["method"] == "line" else LOOPON_FLOP
        return {"bytes": 72.0 * n + 60.0 * _terms(case), "flops": float(per) * n * case["loops"]}
    if kind == "matter":
        return {"bytes": 52.0 * _sites(case), "flops": 20.0 * _sites(case)}
    if kind == "output":
        n = case["atoms"] + case["copies"]
        return {"bytes": (48.0 + 24.0 + 45.0) * n, "flops": 12.0 * n}
    if kind == "batch":
        n = 2.0 * ((case["edge_min"] + case["edge_max"]) / 2.0) ** 3 * case["samples"]
        return {"bytes": 72.0 * n, "flops": LINE_FLOP * n * (1 + case["loops_max"]) / 2.0}
    if kind == "learned":
        n = 4.0 * case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 72.0 * n, "flops": (LINE_FLOP + 2.0 * (14 * 128 + 2 * 128 * 128 + 128 * 3)) * n * case["loops"]}
    rows = case["batch"] * case["steps"]
    return {"bytes": 76.0 * rows + case["steps"] * 7 * 4.0 * 37264, "flops": 6.0 * (14 * 128 + 2 * 128 * 128 + 128 * 3) * rows}


# ---- 64-bit results --------------------------------------------------------------------

EXACT_LIMIT = 3.0e10      # terms that plain torch sums in well under 20 seconds


def _line_exact(pos, lp, box, images, nu, u):
    """Barnett's closed form of one polygonal loop over its images, added to u."""
    V = torch.tensor(np.stack([lp.vx, lp.vy, lp.vz]), device="cuda")                     # (3, k)
    c = torch.tensor([lp.cx, lp.cy, lp.cz], dtype=torch.float64, device="cuda")
    p = lp.phys
    b = torch.tensor([p.bx * p.mx, p.by * p.my, p.bz * p.mz], dtype=torch.float64, device="cuda")
    A, E = torch.roll(V, 1, 1), V
    T = E - A
    Ln = T.norm(dim=0)
    T = T / Ln
    W = torch.linalg.cross(b[:, None].expand_as(T), T, dim=0)
    c3 = 1.0 / (8.0 * math.pi * (1.0 - nu))
    cJ = c3 - 1.0 / (4.0 * math.pi)
    k = V.shape[1]
    step = max(256, int(3e6) // k)

    def dot(a, q):
        return a[0] * q[0] + a[1] * q[1] + a[2] * q[2]

    for i0 in range(0, pos.shape[1], step):
        P0 = pos[:, i0:i0 + step]
        acc = torch.zeros_like(P0)
        for img in range((2 * images + 1) ** 3):
            w = 2 * images + 1
            s = torch.tensor([(img // (w * w) - images) * box[0], (img // w % w - images) * box[1],
                              (img % w - images) * box[2]], dtype=torch.float64, device="cuda")
            P = P0 - s[:, None]
            r = c[:, None] - P                                                           # (3, n)
            l1 = r.norm(dim=0)[:, None]
            v = V[:, None, :] - P[:, :, None]                                            # (3, n, k) ends
            lv = v.norm(dim=0)
            a, la = torch.roll(v, 1, 2), torch.roll(lv, 1, 1)
            rr = r[:, :, None]
            num = dot(rr, torch.linalg.cross(a, v, dim=0))
            ra, rb = dot(rr, a), dot(rr, v)
            den = l1 * la * lv + ra * lv + rb * la + dot(a, v) * l1
            omega = 2.0 * torch.atan2(num, den).sum(1)
            t, ww = T[:, None, :], W[:, None, :]
            sA = dot(a, t)
            sB = sA + Ln
            d = a - sA * t
            d2 = dot(d, d)
            J0 = torch.log1p(2.0 * Ln / (la + lv - Ln))
            K0 = torch.where(sA >= 0, 1.0 / (la * (la + sA)) - 1.0 / (lv * (lv + sB)),
                             torch.where(sB <= 0, 1.0 / (lv * (lv - sB)) - 1.0 / (la * (la - sA)),
                                         (sB / lv - sA / la) / d2))
            K1 = 1.0 / la - 1.0 / lv
            dw = dot(d, ww) * c3
            f = (cJ * J0 * ww - dw * (d * K0 + t * K1)).sum(2)
            acc += b[:, None] * (omega / (4.0 * math.pi)) + f
        u[:, i0:i0 + step] += acc


def _loopon_exact(pos, lp, box, images, nu, u):
    """Kroupa's point loops of one loop over its images, added to u."""
    p = lp.phys
    q = torch.tensor(np.stack([lp.x, lp.y, lp.z]), device="cuda")
    m = torch.tensor([p.mx, p.my, p.mz], dtype=torch.float64, device="cuda")
    n = torch.tensor([p.nx, p.ny, p.nz], dtype=torch.float64, device="cuda")
    b = torch.tensor([p.bx, p.by, p.bz], dtype=torch.float64, device="cuda")
    k1, c2, bn = 1.0 / (8.0 * math.pi * (1.0 - nu)), 1.0 - 2.0 * nu, float((m * n).sum())
    step = max(64, int(6e6) // q.shape[1])
    w = 2 * images + 1
    for i0 in range(0, pos.shape[1], step):
        P0 = pos[:, i0:i0 + step]
        acc = torch.zeros_like(P0)
        for img in range(w ** 3):
            s = torch.tensor([(img // (w * w) - images) * box[0], (img // w % w - images) * box[1],
                              (img % w - images) * box[2]], dtype=torch.float64, device="cuda")
            R = (P0 - s[:, None])[:, :, None] - q[:, None, :]
            r2 = (R * R).sum(0)
            ir = torch.where(r2 < 1e-20, 0.0, r2.rsqrt())
            mr = m[0] * R[0] + m[1] * R[1] + m[2] * R[2]
            nr = n[0] * R[0] + n[1] * R[1] + n[2] * R[2]
            ir3 = ir * ir * ir
            tail = 3.0 * mr * nr * ir3 * ir * ir
            acc += torch.stack([(c2 * ir3 * (n[i] * mr + m[i] * nr - R[i] * bn) + tail * R[i]).sum(1) for i in range(3)])
        u[:, i0:i0 + step] -= k1 * p.dS * b[:, None] * acc


def _field_exact(pos, loops, box, images, nu):
    terms = sum(len(lp.vx) if lp.line else len(lp.x) for lp in loops)
    if pos.shape[1] * terms * (2 * images + 1) ** 3 > EXACT_LIMIT:
        return None
    d = torch.tensor(pos, device="cuda")
    u = torch.zeros_like(d)
    for lp in loops:
        (_line_exact if lp.line else _loopon_exact)(d, lp, box, images, nu, u)
    return u


def _split_params(p):
    at, out = 0, []
    for rows, cols in ((128, 16), (128, 128), (128, 128), (16, 128)):
        out.append(p[at:at + rows * cols].view(rows, cols))
        at += rows * cols
        out.append(p[at:at + rows])
        at += rows
    return out


def _net_exact(parts, X):
    h = X
    for i in (0, 2, 4):
        h = torch.nn.functional.silu(h @ parts[i].T + parts[i + 1])
    return h @ parts[6].T + parts[7]


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("plan", "call"):
        loops, box = _loops(case, rng), _box(case)
        u = _field_exact(_positions(case, rng), loops, box, case["images"], case["nu"])
        return u if u is None or kind == "plan" else list(u)
    if kind == "output":
        pos, u, src, shift, box = _output_inputs(case, seed)
        i = src.long()
        r = torch.cat([pos + u, pos[:, i] + u[:, i] + shift.T], 1)
        Lb = torch.tensor(box, dtype=torch.float64, device="cuda")[:, None]
        r = torch.where(r > Lb / 2, r - Lb, torch.where(r < -Lb / 2, r + Lb, r)) + Lb / 2
        return dict(final=r, text=None, bytes=None)
    if kind == "batch":
        parts = [_field_exact(s[0], s[1], s[2], s[3], 0.29) for s in _batch_samples(case, rng)]
        return None if any(p is None for p in parts) else torch.cat([p.reshape(-1) for p in parts])
    if kind == "learned":
        full = dict(case, lattice="fcc", rmin=10.0, rmax=40.0)
        pos = _positions(full, rng)
        loops, box = _glide_loops(full, rng), _box(full)
        u = _field_exact(pos, loops, box, 1, 0.34)
        if u is None:
            return None
        parts = _split_params(torch.tensor(_net_params(np.random.default_rng(seed + 1)), device="cuda").double())
        norm, d = _far_norm(), torch.tensor(pos, device="cuda")
        mu, isd = (torch.tensor(v, device="cuda").double() for v in (norm.mu, norm.inv_sd))
        Lref = (box[0] * box[1] * box[2]) ** (1.0 / 3.0)
        for lp in loops:
            c = np.array([lp.cx, lp.cy, lp.cz])
            V = np.stack([lp.vx, lp.vy, lp.vz], 1) - c
            A = 0.5 * np.linalg.norm(np.cross(V, np.roll(V, -1, axis=0)).sum(0))
            b, req = lp.burgers(), math.sqrt(A / math.pi)
            n = np.array([lp.phys.nx, lp.phys.ny, lp.phys.nz])
            n = n / np.linalg.norm(n)
            bh = b / np.linalg.norm(b)
            tail = np.concatenate([[req / Lref], n, bh, [box[1] / box[0] - 1, box[2] / box[0] - 1,
                                   np.linalg.norm(V, axis=1).max() / req - 1, float(bh @ n)], [0.0, 0.0]])
            X = torch.cat([((d - torch.tensor(c, device="cuda")[:, None]) / torch.tensor(box, device="cuda").double()[:, None]).T,
                           torch.tensor(tail, device="cuda").expand(d.shape[1], 13)], 1)
            X = (X - mu) * isd
            for i0 in range(0, X.shape[0], 1 << 18):
                y = _net_exact(parts, X[i0:i0 + (1 << 18)])[:, :3].T
                u[:, i0:i0 + (1 << 18)] += y * (norm.out_scale * float(np.linalg.norm(b)) * A / Lref ** 2)
        return u
    if kind == "train":
        X, T, p0 = _train_inputs(case, seed)
        p = torch.tensor(p0, device="cuda").double().requires_grad_(True)
        mask = torch.ones_like(p)
        parts = _split_params(mask)
        parts[0][:, 14:], parts[6][3:], parts[7][3:] = 0.0, 0.0, 0.0
        m, v, b = torch.zeros_like(p), torch.zeros_like(p), case["batch"]
        for i in range(case["steps"]):
            y = _net_exact(_split_params(p), X[i * b:(i + 1) * b].double())[:, :3]
            loss = ((y - T[i * b:(i + 1) * b].double()) ** 2).sum() / b
            g, = torch.autograd.grad(loss, p)
            with torch.no_grad():
                g = g * mask
                m = 0.9 * m + 0.1 * g
                v = 0.999 * v + 0.001 * g * g
                p -= 1e-3 * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
        return dict(params=p.detach(), loss=float(loss))
    return None
