"""The sum by cells (tree.cu) against the plain sum over every image, which an
explicit image split selects, and against the oracle.

Tolerance (line): the cells' interpolation stays below 4e-15 A per loop at
|b| = 2.5 A where theta(q) was set, at most about three levels add at an atom,
and the plain sum itself is within 1e-14 A of the oracle on these sizes: 2e-14
A per loop, plus 2e-14 A.  Loopons: the plain sum over 1e4 to 1e6 terms is
within about 1e-13 A of the reference's, and the squares' interpolation is of
the line's size per loop: 2e-14 A per loop, plus 2e-13 A."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import oracle as O
from disco_b200 import _capi as C
from disco_b200 import backend as B
from disco_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _sum(torch, w, pos, split, precision=C.DISCO_FP64):
    p = B.Plan(w.loops, w.box, precision=precision, images=w.images, nu=w.nu, image_split=split,
               max_atoms=pos.shape[1])
    u = torch.zeros_like(pos)
    p.execute(pos, u)
    p.sync(torch.cuda.current_stream().cuda_stream)
    p.close()
    return u


def _positions(torch, w):
    return torch.tensor(np.stack([w.x, w.y, w.z]), dtype=torch.float64, device="cuda")


def _uneven():
    """A 3 : 2 : 1 box, odd atom count."""
    w = W.batch(nsamples=1, edge=(60, 60), nloops=(6, 6), radius=(6.0, 20.0), images=(2, 2), seed=11)[0]
    keep = (np.abs(w.y) < w.box[1] / 3) & (np.abs(w.z) < w.box[2] / 6)
    keep[::977] = False
    s = w.subset(np.flatnonzero(keep))
    s.box = (w.box[0], w.box[1] * 2 / 3, w.box[2] / 3)
    return s


def _prismatic(cells, n, rmin, rmax, images=1):
    w = W.bcc_prismatic(cells=cells, n_inter=n, n_vac=n, rmin=rmin, rmax=rmax)
    w.images = images
    return w


def _tolerance(w):
    return 2e-14 * len(w.loops) + (2e-14 if w.method == "line" else 2e-13)


CASES = {
    "fcc": lambda: W.fcc_random(cells=36, n_circles=4, n_hex=2, n_rect=2),
    "uneven": _uneven,
    "loopons": lambda: _prismatic(40, 2, 15.0, 40.0),
    "loopons, two shells": lambda: _prismatic(30, 2, 12.0, 30.0, 2),
    "small loopon loops": lambda: _prismatic(24, 4, 6.0, 12.0, 2),
    "large cells": lambda: W.fcc_random(cells=70, images=3, n_circles=2, n_hex=1, n_rect=1),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("form", ["plain", "shifted", "shuffled"])
def test_cells_match_plain_sum(name, form):
    torch = pytest.importorskip("torch")
    w = CASES[name]()
    pos = _positions(torch, w)
    if form == "shifted":
        pos += torch.tensor([[0.5 * w.box[0]], [0.25 * w.box[1]], [-0.4 * w.box[2]]], device="cuda")
    elif form == "shuffled":
        g = torch.Generator(device="cuda")
        g.manual_seed(1)
        pos = pos[:, torch.randperm(pos.shape[1], generator=g, device="cuda")].contiguous()
    tol = _tolerance(w)
    a = _sum(torch, w, pos, 1)
    b = _sum(torch, w, pos, 0)
    c = _sum(torch, w, pos, 0)
    assert float((a - b).abs().max()) <= tol
    assert torch.equal(b, c)                       # same atoms, same bits
    if form == "plain":
        idx = np.random.default_rng(0).permutation(w.n)[:1500]
        s = w.subset(idx)
        ref = np.stack(O.displace(s.x, s.y, s.z, s.loops, s.box, images=s.images, nu=s.nu))
        assert np.abs(b.cpu().numpy()[:, idx] - ref).max() <= tol


@pytest.mark.parametrize("name", ["fcc", "loopons"])
def test_atoms_outside_the_cells(name):
    """Outliers, a NaN and an infinity take every image themselves and leave
    the other atoms alone; atoms that fill a corner of the box only."""
    torch = pytest.importorskip("torch")
    w = CASES[name]()
    pos = _positions(torch, w)
    pos[:, 7] = torch.tensor([5.0, -3.1, 0.2], device="cuda") * w.box[0]
    pos[0, 100] = float("nan")
    pos[2, 4001] = float("inf")
    pos[:, 9000:] = pos[:, 9000:] * 0.45 + 0.1 * w.box[0]
    a, b = _sum(torch, w, pos, 1), _sum(torch, w, pos, 0)
    odd = torch.zeros(pos.shape[1], dtype=torch.bool, device="cuda")
    odd[100] = odd[4001] = True
    assert torch.isfinite(b[:, ~odd]).all()
    assert float((a - b)[:, ~odd].abs().max()) <= _tolerance(w)
    assert torch.equal(torch.isnan(a[:, 100]), torch.isnan(b[:, 100]))


def test_accumulates_and_captures():
    """execute adds into u; a captured stream keeps to the plain kernels."""
    torch = pytest.importorskip("torch")
    w = W.fcc_random(cells=36, n_circles=4, n_hex=2, n_rect=2)
    pos = _positions(torch, w)
    one = _sum(torch, w, pos, 0)
    plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, max_atoms=w.n)
    u = torch.ones_like(pos)
    plan.execute(pos, u)
    torch.cuda.synchronize()
    tol = 2e-14 * len(w.loops) + 2e-14
    assert float((u - 1.0 - one).abs().max()) <= 1e-15 + tol
    v = torch.zeros_like(pos)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.execute(pos, v)
    for _ in range(2):
        v.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert float((v - one).abs().max()) <= tol
    del graph
    plan.close()


def test_two_streams_at_once():
    """Calls in flight on two streams have their own scratch."""
    torch = pytest.importorskip("torch")
    w = W.fcc_random(cells=36, n_circles=4, n_hex=2, n_rect=2)
    pos = _positions(torch, w)
    one = _sum(torch, w, pos, 0)
    plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, max_atoms=w.n)
    streams = [torch.cuda.Stream() for _ in range(2)]
    us = [torch.zeros_like(pos) for _ in streams]
    torch.cuda.synchronize()
    for _ in range(3):
        for s, u in zip(streams, us):
            with torch.cuda.stream(s):
                u.zero_()
                plan.execute(pos, u, s)
    torch.cuda.synchronize()
    for u in us:
        assert torch.equal(u, one)
    plan.close()


def test_loopons_off_one_plane():
    """Loopons that do not lie in one plane have no squares: the plain sum."""
    torch = pytest.importorskip("torch")
    w = _prismatic(30, 2, 12.0, 30.0)
    w.loops[1].z = w.loops[1].z + 0.3 * np.sin(w.loops[1].x)
    pos = _positions(torch, w)
    a, b = _sum(torch, w, pos, 1), _sum(torch, w, pos, 0)
    assert float((a - b).abs().max()) <= _tolerance(w)


def test_threads_with_plans_of_different_shapes():
    """Host threads, each with a plan, a stream and an atom count of its own, so
    that kernels of one instance are launched with different shared memory at
    the same time: every call succeeds and gives the thread's own sum."""
    torch = pytest.importorskip("torch")
    ws = [W.fcc_random(cells=c, n_circles=4, n_hex=2, n_rect=2, images=im) for c, im in ((24, 2), (36, 2), (30, 3), (20, 4))]
    ws += [_prismatic(24, 2, 8.0, 20.0), _prismatic(30, 4, 12.0, 30.0)]
    poss = [_positions(torch, w) for w in ws]
    want = [_sum(torch, w, p, 0) for w, p in zip(ws, poss)]
    failures = []

    def go(w, pos, one):
        try:
            stream = torch.cuda.Stream()
            plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, max_atoms=w.n)
            u = torch.zeros_like(pos)
            torch.cuda.synchronize()
            for _ in range(60):
                with torch.cuda.stream(stream):
                    u.zero_()
                plan.execute(pos, u, stream)
            stream.synchronize()
            if not torch.equal(u, one):
                failures.append("another sum")
            plan.close()
        except Exception as e:
            failures.append(repr(e))
    threads = [threading.Thread(target=go, args=a) for a in list(zip(ws, poss, want)) * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failures == []


def test_beside_a_capture():
    """A call on one stream while another stream is being captured: its first,
    which makes the scratch pool, a repeated one, and the plan's end.  The
    capture goes on, and both results are right."""
    torch = pytest.importorskip("torch")
    code = """
import sys
import numpy as np, torch
from disco_b200 import backend as B, workloads as W
w = W.quadrupole(cells=40)
pos = torch.tensor(np.stack([w.x, w.y, w.z]), device="cuda")
plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, max_atoms=w.n)
u, a = torch.zeros_like(pos), torch.zeros(4, device="cuda")
side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
    a += 1
    for _ in range(2):
        plan.execute(pos, u, side)
    a += 1
graph.replay()
torch.cuda.synchronize()
assert a.tolist() == [2.0] * 4
v = torch.zeros_like(pos)
for _ in range(2):
    plan.execute(pos, v)
torch.cuda.synchronize()
assert float(u.abs().max()) > 0 and torch.equal(u, v)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# (method, loops, radius, atoms, shells) -> summed by cells?  Both sides of the
# line between the cells and the plain sum, measured on one B200 (ms, plain and
# cells): 0.29 / 0.68, 0.49 / 0.58, 7.2 / 17.7, 28.5 / 70.5, 23 / 43; 6.4 / 1.3,
# 9.3 / 5.2, 7.1 / 1.7, 15.4 / 8.7.
LINE_OF_CHOICE = [("line", 1, 6.0, 16000, 2, False), ("line", 1, 6.0, 130000, 1, False),
                  ("loopons", 16, 6.0, 2000, 4, False), ("loopons", 64, 6.0, 2000, 4, False),
                  ("loopons", 64, 11.0, 387471, 0, False),
                  ("line", 2, 9.7, 195821, 2, True), ("line", 16, 12.4, 33529, 2, True),
                  ("loopons", 1, 8.4, 110732, 2, True), ("loopons", 8, 15.0, 8000, 2, True)]


def _random_loops(method, count, radius, edge, seed):
    rng = np.random.default_rng(seed)
    loops = []
    for _ in range(count):
        n = rng.normal(size=3)
        n /= np.linalg.norm(n)
        a = np.array([n[1], -n[0], 0.0]) / np.hypot(n[0], n[1])
        b, c = np.cross(n, a), rng.uniform(-edge / 2, edge / 2, size=3)
        phys = B.LoopPhys(2.5, 2.5, 2.5, *(a if method == "line" else n), *n, 1.0)
        if method == "line":
            t = 2 * np.pi * np.arange(24) / 24
            p = c + radius * (np.cos(t)[:, None] * a + np.sin(t)[:, None] * b)
            loops.append(B.LoopData(phys=phys, line=True, vx=p[:, 0].copy(), vy=p[:, 1].copy(), vz=p[:, 2].copy(),
                                    cx=c[0], cy=c[1], cz=c[2]))
        else:
            k = np.arange(-int(radius), int(radius) + 1)
            i, j = (v.ravel() for v in np.meshgrid(k, k))
            inside = i * i + j * j <= radius * radius
            p = c + i[inside, None] * a + j[inside, None] * b
            loops.append(B.LoopData(x=p[:, 0].copy(), y=p[:, 1].copy(), z=p[:, 2].copy(), phys=phys))
    return loops


@pytest.mark.parametrize("method,count,radius,atoms,images,cells", LINE_OF_CHOICE)
def test_choice_between_cells_and_the_plain_sum(method, count, radius, atoms, images, cells):
    """Sums that the cells would slow down take the plain kernel, the others the
    cells."""
    edge = (atoms / 0.08) ** (1.0 / 3.0)
    plan = B.Plan(_random_loops(method, count, radius, edge, 3), (edge,) * 3, images=images, nu=0.3, max_atoms=atoms)
    levels = plan.cells(atoms)
    plan.close()
    assert (levels > 0) == cells, levels


@pytest.mark.parametrize("name", list(CASES))
def test_these_sizes_go_by_cells(name):
    """What the tests above compare with the plain sum is the sum by cells; a
    caller's image split and far shells alone are not."""
    w = CASES[name]()
    for kw, cells in (({}, True), ({"image_split": 1}, False), ({"image_min": 1}, False)):
        plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, max_atoms=w.n, **kw)
        assert (plan.cells(w.n) > 0) == cells, kw
        assert plan.cells(0) == 0 and plan.cells(1) == 0
        plan.close()


def test_threads_launch_one_kernel_with_other_shared_memory():
    """Two plans whose last kernel is the same instance with 58 and 92 KB of
    shared memory, executed over and over by eight host threads."""
    torch = pytest.importorskip("torch")
    plans = []
    for radius, atoms, images in ((7.1, 38682, 2), (12.1, 14140, 3)):
        edge = (atoms / 0.08) ** (1.0 / 3.0)
        g = torch.Generator(device="cuda")
        g.manual_seed(atoms)
        pos = (torch.rand((3, atoms), dtype=torch.float64, device="cuda", generator=g) - 0.5) * edge
        plans.append((B.Plan(_random_loops("line", 1, radius, edge, 3), (edge,) * 3, images=images, max_atoms=atoms), pos))
    failures = []

    def go(plan, pos):
        try:
            stream = torch.cuda.Stream()
            u = torch.zeros_like(pos)
            torch.cuda.synchronize()
            for _ in range(400):
                plan.execute(pos, u, stream)
            stream.synchronize()
        except Exception as e:
            failures.append(repr(e))
    threads = [threading.Thread(target=go, args=plans[k % 2]) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for plan, _ in plans:
        plan.close()
    assert failures == []


@pytest.mark.parametrize("name", ["fcc", "loopons"])
@pytest.mark.parametrize("left", [0.0, 1.0 / 9.0, 1.0 / 7.0, 1.0 / 5.0, 1.0 / 3.0])
def test_most_atoms_outside_the_cells(name, left):
    """Unwrapped atoms: all but a share on both sides of the eighth (lines) and
    the quarter (loopons) below which the plain kernel takes every atom, several
    box lengths away, every second one of those with a coordinate that is not a
    number."""
    torch = pytest.importorskip("torch")
    w = CASES[name]()
    pos = _positions(torch, w)
    n = pos.shape[1]
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    away = torch.randperm(n, generator=g, device="cuda")[int(left * n):]
    box = torch.tensor(w.box, dtype=torch.float64, device="cuda")
    pos[:, away] += box[:, None] * torch.randint(3, 6, (3, len(away)), generator=g, device="cuda").double()
    nan = away[::2]
    pos[1, nan] = float("nan")
    a, b = _sum(torch, w, pos, 1), _sum(torch, w, pos, 0)
    fine = torch.ones(n, dtype=torch.bool, device="cuda")
    fine[nan] = False
    assert torch.isnan(a[:, nan]).all() and torch.isnan(b[:, nan]).all()
    assert float((a - b)[:, fine].abs().max()) <= _tolerance(w)


def test_unwrapped_atoms_are_no_slower_than_in_the_plain_sum():
    """All atoms several box lengths away: the cells have nothing to sum, and the
    call takes the plain kernel's time (1.18 of it when the near pass summed
    them)."""
    torch = pytest.importorskip("torch")
    w = CASES["loopons, two shells"]()
    pos = _positions(torch, w) + 5.0 * w.box[0]
    times = []
    for split in (1, 0):
        plan = B.Plan(w.loops, w.box, images=w.images, nu=w.nu, image_split=split, max_atoms=w.n)
        u = torch.zeros_like(pos)
        best = 1e300
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.execute(pos, u)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        plan.close()
        times.append(best)
    assert times[1] <= 1.1 * times[0], times


def _circle(radius, chords, center, normal, seed):
    rng = np.random.default_rng(seed)
    n = np.asarray(normal, dtype=float) / np.linalg.norm(normal)
    a = np.cross(n, rng.normal(size=3))
    a /= np.linalg.norm(a)
    b, t = np.cross(n, a), 2 * np.pi * np.arange(chords) / chords
    p = np.asarray(center) + radius * (np.cos(t)[:, None] * a + np.sin(t)[:, None] * b)
    return B.LoopData(phys=B.LoopPhys(2.5, 2.5, 2.5, *a, *n, 1.0), line=True, vx=p[:, 0].copy(), vy=p[:, 1].copy(),
                      vz=p[:, 2].copy(), cx=center[0], cy=center[1], cz=center[2])


def _forms():
    """(loops, atoms, edge, shells, loops of each method): what the cases above
    leave out."""
    edge = (200000 / 0.08) ** (1.0 / 3.0)
    rng = np.random.default_rng(4)
    long = [_circle(30.0, c, rng.uniform(-40, 40, size=3), rng.normal(size=3), c) for c in (257, 600, 1100)]
    mixed = _random_loops("line", 3, 20.0, edge, 1) + _random_loops("loopons", 2, 15.0, edge, 2)
    e0 = (1000000 / 0.08) ** (1.0 / 3.0)
    return {"open pieces": (long, 200000, edge, 2), "both methods": (mixed, 200000, edge, 1),
            "no images": (_random_loops("line", 64, 6.0, e0, 3), 1000000, e0, 0),
            "four shells": (_random_loops("line", 2, 15.0, edge, 5), 200000, edge, 4),
            "eight shells": (_random_loops("line", 2, 10.0, 0.5 * edge, 6), 25000, 0.5 * edge, 8),
            "eight shells, loopons": (_random_loops("loopons", 1, 6.0, 0.5 * edge, 7), 25000, 0.5 * edge, 8)}


@pytest.mark.parametrize("name", ["open pieces", "both methods", "no images", "four shells", "eight shells",
                                  "eight shells, loopons"])
def test_other_forms_match_plain_sum(name):
    """Lines of more than one piece (open ones), a plan with both methods, and the
    ends of the range of shells.  Tolerance as above, its part for the plain sum's
    own rounding with the square root of the terms it adds to an atom per loop,
    from 48 segments and 125 images on."""
    torch = pytest.importorskip("torch")
    loops, atoms, edge, images = _forms()[name]
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    pos = (torch.rand((3, atoms), dtype=torch.float64, device="cuda", generator=g) - 0.5) * edge
    sums = []
    for split in (1, 0):
        plan = B.Plan(loops, (edge,) * 3, images=images, nu=0.3, image_split=split, max_atoms=atoms)
        u = torch.zeros_like(pos)
        plan.execute(pos, u)
        levels = plan.cells(atoms)
        plan.close()
        sums.append(u)
    of = [[lp for lp in loops if lp.line], [lp for lp in loops if not lp.line]]
    each = []
    for some in of:
        if some:
            plan = B.Plan(some, (edge,) * 3, images=images, nu=0.3, max_atoms=atoms)
            each.append(plan.cells(atoms))
            plan.close()
    assert min(each) > 0 and sum(each) == levels
    terms = max(len(lp.vx) if lp.line else len(lp.x) for lp in loops)
    growth = max(1.0, np.sqrt(terms / 48.0 * (2 * images + 1) ** 3 / 125.0))
    base = 2e-14 if all(lp.line for lp in loops) else 2e-13
    assert float((sums[0] - sums[1]).abs().max()) <= 2e-14 * len(loops) + base * growth
