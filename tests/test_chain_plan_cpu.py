"""The chained sweeps' schedules (oneflow_b200/csrc/ofg_chain_plan.h), compiled
for the host: every edge names its neighbour, in the ring or in global memory, and
a neighbour read from global memory is written early enough.  Where it names a ring
slot, no write to that slot is unordered against the read: levels are ordered one
after the other, the cells of a level are not, so what a slot holds is decided only
if the neighbour's is the one position of its level with that slot, and no position
of a later level up to the reader's own has it.  And the cluster's
phases, replayed with warps that lag: every wait ends."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from oneflow_b200 import meshgen

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oneflow_b200", "csrc")
WRAPPER = r"""
#include "ofg_chain_plan.h"
using namespace ofg;
static SweepPlan plan;
extern "C" {
int ring() { return kChainRing; }
int groups() { return kChainGroups; }
int none() { return kChainNone; }
int warps() { return kChainWarps; }
int arrivals() { return kChainArrivals; }
long long make(int n, const int *order, int nlev, const int *off, const int *nbOff, const int *nbl) {
    plan = SweepPlan();
    plan_sweep(n, std::vector<int>(order, order + n), std::vector<int>(off, off + nlev + 1),
               std::vector<int>(nbOff, nbOff + n + 1), std::vector<int>(nbl, nbl + 2 * nbOff[n]), plan);
    return plan.fits ? plan.slots : -1;
}
int far_kind() { return plan.far; }
void get(int *lev, int *ref, int *edge) {
    std::copy(plan.lev.begin(), plan.lev.end(), lev);
    std::copy(plan.ref.begin(), plan.ref.end(), ref);
    std::copy(plan.edge.begin(), plan.edge.end(), edge);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(WRAPPER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "plan.so"), str(d / "plan.cpp")],
                   check=True)
    L = C.CDLL(str(d / "plan.so"))
    L.make.restype = C.c_longlong
    return L


def sweep(mesh, lower):
    """Level order, level offsets and edge lists of a sweep in the cells' own numbering."""
    n, nb = mesh.n_cells, mesh.n_bfaces
    edges = [[] for _ in range(n)]   # in ascending face id
    for f in range(nb, mesh.n_faces):
        a, b = int(mesh.lc[f]), int(mesh.rc[f])
        if (b < a) == lower:
            edges[a].append((f, b))
        else:
            edges[b].append((f - (1 << 31), a))
    lev = np.zeros(n, np.int32)
    for i in (range(n) if lower else range(n - 1, -1, -1)):
        if edges[i]:
            lev[i] = 1 + max(lev[j] for _, j in edges[i])
    order = np.argsort(lev, kind="stable").astype(np.int32)
    off = np.concatenate([[0], np.cumsum(np.bincount(lev))]).astype(np.int32)
    nb_off = np.concatenate([[0], np.cumsum([len(e) for e in edges])]).astype(np.int32)
    nbl = np.array([v for e in edges for p in e for v in p], np.int32)
    return lev, order, off, nb_off, nbl


def plan(L, sw):
    lev, order, off, nb_off, nbl = sw
    p = lambda a: a.ctypes.data_as(C.c_void_p)   # noqa: E731
    slots = L.make(len(order), p(order), len(off) - 1, p(off), p(nb_off), p(nbl))
    assert slots >= 0
    m, ref, edge = np.empty(4 * (len(off) - 1), np.int32), np.empty(slots, np.int32), np.empty(4 * slots, np.int32)
    L.get(p(m), p(ref), p(edge))
    return m.reshape(-1, 4), ref, edge.reshape(-1, 4), L.far_kind()


def mesh_of(name):
    kind, *args = name.split("-")
    m = meshgen.plate_2d(40, 30) if kind == "plate2d" else meshgen.bump_channel(*map(int, args[:2]))
    if "shuffled" in args:
        m = m.renumber_cells(np.random.default_rng(len(name)).permutation(m.n_cells))
    return m


# the widest levels: 30 and 33 cells, 1,300, 1,900; 4,200 and 7,600, wider than the ring
NAMES = ["plate2d", "bump-33-21", "bump-60-40-shuffled", "bump-70-50-shuffled", "bump-110-70-shuffled",
         "bump-140-100-shuffled"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("lower", [True, False])
def test_every_edge_finds_its_neighbour(lib, name, lower):
    sw = sweep(mesh_of(name), lower)
    lev, order, off, nb_off, nbl = sw
    m, ref, edge, far = plan(lib, sw)
    n, ring = len(order), lib.ring()
    pos = np.empty(n, np.int64)
    pos[order] = np.arange(n)
    used = np.flatnonzero(edge[:, 1] >= 0)
    cell, nb, r = edge[used, 2], edge[used, 1], ref[used]
    assert (ref[edge[:, 1] < 0] == lib.none()).all() and (r != lib.none()).all()
    # every edge once, in its cell's order; ring or neighbour
    o = np.argsort(cell, kind="stable")
    assert np.array_equal(np.stack([edge[used, 0], nb], 1)[o].ravel(), nbl)
    near = r >= 0
    assert (~r[~near] == nb[~near]).all() and (r[near] == pos[nb[near]] % ring).all()
    # a copy written after its signal is released by its warp's next arrival, `groups`
    # levels on, and known to the other blocks a level after that
    late = lev[cell[~near]] > lev[nb[~near]] + lib.groups() + 1
    assert far == (0 if near.all() else 1 if late.all() else 2)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("lower", [True, False])
def test_no_slot_of_the_ring_is_read_with_an_unordered_write(lib, name, lower):
    sw = sweep(mesh_of(name), lower)
    lev, order = sw[:2]
    m, ref, edge, _ = plan(lib, sw)
    n, ring = len(order), lib.ring()
    pos = np.empty(n, np.int64)
    pos[order] = np.arange(n)
    near = np.flatnonzero((edge[:, 1] >= 0) & (ref >= 0))
    for c, q in zip(edge[near, 2], edge[near, 1]):
        p = int(pos[q])
        others = np.arange(p % ring, n, ring)
        others = others[others != p]
        at = lev[order[others]]
        # the other writers of the slot: none in the neighbour's level, none after it up to the reader's level
        assert not ((at >= lev[q]) & (at <= lev[c])).any(), (c, q)


def test_levels_wider_than_the_ring_are_among_them(lib):
    widest = [np.diff(sweep(mesh_of(n), True)[2]).max() for n in NAMES]
    assert sum(w > lib.ring() for w in widest) == 2 and min(widest) < 100


def test_a_read_three_levels_on_is_among_them(lib):
    """far neighbours exactly groups + 1 levels back, and none closer"""
    sw = sweep(mesh_of("bump-60-40-shuffled"), True)
    lev, edge, ref = sw[0], plan(lib, sw)[2], plan(lib, sw)[1]
    far = (edge[:, 1] >= 0) & (ref < 0)
    assert (lev[edge[far, 2]] - lev[edge[far, 1]]).min() == lib.groups() + 1


class Barrier:
    """An mbarrier: a phase ends when its arrivals and its bytes (here: messages) are all in."""

    def __init__(self, count):
        self.count, self.phase, self.pending, self.tx = count, 0, count, 0

    def step(self, arrive, tx):
        self.pending -= arrive
        self.tx += tx
        assert self.pending >= 0
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, self.count

    def passed(self, k):   # a wait on the parity of phase k
        return self.phase % 2 != k % 2


@pytest.mark.parametrize("widths", ["wide narrow narrow", "wide wide narrow narrow", "wide narrow"])
def test_every_wait_of_the_cluster_ends(lib, widths):
    """chain_run's waits, arrivals and messages for two blocks, one message a warp with
    cells and one word a block and level; the warps move in a random order, one of
    them rarely."""
    warps, groups, arrivals, blocks = lib.warps(), lib.groups(), lib.arrivals(), 2
    width = widths.split() * 8
    rng = np.random.default_rng(7)
    for lag in range(warps):
        bars = [[Barrier(arrivals) for _ in range(groups)] for _ in range(blocks)]
        todo = {(b, g, w): g for b in range(blocks) for g in range(groups) for w in range(warps)}   # each warp's level
        idle = 0
        while todo:
            live = [k for k in todo if k[2] != lag or rng.random() < 0.01]
            if not live:
                continue
            b, g, w = k = live[rng.integers(len(live))]
            lvl = todo[k]
            mine = bars[b][lvl % groups]
            if (lvl >= groups and not mine.passed(lvl // groups - 1)) or (
                    lvl > 0 and not bars[b][(lvl - 1) % groups].passed((lvl - 1) // groups)):
                idle += 1
                assert idle < 20000, f"warp {k} waits before level {lvl}"
                continue
            idle = 0
            has = width[lvl] == "wide" or (b == 0 and w == 0)
            messages = blocks + (blocks * warps if width[lvl] == "wide" else 1)   # this block receives
            if w == 0 or arrivals > 1:
                mine.step(1, messages if w == 0 else 0)
            for peer in range(blocks):
                bars[peer][lvl % groups].step(0, -(has + (w == 0)))
            todo[k] += groups
            if todo[k] >= len(width):
                del todo[k]
