"""Octrees that are no lattice of depth 15 (no leaf records): the walkers on the node arrays.

A tree whose walls are not the 2^L + 1 coordinates of a halved box per axis, or that is deeper than 15, is
walked on its node arrays in either precision. Here: the split of one subtree moved by an ulp, uneven splits
everywhere, a chain of 16 levels towards a corner; and the halved tree that has records, for comparison. All
against the CPU oracle: path segments bit for bit (both precisions walk in FP64), optical depths (FP32 sums to
1e-5), the life cycle history by history, pipelined and plain passes.
"""
import numpy as np
import pytest

from skgpu import abi, workloads
from test_gpu_parity import assert_close_runs, run_both
from test_gpu_passes import assert_passes_agree

pytestmark = pytest.mark.gpu

KINDS = ["lattice", "ulp", "uneven", "deep"]


def build(kind, ext):
    """Nodes with eight consecutive children each, and per leaf wall the leaves that touch it, by overlap."""
    rng = np.random.default_rng(3)
    depth = 16 if kind == "deep" else 3
    bounds, child, level = [np.array(ext, float)], [-1], [0]
    q = 0
    while q < len(bounds):
        b = bounds[q]
        corner = np.array_equal(b[3:], bounds[0][3:])
        if level[q] < (depth if kind != "deep" else 2) or (kind == "deep" and corner and level[q] < depth):
            c = 0.5 * (b[:3] + b[3:])
            if kind == "uneven":
                c = b[:3] + rng.uniform(0.3, 0.7, 3) * (b[3:] - b[:3])
            if kind == "ulp" and q == 5:
                c = np.nextafter(c, np.inf)
            child[q] = len(bounds)
            for o in range(8):
                up = np.array([(o >> a) & 1 for a in range(3)], bool)
                bounds.append(np.r_[np.where(up, c, b[:3]), np.where(up, b[3:], c)])
                child.append(-1)
                level.append(level[q] + 1)
        q += 1
    b, child = np.array(bounds), np.array(child)
    leaves = np.flatnonzero(child < 0)
    cell = np.full(len(b), -1, np.int32)
    cell[leaves] = np.arange(len(leaves))
    begin, lists = np.zeros(6 * len(b) + 1, np.int32), []
    lb = b[leaves]
    for n in range(len(b)):
        for wall in range(6):
            if child[n] < 0:
                a, upper = wall // 2, wall % 2
                touch = lb[:, a if upper else 3 + a] == b[n, 3 + a if upper else a]
                area = np.ones(len(leaves))
                for o in (x for x in range(3) if x != a):
                    d = np.minimum(lb[:, 3 + o], b[n, 3 + o]) - np.maximum(lb[:, o], b[n, o])
                    touch &= d >= 0
                    area *= np.maximum(d, 0)
                nb = np.flatnonzero(touch)
                lists += list(leaves[nb[np.argsort(-area[nb], kind="stable")]])
            begin[6 * n + wall + 1] = len(lists)
    inner = child >= 0
    return dict(bounds=b, cell_index=cell, child_begin=(np.cumsum(8 * inner) - 8 * inner).astype(np.int32),
                child_count=(8 * inner).astype(np.int32),
                child_index=np.concatenate([child[n] + np.arange(8) for n in np.flatnonzero(inner)]).astype(np.int32),
                nb_begin=begin, nb_index=np.array(lists, np.int32)), len(leaves)


def scene(kind):
    sc = workloads.galaxy_octree(npix=32, nlambda=4, max_level=3, max_dust_fraction=1e-2)
    tree, cells = build(kind, sc.grid["extent"])
    mean = sc.density.mean()
    sc.grid = dict(sc.grid, **tree)
    sc.density = mean * np.random.default_rng(4).uniform(0.2, 2.0, cells)
    return sc


def rays_for(sc):
    rng = np.random.default_rng(5)
    lo, hi = sc.grid["extent"][:3], sc.grid["extent"][3:]
    p = rng.uniform(lo, hi, (300, 3))
    k = rng.normal(size=(300, 3))
    p[:60] = rng.choice(sc.grid["bounds"], 60)[:, :3]     # from corners of nodes
    k[60:120] = np.eye(3)[rng.integers(0, 3, 60)] * rng.choice([-1.0, 1.0], (60, 1))  # along the axes
    k[:30] = p[30:60] - p[:30]                             # from corner to corner
    k[np.all(k == 0, axis=1)] = (0.0, 0.0, 1.0)
    return np.hstack([p, k / np.linalg.norm(k, axis=1)[:, None]])


@pytest.mark.parametrize("kind", KINDS)
def test_paths_equal_oracle(gpu_backend, oracle_backend, kind):
    sc = scene(kind)
    sc.upload(gpu_backend)
    sc.upload(oracle_backend)
    rays = rays_for(sc)
    ref = oracle_backend.trace_paths(rays, 512)
    assert (ref[0] > 0).mean() > 0.8 and ref[0].max() < 512  # a corner's ray may leave at once
    tau = oracle_backend.optical_depths(rays, 0.55e-6)
    for precision in (abi.PREC_FP64_EXACT, abi.PREC_FP32):
        got = gpu_backend.trace_paths(rays, 512, precision=precision)
        assert np.array_equal(got[0], ref[0])
        for r, n in enumerate(ref[0]):
            assert np.array_equal(got[1][r, :n], ref[1][r, :n]) and np.array_equal(got[2][r, :n], ref[2][r, :n]), r
        t = gpu_backend.optical_depths(rays, 0.55e-6, precision=precision)
        assert np.array_equal(t, tau) if precision == abi.PREC_FP64_EXACT else np.allclose(t, tau, rtol=1e-5, atol=1e-9)


@pytest.mark.parametrize("kind", KINDS)
def test_runs_equal_oracle(gpu_backend, oracle_backend, kind):
    sc = scene(kind)
    rg, ro = run_both(sc, gpu_backend, oracle_backend, 3000, seed=17)
    assert_close_runs(rg, ro, frac=0.99)
    for precision in (abi.PREC_FP64_EXACT, abi.PREC_FP32):
        a, _ = assert_passes_agree(gpu_backend, lambda: sc.run(gpu_backend, 3000, seed=17, precision=precision))
        # FP32 depths move interaction points by 1e-6 of a path, across a wall now and then
        rel = 1e-12 if precision == abi.PREC_FP64_EXACT else 2e-3
        assert a.counters["crossings"] == pytest.approx(rg.counters["crossings"], rel=rel)
        assert a.rf.sum() == pytest.approx(rg.rf.sum(), rel=rel)
