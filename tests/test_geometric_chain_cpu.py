"""The distance chains of the geometric reinitialisation on the CPU: the
kernels' own device code (csrc/lsm_geometric_dev.cuh) on a warp of host fibers
against the sequential loops, bit for bit, and its FP32 enclosures against the
FP64 distances that they have to hold.  The surfaces pass close to a node at
the coordinate origin (corner or middle of the grid), where the point's
coordinates and its distance are small while the triangles are a cell wide, on
cells of aspect 1 to 100, smooth and rough; and layers of many nearly equal
distances.  No queued item may be without tasks."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SEEDS = (693240, 218490, 327034, 345658, 4699, 5467, 17083, 125244, 126044, 141148, 253, 701, 1021, 2110, 42718, 52254)
CSRC = os.path.join(os.path.dirname(HERE), "ns-lsm-single-phase_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    out = str(tmp_path_factory.mktemp("geo") / "libgeo.so")
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I",
                        os.path.join(HERE, "simt"), "-I", CSRC, os.path.join(HERE, "geo_chain_harness.cpp"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    d = C.CDLL(out)
    d.geo_enclosures.restype = C.c_long
    return d


def ptr(a):
    return C.c_void_p(a.ctypes.data)


def chains(lib, x, y, z, phi, pc, at, reach):
    """(nodes, signed distances and |v| that differ, items without tasks, largest difference)"""
    x, y, z, phi, pc = (np.asfortranarray(a, dtype=np.float64) for a in (x, y, z, phi, pc))
    n = np.zeros(5)
    lib.geo_chains(*phi.shape, ptr(phi), ptr(x), ptr(y), ptr(z), ptr(pc), *at, reach, ptr(n))
    return n


def grid(n, at, h, shift=(0.0, 0.0, 0.0)):
    """Coordinates of n^3 nodes, spacing h per axis, (0, 0, 0) + shift at node `at`."""
    return np.meshgrid(*((np.arange(n) - at) * h[c] + shift[c] for c in range(3)), indexing="ij")


def rough(rng, n, at, h, off, amp):
    """A surface `off` cells from node `at`, noisy by `amp` cells."""
    X, Y, Z = np.meshgrid(*(np.arange(n) - float(at),) * 3, indexing="ij")
    s = rng.standard_normal(2) * 0.6
    f = (Z + s[0] * X + s[1] * Y - off) * min(h)
    return f + amp * min(h) * rng.standard_normal((n,) * 3) * (np.abs(X) + np.abs(Y) + np.abs(Z) > 0)


@pytest.mark.parametrize("place", ["corner", "middle"])
@pytest.mark.parametrize("aspect", [1, 10, 100])
def test_surfaces_near_an_origin_node(lib, place, aspect):
    n, at = (9, 0) if place == "corner" else (11, 5)
    total = np.zeros(5)
    for off in (0.3, 0.03, 0.003):
        for amp in (0.0, 0.3, 2.0):
            for s in range(4):
                rng = np.random.default_rng([s, aspect, int(off * 1000), int(amp * 10)])
                h = np.array([1.0, 1.0, 1.0 / aspect]) * rng.choice([0.02, 1.0])
                pc = rng.standard_normal((n,) * 3) * rng.choice([20.0, 0.1, 9.9])
                total += chains(lib, *grid(n, at, h), rough(rng, n, at, h, off, amp), pc, (at,) * 3, 1)
    assert total[0] > 200
    assert (total[1:4] == 0).all(), total


def layers(rng, n, h):
    X, Y, Z = np.meshgrid(*(np.arange(n) - 0.3,) * 3, indexing="ij")
    return np.sin(2.1 * Z + 0.02 * X) * 0.3 * min(h) + 0.01 * min(h) * rng.standard_normal((n,) * 3)


@pytest.mark.parametrize("aspect", [1, 100])
def test_many_nearly_equal_distances(lib, aspect):
    """Flat and rippled layers, near and far from the origin: queues that fill."""
    n, total = 11, np.zeros(5)
    for s in range(10):
        rng = np.random.default_rng([s, aspect])
        h = np.array([1.0, 1.0, 1.0 / aspect])
        shift = rng.choice([0.0, 3000.0]) * np.array([1.0, -0.3, 0.05])
        f = layers(rng, n, h) if s % 2 else rough(rng, n, 5, h, 0.4, 0.02)
        total += chains(lib, *grid(n, 5, h, shift), f, np.full((n,) * 3, -9.9), (5, 5, 5), 2)
    assert total[0] > 300
    assert (total[1:4] == 0).all(), total


@pytest.mark.parametrize("h", [1e-3, 1e-6, 1e-8])
def test_short_edges(lib, h):
    """Cells whose triangles' edges are too short for the enclosures: bounding boxes alone."""
    total = np.zeros(5)
    for s in range(6):
        rng = np.random.default_rng(s)
        n = 11
        f = (layers(rng, n, (1, 1, 1)) if s % 2 else rough(rng, n, 5, (1, 1, 1), 0.4, 0.2)) * h
        total += chains(lib, *grid(n, 5, (h, h, h)), f, np.full((n,) * 3, -9.9), (5, 5, 5), 2)
    assert total[0] > 300
    assert (total[1:4] == 0).all(), total


@pytest.mark.parametrize("at", [(23, 0, 22), (27, 0, 21), (33, 0, 19), (35, 0, 18)])
def test_flush_between_pnodes(lib, at):
    """Nodes on a wall whose queue fills just before a pnode out of reach: an item
    without tasks there changes the last bits."""
    X, Y, Z = np.meshgrid(*(np.linspace(0, 1, m) for m in (64, 48, 40)), indexing="ij")
    phi = (Z - 0.48 - 0.1 * np.sin(6 * X) * np.cos(4 * Y)) * 1e-5
    c = chains(lib, X * 1e-5, Y * 1e-5, Z * 1e-5, phi, np.where(phi < 0, -9.9, 9.9), at, 0)
    assert c[0] == 1 and (c[1:4] == 0).all(), c


def test_values_of_any_size_before(lib):
    """|v| of the nodes without a distance: not a number, infinite, huge, about
    10, tiny and zero, of either sign."""
    total = np.zeros(5)
    for s in range(6):
        rng = np.random.default_rng(s)
        n, h = 9, (1.0, 1.0, 1.0)
        v = np.array([np.nan, -np.nan, np.inf, -np.inf, 1e300, -3e38, 10.0, 9.9999, -10.000001, 1e-300, 0.0, -0.0])
        total += chains(lib, *grid(n, 4, h), rough(rng, n, 4, h, 0.4, 0.2), rng.choice(v, (n,) * 3), (4,) * 3, 2)
    assert total[0] > 500
    assert (total[1:4] == 0).all(), total


def deciding(seed):
    rng = np.random.default_rng([seed, 5])
    n, at = ((5, 0), (9, 4))[seed & 1]
    off, amp = (0.03, 0.01, 0.003, 0.001)[(seed >> 1) & 3], (0.01, 0.1, 0.3, 1.0)[(seed >> 3) & 3]
    h = np.array([1.0, 1.0, 1.0 / (1, 10)[(seed >> 5) & 1]])
    return n, at, grid(n, at, h), rough(rng, n, at, h, off, amp)


@pytest.mark.parametrize("seed", SEEDS)
def test_surfaces_that_decide_by_an_enclosure(lib, seed):
    """Rough surfaces within 0.03 cells of a node at the origin: the last bits of
    its distance depend on triangles that an enclosure without the triangle's size loses."""
    n, at, xyz, phi = deciding(seed)
    c = chains(lib, *xyz, phi, np.full((n,) * 3, -9.9), (at,) * 3, 0)
    assert c[0] == 1 and (c[1:4] == 0).all(), c


@pytest.mark.parametrize("seed", range(4))
def test_enclosures_hold_the_distance(lib, seed):
    """Random triangles of all shapes and points at all distances and offsets
    from the origin; the point at or near a vertex, an edge, the plane."""
    rng = np.random.default_rng(seed)
    n = 400000
    size = 10.0 ** rng.uniform(-3, 3, (n, 1, 1))
    T = rng.standard_normal((n, 3, 3)) * size * 10.0 ** rng.uniform(-3, 0, (n, 1, 3))
    k = rng.integers(0, 4, n)
    T[k == 1, 2] = T[k == 1, 1] + 1e-3 * (T[k == 1, 2] - T[k == 1, 1])            # short edges
    T[k == 2, 2] = T[k == 2, 0] + 0.6 * (T[k == 2, 1] - T[k == 2, 0]) + 1e-3 * T[k == 2, 2]   # slivers
    w = rng.dirichlet((0.5, 0.5, 0.5), n)[:, :, None]
    d = rng.standard_normal((n, 3)) * size[:, 0] * 10.0 ** rng.uniform(-7, 1, (n, 1))
    on = np.where(rng.random((n, 1)) < 0.5, (T * w).sum(1), T[np.arange(n), rng.integers(0, 3, n)])
    P = on + d
    m = rng.integers(0, 3, n)
    o = np.where((m == 0)[:, None], P, 0.0)                                       # the point at the origin
    o = np.where((m == 1)[:, None], P + rng.standard_normal((n, 3)) * size[:, 0] * 10.0 ** rng.uniform(-7, 3, (n, 1)), o)
    T, P = np.ascontiguousarray(T - o[:, None]), np.ascontiguousarray(P - o)
    width = np.zeros(1)
    missed = lib.geo_enclosures(n, ptr(T), ptr(P), ptr(width))
    assert missed == 0, missed
