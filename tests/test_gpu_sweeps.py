"""GPU parity tests of the sweep kernels at the edges of their tiles and
remainders (bit-exact against the CPU oracle; the arithmetic is the same
operations in the same order, so there is no tolerance)."""
import ctypes as C

import numpy as np
import pytest

from charming_b200.jacobi import Jacobi2D, Problem
from oracle import jacobi as oj

pytestmark = pytest.mark.gpu


def oracle(grid, sweeps):
    if grid.dtype == np.float64:
        return oj.jacobi2d(grid, sweeps)
    g = np.ascontiguousarray(grid).copy()
    oj.lib().oracle_jacobi2d_f32(g.ctypes.data_as(C.POINTER(C.c_float)), g.shape[1] - 2, g.shape[0] - 2, sweeps, 0)
    return g


def same_bits(a, b):
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


# widths around whole vectors (2 or 4 values) and strips (a warp owns 32 less
# the vectors its edges lose), heights around the steady loop's turns of 4
# rows after the fill of 2 * depth rows, one chare and split ones
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("depth", [2, 5, 6, 8])
def test_multi_sweep_pass_tile_edges(rt, dtype, depth):
    rng = np.random.default_rng(depth)
    npdt = np.float64 if dtype == "f64" else np.float32
    sizes = [(w, h) for w in (9, 48, 53, 104, 111, 117) for h in (8, 4 * depth + 1, 4 * depth + 2, 4 * depth + 3, 131)]
    probs, grids = [], []
    for k, (w, h) in enumerate(sizes):
        px, py = ((1, 1), (1, 1), (2, 1), (1, 2), (2, 3))[k % 5]
        if w // px < depth or h // py < depth:
            px = py = 1
        probs.append(Problem(w, h, 2 * depth + 3, px=px, py=py))
        grids.append(rng.random((h + 2, w + 2)).astype(npdt))
    with Jacobi2D(probs, dtype=dtype, depth=depth) as j:
        for p, g in enumerate(grids):
            j.load(p, g)
        j.run()
        for p, g in enumerate(grids):
            assert same_bits(j.store(p), oracle(g, probs[p].max_sweeps)), sizes[p]


# Halos written into the neighbours' ghost zones: side halos of whole vectors
# on both sides, of odd columns or at odd offsets (element copies), one to four
# neighbours, chares no deeper than the halo
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("depth", [1, 2, 3, 4, 7, 8])
def test_put_halos_units(rt, dtype, depth):
    rng = np.random.default_rng(100 + depth)
    npdt = np.float64 if dtype == "f64" else np.float32
    shapes = [(24, 24, 3, 3), (64, 48, 4, 2), (65, 47, 4, 2), (67, 50, 3, 3), (200, 9, 5, 1), (11, 160, 1, 7),
              (301, 77, 2, 2), (512, 96, 1, 3)]
    probs, grids = [], []
    for nx, ny, px, py in shapes:
        probs.append(Problem(nx, ny, 3 * depth + 2, px=px, py=py))
        grids.append(rng.random((ny + 2, nx + 2)).astype(npdt))
    with Jacobi2D(probs, dtype=dtype, depth=depth) as j:
        for p, g in enumerate(grids):
            j.load(p, g)
        j.run()
        for p, g in enumerate(grids):
            assert same_bits(j.store(p), oracle(g, probs[p].max_sweeps)), shapes[p]
        # the same again: nothing of the first run is left in the ghost zones
        j.load(0, grids[0] * 0.5)
        for p in range(1, len(grids)):
            j.load(p, grids[p])
        j.run()
        assert same_bits(j.store(0), oracle((grids[0] * npdt(0.5)).astype(npdt), probs[0].max_sweeps))


# charming_jacobi2d_sweeps_noalloc: pass lengths 1..8 and their splits, vector
# rows and element rows (odd widths, grids one element off a 16-byte
# boundary), strip and row-run remainders, the smallest and largest grids
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,sweeps,shift", [
    (1, 1, 3, 0), (2, 5, 1, 0), (3, 2, 9, 1), (6, 300, 7, 0), (301, 4, 8, 0), (46, 33, 2, 1), (54, 61, 13, 0),
    (110, 130, 17, 0), (111, 97, 23, 1), (510, 254, 20, 0), (1022, 1020, 11, 0), (1445, 1441, 10, 1),
    # rows of at most 16 vectors: groups of 1 to 16 lanes (2, 4, 8, 16 and 32
    # items a warp), the widest of each type, and the next wider grid in strips
    (1, 5000, 8, 0), (2, 777, 5, 1), (4, 4001, 8, 0), (6, 33, 3, 0), (12, 2503, 20, 1), (14, 900, 7, 0),
    (28, 129, 6, 0), (30, 1000, 16, 0), (31, 1000, 8, 0), (61, 700, 9, 1), (62, 701, 8, 0), (63, 702, 8, 0),
])
def test_noalloc_pass_edges(rt, dtype, nx, ny, sweeps, shift):
    torch = pytest.importorskip("torch")
    from charming_b200 import _lib
    npdt = np.float64 if dtype == "f64" else np.float32
    n = (nx + 2) * (ny + 2)
    g = np.random.default_rng(nx * 7 + ny).random((ny + 2, nx + 2)).astype(npdt)
    tdt = torch.float64 if dtype == "f64" else torch.float32
    d_in = torch.empty(n + 4, dtype=tdt, device="cuda")
    d_out = torch.full((n + 4,), float("nan"), dtype=tdt, device="cuda")
    d_in[shift:shift + n] = torch.from_numpy(g.reshape(-1)).cuda()
    esz = g.itemsize
    _lib.check(rt.lib.charming_jacobi2d_sweeps_noalloc(_lib.F64 if dtype == "f64" else _lib.F32, nx, ny, sweeps,
                                                       d_in.data_ptr() + shift * esz, d_out.data_ptr() + shift * esz))
    out = d_out.cpu().numpy()
    assert same_bits(out[shift:shift + n].reshape(g.shape).copy(), oracle(g, sweeps))
    assert np.isnan(out[:shift]).all() and np.isnan(out[shift + n:]).all()  # nothing beyond the grid is written
    assert same_bits(d_in[shift:shift + n].cpu().numpy().reshape(g.shape), g)


# charming_jacobi3d: grids smaller than a warp's strip and rows, strip (60
# columns for two sweeps, 62 for one) and row remainders, odd widths (element
# copies), runs of planes, odd sweep counts (a last pass of one sweep)
@pytest.mark.parametrize("nx,ny,nz,sweeps", [
    (1, 1, 1, 3), (3, 2, 5, 4), (58, 44, 9, 2), (59, 45, 10, 3), (61, 46, 33, 1), (62, 5, 70, 6), (120, 100, 40, 4),
    (257, 31, 12, 5), (20, 300, 16, 2), (124, 90, 130, 7),
    # rows of at most 16 vectors: groups of 2 to 16 lanes; more than 64 runs
    (1, 400, 5, 4), (2, 3, 700, 6), (4, 97, 12, 3), (5, 41, 9, 2), (6, 200, 20, 7), (13, 500, 3, 6), (14, 9, 900, 3),
    (29, 77, 33, 5), (30, 64, 20, 6), (31, 64, 20, 6),
])
def test_jacobi3d_tile_edges(rt, nx, ny, nz, sweeps):
    g = np.random.default_rng(nx + ny + nz).random((nz + 2, ny + 2, nx + 2))
    out, _ms = rt.jacobi3d(g, sweeps)
    assert same_bits(out, oj.jacobi3d(g, sweeps))


def test_jacobi3d_time_covers_the_row_copies(rt):
    """Odd widths are copied to rows of whole vectors and back: the reported
    device time has both copies in it (with no sweeps it is nothing but them).
    Each reads and writes the grid, at no more than 20 TB/s (L2 included)."""
    nx, ny, nz = 299, 300, 300
    g = np.random.default_rng(1).random((nz + 2, ny + 2, nx + 2))
    out, ms = rt.jacobi3d(g, 0)
    assert same_bits(out, g)
    assert ms > 4 * g.nbytes / 20e12 * 1e3


# load and store of grids: narrow and wide ones, one chare and many, chares of
# a few cells, columns beyond one block and chares that a block's columns share
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,px,py", [
    (1, 1, 1, 1), (3, 700, 1, 1), (5, 300, 2, 7), (900, 2, 1, 1), (5000, 3, 9, 2), (62, 40, 3, 3), (63, 63, 63, 1),
    (64, 64, 8, 8), (131, 77, 16, 11), (300, 260, 60, 65), (257, 1030, 1, 1), (4100, 300, 2, 1),
])
def test_load_store_round_trip(rt, dtype, nx, ny, px, py):
    npdt = np.float64 if dtype == "f64" else np.float32
    g = np.random.default_rng(nx * 3 + ny).random((ny + 2, nx + 2)).astype(npdt)
    with Jacobi2D([Problem(nx, ny, 3, px=px, py=py)], dtype=dtype) as j:
        j.load(0, g)
        assert same_bits(j.store(0), g)
        j.run()  # and from the other buffer
        assert same_bits(j.store(0), oracle(g, 3))
