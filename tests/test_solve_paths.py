"""The resident pressure solve against the streaming kernel, each run known to have taken the one or
the other (Batch.solve_resident): around the limits of what fits, where a scene's neighbours in other
blocks find no room, and in batches of which a part is resident.  Both kernels add the same numbers
in the same order, so pressures, iterations and residuals must be equal to the bit.  A scene streams
when `pcg_grid_blocks` leaves too few blocks for it, and small ones where another scene streams."""
import numpy as np
import pytest

from ariel_b200 import _abi as A
from ariel_b200._lib import lib
from ariel_b200.flipsim import Batch

from helpers import dambreak, params

BOTH = [A.PREC_MIXED, A.PREC_FP64]


def _first(n, cells):
    """The first `cells` cells of an n^3 grid in (i, j, k) order, as (n, fluid)."""
    return n, (np.arange(n ** 3) < cells).reshape(n, n, n)


def _sheets(n):
    """Pairs of planes on both sides of the list bricks' x faces: over one neighbour in another block
    for each cell, where blocks of four full chunks have one slot a cell."""
    m = np.zeros((n, n, n), bool)
    m[np.arange(n) % 8 % 7 == 0] = True
    return n, m


def _solve(scenes, precision, blocks=0):
    """Per scene: (pressures, iterations, residual), and which scenes were resident."""
    descs = []
    for n, _ in scenes:
        d = A.scene_dambreak(n)
        d.n_liquid = 0
        descs.append(d)
    b = Batch(descs, params(precision=precision, stop=A.STOP_REL, tol=1e-5, pcg_grid_blocks=blocks))
    b.init()
    assert not any(b.solve_resident(s) for s in range(len(scenes)))
    for s, (n, fluid) in enumerate(scenes):
        rng = np.random.default_rng(n + int(fluid.sum()) % 1000)
        b.set_grid(A.GRID_A, fluid.astype(np.int32), s)
        b.set_grid(A.GRID_L, np.where(fluid, -3.0 + rng.random((n, n, n), np.float32), np.float32(1.6)), s)
        b.set_grid(A.GRID_D, np.where(fluid, rng.standard_normal((n, n, n), np.float32), np.float32(0.0)), s)
        b.set_grid(A.GRID_P64, np.zeros((n, n, n)), s)
    b.stage(A.STAGE_SOLVE)
    out = []
    for s, (n, fluid) in enumerate(scenes):
        st = b.stats(s)
        assert st.n_fluid_cells == fluid.sum() and st.pcg_converged == 1
        out.append((b.get_grid(A.GRID_P64, s), b.get_grid(A.GRID_P, s), st.pcg_iterations, st.pcg_rel_residual))
    where = [b.solve_resident(s) for s in range(len(scenes))]
    b.close()
    return out, where


def _assert_same(got, want):
    assert got[2:] == want[2:]
    for g, w in zip(got[:2], want[:2]):
        np.testing.assert_array_equal(g.view(np.uint8), w.view(np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", BOTH)
@pytest.mark.parametrize("cells", [0, 1, 2, 511, 512, 513, 1024])
def test_smallest_scenes(cells, precision):
    scene = _first(20, cells)
    alone, where = _solve([scene], precision)
    assert where == [True]
    beside, where = _solve([scene, _first(20, 5000)], precision, 1)  # 10 chunks: too many for one block
    assert where == [False, False]
    _assert_same(alone[0], beside[0])


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n,cells,resident", [
    # one chunk per half block and two, of 512 cells; the largest FP64 chunks that fit two to a block, and one
    # cell more; MIXED: two full chunks a block, up to four, and one cell more
    (A.PREC_FP64, 60, 148 * 512 + 1, True), (A.PREC_FP64, 76, 296 * 1472, True), (A.PREC_FP64, 76, 296 * 1472 + 1, False),
    (A.PREC_MIXED, 60, 148 * 512 + 1, True), (A.PREC_MIXED, 86, 296 * 2048, True),
    (A.PREC_MIXED, 107, 592 * 2048, True), (A.PREC_MIXED, 107, 592 * 2048 + 1, False)])
def test_limits_of_what_fits(precision, n, cells, resident):
    scene = _first(n, cells)
    got, where = _solve([scene], precision)
    assert where == [resident]
    want, where = _solve([scene], precision, 24)
    assert where == [False]
    _assert_same(got[0], want[0])


@pytest.mark.gpu
@pytest.mark.parametrize("precision,scene", [
    # FP64: the list in the grid's order, 2 neighbours in other planes and 2 x 288 of 2,944 in other rows: 6,464
    # a block, for 6,437 slots
    (A.PREC_FP64, lambda: _first(288, 432000)), (A.PREC_MIXED, lambda: _sheets(160))])
def test_neighbours_without_room(precision, scene):
    scene = scene()
    got, where = _solve([scene], precision)  # by its cells resident, handed over
    assert where == [False]
    want, where = _solve([scene], precision, 24)
    assert where == [False]
    _assert_same(got[0], want[0])


@pytest.mark.gpu
@pytest.mark.parametrize("last", [1, 33, 700, 2048, 3001, 4095, 4096, 4097, 6000, 8191])
def test_big_scene_with_a_short_last_block(last):
    # 74 blocks of four full chunks and one of `last` cells, whose neighbours are mostly not its own
    scene = _first(90, 296 * 2048 + last)
    got, where = _solve([scene], A.PREC_MIXED)
    assert where == [True]
    want, where = _solve([scene], A.PREC_MIXED, 24)
    assert where == [False]
    _assert_same(got[0], want[0])


MIX = {
    "shared": lambda: _first(58, 296 * 640),      # chunks of 640 cells, four to a block
    "pair": lambda: _first(69, 296 * 1100),       # two to a block, all blocks
    "pair2": lambda: _first(70, 296 * 1150),      # and a second group of blocks
    "small": lambda: _first(20, 5000),
    "empty": lambda: _first(9, 0),
    "big": lambda: _first(90, 700000),            # up to four full chunks a block
    "sheets": lambda: _sheets(160),               # hands over to the streaming kernel
    "huge": lambda: _first(107, 592 * 2048 + 1),  # never resident
}


@pytest.mark.gpu
@pytest.mark.parametrize("names,stream", [
    (("shared", "pair", "small", "empty", "big", "pair2"), ()),
    (("sheets", "shared", "pair", "small", "empty", "big"), ("sheets",)),
    # where a scene streams from the start, those of the smallest chunks join it
    (("shared", "pair", "small", "huge", "empty", "big"), ("huge", "small", "empty"))])
def test_batches_partly_resident(names, stream):
    scenes = [MIX[m]() for m in names]
    got, where = _solve(scenes, A.PREC_MIXED)
    assert where == [m not in stream for m in names]
    for m, scene, g in zip(names, scenes, got):
        want, w = _solve([scene], A.PREC_MIXED, 24)
        assert w == [m in ("small", "empty")]
        _assert_same(g, want[0])


def _steps(descs, blocks, graph):
    b = Batch(descs, params(precision=A.PREC_MIXED, stop=A.STOP_REL, tol=1e-5, graph=graph, pcg_grid_blocks=blocks))
    b.init()
    b.step(3)
    out = [(b.get_particles(s), b.stats(s).pcg_iterations, b.stats(s).pcg_outer) for s in range(len(descs))]
    where = [b.solve_resident(s) for s in range(len(descs))]
    b.close()
    return out, where


@pytest.mark.gpu
@pytest.mark.parametrize("descs,blocks,graph", [
    # at the bench sizes, chunks streamed past the one that a block caches, in alternate directions
    (lambda: [A.scene_dambreak(64)], (24, 7), 1), (lambda: [A.scene_dambreak(128)], (64,), 1),
    # uneven scenes through one pipeline, across the borders of scenes and past those that end early
    (lambda: [dambreak(40, seed=2), dambreak(12, seed=3), dambreak(48, seed=4, hi=(0.3, 0.5, 1.0))], (1, 3), 0)])
def test_steps_streamed(descs, blocks, graph):
    want, where = _steps(descs(), 0, graph)
    assert all(where)
    for nb in blocks:
        got, where = _steps(descs(), nb, graph)
        assert not any(where)
        for (p, *counts), (q, *counts0) in zip(got, want):
            assert counts == counts0
            for key in ("pos", "vel"):
                np.testing.assert_array_equal(p[key].view(np.uint8), q[key].view(np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("timeout_ms", [0.0, 0.05, 1.0, 200.0])
def test_bounded_waits_at_any_limit(timeout_ms):
    assert lib().ariel_selftest_barrier_timeout(timeout_ms) == A.ARIEL_ERR_DEVICE_TIMEOUT
