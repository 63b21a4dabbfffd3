"""The resident pressure solve (one or two chunks of a scene per SM, state on chip) against the
streaming kernel: a scene takes the one or the other by its FLUID count and the number of blocks,
and both evaluate the same sums in the same order, so the pressures must be equal bit for bit.
`pcg_grid_blocks` caps the blocks, which sends a scene of more than two chunks per block to the
streaming kernel.  The streaming kernel's own answers are held to the FP64 oracle in test_pcg.py.
"""
import numpy as np
import pytest

from ariel_b200 import _abi as A
from ariel_b200.flipsim import Batch

from helpers import params


def _solve(n, fluid, precision, blocks, seed=3, tol=1e-5):
    rng = np.random.default_rng(seed)
    d = A.scene_dambreak(n)
    d.n_liquid = 0
    b = Batch([d], params(precision=precision, stop=A.STOP_REL, tol=tol, pcg_grid_blocks=blocks))
    b.init()
    b.set_grid(A.GRID_A, fluid.astype(np.int32))
    b.set_grid(A.GRID_L, np.where(fluid, -3.0 + rng.random((n, n, n)), 1.6).astype(np.float32))
    b.set_grid(A.GRID_D, np.where(fluid, rng.standard_normal((n, n, n)), 0.0).astype(np.float32))
    b.set_grid(A.GRID_P64, np.zeros((n, n, n)))
    b.stage(A.STAGE_SOLVE)
    out = b.get_grid(A.GRID_P64), b.get_grid(A.GRID_P), b.stats()
    b.close()
    return out


def _first(n, cells):
    """The first `cells` cells of the grid in (i, j, k) order."""
    return (np.arange(n ** 3) < cells).reshape(n, n, n)


def _slabs(n):
    """Pairs of planes on both sides of the list bricks' x borders: every cell has its x neighbour
    in another brick, more neighbours in other blocks than a block of this size has slots for."""
    m = np.zeros((n, n, n), bool)
    m[np.arange(n) % 8 % 7 == 0] = True
    return m


CASES = [
    # FLUID counts around one chunk, the smallest chunks' end, and blocks of one and two chunks
    (20, _first(20, 0)), (20, _first(20, 1)), (20, _first(20, 511)), (20, _first(20, 513)),
    (33, _first(33, 33 ** 3 - 700)), (60, _first(60, 148 * 512)), (60, _first(60, 148 * 512 + 1)),
    (61, _first(61, 296 * 512)), (61, _first(61, 296 * 512 + 1)),
    # two full-size chunks per block, one cell more (up to four), four, and one cell too many
    (86, _first(86, 296 * 2048)), (86, _first(86, 296 * 2048 + 1)),
    (107, _first(107, 592 * 2048)), (107, _first(107, 592 * 2048 + 1)),
    (134, _slabs(134)), (160, _slabs(160)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [A.PREC_MIXED, A.PREC_FP64])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_resident_equals_streaming(case, precision):
    n, fluid = CASES[case]
    p64, p, st = _solve(n, fluid, precision, 0)
    q64, q, su = _solve(n, fluid, precision, 1 if n < 61 else 24)
    assert st.n_fluid_cells == su.n_fluid_cells == fluid.sum()
    assert st.pcg_converged == 1 and st.pcg_iterations == su.pcg_iterations
    assert st.pcg_rel_residual == su.pcg_rel_residual
    np.testing.assert_array_equal(p64, q64)
    np.testing.assert_array_equal(p, q)
