"""The density over pair records (csrc/particles.cu, k_density) bit for bit against the oracle:
cells of few and odd numbers of particles up to the walls, solid particles among them, grids with
and without a power-of-two kernel radius, and a radius far out of range; and the records rebuilt
where the last sort was the resampler's, which leaves them out."""
import numpy as np
import pytest

from ariel_b200 import _abi as A
from ariel_b200.flipsim import Batch

from helpers import assert_bits, dambreak, params


@pytest.mark.gpu
@pytest.mark.parametrize("n,count,density", [(2, 1, 0.5), (2, 9, 0.5), (5, 2, 0.5), (16, 3000, 0.5), (31, 20001, 0.5),
                                             (33, 40000, 0.3), (16, 500, 1e12), (12, 400, 1e-12)])
def test_density_bits(n, count, density):
    from oracle.pyoracle import RefSim
    rng = np.random.default_rng(n + count)
    desc = A.scene_dambreak(n, density=density)
    prm = params()
    pos = rng.random((count, 3)).astype(np.float32)
    pos[rng.random(count) < 0.3] *= np.float32(0.2)  # crowded corner
    pos[: count // 20] = np.round(pos[: count // 20])  # on the walls and in the corners
    vel = np.zeros((count, 3), np.float32)
    typ = np.where(rng.random(count) < 0.1, A.SOLID, A.FLUID).astype(np.int32)
    mass = np.where(typ == A.SOLID, 10.0, 1.0 + rng.random(count)).astype(np.float32)
    got = []
    for make in (lambda: Batch([desc], prm), lambda: RefSim(desc, prm)):
        s = make()
        s.set_particles(pos, vel, mass, typ)
        s.stage(A.STAGE_SORT)
        s.stage(A.STAGE_DENSITY)
        got.append(s.get_particles()["density"])
        s.close()
    assert_bits("density", got[0], got[1])


@pytest.mark.gpu
@pytest.mark.parametrize("density", [1e25, 1e19, 1e-25])
@pytest.mark.parametrize("count", [1, 2, 301])
def test_density_bits_where_the_squared_radius_leaves_the_range(count, density):
    """A kernel radius whose square overflows (every particle near counts with its whole mass) or
    is zero (no number): cells of odd counts, whose last pair record is filled up."""
    from oracle.pyoracle import RefSim
    rng = np.random.default_rng(count)
    desc = A.scene_dambreak(4, density=density)
    pos = rng.random((count, 3)).astype(np.float32)
    got = []
    for make in (lambda: Batch([desc], params()), lambda: RefSim(desc, params())):
        s = make()
        s.set_particles(pos, np.zeros_like(pos), np.ones(count, np.float32), np.full(count, A.FLUID, np.int32))
        s.stage(A.STAGE_SORT)
        s.stage(A.STAGE_DENSITY)
        got.append(s.get_particles()["density"])
        s.close()
    if density > 1:
        assert not np.isnan(got[1]).any()
    assert_bits("density", got[0], got[1])


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [0, 1])
def test_density_after_the_resamplers_sort(graph):
    # no resampling: the step's last sort leaves every particle where a fresh sort finds it
    b = Batch([dambreak(20), dambreak(13, seed=3)], params(graph=graph, resample_every=0))
    b.init()
    b.step(3)
    b.stage(A.STAGE_DENSITY)
    stale = [b.get_particles(s)["density"] for s in range(2)]
    b.stage(A.STAGE_SORT)
    b.stage(A.STAGE_DENSITY)
    for s in range(2):
        assert_bits("scene %d" % s, b.get_particles(s)["density"], stale[s])
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [13, 20])
def test_density_after_a_resampling_that_moved_particles(n):
    """The resampler sorts the advected particles and then moves them; the records made after it are
    those of its sort, so the density is that of a sort and a density in the resampler's place."""
    got = []
    for stages in ((A.STAGE_SORT, A.STAGE_DENSITY), (A.STAGE_RESAMPLE, A.STAGE_DENSITY)):
        b = Batch([dambreak(n), dambreak(n - 4, seed=3)], params())
        b.init()
        b.step(2)
        for g in range(A.STAGE_RESAMPLE):
            b.stage(g)
        for g in stages:
            b.stage(g)
        got.append([b.get_particles(s) for s in range(2)])
        b.close()
    for s in range(2):
        assert (got[0][s]["pos"] != got[1][s]["pos"]).any()
        assert_bits("scene %d" % s, got[1][s]["density"], got[0][s]["density"])
