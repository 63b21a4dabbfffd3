"""The bytes of a handle's state (ariel_state_bytes, what the request server admits by): the density's
pair records take no memory of their own, so a scene needs no more than it did without them (the
bytes below), and a server with a given budget accepts what it accepted.  Where the records share
memory with the solver or the host I/O staging area, a density after either is that of a fresh
sort."""
import numpy as np
import pytest

from ariel_b200 import _abi as A
from ariel_b200 import workloads
from ariel_b200.flipsim import Batch, state_bytes

from helpers import assert_bits, params

# per scene set: bytes in REF32, FP64 and MIXED without pair records
SETS = {
    "16": (lambda: [A.scene_dambreak(16)], (1721856, 2016768, 1771008)),
    "64": (lambda: [A.scene_dambreak(64)], (109106432, 127980800, 112252160)),
    "full": (lambda: [A.scene_dambreak(48, liquid_hi=(1.0, 1.0, 1.0))], (129459712, 137422336, 130786816)),
    "thin": (lambda: [A.scene_dambreak(40, liquid_hi=(0.05, 0.6, 1.0))], (13344512, 17952512, 14112512)),
    "sphere": (lambda: [workloads.sphere_dambreak(48)], (46345472, 54308096, 47672576)),
    "batch": (lambda: [A.scene_dambreak(32), A.scene_dambreak(21, liquid_hi=(0.9, 0.9, 1.0)), A.scene_dambreak(5)],
              (22942976, 25978880, 23449088)),
}


@pytest.mark.parametrize("name", sorted(SETS))
def test_no_memory_for_pair_records(name):
    make, old = SETS[name]
    for precision in (A.PREC_REF32, A.PREC_FP64, A.PREC_MIXED):
        assert state_bytes(make(), params(precision=precision)) <= old[precision]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [A.PREC_REF32, A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("hi", [(1.0, 1.0, 1.0), (0.3, 0.3, 0.3), (0.1, 0.05, 0.1)])
def test_density_after_what_shares_its_memory(hi, precision):
    descs = [A.scene_dambreak(13, liquid_hi=hi), A.scene_dambreak(18, liquid_hi=hi, seed=5)]
    b = Batch(descs, params(precision=precision, stop=A.STOP_REL))
    b.init()
    b.stage(A.STAGE_SORT)
    b.stage(A.STAGE_DENSITY)
    want = [b.get_particles(s) for s in range(2)]
    frame = [(np.empty_like(w["pos"]), np.empty_like(w["vel"])) for w in want]

    def up():
        for s in range(2):
            b.upload_state(want[s]["pos"], want[s]["vel"], s)

    between = [lambda: None, lambda: b.get_particles(1), lambda: b.download_state(*frame[0], 0), up,
               lambda: b.stage(A.STAGE_SOLVE)]
    for f in between:
        b.stage(A.STAGE_SORT)
        f()
        for _ in range(2):
            b.stage(A.STAGE_DENSITY)
            for s in range(2):
                assert_bits("scene %d" % s, b.get_particles(s)["density"], want[s]["density"])
    b.step(2)  # and a step goes on from there
    b.synchronize()
    b.close()
