"""A context of one replica (its kernels take the block tables' entries from their parameters, and load
rows before their lengths are known) against the same system twice in one context (tables in memory):
the same arithmetic in the same order, so the same bits.  Sizes around the blocks of 128 / lanes metal
atoms, 32 carbon atoms, 128 atoms and 1,024 reduced atoms, metal only, one metal atom."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, workloads
from surfacegrowthconsole_gb300.engine import Simulation, build_workload

pytestmark = pytest.mark.gpu


def sheet(ux, uy, clusters, seed):
    return build_workload(ux, uy, clusters, 500.0, seed, step_limit=10 ** 6, delta_t=0.005)


CASES = {"one_metal": lambda: sheet(4, 8, [1], 3), "below_block": lambda: sheet(4, 8, [31], 4),
         "whole_blocks": lambda: sheet(4, 8, [128], 5), "above_block": lambda: sheet(5, 8, [129], 6),
         "metal_1025": lambda: sheet(8, 12, [1025], 7), "metal_only": lambda: workloads.bulk_metal(7, seed=3)}


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("lanes", [4, 16])
@pytest.mark.parametrize("name", CASES)
def test_one_replica_matches_two(name, lanes, mode):
    p, r, v = CASES[name]()
    a = np.zeros((p.nMol, 3), np.float32)
    one, two = Simulation([p], mode=mode, metal_lanes=lanes), Simulation([p, p], mode=mode, metal_lanes=lanes)
    one.set_state(r, v, a)
    two.set_state(np.concatenate([r, r]), np.concatenate([v, v]), np.concatenate([a, a]))
    for sim in (one, two):
        sim.step(12)  # the lists are built, kept and built again
    got = one.get_state()
    for rep in (0, 1):
        for x, y in zip(got, two.get_state(rep)):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    if mode == MODE_PLAIN:  # MIXED sums its blocks of 256 to 2,048 atoms by the size of the whole context
        t = one.thermo(0)
        for rep in (0, 1):
            s = two.thermo(rep)
            for f in ("kinEnergy", "potEnergy", "totEnergy", "vvSum", "uSum", "vvMax"):
                assert getattr(t, f) == getattr(s, f), f
    one.close()
    two.close()
