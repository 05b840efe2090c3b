"""Steps launched several to a graph against steps launched one by one: the same kernels in the same
order, so the same bits.  A variant of the step goes into groups after 64 single ones; the counts asked
for end groups of 8, 4 and 2 steps early, with and without the last one's publish, across RDF samples and
the start of the shear drive."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, workloads
from surfacegrowthconsole_gb300.engine import Simulation

pytestmark = pytest.mark.gpu


def system(rdf, shear_at):
    p, r, v = workloads.small(seed=44)
    p.bRdf, p.stepRdf, p.limitRdf = int(rdf), 13, 3
    if shear_at:
        p.stepEquil, p.stepCool = 0, shear_at
        p.deltaF = np.float32(2.0) * np.float32(p.forceU) * np.float32(0.001)
    return p, r, v


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("rdf,shear_at", [(False, 0), (True, 0), (False, 90)], ids=["plain_steps", "rdf", "shear"])
def test_groups_match_single_steps(mode, rdf, shear_at):
    p, r, v = system(rdf, shear_at)
    a = np.zeros((p.nMol, 3), np.float32)
    one, many = Simulation(p, mode=mode), Simulation(p, mode=mode)
    for sim in (one, many):
        sim.set_state(r, v, a)
    for n in (65, 10, 1, 2, 3, 7, 8, 9, 33, 12, 80):
        for _ in range(n):
            one.step(1)
        many.step(n)
        x, y = one.thermo(0), many.thermo(0)
        for f in ("stepCount", "kinEnergy", "potEnergy", "vvSum", "uSum", "vvMax", "countRdf"):
            if hasattr(x, f):
                assert getattr(x, f) == getattr(y, f), (n, f)
        for x, y in zip(one.get_state(), many.get_state()):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), n
        if rdf:
            assert np.array_equal(one.rdf(0), many.rdf(0))
    one.close()
    many.close()


def test_kernels_per_step_after_a_group():
    p, r, v = system(False, 0)
    a = np.zeros((p.nMol, 3), np.float32)
    counts = []
    for steps in (1, 72):  # a single step; 64 single ones and a group of 8 that ends with the publish
        sim = Simulation(p)
        sim.set_state(r, v, a)
        sim.step(steps)
        counts.append(sim.kernels_per_step())
        sim.close()
    assert counts[0] == counts[1] > 0
