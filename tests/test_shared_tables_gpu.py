"""Replicas of one metal share an EAM table (MIXED): each replica of a context of several metals against
the same system alone, and a fitted model loaded into one replica, which must leave its former sharers as
they were.  The same table values and arithmetic either way: the same bits."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, workloads
from surfacegrowthconsole_gb300.engine import Simulation, diff_init_theta

pytestmark = pytest.mark.gpu


def forces(systems, load=None):
    sim = Simulation([s[0] for s in systems], mode=MODE_MIXED)
    sim.set_state(np.concatenate([s[1] for s in systems]), np.concatenate([s[2] for s in systems]),
                  np.zeros((sum(s[0].nMol for s in systems), 3), np.float32))
    if load:
        sim.load_diff_theta(*load)
    sim.build_lists()
    sim.compute_forces()
    out = [(sim.get_state(k)[0][:, 3], sim.get_state(k)[2], sim.rho(k)) for k in range(len(systems))]
    sim.close()
    return out


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


@pytest.mark.parametrize("metals", [(3, 3, 3), (3, 2, 3), (2, 3, 0)], ids=["one", "two", "three"])
def test_metals_in_one_context(metals):
    systems = [workloads.bulk_metal(5, seed=10 + k, material=m) for k, m in enumerate(metals)]
    for got, s in zip(forces(systems), systems):
        assert same(got, forces([s])[0])


@pytest.mark.parametrize("rep", [0, 1, 2])
def test_model_loaded_into_one_of_the_sharers(rep):
    systems = [workloads.bulk_metal(5, seed=20 + k) for k in range(3)]
    theta = diff_init_theta(systems[0][0])
    theta[2:] *= 1.01
    before, after = forces(systems), forces(systems, (theta, rep))
    for k in range(3):
        assert same(before[k], after[k]) == (k != rep), k
    assert same(after[rep], forces([systems[rep]], (theta, 0))[0])
