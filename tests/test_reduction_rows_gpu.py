"""The step's sums (PLAIN) over the numbers of 1,024-atom blocks where their final tree changes form (32,
64 and 128 blocks), against the reference's stride-halving tree restated in FP32 on the downloaded state:
bit for bit, and the metal centre-of-mass velocity of the same sizes."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_PLAIN, workloads
from surfacegrowthconsole_gb300.engine import Simulation

pytestmark = pytest.mark.gpu


def tree(x):
    """Blocks of 1,024 values, zero-padded and halved; then the block sums the same way."""
    x = np.pad(np.asarray(x, np.float32), (0, -len(x) % 1024)).reshape(-1, 1024)
    while x.shape[1] > 1:
        h = x.shape[1] // 2
        x = x[:, :h] + x[:, h:]
    return x[0, 0] if len(x) == 1 else tree(x[:, 0])


@pytest.mark.parametrize("cells", [6, 7, 20, 21, 25, 26, 32, 33])  # 1, 2, 32, 37, 62, 69, 128 and 141 blocks
def test_sums_match_the_reference_tree(cells):
    p, r, v = workloads.bulk_metal(cells)
    r[:, :3] += np.random.RandomState(3).normal(0, 0.02, size=(p.nMol, 3)).astype(np.float32)
    sim = Simulation(p, mode=MODE_PLAIN)
    sim.set_state(r, v, np.zeros((p.nMol, 3), np.float32))
    sim.step(2)
    rg, vg, _ = sim.get_state()
    t = sim.thermo(0)
    sq = vg[:, 0] * vg[:, 0] + vg[:, 1] * vg[:, 1] + vg[:, 2] * vg[:, 2]
    assert np.float32(t.vvSum) == tree(np.float32(p.massMe) * sq)
    assert np.float32(t.uSum) == tree(rg[:, 3])
    assert np.float32(t.vvMax) == sq.max()
    for got, c in zip((t.cmVel.x, t.cmVel.y, t.cmVel.z), vg.T):
        assert np.float32(got) == tree(c)
    sim.close()
