"""The differentiation form with rows far longer than what a block's shared memory could hold of them,
as many entries as a frame has atoms, against the same frames with the usual rows."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300.engine import DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu


def evaluate(rows):
    frames, r = [], []
    for k, (ux, uy, cl) in enumerate([(7, 9, [57]), (10, 11, [3])]):
        p, x, _ = build_workload(ux, uy, cl, 300.0, 30 + k)
        x[:, :3] += np.random.RandomState(k).normal(0, 0.03, size=(p.nMol, 3)).astype(np.float32)
        q = diff_frame_params(p)
        q.iNebrMax = rows
        frames.append(q)
        r.append(x)
    model = DiffModel(frames, np.concatenate(r))
    theta = diff_init_theta(frames[0])
    ref = np.random.RandomState(9).normal(0, 1.0, size=(model.n, 3)).astype(np.float32)
    e, gE = model.energy(theta)
    loss, gL = model.force_matching(theta, ref)
    out = [e, gE, model.forces(theta), np.array([loss]), gL]
    model.close()
    return out


# frames of 2,073 and 3,523 atoms: four rows a block to 3,072 entries, then one; rows past an SM's memory
@pytest.mark.parametrize("rows", [3072, 3076, 60000])
def test_long_rows(rows):
    # the order of the FP64 additions varies from run to run, and nothing else
    for x, y in zip(evaluate(rows), evaluate(192)):
        assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max()
