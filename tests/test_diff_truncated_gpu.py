"""The differentiation form on lists that did not fit their rows (iNebrMax too small: set_positions
reports it and goes on with the truncated rows): the energy and its gradient still belong to one
function, taken by finite differences of the energy."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import _lib as L
from surfacegrowthconsole_gb300.engine import DIFF_NPARAM, DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu

PHI, DEN = slice(2, 34), slice(34, 66)
# E is linear in phi's coefficients: a difference over a step of 1 is the derivative but for the FP32
# of two energies (1e-5 of an energy that the step changes by its own order)
PHI_REL = 1e-4
# a central difference over f's coefficients scaled by 1 +- 0.01: 1e-5 / 0.02 from FP32, a few 0.01^2
# from the curvature
DEN_REL = 3e-3


def squeezed(rows):
    """Two frames, one with a cluster pressed to 0.65 of its size, whose atoms have up to 336 entries (98
    of them more than 192, the fewest a frame's rows hold)."""
    frames, r = [], []
    for k, (ux, uy, cl, size) in enumerate([(8, 10, [400], 0.65), (7, 9, [57], 1.0)]):
        p, x, _ = build_workload(ux, uy, cl, 300.0, 20 + k)
        mid = x[:p.nMolMe, :3].mean(0)
        x[:p.nMolMe, :3] = mid + (x[:p.nMolMe, :3] - mid) * np.float32(size)
        x[:, :3] += np.random.RandomState(k).normal(0, 0.03, size=(p.nMol, 3)).astype(np.float32)
        p.iNebrMax, p.blockSize = rows, 256  # cells with room for them
        frames.append(diff_frame_params(p))
        r.append(x)
    arr, h = (L.SimParams * len(frames))(*frames), C.c_void_p()
    L.check(L.lib().sg_diff_create(arr, len(frames), 0, C.byref(h)))
    model = DiffModel.__new__(DiffModel)
    model._h, model.nframes, model.n = h, len(frames), sum(q.nMol for q in frames)
    r = np.ascontiguousarray(np.concatenate(r))
    return model, frames[0], L.lib().sg_diff_set_positions(h, C.c_void_p(r.ctypes.data))


@pytest.mark.parametrize("rows", [192, 256, 400])
def test_gradient_of_the_energy_over_truncated_rows(rows):
    model, p, rc = squeezed(rows)
    assert (rc != 0) == (rows < 400)
    theta = diff_init_theta(p) * (1 + 0.02 * np.random.RandomState(5).normal(size=DIFF_NPARAM))
    e0, g = model.energy(theta)
    diff = np.zeros(32)
    for k in range(32):
        t = theta.copy()
        t[2 + k] += 1.0
        diff[k] = (model.energy(t, grad=False) - e0).sum()
    assert np.abs(g[PHI] - diff).max() <= PHI_REL * np.abs(diff).max()
    up, down = theta.copy(), theta.copy()
    up[DEN] *= 1.01
    down[DEN] *= 0.99
    slope = (model.energy(up, grad=False) - model.energy(down, grad=False)).sum() / 0.02
    assert abs((g[DEN] * theta[DEN]).sum() - slope) <= DEN_REL * abs(slope)
    model.close()
