"""Reference forces whose squares overflow: the loss is infinite, whichever atom they belong to (one
with pairs, one without; first and last; whatever the array's alignment), and not a NaN."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300.engine import DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [1e25, float("inf")])
@pytest.mark.parametrize("shift", [0, 1])
def test_overflowing_reference_forces(value, shift):
    p, r, _ = build_workload(7, 9, [57], 300.0, 31)
    q = diff_frame_params(p)
    model = DiffModel([q], r)
    theta = diff_init_theta(q)
    n = q.nMol
    buf = np.zeros(3 * n + 8, np.float32)
    o = (-buf.ctypes.data % 16) // 4 + shift
    ref = buf[o:o + 3 * n].reshape(n, 3)
    for atom in (0, 1, 2, 3, n - 1):  # metal atoms, with pairs; a carbon atom far from the cluster
        for c in range(3):
            ref[atom, c] = value
            assert model.force_matching(theta, ref, grad=False) == np.inf
            ref[atom, c] = 0
    assert np.isfinite(model.force_matching(theta, ref, grad=False))
    model.close()
