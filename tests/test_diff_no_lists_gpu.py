"""A set of positions whose pair lists could not be made: the evaluations answer with the error, not with
zeros, until positions are set that have some."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import _lib as L
from surfacegrowthconsole_gb300.engine import DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu


def limit(model, places):
    f = L.lib()._Z20sg_diff_limit_placesP7sg_diffy
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_ulonglong]
    assert f(model._h, places) == 0


def test_no_lists_no_results():
    p, r, _ = build_workload(7, 9, [57], 300.0, 61)
    model = DiffModel([diff_frame_params(p)], r)
    theta = diff_init_theta(p)
    ref = np.zeros((model.n, 3), np.float32)
    e, loss, f = model.energy(theta, grad=False), model.force_matching(theta, ref, grad=False), model.forces(theta)
    limit(model, 64)  # fewer than any slice of the set has
    for call in (lambda: model.set_positions(r), lambda: model.energy(theta), lambda: model.forces(theta),
                 lambda: model.force_matching(theta, ref), lambda: model.energy(theta, grad=False)):
        with pytest.raises(L.SgError, match="SG_ERR_NOMEM"):
            call()
    limit(model, 0)
    model.set_positions(r)
    # the order of the sums varies
    assert np.abs(model.energy(theta, grad=False) - e).max() <= 1e-6 * np.abs(e).max()
    assert abs(model.force_matching(theta, ref, grad=False) - loss) <= 1e-6 * loss
    assert np.abs(model.forces(theta) - f).max() <= 1e-6 * np.abs(f).max()
    model.close()
