"""Sets of frames whose pairs are more than can be laid out at once: the passes over them in batches give
what one layout gives."""
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


def frames(iNebrMax):
    out = []
    for k, (ux, uy, cl, size) in enumerate([(7, 9, [201], 1.0), (8, 10, [1], 1.0), (8, 10, [400], 0.65), (7, 11, [57], 1.0)]):
        p, r, _ = build_workload(ux, uy, cl, 300.0, 60 + k)
        mid = r[:p.nMolMe, :3].mean(0)
        r[:p.nMolMe, :3] = mid + (r[:p.nMolMe, :3] - mid) * np.float32(size)
        r[:, :3] += np.random.RandomState(k).normal(0, 0.03, size=(p.nMol, 3)).astype(np.float32)
        p.iNebrMax, p.blockSize = iNebrMax, 256
        out.append((diff_frame_params(p), r))
    return [f[0] for f in out], np.ascontiguousarray(np.concatenate([f[1] for f in out]))


def evaluate(model, theta, ref):
    e, gE = model.energy(theta)
    loss, gL = model.force_matching(theta, ref)
    return [e, model.energy(theta, grad=False), gE, model.forces(theta), np.array([loss]), gL,
            np.array([model.force_matching(theta, ref, grad=False)])]


@pytest.mark.parametrize("rows", [400, 192])  # 192: truncated rows
def test_batches_equal_one_layout(rows):
    params, r = frames(rows)
    model = DiffModel.__new__(DiffModel)
    arr, h = (L.SimParams * len(params))(*params), C.c_void_p()
    L.check(L.lib().sg_diff_create(arr, len(params), 0, C.byref(h)))
    model._h, model.nframes, model.n = h, len(params), len(r)
    theta = diff_init_theta(params[0])
    ref = np.random.RandomState(9).normal(0, 1.0, size=(model.n, 3)).astype(np.float32)
    whole = None
    # the widest slice has up to 32 (336 + a few) places; the set some 100,000
    for places in (0, 12000, 12345, 40000, 10 ** 6, 0):
        limit(model, places)
        rc = L.lib().sg_diff_set_positions(h, C.c_void_p(r.ctypes.data))
        assert (rc != 0) == (rows == 192)
        got = evaluate(model, theta, ref)
        whole = whole or got
        for x, y in zip(got, whole):  # the order of the FP64 sums and which pairs share a column vary
            assert np.abs(x - y).max() <= 3e-6 * np.abs(y).max()
    model.close()

