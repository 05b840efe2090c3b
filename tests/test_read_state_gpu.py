"""sg_get_state's one-launch download against its copying route (taken when r is not 16-byte
aligned) on the same state: all replicas and single ones, with and without a pending thermostat
rescale, partial requests, sizes around the blocks of 128 atoms; and that a download changes nothing
a later step sees."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, _lib as L
from surfacegrowthconsole_gb300.engine import Simulation, build_workload

pytestmark = pytest.mark.gpu


def systems():
    out = []
    for k, (ux, uy, cl) in enumerate([(4, 8, [53]), (4, 9, [128]), (5, 8, [1]), (4, 8, [96])]):  # 1,077 .. 1,281 atoms
        out.append(build_workload(ux, uy, cl, 500.0, 70 + k, step_limit=10 ** 6, delta_t=0.005))
    return out


def download(sim, rep, want, shift):
    """(r, v, a) through pointers `shift` bytes past a 16-byte boundary; None where not wanted."""
    n = sim.natoms(rep)
    bufs = [np.full(n * w + 8, np.float32(-7)) for w in (4, 3, 3)]
    bases = [(-b.ctypes.data) % 16 + shift for b in bufs]
    ptr = [C.c_void_p(b.ctypes.data + o) if use else None for b, o, use in zip(bufs, bases, want)]
    L.check(L.lib().sg_get_state(sim.handle, rep, *ptr))
    return [b.view(np.uint8)[o:o + 4 * n * w].view(np.float32).reshape(n, w).copy() if use else None
            for b, o, w, use in zip(bufs, bases, (4, 3, 3), want)]


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("steps", [24, 25])  # the thermostat decides a rescale in step 25
def test_download_routes_agree(mode, steps):
    reps = systems()
    sims = []
    for _ in range(2):
        sim = Simulation([s[0] for s in reps], mode=mode)
        sim.set_state(np.concatenate([s[1] for s in reps]), np.concatenate([s[2] for s in reps]),
                      np.zeros((sum(s[0].nMol for s in reps), 3), np.float32))
        sim.step(steps)
        sims.append(sim)
    direct, copied = sims
    # every direct download before the copying route, which applies the rescale on the device
    for want in ((1, 1, 1), (0, 1, 0), (1, 0, 1)):
        for rep in (-1, 0, 2, len(reps) - 1):
            got = download(direct, rep, want, 0)
            ref = download(copied, rep, want, 4 if want[0] else 0)
            for g, r in zip(got, ref):
                assert (g is None) == (r is None)
                assert g is None or np.array_equal(g, r)
    direct.step(5)
    copied.step(5)
    for g, r in zip(direct.get_state(), copied.get_state()):
        assert np.array_equal(g, r)
    for sim in sims:
        sim.close()
