"""Velocities that a download has returned are the ones the context goes on with: a download at a
thermostat step, then an upload that leaves velocities alone (positions only, one replica of several,
one step from one replica's host arrays), by the one-launch route and by the copying one (r not
16-byte aligned), whose later steps agree bit for bit."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, _lib as L
from surfacegrowthconsole_gb300.engine import Simulation, build_workload

pytestmark = pytest.mark.gpu

STEPS = 25  # the thermostat decides a rescale in step 25, applied when the velocities are next read


def systems(count):
    shapes = [(4, 8, [53]), (4, 9, [128]), (5, 8, [1])]
    return [build_workload(ux, uy, cl, 500.0, 90 + k, step_limit=10 ** 6, delta_t=0.005)
            for k, (ux, uy, cl) in enumerate(shapes[:count])]


def start(mode, count):
    reps = systems(count)
    sim = Simulation([s[0] for s in reps], mode=mode)
    sim.set_state(np.concatenate([s[1] for s in reps]), np.concatenate([s[2] for s in reps]),
                  np.zeros((sum(s[0].nMol for s in reps), 3), np.float32))
    sim.step(STEPS)
    return sim


def download(sim, rep, shift):
    """r, v, a of a replica; r at `shift` bytes past a 16-byte boundary."""
    n = sim.natoms(rep)
    buf = np.zeros(4 * n + 8, np.float32)
    o = ((-buf.ctypes.data) % 16 + shift) // 4
    r, v, a = buf[o:o + 4 * n].reshape(n, 4), np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
    L.check(L.lib().sg_get_state(sim.handle, rep, *(C.c_void_p(x.ctypes.data) for x in (r, v, a))))
    return r.copy(), v, a


@pytest.mark.parametrize("shift", [0, 4], ids=["direct", "copied"])
@pytest.mark.parametrize("count", [1, 3])
@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
def test_upload_of_positions_keeps_the_returned_velocities(mode, count, shift):
    sim = start(mode, count)
    r, v, _ = download(sim, -1, shift)
    sim.set_state(r + np.float32(0.001))
    assert np.array_equal(download(sim, -1, shift)[1], v)
    sim.close()


@pytest.mark.parametrize("shift", [0, 4], ids=["direct", "copied"])
@pytest.mark.parametrize("of", [-1, 0, 2])  # the download: all replicas, the uploaded one, another
@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
def test_upload_of_one_replica_keeps_the_others(mode, of, shift):
    sim, before = start(mode, 3), start(mode, 3)
    offs = np.cumsum([0] + [before.natoms(k) for k in range(3)])
    want = download(before, -1, shift)[1]
    download(sim, of, shift)
    r0, v0, a0 = download(sim, 0, shift)
    sim.set_state(r0, v0, a0, rep=0)
    for k in range(3):
        assert np.array_equal(download(sim, k, shift)[1], want[offs[k]:offs[k + 1]])
    sim.close()
    before.close()


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
def test_later_steps_do_not_depend_on_the_route(mode):
    out = []
    for shift in (0, 4):
        sim = start(mode, 3)
        r, v, a = download(sim, 1, shift)
        sim.step_from_host(r, v, a, rep=1)
        r, v, a = download(sim, -1, shift)
        sim.set_state(r)
        sim.step(STEPS)  # past the next rescale
        download(sim, 2, shift)
        sim.step(3)
        out.append(download(sim, -1, shift))
        sim.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
