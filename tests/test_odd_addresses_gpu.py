"""Host arrays at addresses that are no multiple of four (views into byte buffers), which kernels cannot
read or write in place: downloads, uploads, steps from host arrays and reference forces give what they
give at aligned addresses."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, _lib as L
from surfacegrowthconsole_gb300.engine import DiffModel, Simulation, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu


class At:
    """A float array of n rows of w, `shift` bytes past a 16-byte boundary."""

    def __init__(self, n, w, shift, x=None):
        self.n, self.w = n, w
        self.buf = np.zeros(4 * n * w + 32, np.uint8)
        self.o = -self.buf.ctypes.data % 16 + shift
        if x is not None:
            self.buf[self.o:self.o + 4 * n * w] = np.ascontiguousarray(x, np.float32).view(np.uint8).ravel()
        self.ptr = C.c_void_p(self.buf.ctypes.data + self.o)

    def get(self):
        return self.buf[self.o:self.o + 4 * self.n * self.w].copy().view(np.float32).reshape(self.n, self.w)


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("shifts", [(0, 1, 0), (0, 0, 2), (0, 3, 3), (1, 2, 3)])
def test_states_at_odd_addresses(mode, shifts):
    p, r, v = build_workload(4, 9, [128], 500.0, 77, step_limit=10 ** 6, delta_t=0.005)
    a = np.random.RandomState(1).normal(0, 0.1, size=(p.nMol, 3)).astype(np.float32)
    out = []
    for at in ((0, 0, 0), shifts):
        sim = Simulation(p, mode=mode)
        x = [At(p.nMol, w, s, y) for w, s, y in zip((4, 3, 3), at, (r, v, a))]
        L.check(L.lib().sg_set_state(sim.handle, -1, *(y.ptr for y in x)))
        sim.step(3)
        L.check(L.lib().sg_step_from_host(sim.handle, -1, *(y.ptr for y in x), 1, 0, None))
        got = [At(p.nMol, w, s) for w, s in zip((4, 3, 3), at)]
        L.check(L.lib().sg_get_state(sim.handle, -1, *(y.ptr for y in got)))
        only = At(p.nMol, 3, at[1])
        L.check(L.lib().sg_get_state(sim.handle, 0, None, only.ptr, None))
        out.append([y.get() for y in got] + [only.get()])
        sim.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_reference_forces_at_odd_addresses(shift):
    p, r, _ = build_workload(7, 9, [57], 300.0, 31)
    q = diff_frame_params(p)
    model = DiffModel([q], r)
    theta = diff_init_theta(q)
    ref = np.random.RandomState(2).normal(0, 1.0, size=(p.nMol, 3))
    loss = []
    for s in (0, shift):
        x, y = At(p.nMol, 3, s, ref), C.c_double()
        L.check(L.lib().sg_diff_force_matching(model._h, C.c_void_p(theta.ctypes.data), x.ptr, C.byref(y), None))
        loss.append(y.value)
    assert abs(loss[1] - loss[0]) <= 1e-6 * loss[0]  # the order of the sums varies
    model.close()
