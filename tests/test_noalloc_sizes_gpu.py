"""sg_compute_forces_noalloc over the sizes where its sort, work items and launches change shape,
against the context path (sg_build_lists + sg_compute_forces) on the same input: one and several
blocks of cells, the largest system, metal only, atoms outside the grid, a crowded cell."""
import ctypes as C

import numpy as np
import pytest

from surfacegrowthconsole_gb300 import _lib as L
from surfacegrowthconsole_gb300 import workloads
from surfacegrowthconsole_gb300.engine import Simulation, build_workload

pytestmark = pytest.mark.gpu

FORCE_RTOL, FORCE_ATOL = 2e-5, 1e-6  # tests/test_zz_no_alloc.py


def sheet(ux, uy, clusters, seed):
    p, r, _ = build_workload(ux, uy, clusters, 300.0, seed)
    return p, r


def bulk():
    p, r, _ = workloads.bulk_metal(10, seed=3)
    return p, r


def largest():
    # 15,872 C + 512 Ni = 16,384 atoms
    p, r = sheet(16, 31, [512], 5)
    assert p.nMol == 16384
    return p, r


def outside():
    p, r = sheet(7, 9, [201], 6)
    r[5, 2] = 10 * p.region.z     # a metal atom above the grid
    r[300, 0] = np.nan            # a carbon atom without a position
    return p, r


CASES = {"small": lambda: sheet(7, 9, [201], 4), "one_metal": lambda: sheet(8, 8, [1], 7),
         "several_blocks": lambda: sheet(19, 24, [1291], 8), "largest": largest, "metal_only": bulk, "outside": outside}


@pytest.mark.parametrize("name", CASES)
def test_sizes_match_the_context_path(name):
    import torch
    p, r = CASES[name]()
    rng = np.random.RandomState(11)
    r[:, :3] += rng.normal(0, 0.03, size=(p.nMol, 3)).astype(np.float32)
    r[:, 3] = 0
    sim = Simulation(p)
    sim.set_state(r, np.zeros((p.nMol, 3), np.float32), np.zeros((p.nMol, 3), np.float32))
    sim.build_lists()
    sim.compute_forces()
    rc, _, ac = sim.get_state()
    sim.close()
    pos = torch.from_numpy(r).cuda()
    acc = torch.full((p.nMol, 4), float("nan"), device="cuda")
    for _ in range(2):  # the second call starts from the first one's scratch
        L.check(L.lib().sg_compute_forces_noalloc(C.byref(p), C.c_void_p(pos.data_ptr()), C.c_void_p(acc.data_ptr()),
                                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        for got, want in ((acc.cpu().numpy()[:, :3], ac), (pos.cpu().numpy()[:, 3], rc[:, 3])):
            bad = ~np.isfinite(want)
            assert np.array_equal(bad, ~np.isfinite(got))
            scale = np.abs(want[~bad]).max()
            assert np.abs(got[~bad].astype(np.float64) - want[~bad]).max() <= FORCE_RTOL * scale + FORCE_ATOL


def test_crowded_cell_is_reported():
    import torch
    p, r = sheet(7, 9, [201], 9)
    rng = np.random.RandomState(1)
    r[400:480, :3] = r[400, :3] + rng.uniform(0, 0.4, size=(80, 3)).astype(np.float32)  # 81 atoms near one place
    pos = torch.from_numpy(r).cuda()
    acc = torch.zeros((p.nMol, 4), device="cuda")
    with pytest.raises(L.SgError) as e:
        L.check(L.lib().sg_compute_forces_noalloc(C.byref(p), C.c_void_p(pos.data_ptr()), C.c_void_p(acc.data_ptr()),
                                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert e.value.code in (5, 11)  # more than 64 atoms in a cell; their lists may overflow too
