"""The differentiation form where its packed pair lists and its grids change shape, against the
FP64 restatement (oracle.diff_eval): uneven frames, one of a single metal atom, atoms with more pairs
than a lane group keeps in registers, and a set large enough that the reference forces stream in
their own launch; a second set of positions on the same model."""
import numpy as np
import pytest

import oracle
from surfacegrowthconsole_gb300.engine import DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu

# as tests/test_diff_gpu.py: energies, forces (RMS), loss and gradients relative
ENERGY_REL, FORCE_REL, LOSS_REL, GRAD_REL = 1e-5, 1e-5, 1e-4, 1e-4


def frame(ux, uy, clusters, seed, squeeze=1.0):
    p, r, _ = build_workload(ux, uy, clusters, 300.0, seed)
    rng = np.random.RandomState(seed)
    m = p.nMolMe
    if m:
        mid = r[:m, :3].mean(0)
        r[:m, :3] = mid + (r[:m, :3] - mid) * np.float32(squeeze)
    r[:, :3] += rng.normal(0, 0.03, size=(p.nMol, 3)).astype(np.float32)
    r[:, 3] = 0
    return diff_frame_params(p), r


def uneven(seed):
    return [frame(7, 9, [201], seed), frame(8, 10, [7], seed + 1), frame(9, 9, [1], seed + 2), frame(7, 11, [57], seed + 3)]


def dense(seed):
    return [frame(8, 10, [400], seed, squeeze=0.85)]


def large(seed):
    return [frame(24, 24, [333], seed), frame(25, 24, [801], seed + 1), frame(24, 24, [97], seed + 2),
            frame(30, 24, [2], seed + 3)]


@pytest.mark.parametrize("frames_of", [uneven, dense, large])
def test_evaluations_match_the_fp64_model(frames_of):
    model = None
    for seed in (3, 40):  # the second set of positions replaces the first one's lists
        frames = frames_of(seed)
        params, r = [f[0] for f in frames], np.concatenate([f[1] for f in frames])
        if model is None:
            model = DiffModel(params, r)
        else:
            model.set_positions(r)
        rng = np.random.RandomState(seed)
        theta = diff_init_theta(params[0]) * (1 + 0.02 * rng.normal(size=66))
        ref = rng.normal(0, 1.0, size=(len(r), 3)).astype(np.float32)
        e64, f64, gE64, L64, gL64 = oracle.diff_eval(params, r, theta, ref)
        e, gE = model.energy(theta)
        assert np.abs(e - e64).max() <= ENERGY_REL * np.abs(e64).max()
        assert np.abs(model.energy(theta, grad=False) - e64).max() <= ENERGY_REL * np.abs(e64).max()
        assert np.abs(gE - gE64).max() <= GRAD_REL * np.abs(gE64).max()
        f = model.forces(theta)
        assert np.linalg.norm(f - f64) <= FORCE_REL * np.linalg.norm(f64)
        assert np.array_equal(np.abs(f).sum(1) == 0, np.abs(f64).sum(1) == 0)  # atoms without a pair
        # reference forces at any 4-byte alignment
        for shift in (0, 1):
            buf = np.zeros(3 * len(r) + 4, np.float32)
            mine = buf[shift:shift + 3 * len(r)].reshape(-1, 3)
            mine[:] = ref
            L, gL = model.force_matching(theta, mine)
            assert abs(L - L64) <= LOSS_REL * L64
            assert np.abs(gL - gL64).max() <= GRAD_REL * np.abs(gL64).max()
            assert abs(model.force_matching(theta, mine, grad=False) - L64) <= LOSS_REL * L64
    model.close()
