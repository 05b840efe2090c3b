"""Sums over sets of frames so large that a thread adds many terms: large terms first, then many that a
plain FP32 sum of them would lose, so that what is lost grows with the set."""
import numpy as np
import pytest

from surfacegrowthconsole_gb300 import workloads
from surfacegrowthconsole_gb300.engine import DiffModel, build_workload, diff_frame_params, diff_init_theta

pytestmark = pytest.mark.gpu

# the FP32 roundings a loss keeps however many terms it has: of a term (2), of a thread's compensated sum
# (2), of the tree over a warp (5), each 2^-24; the gradients': the columns' few dozen terms and their tree
LOSS_REL, GRAD_REL = 9 / 2 ** 24, 32 / 2 ** 24
BIG = 4096.0  # its square is 2^24


def test_loss_of_atoms_without_pairs():
    p, r, _ = build_workload(24, 24, [1], 300.0, 5)
    frames = 64
    model = DiffModel([diff_frame_params(p)] * frames, np.concatenate([r] * frames))
    ref = np.ones(3 * model.n, np.float32)
    ref[:len(ref) // 24] = BIG  # 1.4e-6 of the loss is in the others
    theta = diff_init_theta(p)
    loss = model.force_matching(theta, ref.reshape(-1, 3), grad=False)
    want = (ref.astype(np.float64) ** 2).mean()
    assert abs(loss - want) <= LOSS_REL * want
    model.close()


@pytest.fixture(scope="module")
def bulk():
    """A lattice of 55,296 atoms (and one with its atoms displaced), alone and 24 times."""
    p, r, _ = workloads.bulk_metal(24, 300.0, seed=1, material=2)
    q = diff_frame_params(p)
    moved = r.copy()
    moved[:, :3] += np.random.RandomState(3).normal(0, 0.05, size=(q.nMol, 3)).astype(np.float32)
    one, many = DiffModel([q], r), DiffModel([q] * 24, np.concatenate([r] * 24))
    yield q, r, moved, one, many
    one.close()
    many.close()


def test_loss_of_metal_atoms(bulk):
    q, r, _, _, model = bulk  # a perfect lattice: no forces beside the reference's
    model.set_positions(np.concatenate([r] * 24))
    ref = np.ones((model.n, 3), np.float32)
    ref[:q.nMol] = BIG
    loss = model.force_matching(diff_init_theta(q), ref, grad=False)
    want = (ref.astype(np.float64) ** 2).mean()
    assert abs(loss - want) <= LOSS_REL * want


def test_many_frames_are_as_many_times_one(bulk):
    q, _, moved, one, many = bulk
    one.set_positions(moved)
    many.set_positions(np.concatenate([moved] * 24))
    theta = diff_init_theta(q)
    e1, g1 = one.energy(theta)
    e, g = many.energy(theta)
    assert np.abs(e - e1).max() <= 1e-7 * np.abs(e1).max()
    assert np.abs(g - 24 * g1).max() <= GRAD_REL * np.abs(24 * g1).max()
    l1, h1 = one.force_matching(theta, np.zeros((one.n, 3), np.float32))
    l, h = many.force_matching(theta, np.zeros((many.n, 3), np.float32))
    assert abs(l - l1) <= LOSS_REL * l1
    assert np.abs(h - h1).max() <= GRAD_REL * np.abs(h1).max()
