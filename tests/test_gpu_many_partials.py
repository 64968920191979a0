"""Statistics of worlds whose step is cut into more blocks than one warp of the
last block adds up at once: long stacks of small planes, many short rows; one
and several channels, odd counts of partials.  Two Euler steps against the
float64 oracle (statistics.py:36-126)."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import random_multichannel_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('world', [(1024, 8, 8), (257, 6, 10), (4096, 4, 4), (512, 16, 9), (500, 500), (515, 24),
                                   (1031, 20)])
@pytest.mark.parametrize('n,C,per', [(1, 1, 1), (3, 1, 1), (1, 3, 2)])
def test_statistics_match_the_oracle(cuda, world, n, C, per):
    R = 2.0 if min(world) < 9 else 4.0
    kp = random_multichannel_params(C, per, seed=3, R_range=(0.7 * R, R), world_R=R)
    for p in kp:
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, cuda)
    rng = np.random.Generator(np.random.PCG64(sum(world)))
    cells = rng.random((n, C) + world, dtype=np.float32)
    w = (0.2 + 0.8 * rng.random((C, len(kp)))).astype(np.float32)
    upd = helpers.build_update_fn(K.shape, mp, 'v1', True)
    x = torch.from_numpy(cells).to(cuda)
    *_, sd = runner.run_scan(None, x, K, mp.get_gf_params(cuda), torch.from_numpy(w).to(cuda), torch.tensor(10.0), 2, R,
                             upd, statistics.ComputeStatsFn(list(world), R, 10.0), engine='nd')
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, np.float64)
    ref, masses, growths, chan = cells.astype(np.float64), [], [], []
    for _ in range(2):
        masses.append(ref.reshape(n, -1).sum(1) / R**2)
        chan.append(ref.reshape(n, C, -1).sum(2) / R**2)
        ref, f, _ = O.update(ref, Ko, mpo['gf_params'], w.astype(np.float64), 0.1, O.Model(mpo, 'v1', True))
        growths.append(np.maximum(f, 0).reshape(n, -1).sum(1) / R**2)
    # sums of positive float32 terms, at most 64 added one after the other by a thread: below 1e-5
    np.testing.assert_allclose(sd['mass'].cpu().numpy(), np.stack(masses), rtol=1e-5)
    np.testing.assert_allclose(sd['channel_mass'].cpu().numpy(), np.stack(chan), rtol=1e-5)
    # the mean positive growth of a cell: a potential's roundings (below 1e-6) times the growth's slope
    # (at most 2 e^-0.5 / s < 41)
    cell = R**2 / cells[0].size
    mean = np.stack(growths) * cell
    assert (np.abs(sd['growth'].cpu().numpy() * cell - mean) <= 41e-6 * np.maximum(mean, 1) + 1e-5 * mean).all()


@pytest.mark.parametrize('world', [(4096, 4, 4), (1024, 8, 8), (2048, 6, 4), (1000, 1000)])
@pytest.mark.parametrize('value', [0.1, 0.37, 0.7, 0.9])
def test_masses_of_constant_worlds(cuda, world, value):
    # equal terms round the same way in a chain; by pairs a sum of n blocks is log2(n) roundings deep.  At most
    # 64 roundings from a cell to its world's mass: a thread's cells, a warp, a block's warps, the partials
    R = 2.0
    kp = random_multichannel_params(1, 1, seed=3, R_range=(0.7 * R, R), world_R=R)
    K, mp = kernels.get_kernels_and_mapping(kp, list(world), 1, R, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp, 'v1', True)
    cells = torch.full((1, 1) + world, value, device=cuda)
    *_, sd = runner.run_scan(None, cells, K, mp.get_gf_params(cuda), mp.get_kernels_weight_per_channel(cuda),
                             torch.tensor(10.0), 1, R, upd, statistics.ComputeStatsFn(list(world), R, 10.0), engine='nd')
    mass = float(np.float32(value)) * np.prod(world) / R**2
    assert abs(float(sd['mass'][0, 0]) / mass - 1) <= 64 * 2.0**-24
