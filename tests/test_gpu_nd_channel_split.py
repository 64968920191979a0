"""The N-D epilogue with a block per output channel and with blocks that walk
all channels, at the batch sizes on both sides of its rule: packed rows with
the fields on chip and in memory, whole z-planes, y passes of their own; weight
tables whose kernels feed several channels, one or none (their potentials still
count), and channels that no kernel feeds.  Two Euler steps against the float64
oracle (core.py:13-49, 202-242; statistics.py:131-138)."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import random_multichannel_params

pytestmark = pytest.mark.gpu

# Two steps of dt |field error|: potentials a few float32 roundings below 1e-6,
# growth slopes below 41 (gaussian, s >= 0.03; poly_quad4 stays below it), the
# weights of a channel sum to at most 1, dt = 0.1: 2 * 0.1 * 41e-6 < 1e-5.
TOL = 1e-5

# world, C, kernels per channel, last batch with a block per channel
CASES = [
    ([36, 50], 2, 3, 303),
    ([35, 29], 3, 11, 303),      # odd sides, Bluestein lines, more than 32 kernels
    ([6, 4000], 2, 2, 101),      # fields in memory, one row pair a tile
    ([6, 10, 12], 2, 2, 50),     # whole z-planes
    ([4, 60, 70], 2, 2, 101),    # y transforms of their own
]


def _weights(C, K, seed, rng):
    """Mostly one channel a kernel; kernel 0 feeds every channel, the last one none, and with a second
    pattern channel 0 is fed by nothing."""
    w = np.zeros((C, K), np.float32)
    for k in range(K):
        w[int(rng.integers(0, C)), k] = 0.2 + 0.8 * rng.random()
    w[:, 0] = 0.2 + 0.8 * rng.random(C)
    w[:, K - 1] = 0.0
    if seed:
        w[0] = 0.0
    return (w / np.maximum(w.sum(1, keepdims=True), 1e-6)).astype(np.float32)


@pytest.mark.parametrize('world,C,per,limit', CASES)
@pytest.mark.parametrize('which', ['one', 'limit', 'past'])
@pytest.mark.parametrize('seed', [0, 1])
def test_two_steps_match_the_oracle(cuda, world, C, per, limit, which, seed):
    n = {'one': 1, 'limit': limit, 'past': limit + 1}[which]
    R = 2.0 if len(world) == 3 else 2.5
    rng = np.random.Generator(np.random.PCG64(sum(world) + 10 * C + seed))
    kp = random_multichannel_params(C, per, seed=seed + 1, R_range=(0.7 * R, R), world_R=R)
    for i, p in enumerate(kp):
        p['gf_slug'] = ('gaussian', 'poly_quad4')[i % 2]
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], world, C, R, True, cuda)
    mean = not seed  # the mean of a channel that no kernel feeds is 0 / 0
    w = _weights(C, len(kp), seed, rng)
    upd = helpers.build_update_fn(K.shape, mp, 'v1', mean)
    base = rng.random((min(n, 3), C) + tuple(world), dtype=np.float32)  # the oracle runs these; they repeat over the batch
    idx = np.arange(n) % len(base)
    stats_fn = statistics.ComputeStatsFn(world, R, 10.0)
    wt = torch.from_numpy(w).to(cuda)
    cells = torch.from_numpy(base[idx]).to(cuda)
    got, field, pot, sd = runner.run_scan(None, cells, K, mp.get_gf_params(cuda), wt, torch.tensor(10.0), 2, R, upd,
                                          stats_fn, engine='nd')
    _, fin = runner.run_scan_mem_optimized(None, cells[None], K[None], mp.get_gf_params(cuda)[None], wt[None],
                                           torch.tensor([10.0]), 2, R, upd, stats_fn, engine='nd')
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], world, C, R, True, np.float64)
    model = O.Model(mpo, 'v1', mean)
    ref, states, pots, fields = base.astype(np.float64), [], [], []
    for _ in range(2):
        states.append(ref)
        ref, f, u = O.update(ref, Ko, mpo['gf_params'], w.astype(np.float64), 0.1, model)
        pots.append(u)
        fields.append(f)
    assert np.abs(got[1].cpu().numpy() - states[1][idx]).max() <= TOL
    assert np.abs(fin[0].cpu().numpy() - ref[idx]).max() <= TOL
    assert np.abs(pot[1].cpu().numpy() - pots[1][idx]).max() <= TOL
    assert np.abs(field[1].cpu().numpy() - fields[1][idx]).max() <= 10 * TOL  # no dt factor
    mass = np.stack([s.reshape(len(base), C, -1).sum(2) for s in states])[:, idx] / R**2
    np.testing.assert_allclose(sd['channel_mass'].cpu().numpy(), mass, rtol=1e-5)
    # the potential's support is counted once a kernel, whatever it feeds
    count = (pot > 1e-7).flatten(2).sum(2).float() / R**2
    np.testing.assert_allclose(sd['potential_volume'].cpu().numpy(), count.cpu().numpy(), rtol=1e-6)
