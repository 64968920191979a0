"""The streamed engine's row inverse split over channels and kernels, at the
batch sizes on both sides of its rule and for the weight tables it sorts by
bit masks: kernels that feed several channels, one or none (their potentials
still count), channels that no kernel feeds, more than 32 kernels, fewer
kernels than a block has warps, mixed growth functions.  Two Euler steps (the
second starts from the spectra the first one emitted) against the float64
oracle (core.py:13-49, 202-242; statistics.py:131-138)."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import random_multichannel_params

pytestmark = pytest.mark.gpu

# Two steps of at most dt |field error| each: the potential carries a few
# float32 roundings (below 1e-6 of max |u| <= 1), a growth multiplies it by at
# most 2 e^-0.5 / s < 41 (gaussian, s = 0.03; poly_quad4 stays below it), the
# weights of a channel sum to at most 1, dt = 0.1: 2 * 0.1 * 41e-6 < 1e-5.
TOL = 1e-5

# side, C, kernels per channel, growth slugs, last world count that is split
CASES = [
    (32, 4, 10, ('gaussian', 'poly_quad4'), 128),
    (64, 3, 5, ('gaussian', ), 128),
    (128, 2, 2, ('poly_quad4', ), 32),
    (256, 1, 3, ('gaussian', ), 8),
    (512, 2, 1, ('gaussian', 'poly_quad4'), 2),
]


def _weights(C, K, seed, rng):
    """Mostly one channel a kernel; kernel 0 feeds every channel, the last one none, and with a second
    pattern channel 0 is fed by nothing."""
    w = np.zeros((C, K), np.float32)
    for k in range(K):
        w[int(rng.integers(0, C)), k] = 0.2 + 0.8 * rng.random()
    w[:, 0] = 0.2 + 0.8 * rng.random(C)
    if K > 2:
        w[:, K - 1] = 0.0
    if seed and C > 1:
        w[0] = 0.0
    return (w / np.maximum(w.sum(1, keepdims=True), 1e-6)).astype(np.float32)


@pytest.mark.parametrize('side,C,per,slugs,limit', CASES)
@pytest.mark.parametrize('which', ['one', 'limit', 'past'])
@pytest.mark.parametrize('seed', [0, 1])
def test_two_steps_match_the_oracle(cuda, side, C, per, slugs, limit, which, seed):
    n = {'one': 1, 'limit': limit, 'past': limit + 1}[which]
    R, world = 5.0, [side, side]
    rng = np.random.Generator(np.random.PCG64(100 * side + 10 * C + seed))
    kp = random_multichannel_params(C, per, seed=seed + 1, R_range=(3.0, R), world_R=R)
    for i, p in enumerate(kp):
        p['gf_slug'] = slugs[i % len(slugs)]
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], world, C, R, True, cuda)
    nk = len(kp)
    mean = not seed  # the mean of a channel that no kernel feeds is 0 / 0
    w = _weights(C, nk, seed, rng)
    upd = helpers.build_update_fn(K.shape, mp, 'v1', mean)
    base = rng.random((min(n, 3), C) + tuple(world), dtype=np.float32)  # the oracle runs these; they repeat over the batch
    cells = base[np.arange(n) % len(base)]
    stats_fn = statistics.ComputeStatsFn(world, R, 10.0)
    wt = torch.from_numpy(w).to(cuda)
    got, field, pot, sd = runner.run_scan(None, torch.from_numpy(cells).to(cuda), K, mp.get_gf_params(cuda), wt,
                                          torch.tensor(10.0), 2, R, upd, stats_fn, engine='streamed')
    _, fin = runner.run_scan_mem_optimized(None, torch.from_numpy(cells[None]).to(cuda), K[None],
                                           mp.get_gf_params(cuda)[None], wt[None], torch.tensor([10.0]), 2, R, upd,
                                           stats_fn, engine='streamed')
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], world, C, R, True, np.float64)
    model = O.Model(mpo, 'v1', mean)
    ref, states, pots, fields = base.astype(np.float64), [], [], []
    for _ in range(2):
        states.append(ref)
        ref, f, u = O.update(ref, Ko, mpo['gf_params'], w.astype(np.float64), 0.1, model)
        pots.append(u)
        fields.append(f)
    idx = np.arange(n) % len(base)
    assert np.abs(got[1].cpu().numpy() - states[1][idx]).max() <= TOL
    assert np.abs(fin[0].cpu().numpy() - ref[idx]).max() <= TOL
    assert np.abs(pot[1].cpu().numpy() - pots[1][idx]).max() <= TOL
    assert np.abs(field[1].cpu().numpy() - fields[1][idx]).max() <= 10 * TOL  # no dt factor
    mass = np.stack([s.reshape(len(base), -1).sum(1) for s in states])[:, idx] / R**2
    np.testing.assert_allclose(sd['mass'].cpu().numpy(), mass, rtol=1e-5)
    # the potential's support is counted once a kernel, whatever it feeds
    count = (pot > 1e-7).flatten(2).sum(2).float() / R**2
    np.testing.assert_allclose(sd['potential_volume'].cpu().numpy(), count.cpu().numpy(), rtol=1e-6)
