"""The N-D engine's line transforms at the sizes where a plan, a tile or a
dispatch changes: one-, two-, three- and more-stage lines, lone last rows,
prime (Bluestein) lines along each axis, planes that just fit a tile and
planes that do not, fields on chip and in memory.  Two Euler steps (the second
starts from the spectra the first one emitted) against the float64 oracle
(core.py:13-49, runner.py:119-164)."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import bump_kernel_params, random_multichannel_params

pytestmark = pytest.mark.gpu

# Two steps of at most dt |field error| each: the potential carries a few
# float32 roundings (below 1e-6 of max |u| <= 1), growth multiplies it by at
# most 2 e^-0.5 / s < 41 at s = 0.03, dt = 0.1: 2 * 0.1 * 41e-6 < 1e-5.
TOL = 1e-5

# world, C, kernels per channel, R
CASES = [
    ([8, 10], 1, 1, 3.0),       # one-stage lines
    ([9, 16], 1, 1, 4.0),       # lone last row, 16 = 4 x 4
    ([81, 96], 1, 1, 9.0),      # 9 x 9, 8 x 12 as three stages
    ([33, 343], 1, 1, 9.0),     # Bluestein columns, 7 x 7 x 7 rows
    ([250, 37], 1, 1, 9.0),     # 5 x 5 x 10 columns, Bluestein rows
    ([29, 31], 2, 2, 7.0),      # both axes Bluestein, several kernels a channel
    ([24, 1000], 3, 2, 6.0),    # fields of three channels on chip
    ([12, 2048], 3, 1, 5.0),    # ... and in memory
    ([8, 64, 64], 1, 1, 3.0),   # the largest plane tile
    ([8, 60, 70], 1, 1, 3.0),   # past it: y transforms of their own
    ([6, 130, 20], 1, 1, 2.5),  # more row pairs than a plane tile holds
    ([11, 13, 14], 2, 1, 4.0),  # Bluestein z and y
    ([5, 9, 15], 3, 2, 2.0),    # odd everywhere, lone rows, several channels
]


@pytest.mark.parametrize('world,C,per,R', CASES)
@pytest.mark.parametrize('n', [1, 3])
def test_two_steps_match_the_oracle(cuda, world, C, per, R, n):
    kp = bump_kernel_params(s=0.03) if C == 1 else random_multichannel_params(C, per, seed=3, R_range=(0.6 * R, R),
                                                                                world_R=R)
    for p in kp:
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, cuda)
    mean = C == 1 or per > 1  # the mean of a channel that no kernel feeds is 0 / 0
    upd = helpers.build_update_fn(K.shape, mp, 'v1', mean)
    rng = np.random.Generator(np.random.PCG64(sum(world) + C))
    cells = rng.random((n, C) + tuple(world), dtype=np.float32)
    stats_fn = statistics.ComputeStatsFn(world, R, 10.0)
    got, _, pot, sd = runner.run_scan(None, torch.from_numpy(cells).to(cuda), K, mp.get_gf_params(cuda),
                                      mp.get_kernels_weight_per_channel(cuda), torch.tensor(10.0), 2, R, upd, stats_fn,
                                      engine='nd')
    _, fin = runner.run_scan_mem_optimized(None, torch.from_numpy(cells[None]).to(cuda), K[None],
                                           mp.get_gf_params(cuda)[None], mp.get_kernels_weight_per_channel(cuda)[None],
                                           torch.tensor([10.0]), 2, R, upd, stats_fn, engine='nd')
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, np.float64)
    model = O.Model(mpo, 'v1', mean)
    ref, states = cells.astype(np.float64), []
    for _ in range(2):
        states.append(ref)
        ref, _, u = O.update(ref, Ko, mpo['gf_params'], mpo['weights'], 0.1, model)
    assert np.abs(got[1].cpu().numpy() - states[1]).max() <= TOL
    assert np.abs(fin[0].cpu().numpy() - ref).max() <= TOL
    assert np.abs(pot[1].cpu().numpy() - u).max() <= TOL
    mass = np.stack([s.reshape(n, -1).sum(1) for s in states]) / R**2
    np.testing.assert_allclose(sd['mass'].cpu().numpy(), mass, rtol=1e-5)

