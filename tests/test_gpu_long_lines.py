"""The N-D engine's long lines: axes whose transforms take the wide radices
(8..10, 12, 14, 15, 16 at the ends) along x, along y and along both, next to
lengths just short of them, for one kernel and for several; states against the
float64 oracle (core.py:13-49) and gradients against float64 autograd."""
import numpy as np
import pytest
import torch

from leniax_gb300 import grad as lgrad
from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_grad_oracle as GO
from oracle import lenia_oracle as O
from tests.cases import bump_kernel_params, random_multichannel_params

pytestmark = pytest.mark.gpu

# As for the shorter lines: two steps of dt |field error|, the potential a few
# float32 roundings below 1e-6, growth slopes below 41 (s >= 0.03), dt = 0.1.
TOL = 1e-5

WORLDS = [[12, 768], [768, 12], [9, 1024], [1024, 9], [1400, 10], [8, 2048], [1024, 1344], [12, 4096], [3072, 8],
          [800, 10], [10, 729]]


def _model(C, per, R):
    kp = bump_kernel_params(s=0.03) if C == 1 else random_multichannel_params(C, per, seed=3, R_range=(0.6 * R, R),
                                                                                world_R=R)
    for p in kp:
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    return kp


@pytest.mark.parametrize('world', WORLDS)
@pytest.mark.parametrize('C,per', [(1, 1), (2, 2)])
def test_two_steps_match_the_oracle(cuda, world, C, per):
    R = 3.0
    kp = _model(C, per, R)
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp, 'v1', True)
    rng = np.random.Generator(np.random.PCG64(sum(world) + C))
    cells = rng.random((2, C) + tuple(world), dtype=np.float32)
    stats_fn = statistics.ComputeStatsFn(world, R, 10.0)
    sd, fin = runner.run_scan_mem_optimized(None, torch.from_numpy(cells[None]).to(cuda), K[None],
                                            mp.get_gf_params(cuda)[None], mp.get_kernels_weight_per_channel(cuda)[None],
                                            torch.tensor([10.0]), 2, R, upd, stats_fn, engine='nd')
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, np.float64)
    model = O.Model(mpo, 'v1', True)
    ref = cells.astype(np.float64)
    for _ in range(2):
        ref, _, _ = O.update(ref, Ko, mpo['gf_params'], mpo['weights'], 0.1, model)
    assert np.abs(fin[0].cpu().numpy() - ref).max() <= TOL


@pytest.mark.parametrize('world', [[16, 768], [1024, 12], [1024, 1024]])
def test_gradients_match_float64_autograd(cuda, world):
    R, m, s, steps, T = 3.0, 0.15, 0.05, 2, 10.0
    K, mp = kernels.get_kernels_and_mapping(bump_kernel_params(m=m, s=s), world, 1, R, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp)
    k_real = lgrad.ring_kernel(R, 1.0, torch.tensor([1.0], device=cuda), 'gauss_bump', [1.0], world)
    rng = np.random.Generator(np.random.PCG64(sum(world)))
    cells = rng.random((1, 1) + tuple(world), dtype=np.float32) * 0.5
    target = rng.random((1, 1) + tuple(world), dtype=np.float32) * 0.5
    c0 = torch.from_numpy(cells[None]).to(cuda).requires_grad_(True)
    kr = k_real[None].detach().requires_grad_(True)
    fin = lgrad.rollout(c0, kr, torch.tensor([[[m, s]]], device=cuda), torch.ones(1, 1, 1, device=cuda),
                        torch.tensor([T]), upd, steps, 2, 'ste', engine='nd')
    ((fin - torch.from_numpy(target[None]).to(cuda))**2).mean().backward()
    _, (rc, rk, *_) = GO.loss_and_grads(cells.astype(np.float64), k_real.detach().cpu().double().numpy(), m, s, 1.0,
                                        1 / T, steps, target, clip='ste')
    # growth' moves by |u - m| / s^2 * du < 400 * 1e-6 where it is not small
    for got, want in ((c0.grad[0], rc), (kr.grad[0], rk)):
        got = got.cpu().double().numpy()
        assert np.linalg.norm(got - np.reshape(want, got.shape)) <= 4e-4 * np.linalg.norm(want)
