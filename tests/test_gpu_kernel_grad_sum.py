"""The one-kernel adjoint's sum of kernel-gradient spectra over a solution's
initial states, whose worlds a block's eight warps take in turn: fewer worlds
than warps, as many, one more and more than two rounds, for two solutions at
every side, against float64 autograd of the same step (runner.py:363-448)."""
import numpy as np
import pytest
import torch

from leniax_gb300 import grad as lgrad
from leniax_gb300 import helpers, kernels
from oracle import lenia_grad_oracle as GO
from tests.cases import bump_kernel_params, patch_init

pytestmark = pytest.mark.gpu

# One step's kernel gradient is linear in lam * growth'(u): growth' moves by at
# most |d growth' / growth'| ~ |u - m| / s^2 * du < 400 * 1e-7 where it is not
# small, the transforms and the sum over worlds add a few 1e-7.
TOL = 1e-4


@pytest.mark.parametrize('size', [32, 64, 128, 256])
@pytest.mark.parametrize('inits', [1, 7, 8, 9, 17])
def test_kernel_gradient_sums_over_initial_states(cuda, size, inits):
    R, T, m, s = 5, 10.0, 0.15, 0.05
    K, mp = kernels.get_kernels_and_mapping(bump_kernel_params(m=m, s=s), [size, size], 1, R, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp)
    k_real = lgrad.ring_kernel(R, 1.0, torch.tensor([1.0], device=cuda), 'gauss_bump', [1.0], [size, size])
    cells = np.stack([patch_init(inits, size, size // 2, seed=size + i, scale_range=(0.4, 1.0)) for i in (0, 50)])
    target = np.stack([0.5 * patch_init(inits, size, size // 2, seed=size + i) for i in (100, 150)])
    kr = torch.stack([k_real, k_real.flip(0) * 0.9]).detach().requires_grad_(True)
    gf = torch.tensor([[[m, s]], [[m, s]]], device=cuda)
    fin = lgrad.rollout(torch.from_numpy(cells).to(cuda), kr, gf, torch.ones(2, 1, 1, device=cuda),
                        torch.tensor([T, T]), upd, 1, 1, 'ste')
    ((fin - torch.from_numpy(target).to(cuda))**2).mean().backward()
    got = kr.grad.cpu().double().numpy()
    for i in range(2):
        kref = kr.detach()[i].cpu().double().numpy()
        _, (_, rk, *_) = GO.loss_and_grads(cells[i].astype(np.float64), kref, m, s, 1.0, 1 / T, 1, target[i],
                                           clip='ste')
        rk = 0.5 * np.reshape(rk, got[i].shape)  # the engine's mean runs over both solutions
        assert np.linalg.norm(got[i] - rk) <= TOL * np.linalg.norm(rk)
