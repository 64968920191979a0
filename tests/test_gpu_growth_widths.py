"""Gaussian growth at widths and potentials where float32 has no finite
coefficient 1 / (2 s^2) or square: leniax's exp(-((u - m) / s)^2 / 2) still
gives -1 (s = 0 or tiny, u far off) or +1 (s huge), on every route to the N-D
step."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import bump_kernel_params, random_multichannel_params

pytestmark = pytest.mark.gpu

# one step of dt = 0.1: the growths are exactly -1 or +1, so the weighted field
# carries the rounding of its at most 8 weights' sum and the state that of one fma
FIELD, STATE = 16 * 6e-8, 4 * 6e-8

# (world, worlds, channels, kernels a channel)
WORLDS = [((48, 48), 4, 1, 1), ((100, 100), 1, 1, 1), ((100, 100), 4, 1, 1), ((45, 45), 2, 2, 4), ((33, 62), 3, 1, 1),
          ((32, 32, 32), 2, 1, 1), ((64, 64, 64), 1, 1, 1), ((24, 20, 36), 2, 1, 1), ((16, 18, 20), 1, 2, 2),
          ((600, 600), 1, 1, 1)]


def _model(cuda, world, C, per, width):
    R = 5.0
    kp = bump_kernel_params(s=width) if C == 1 else random_multichannel_params(C, per, seed=3, R_range=(0.6 * R, R),
                                                                                  world_R=R)
    for p in kp:
        p['gf_params'] = [p['gf_params'][0], width]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, cuda)
    Ko, mpo = O.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, np.float64)
    mpo['gf_params'] = np.asarray(mpo['gf_params'], np.float32).astype(np.float64)
    return K, mp, helpers.build_update_fn(K.shape, mp), Ko, mpo


def _step(Ko, mpo, cells):
    with np.errstate(all='ignore'):
        return O.update(cells.astype(np.float64), Ko, mpo['gf_params'], mpo['weights'], 0.1, O.Model(mpo, 'v1', True))


@pytest.mark.parametrize('world,n,C,per', WORLDS)
@pytest.mark.parametrize('width', [0.0, 1e-30, 1e-18, 1e-12, 1e16, 1e25, float('inf')])
def test_extreme_widths(cuda, world, n, C, per, width):
    K, mp, upd, Ko, mpo = _model(cuda, world, C, per, width)
    rng = np.random.Generator(np.random.PCG64(5))
    cells = (0.2 + 0.6 * rng.random((n, C) + world)).astype(np.float32)
    gf, w = mp.get_gf_params(cuda), mp.get_kernels_weight_per_channel(cuda)
    so, fo, _ = _step(Ko, mpo, cells)
    assert np.isfinite(fo).all()
    x = torch.from_numpy(cells).to(cuda)
    s, f, _ = upd(None, x, K, gf, w, 0.1)
    assert np.abs(f.cpu().numpy() - fo).max() <= FIELD
    assert np.abs(s.cpu().numpy() - so).max() <= STATE
    for engine in ('auto', 'nd'):
        _, final = runner.run_scan_mem_optimized(None, x[None], K[None], gf[None], w[None], torch.tensor([10.0]), 1, 5.0,
                                                 upd, statistics.ComputeStatsFn(list(world), 5.0, 10.0), engine=engine)
        assert np.abs(final[0].cpu().numpy() - so).max() <= STATE


@pytest.mark.parametrize('world,n,C,per', WORLDS)
@pytest.mark.parametrize('width', [0.015, 0.05, 0.07, 0.09, 0.13, -0.05, -0.09])
def test_potentials_with_infinite_squares(cuda, world, n, C, per, width):
    K, mp, upd, Ko, mpo = _model(cuda, world, C, per, width)
    rng = np.random.Generator(np.random.PCG64(6))
    cells = (1e21 * (0.2 + 0.6 * rng.random((n, C) + world))).astype(np.float32)
    s, f, _ = upd(None, torch.from_numpy(cells).to(cuda), K, mp.get_gf_params(cuda),
                  mp.get_kernels_weight_per_channel(cuda), 0.1)
    so, fo, _ = _step(Ko, mpo, cells)
    assert np.abs(fo + 1).max() <= 1e-12
    assert np.abs(f.cpu().numpy() - fo).max() <= FIELD
    assert np.abs(s.cpu().numpy() - so).max() <= STATE
