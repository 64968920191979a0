"""Fields, potentials and states of a world are the same bits whatever the
batch it runs in, on both sides of the streamed engine's rule for few worlds
and for every batch of the N-D engine."""
import numpy as np
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from tests.cases import random_multichannel_params

pytestmark = pytest.mark.gpu


def _run(cuda, world, C, per, slugs, mean, cells, engine):
    R = 5.0
    kp = random_multichannel_params(C, per, seed=7, R_range=(3.0, R), world_R=R)
    for i, p in enumerate(kp):
        p['gf_slug'] = slugs[i % len(slugs)]
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping(kp, list(world), C, R, True, cuda)
    nk = len(kp)
    w = np.random.Generator(np.random.PCG64(nk)).random((C, nk)).astype(np.float32)
    w[:, 1::3] *= np.arange(C)[:, None] == 0  # some kernels feed channel 0 alone
    if nk > 2:
        w[:, -1] = 0.0  # and one feeds none
    upd = helpers.build_update_fn(K.shape, mp, 'v1', mean)
    *traj, _ = runner.run_scan(None, cells, K, mp.get_gf_params(cuda), torch.from_numpy(w).to(cuda),
                               torch.tensor(10.0), 3, R, upd, statistics.ComputeStatsFn(list(world), R, 10.0),
                               engine=engine)
    return traj  # states, fields, potentials [steps, n, ...]


# side, channels, kernels a channel, growths, last world count of the split row inverse
SPLIT = [(32, 4, 10, ('gaussian', 'poly_quad4'), 128), (64, 3, 5, ('gaussian', ), 128),
         (128, 3, 5, ('gaussian', ), 32), (128, 1, 20, ('poly_quad4', ), 32), (256, 1, 3, ('gaussian', ), 8),
         (256, 2, 6, ('triangle', 'step'), 8), (512, 2, 2, ('gaussian', ), 2), (128, 1, 1, ('gaussian', ), 32)]


@pytest.mark.parametrize('side,C,per,slugs,limit', SPLIT)
@pytest.mark.parametrize('mean', [True, False])
def test_streamed_worlds(cuda, side, C, per, slugs, limit, mean):
    rng = np.random.Generator(np.random.PCG64(side + C))
    cells = torch.from_numpy(rng.random((limit + 1, C, side, side), dtype=np.float32)).to(cuda)
    past = _run(cuda, (side, side), C, per, slugs, mean, cells, 'streamed')
    for n in (1, limit):
        few = _run(cuda, (side, side), C, per, slugs, mean, cells[:n], 'streamed')
        assert all(torch.equal(a, b[:, :n]) for a, b in zip(few, past))


@pytest.mark.parametrize('world,C,per,most', [((45, 45), 1, 1, 400), ((100, 100), 3, 3, 65), ((250, 250), 1, 1, 20),
                                              ((66, 40), 2, 2, 100), ((1024, 1024), 1, 1, 3), ((24, 24, 24), 1, 1, 40),
                                              ((48, 48, 48), 2, 2, 9), ((40, 80, 72), 1, 1, 5), ((128, 512), 1, 1, 32),
                                              ((224, 224), 1, 1, 64), ((480, 480), 1, 1, 13),
                                              ((576, 576), 1, 1, 9), ((16, 4096), 1, 1, 30)])
@pytest.mark.parametrize('mean', [True, False])
def test_nd_worlds(cuda, world, C, per, most, mean):
    rng = np.random.Generator(np.random.PCG64(sum(world)))
    cells = torch.from_numpy(rng.random((most, C) + world, dtype=np.float32)).to(cuda)
    whole = _run(cuda, world, C, per, ('gaussian', ), mean, cells, 'nd')
    for n in (1, 2, most // 2):
        few = _run(cuda, world, C, per, ('gaussian', ), mean, cells[:n], 'nd')
        assert all(torch.equal(a, b[:, :n]) for a, b in zip(few, whole))


@pytest.mark.parametrize('side,C,per', [(24, 1, 1), (100, 1, 1), (126, 2, 2), (360, 1, 3), (500, 1, 1)])
def test_update_steps_on_even_squares(cuda, side, C, per):
    kp = random_multichannel_params(C, per, seed=7, R_range=(3.0, 5.0), world_R=5.0)
    K, mp = kernels.get_kernels_and_mapping(kp, [side, side], C, 5.0, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp)
    rng = np.random.Generator(np.random.PCG64(side))
    cells = torch.from_numpy(rng.random((9, C, side, side), dtype=np.float32)).to(cuda)
    args = (K, mp.get_gf_params(cuda), mp.get_kernels_weight_per_channel(cuda), 0.1)
    whole = upd(None, cells, *args)
    for n in (1, 2, 3):
        assert all(torch.equal(a, b[:n]) for a, b in zip(upd(None, cells[:n], *args), whole))
