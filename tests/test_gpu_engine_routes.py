"""Calls that take the N-D step by the size of their batch: small batches of
32^3 and 64^3 worlds, and update steps on even squares that are no power of
two.  Both sides of each rule against the general form of the same call, the
workspaces either engine asks for, and the inputs that are refused."""
import ctypes

import numpy as np
import pytest
import torch

from leniax_gb300 import _lib, helpers, kernels, runner, statistics
from oracle import lenia_oracle as O
from tests.cases import bump_kernel_params, random_multichannel_params

pytestmark = pytest.mark.gpu

# As elsewhere: steps of dt |field error|, potentials within 1e-6, growth slopes
# below 41 (s >= 0.03), dt = 0.1.  Two float32 engines: twice that.
STEP = 0.1 * 41e-6


def _model(cuda, world, C=1, per=1, R=5.0):
    kp = bump_kernel_params(s=0.05) if C == 1 else random_multichannel_params(C, per, seed=3, R_range=(0.6 * R, R),
                                                                                world_R=R)
    for p in kp:
        p['gf_params'] = [p['gf_params'][0], max(p['gf_params'][1], 0.03)]
    K, mp = kernels.get_kernels_and_mapping([dict(p) for p in kp], list(world), C, R, True, cuda)
    return kp, K, mp, helpers.build_update_fn(K.shape, mp)


@pytest.mark.parametrize('side,n', [(32, 1), (32, 40), (32, 41), (64, 1), (64, 84), (64, 85), (64, 153)])
def test_3d_batches_match_both_engines(cuda, side, n):
    _, K, mp, upd = _model(cuda, [side] * 3)
    g = torch.Generator(device='cpu').manual_seed(side + n)
    cells = torch.rand((1, n, 1) + (side, ) * 3, generator=g).to(cuda)
    stats_fn = statistics.ComputeStatsFn([side] * 3, 5.0, 10.0)
    out = {}
    for engine in ('auto', 'cta', 'nd'):
        out[engine] = runner.run_scan_mem_optimized(None, cells, K[None], mp.get_gf_params(cuda)[None],
                                                    mp.get_kernels_weight_per_channel(cuda)[None],
                                                    torch.tensor([10.0]), 2, 5.0, upd, stats_fn, engine=engine,
                                                    with_box=True, with_centroid=True)
    for other in ('cta', 'nd'):
        assert (out['auto'][1] - out[other][1]).abs().max() <= 4 * STEP
        assert torch.equal(out['auto'][0]['N'], out[other][0]['N'])
        torch.testing.assert_close(out['auto'][0]['mass'], out[other][0]['mass'], rtol=1e-5, atol=0)


@pytest.mark.parametrize('side', [32, 64])
def test_3d_states_off_the_16_byte_grid_match_those_on_it(cuda, side):
    # one world per CTA: state planes by bulk copies where their addresses
    # allow, by the lanes' own loads elsewhere; the arithmetic is the same
    _, K, mp, upd = _model(cuda, [side] * 3)
    g = torch.Generator(device='cpu').manual_seed(side)
    flat = torch.rand(2 * side**3 + 1, generator=g).to(cuda)
    on = flat[1:].clone().view(1, 2, 1, side, side, side)
    off = flat[1:].view(1, 2, 1, side, side, side)
    assert on.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 4
    stats_fn = statistics.ComputeStatsFn([side] * 3, 5.0, 10.0)
    a, b = (runner.run_scan_mem_optimized(None, c, K[None], mp.get_gf_params(cuda)[None],
                                          mp.get_kernels_weight_per_channel(cuda)[None], torch.tensor([10.0]), 3, 5.0,
                                          upd, stats_fn, engine='cta') for c in (on, off))
    assert torch.equal(a[1], b[1])
    assert all(torch.equal(a[0][k], b[0][k]) for k in a[0])


@pytest.mark.parametrize('side,n', [(32, 1), (32, 41), (64, 2)])
@pytest.mark.parametrize('per_world', [False, True])
def test_3d_update_matches_the_oracle(cuda, side, n, per_world):
    kp, K, mp, upd = _model(cuda, [side] * 3)
    rng = np.random.Generator(np.random.PCG64(side + n))
    cells = rng.random((n, 1) + (side, ) * 3, dtype=np.float32)
    dt = (0.05 + 0.05 * rng.random(n)).astype(np.float32) if per_world else np.full(n, 0.1, np.float32)
    s, f, p = upd(None, torch.from_numpy(cells).to(cuda), K, mp.get_gf_params(cuda),
                  mp.get_kernels_weight_per_channel(cuda), torch.from_numpy(dt).to(cuda) if per_world else 0.1)
    Ko, mpo = O.get_kernels_and_mapping([dict(q) for q in kp], [side] * 3, 1, 5.0, True, np.float64)
    for i in range(min(n, 3)):
        so, fo, po = O.update(cells[i:i + 1].astype(np.float64), Ko, mpo['gf_params'], mpo['weights'], float(dt[i]),
                              O.Model(mpo, 'v1', True))
        assert np.abs(s[i:i + 1].cpu().numpy() - so).max() <= 2 * STEP
        assert np.abs(p[i:i + 1].cpu().numpy() - po).max() <= 2e-6


@pytest.mark.parametrize('side', [24, 48, 100, 126, 360])
@pytest.mark.parametrize('n,C,per', [(1, 1, 1), (2, 1, 1), (3, 1, 1), (1, 3, 2), (4, 2, 3)])
@pytest.mark.parametrize('per_world', [False, True])
def test_update_on_even_squares_matches_the_oracle(cuda, side, n, C, per, per_world):
    kp, K, mp, upd = _model(cuda, [side] * 2, C, per)
    rng = np.random.Generator(np.random.PCG64(side + n + C))
    cells = rng.random((n, C, side, side), dtype=np.float32)
    dt = (0.05 + 0.05 * rng.random(n)).astype(np.float32) if per_world else np.full(n, 0.1, np.float32)
    s, f, p = upd(None, torch.from_numpy(cells).to(cuda), K, mp.get_gf_params(cuda),
                  mp.get_kernels_weight_per_channel(cuda), torch.from_numpy(dt).to(cuda) if per_world else 0.1)
    Ko, mpo = O.get_kernels_and_mapping([dict(q) for q in kp], [side] * 2, C, 5.0, True, np.float64)
    for i in range(n):
        so, fo, po = O.update(cells[i:i + 1].astype(np.float64), Ko, mpo['gf_params'], mpo['weights'], float(dt[i]),
                              O.Model(mpo, 'v1', True))
        assert np.abs(s[i:i + 1].cpu().numpy() - so).max() <= 2 * STEP
        assert np.abs(p[i:i + 1].cpu().numpy() - po).max() <= 2e-6


def _raw_update(upd, n, state, kh, gf, w, dt, ws):
    m = upd.model
    lib = _lib.load()
    out, field = torch.empty_like(state), torch.empty_like(state)
    pot = torch.empty((n, m.K) + m.world, device=state.device)
    rc = lib.lgx_update(m.plan.handle, n, state.data_ptr(), kh.data_ptr(), gf.data_ptr(), w.data_ptr(), dt.data_ptr(),
                        0, out.data_ptr(), field.data_ptr(), pot.data_ptr(), ws.data_ptr(), ws.numel(),
                        torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc, out


def test_update_workspaces_and_refusals(cuda):
    side, n = 100, 4
    _, K, mp, upd = _model(cuda, [side] * 2)
    m, lib = upd.model, _lib.load()
    kh = upd.spectra(K, (side, side))
    gf, w = mp.get_gf_params(cuda).contiguous(), mp.get_kernels_weight_per_channel(cuda).contiguous()
    dt = torch.tensor([0.1], device=cuda)
    state = torch.rand((n, 1, side, side), device=cuda)
    need = lib.lgx_update_workspace_bytes(m.plan.handle, n)
    rc, ref = _raw_update(upd, n, state, kh, gf, w, dt, torch.empty(need, dtype=torch.uint8, device=cuda))
    assert rc == 0
    # a workspace that holds the streamed step alone is taken as before, a smaller one refused
    sizes = [b for b in range(256, need, 4096)]
    taken = []
    for b in sizes[::max(1, len(sizes) // 12)] + [need - 1]:
        rc, out = _raw_update(upd, n, state, kh, gf, w, dt, torch.empty(b, dtype=torch.uint8, device=cuda))
        if rc == 0:
            taken.append(b)
            assert (out - ref).abs().max() <= 2 * STEP
        else:
            assert rc == _lib.LGX_ERR_WORKSPACE
            assert not taken  # every size from the smallest that is taken
    # states off the 16-byte grid are refused by every even square's step
    flat = torch.rand(n * side * side + 1, device=cuda)
    rc, _ = _raw_update(upd, n, flat[1:].view(n, 1, side, side), kh, gf, w, dt,
                        torch.empty(need, dtype=torch.uint8, device=cuda))
    assert rc == _lib.LGX_ERR_CUDA
