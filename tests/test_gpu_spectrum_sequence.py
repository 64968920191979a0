"""Kernel spectra of worlds with prime sides built one behind the other on one
stream and in one workspace: each call's first pass is a dependent launch of
the kernel that writes its Bluestein tables, over the last call's."""
import ctypes

import pytest
import torch

from leniax_gb300 import _lib, grad

pytestmark = pytest.mark.gpu

WORLDS = [(31, 37), (127, 66), (11, 13, 17), (37, 31), (254, 26), (22, 26, 34)]


def test_alternating_prime_sides_in_one_workspace(cuda):
    lib = grad._bind(_lib.load())
    dims = [(ctypes.c_int * 3)(*w) for w in WORLDS]
    need = max(lib.lgx_kernel_spectrum_nd_workspace_bytes(len(w), d, 1) for w, d in zip(WORLDS, dims))
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)
    g = torch.Generator(device='cpu').manual_seed(3)
    real = [torch.rand(w, generator=g).to(cuda) for w in WORLDS]
    out = [[torch.full(w[:-1] + (w[-1] // 2 + 1, ), float('nan'), dtype=torch.complex64, device=cuda) for w in WORLDS]
           for _ in range(40)]
    st = torch.cuda.current_stream().cuda_stream
    for row in out:
        for w, d, x, y in zip(WORLDS, dims, real, row):
            _lib.check(lib.lgx_kernel_spectrum_nd(len(w), d, 1, x.data_ptr(), y.data_ptr(), ws.data_ptr(), need, st))
    for i, x in enumerate(real):
        ref = torch.fft.rfftn(x.double(), dim=tuple(range(x.dim())))
        # as the other spectra's: 1e-5 of the largest coefficient
        assert (out[0][i] - ref).abs().max() <= 1e-5 * ref.abs().max()
        assert all(torch.equal(torch.view_as_real(row[i]), torch.view_as_real(out[0][i])) for row in out)
