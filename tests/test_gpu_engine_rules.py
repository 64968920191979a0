"""The engine that lgx_run takes by default for 3D batches: the same bits as
the one its rule names, on both sides of the rule, for the SMs of the device at
hand."""
import pytest
import torch

from leniax_gb300 import helpers, kernels, runner, statistics
from tests.cases import bump_kernel_params

pytestmark = pytest.mark.gpu


def _limits(side, sms):
    """(batch, engine): the last batch of N-D steps and the first of one world per CTA, in the first round of
    worlds and, for 64^3, at both ends of the second."""
    if side == 32:
        last = 40 * sms // 152
        return [(last, 'nd'), (last + 1, 'cta')]
    one, two = 84 * sms // 152, 84 * sms * 2 // 152
    return [(one, 'nd'), (one + 1, 'cta'), (sms, 'cta'), (sms + 1, 'nd'), (two, 'nd'), (two + 1, 'cta')]


@pytest.mark.parametrize('side', [32, 64])
def test_default_engine_of_3d_batches(cuda, side):
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    limits = _limits(side, sms)
    K, mp = kernels.get_kernels_and_mapping(bump_kernel_params(s=0.05), [side] * 3, 1, 5.0, True, cuda)
    upd = helpers.build_update_fn(K.shape, mp)
    g = torch.Generator(device='cpu').manual_seed(side)
    cells = torch.rand((1, max(n for n, _ in limits), 1) + (side, ) * 3, generator=g).to(cuda)
    stats_fn = statistics.ComputeStatsFn([side] * 3, 5.0, 10.0)

    def run(n, engine):
        return runner.run_scan_mem_optimized(None, cells[:, :n], K[None], mp.get_gf_params(cuda)[None],
                                             mp.get_kernels_weight_per_channel(cuda)[None], torch.tensor([10.0]), 2,
                                             5.0, upd, stats_fn, engine=engine)

    for n, engine in limits:
        auto, same, other = run(n, 'auto'), run(n, engine), run(n, 'cta' if engine == 'nd' else 'nd')
        assert torch.equal(auto[1], same[1]) and not torch.equal(auto[1], other[1])
        assert all(torch.equal(auto[0][k], same[0][k]) for k in auto[0])
