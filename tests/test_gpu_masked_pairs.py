"""CTA pairs in the masked layout: groups on either side of 128 rows, the second CTA of a pair with no rows of its group."""

import pytest
import torch

import deep_gemm
from helpers import assert_close, seed_all, uniform_fp8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [136, 512])
@pytest.mark.parametrize('config', [None, {'cta_group': 2, 'block_n': 256}, {'cta_group': 2, 'block_n': 224},
                                    {'cta_group': 2, 'block_n': 96}, {'cta_group': 1, 'block_n': 256}])
@pytest.mark.parametrize('out', [torch.bfloat16, torch.float32])
def test_masked_pairs(n, config, out):
    seed_all(n)
    sizes, slots, k = [0, 1, 127, 128, 129, 255, 256, 200, 3, 300], 300, 640
    g = len(sizes)
    parts = [(uniform_fp8((slots, k), (1, 32)), uniform_fp8((n, k), (1, 32))) for _ in range(g)]
    stack = lambda i, j: torch.stack([p[i][j].view(torch.uint8) if j == 0 else p[i][j] for p in parts]).cuda()  # noqa: E731
    a, b = (stack(0, 0).view(torch.float8_e4m3fn), stack(0, 1)), (stack(1, 0).view(torch.float8_e4m3fn), stack(1, 1))
    d = torch.full((g, slots, n), 7.0, dtype=out, device='cuda')
    rows = torch.tensor(sizes, dtype=torch.int32, device='cuda')
    deep_gemm.m_grouped_fp8_gemm_nt_masked(a, b, d, rows, 140, recipe=(1, 1, 32), config=config)
    assert deep_gemm.device_status() == 0
    for i, r in enumerate(sizes):
        if r:
            assert_close(d[i, :r], (parts[i][0][2][:r].float() @ parts[i][1][2].float().t()).to(out), f'group {i} of {r} rows, {config}')
        assert (d[i, (r + 127) // 128 * 128:] == 7.0).all()          # rows beyond the last 128-row block are not written
