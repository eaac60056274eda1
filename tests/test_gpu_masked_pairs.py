"""CTA pairs in the masked layout: groups on either side of 128 rows, the second CTA of a pair with no rows of its group."""

import pytest
import torch

import deep_gemm
from helpers import assert_close, seed_all, uniform_fp4, uniform_fp8

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


@pytest.mark.parametrize('kind,k', [('mixed', 640), ('decoded', 608), ('fp4', 768), ('bf16', 320)])
@pytest.mark.parametrize('block_n', [128, 256])
def test_masked_pairs_of_other_operands(kind, k, block_n):
    """The second CTA of a pair without rows of its group fetches its half of B only. How many bytes that is depends on the operands:
    E2M1 B unpacked by TMA or (K no multiple of 128) by the decoder warps, packed pairs with two words of scales a stage, BF16 without scales."""
    seed_all(k + block_n)
    n, slots, sizes = 264, 300, [0, 1, 128, 129, 256, 3, 300, 127]
    out = torch.bfloat16
    parts = []
    for _ in sizes:
        if kind == 'bf16':
            a, b = torch.randn(slots, k).bfloat16(), torch.randn(n, k).bfloat16()
            parts.append(((a, torch.zeros(1, 1), a.float()), (b, torch.zeros(1, 1), b.float())))
        else:
            parts.append((uniform_fp4(slots, k, (1, 32), False) if kind == 'fp4' else uniform_fp8((slots, k), (1, 32)), uniform_fp4(n, k, (1, 32), False)))
    stack = lambda i, j: torch.stack([p[i][j].view(torch.uint8) if p[i][j].dtype == torch.float8_e4m3fn else p[i][j] for p in parts]).cuda()  # noqa: E731
    a, b = stack(0, 0), stack(1, 0)
    if a.dtype == torch.uint8:
        a = a.view(torch.float8_e4m3fn)
    d = torch.full((len(sizes), slots, n), 7.0, dtype=out, device='cuda')
    rows = torch.tensor(sizes, dtype=torch.int32, device='cuda')
    deep_gemm.m_grouped_fp8_fp4_gemm_nt_masked((a, stack(0, 1)), (b, stack(1, 1)), d, rows, 140, recipe=(1, 1, 32),
                                               config={'cta_group': 2, 'block_n': block_n})
    assert deep_gemm.device_status() == 0
    for i, r in enumerate(sizes):
        if r:
            assert_close(d[i, :r], (parts[i][0][2][:r].float() @ parts[i][1][2].float().t()).to(out), f'{kind} group {i} of {r} rows')
        assert (d[i, (r + 127) // 128 * 128:] == 7.0).all()


@pytest.mark.parametrize('config', [None, {'cta_group': 1, 'block_n': 256}, {'cta_group': 1, 'block_n': 96}, {'cta_group': 2, 'block_n': 256}])
@pytest.mark.parametrize('out,n,slots', [(torch.bfloat16, 264, 168), (torch.float32, 520, 168), (torch.bfloat16, 131, 168), (torch.bfloat16, 264, 64), (torch.bfloat16, 264, 40)])
def test_quarters_of_a_tile_without_rows(config, out, n, slots):
    """The last row of a group at every edge of 32 rows: what lies behind its 32 rows is neither written nor has to be fetched (TMA stores, and
    plain ones for an odd N; slots that are and are not a multiple of 32)."""
    if slots <= 128 and config and config['cta_group'] == 2:
        pytest.skip('no pairs for at most 128 slots')
    seed_all(n + slots)
    sizes, k = [min(r, slots) for r in (0, 1, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 160, 161)], 640
    parts = [(uniform_fp8((slots, k), (1, 32)), uniform_fp8((n, k), (1, 32))) for _ in sizes]
    stack = lambda i, j: torch.stack([p[i][j].view(torch.uint8) if j == 0 else p[i][j] for p in parts]).cuda()  # noqa: E731
    a, b = (stack(0, 0).view(torch.float8_e4m3fn), stack(0, 1)), (stack(1, 0).view(torch.float8_e4m3fn), stack(1, 1))
    d = torch.full((len(sizes), slots, n), 7.0, dtype=out, device='cuda')
    rows = torch.tensor(sizes, dtype=torch.int32, device='cuda')
    for _ in range(2):
        deep_gemm.m_grouped_fp8_gemm_nt_masked(a, b, d, rows, 80, recipe=(1, 1, 32), config=config)
    assert deep_gemm.device_status() == 0
    for i, r in enumerate(sizes):
        if r:
            assert_close(d[i, :r], (parts[i][0][2][:r].float() @ parts[i][1][2].float().t()).to(out), f'group {i} of {r} rows, {config}')
        assert (d[i, (r + 31) // 32 * 32:] == 7.0).all()
