"""Fewer than 128 rows: a pipeline stage holds only the rows there are (rounded up to 8), while the MMA reads 128 rows of shared
memory. What lies behind them must never show: the kernels run behind a product of NaN operands, with guard rows after D."""

import pytest
import torch

import deep_gemm
import oracle
from helpers import assert_close, seed_all, uniform_fp8

pytestmark = pytest.mark.gpu


def _poison():
    """Leaves NaN bit patterns in the shared memory of every SM."""
    nan = torch.full((4096, 1024), 0x7F, dtype=torch.uint8, device='cuda').view(torch.float8_e4m3fn)
    sf = torch.full((4096, 32), 1.0, device='cuda')
    d = torch.empty((4096, 4096), dtype=torch.bfloat16, device='cuda')
    deep_gemm.fp8_gemm_nt((nan, sf), (nan, sf), d, recipe=(1, 1, 32))


@pytest.mark.parametrize('m', [1, 7, 8, 9, 33, 64, 65, 127])
@pytest.mark.parametrize('n,k,config', [
    (320, 1024, None), (200, 4096, {'block_n': 32, 'split_k': 8, 'cluster_split': 1}), (640, 3072, {'block_n': 160, 'split_k': 3, 'cluster_split': 1}),
    (256, 2048, {'block_n': 128, 'split_k': 4, 'cluster_split': 1}), (448, 512, {'block_n': 224, 'num_stages': 2}),
    (72, 256, {'block_n': 32, 'num_stages': 1}), (264, 384, {'block_n': 64, 'num_stages': 1}), (200, 640, {'block_n': 96, 'num_stages': 1}),
    (96, 512, {'block_n': 64, 'num_stages': 2}), (160, 2048, {'block_n': 32, 'split_k': 4, 'cluster_split': 1, 'num_stages': 6}),
    (256, 1024, {'block_n': 96, 'split_k': 4, 'cluster_split': 1, 'num_stages': 3, 'store_bufs': 1}), (130, 8192, {'block_n': 64, 'split_k': 4})])
def test_dense(m, n, k, config):
    seed_all(m + n)
    a, sfa, a_ref = uniform_fp8((m, k), (1, 32))
    b, sfb, b_ref = uniform_fp8((n, k), (1, 32))
    a, sfa, b, sfb = a.cuda(), sfa.cuda(), b.cuda(), sfb.cuda()
    bias = torch.randn(1, n)
    for out, kw in ((torch.bfloat16, {}), (torch.float32, {}), (torch.float32, {'bias': bias})):
        d = torch.full((m + 8, n), 7.0, dtype=out, device='cuda')
        _poison()
        deep_gemm.fp8_gemm_nt((a, sfa), (b, sfb), d[:m], c=bias.cuda() if kw else None, recipe=(1, 1, 32), config=config)
        assert deep_gemm.device_status() == 0
        assert_close(d[:m], oracle.gemm_ref(a_ref, b_ref, out, **kw), f'{m}x{n}x{k} {out} {config}')
        assert (d[m:] == 7.0).all()
    d = torch.full((m, n), 1.0, dtype=torch.float32, device='cuda')
    if config is None or config.get('split_k', 1) == 1 or 'cluster_split' in config:
        deep_gemm.fp8_gemm_nt((a, sfa), (b, sfb), d, c=d, recipe=(1, 1, 32), config=config)
        assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.float32, c=torch.ones(m, n)), f'{m}x{n}x{k} accumulate {config}')


@pytest.mark.parametrize('m', [3, 40, 120])
def test_bf16_batched_and_masked(m):
    seed_all(m)
    g, n, k = 5, 288, 640
    a, b = torch.randn(m, k).bfloat16(), torch.randn(n, k).bfloat16()
    d = torch.full((m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    _poison()
    deep_gemm.bf16_gemm_nt(a.cuda(), b.cuda(), d)
    assert_close(d, (a.float() @ b.float().t()).bfloat16(), f'bf16 {m}')

    parts = [(uniform_fp8((m, k), (1, 32)), uniform_fp8((n, k), (1, 32))) for _ in range(g)]
    stack = lambda i, j: torch.stack([p[i][j].view(torch.uint8) if j == 0 else p[i][j] for p in parts]).cuda()  # noqa: E731
    a_arg = (stack(0, 0).view(torch.float8_e4m3fn), stack(0, 1))
    b_arg = (stack(1, 0).view(torch.float8_e4m3fn), stack(1, 1))
    ref = torch.stack([p[0][2].float() @ p[1][2].float().t() for p in parts]).bfloat16()
    d = torch.full((g, m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    _poison()
    deep_gemm.fp8_bmm(a_arg, b_arg, d)
    assert_close(d, ref, f'batched {m}')

    rows = torch.tensor([m, 0, 1, m - 1, 2], dtype=torch.int32, device='cuda')
    d = torch.full((g, m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    _poison()
    deep_gemm.m_grouped_fp8_gemm_nt_masked(a_arg, b_arg, d, rows, max(1, m // 2), recipe=(1, 1, 32))
    for i, r in enumerate(rows.tolist()):
        if r:
            assert_close(d[i, :r], ref[i, :r], f'masked {m} group {i}')
    assert deep_gemm.device_status() == 0
