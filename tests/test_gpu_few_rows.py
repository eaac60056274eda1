"""The kernel for a handful of rows of A against the oracle, at the edges of its tiles (8 rows of A, 16 rows of B, pieces of 1024 K
shared out among 8 warps, one ring of pieces that is used again where K has more of them than shared memory holds) and of its rule, and
against the tensor-core kernel, which a forced tiling selects."""
# (The head describes the kernel's first form. It now takes up to 16 rows of A, pieces of 1024, 2048 or 4096 of K and 8 or 16 warps; which sizes use
# which ring again, and how often, is asked of the library and tested in test_gpu_few_rows_rings.py.)

import ctypes

import pytest
import torch

import deep_gemm
import oracle
from deep_gemm import _lib as L
from helpers import assert_close, normal_fp8, seed_all, uniform_fp4, uniform_fp8

pytestmark = pytest.mark.gpu


def _operands(m, n, k, kind, dist=uniform_fp8):
    seed_all(m * 31 + n + k)
    a, sfa, a_ref = dist((m, k), (1, 32))
    b, sfb, b_ref = uniform_fp4(n, k, (1, 32), False) if kind == 'fp4' else dist((n, k), (1, 32))
    return (a.cuda(), sfa.cuda()), (b.cuda(), sfb.cuda()), a_ref, b_ref


@pytest.mark.parametrize('kind', ['fp8', 'fp4'])
@pytest.mark.parametrize('m', [1, 2, 7, 8, 9])
@pytest.mark.parametrize('n,k', [(1, 32), (17, 96), (512, 1024), (2112, 7168), (200, 3168), (3000, 256), (40, 16384), (2500, 4448)])
def test_against_the_oracle(kind, m, n, k):
    a, b, a_ref, b_ref = _operands(m, n, k, kind)
    gemm = deep_gemm.fp8_fp4_gemm_nt if kind == 'fp4' else deep_gemm.fp8_gemm_nt
    kw = dict(recipe_a=(1, 32), recipe_b=(1, 32))
    for out in (torch.bfloat16, torch.float32):
        d = torch.full((m + 1, n), float('nan'), dtype=out, device='cuda')
        gemm(a, b, d[:m], **kw)
        assert deep_gemm.device_status() == 0
        assert_close(d[:m], oracle.gemm_ref(a_ref, b_ref, out), f'{kind} {m}x{n}x{k} {out}')
        assert torch.isnan(d[m]).all()
    bias = torch.randn(1, n).bfloat16()
    d = torch.full((m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    gemm(a, b, d, c=bias.cuda(), **kw)
    assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.bfloat16, bias=bias), f'{kind} {m}x{n}x{k} bias')
    gemm(a, b, d, alpha=-0.75, **kw)
    assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.bfloat16, alpha=-0.75), f'{kind} {m}x{n}x{k} alpha')


@pytest.mark.parametrize('kind,m,n,k', [
    ('fp8', 9, 40, 1024), ('fp8', 16, 33, 1056), ('fp8', 12, 512, 4096),             # two column sides: a whole small piece, a remainder of one block
    ('fp8', 16, 4096, 4096), ('fp8', 13, 512, 7200), ('fp8', 16, 2368, 8192),          # small pieces (no room for two large ones), a ring used several times
    ('fp8', 7, 4096, 7168), ('fp8', 8, 4096, 7168), ('fp8', 3, 512, 8192),             # large pieces, small pieces, sixteen warps
    ('fp8', 1, 520, 16384), ('fp8', 8, 2112, 12288), ('fp8', 6, 600, 10528),           # more than 8192 of K
    ('fp8', 2, 12288, 4096), ('fp8', 1, 24576, 544),                                   # several CTAs one after the other on an SM
    ('fp4', 16, 3072, 4096), ('fp4', 9, 1031, 8160), ('fp4', 5, 4096, 8192), ('fp4', 8, 8192, 2048)])
def test_edges_of_pieces_and_rows(kind, m, n, k):
    """Every instantiation at the edges of its pieces (1024, 2048 and 4096 of K), with one row of A less and with all of them, and nothing written
    behind the last row; packed scales as they lie."""
    desc = L.GemmDesc(m=m, n=n, k=k, a_dtype=L.E4M3, b_dtype=L.E2M1X2 if kind == 'fp4' else L.E4M3, d_dtype=L.F32)
    assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 1
    (a, sfa), (b, sfb), a_ref, b_ref = _operands(m, n, k, kind)
    packed = [deep_gemm.transform_sf_into_required_layout(s, mn, k, (1, 32)) for s, mn in ((sfa, m), (sfb, n))]
    d = torch.full((m + 1, n), float('nan'), dtype=torch.float32, device='cuda')
    for _ in range(2):
        deep_gemm.fp8_fp4_gemm_nt((a, packed[0]), (b, packed[1]), d[:m])
    assert deep_gemm.device_status() == 0
    exact = a_ref.double() @ b_ref.double().t()
    # (FP32 sums of k terms in blocks of 32: 1e-7 measured)
    assert ((d[:m].cpu().double() - exact).norm() / exact.norm()).item() < 1e-6
    assert torch.isnan(d[m]).all()


# (By now: one slot for eight pieces, two for seven, and two pieces of 4096 in two.)
@pytest.mark.parametrize('n,k', [(2500, 8192), (2500, 7168), (2048, 8192)])
def test_a_ring_used_several_times(n, k):
    """Eight rows and more CTAs than SMs: two slots for seven and eight pieces, each used four times with both parities of its
    barriers (fewer CTAs: eight slots for eight pieces)."""
    a, b, a_ref, b_ref = _operands(8, n, k, 'fp8')
    desc = L.GemmDesc(m=8, n=n, k=k, a_dtype=L.E4M3, b_dtype=L.E4M3, d_dtype=L.F32)
    assert L.lib().dg_gemm_few_rows(ctypes.byref(desc)) == 1
    d = torch.full((8, n), float('nan'), dtype=torch.float32, device='cuda')
    for _ in range(3):
        deep_gemm.fp8_gemm_nt(a, b, d, recipe_a=(1, 32), recipe_b=(1, 32))
    assert deep_gemm.device_status() == 0
    assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.float32), f'{n}x{k}')


@pytest.mark.parametrize('m', [1, 3, 8])
def test_scales_in_any_layout_and_error_against_64_bits(m):
    """Packed scales as they lie (M rows: no multiple of 16 bytes) and FP32 ones give the same bits; the FP32 result is no further
    from 64-bit sums than the tensor-core kernel's (1e-6 of the norm: FP32 sums of 7168 terms)."""
    n, k = 1040, 7168
    a, b, a_ref, b_ref = _operands(m, n, k, 'fp8', normal_fp8)
    packed = [(x, deep_gemm.transform_sf_into_required_layout(s, x.size(0), k, (1, 32))) for x, s in (a, b)]
    out = []
    for lhs, rhs, cfg in ((a, b, None), (*packed, None), (a, b, {'block_n': 128})):
        d = torch.full((m, n), float('nan'), dtype=torch.float32, device='cuda')
        deep_gemm.fp8_gemm_nt(lhs, rhs, d, config=cfg)
        out.append(d.cpu())
    assert torch.equal(out[0], out[1])
    exact = a_ref.double() @ b_ref.double().t()
    few, tiled = [((o.double() - exact).norm() / exact.norm()).item() for o in (out[0], out[2])]
    print(f'relative error: {few:.3g}, tensor-core kernel {tiled:.3g}')
    assert few < max(1e-6, 1.05 * tiled)


def test_scales_at_the_ends_of_their_range():
    """UE8M0 0 is 2^-127 and 255 is NaN, in one row or block only; the operands' zeros stay zeros under any finite scale."""
    m, n, k = 3, 32, 128
    a = torch.full((m, k), 0x38, dtype=torch.uint8, device='cuda').view(torch.float8_e4m3fn)        # 1.0
    b = torch.full((n, k), 0x38, dtype=torch.uint8, device='cuda').view(torch.float8_e4m3fn)
    ea, eb = torch.full((m, 4), 127), torch.full((n, 4), 127)
    ea[0], eb[5] = 0, 254
    ea[2, 3], eb[7, 1] = 255, 255
    pack = lambda e: (e[:, 0::2] | (e[:, 1::2] << 8)).to(torch.int16).cuda().t().contiguous().t()  # noqa: E731
    d = torch.zeros((m, n), dtype=torch.float32, device='cuda')
    deep_gemm.fp8_gemm_nt((a, pack(ea)), (b, pack(eb)), d)
    d = d.cpu()
    assert torch.isnan(d[2]).all() and torch.isnan(d[:, 7]).all()
    assert d[0, 5].item() == 128.0 and d[1, 0].item() == 128.0           # 2^-127 x 2^127; ones
    zero = torch.zeros_like(a)
    d = torch.ones((m, n), dtype=torch.float32, device='cuda')
    deep_gemm.fp8_gemm_nt((zero, pack(torch.full((m, 4), 254))), (b, pack(torch.full((n, 4), 254))), d)
    assert (d == 0).all()


@pytest.mark.parametrize('m', [1, 3, 8])
def test_fp32_scales_take_one_launch_more(m):
    """FP32 scales of both operands are brought to the packed layout by one launch in front of the GEMM, whatever the number of rows."""
    a, b, a_ref, b_ref = _operands(m, 1040, 2048, 'fp8')
    d = torch.empty((m, 1040), dtype=torch.bfloat16, device='cuda')
    before = L.lib().dg_kernel_launch_count()
    deep_gemm.fp8_gemm_nt(a, b, d)
    assert L.lib().dg_kernel_launch_count() - before == 2
    assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.bfloat16), f'{m} rows')


@pytest.mark.parametrize('kind', ['fp8', 'fp4'])
@pytest.mark.parametrize('k', [160, 1536])
def test_scales_far_apart(kind, k):
    """The scales of A and B at opposite ends of their range, in either order: every product is an ordinary number although neither
    factor is. Against 64-bit sums; FP32 sums of K terms are within K 2^-24 of the sum of the terms' magnitudes."""
    m, n = 8, 40
    blocks = -(-k // 32)
    gen = torch.Generator().manual_seed(k)
    low = torch.randint(0, 2, (1, blocks), generator=gen)                       # per K block: A low and B high, or the other way
    far = torch.randint(90, 128, (1, blocks), generator=gen)
    ea = (127 + torch.where(low == 1, -far, far) + torch.randint(-2, 3, (m, blocks), generator=gen)).clamp(0, 254)
    eb = (127 + torch.where(low == 1, far, -far) + torch.randint(-2, 3, (n, blocks), generator=gen)).clamp(0, 254)
    ea[0], eb[0] = 254, 0
    ea[1], eb[1] = 0, 254
    # 2^-127 to 2^127 everywhere would overflow in the pairs that do not belong together: those are not compared
    ones = torch.full((m, k), 0x38, dtype=torch.uint8, device='cuda').view(torch.float8_e4m3fn)
    b_ones = torch.full((n, k // 2), 0x22, dtype=torch.int8, device='cuda') if kind == 'fp4' else torch.full((n, k), 0x38, dtype=torch.uint8, device='cuda').view(torch.float8_e4m3fn)
    pad = lambda e: torch.nn.functional.pad(e, (0, e.size(1) % 2), value=0)  # noqa: E731
    pack = lambda e: (pad(e)[:, 0::2] | (pad(e)[:, 1::2] << 8)).to(torch.int16).cuda().t().contiguous().t()  # noqa: E731
    d = torch.zeros((m, n), dtype=torch.float32, device='cuda')
    deep_gemm.fp8_fp4_gemm_nt((ones, pack(ea)), (b_ones, pack(eb)), d)
    per_block = torch.full((blocks,), 32.0, dtype=torch.float64)
    terms = per_block * torch.exp2((ea[:, None] + eb[None] - 254).double())
    exact = terms.sum(-1)
    fits = exact < 2.0 ** 127
    assert fits[0, 0] and fits[1, 1] and fits.float().mean() > 0.5
    assert ((d.cpu().double() - exact).abs() <= blocks * 2.0 ** -24 * exact + 2.0 ** -126)[fits].all()
    assert d[0, 0].item() == d[1, 1].item() == k


def test_a_limit_on_the_sms_keeps_the_tiled_kernel():
    a, b, a_ref, b_ref = _operands(4, 256, 512, 'fp8')
    d = torch.empty((4, 256), dtype=torch.bfloat16, device='cuda')
    deep_gemm.set_num_sms(20)
    try:
        deep_gemm.fp8_gemm_nt(a, b, d)
    finally:
        deep_gemm.set_num_sms(0)
    assert_close(d, oracle.gemm_ref(a_ref, b_ref, torch.bfloat16), 'limited')
