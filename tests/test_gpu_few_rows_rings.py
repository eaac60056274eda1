"""The kernel for a few rows where its ring of pieces is used again, and where one scale is far from 1: sizes chosen by the tile and the number of
slots that the library reports for them, results against sums in 64 bits."""

import ctypes

import pytest
import torch

import deep_gemm
from deep_gemm import _lib as L
from helpers import seed_all, uniform_fp4, uniform_fp8

pytestmark = pytest.mark.gpu


def _layout(kind, m, n, k):
    desc = L.GemmDesc(m=m, n=n, k=k, a_dtype=L.E4M3, b_dtype=L.E2M1X2 if kind == 'fp4' else L.E4M3, d_dtype=L.F32)
    out = L.FewRowsLayout()
    assert L.lib().dg_gemm_few_rows_layout(ctypes.byref(desc), ctypes.byref(out)) == 0, L.last_error()
    return out


def _check(d, a, b):
    """Sums of 32 products by the matrix instruction, then K / 32 of them one after the other and over the warps: each addition rounds by at most 2^-24 of
    the terms' magnitudes (2^-23 within the instruction)."""
    exact, size = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    assert ((d.cpu().double() - exact).abs() <= (64 + a.size(1) // 32) * 2.0 ** -24 * size).all()


# (kind, m, n, k), then warps, K of a piece and slots: as many pieces as the slots hold and more of them
RINGS = [
    ('fp8', 1, 2500, 8192, 8, 2048, 2), ('fp8', 2, 2400, 8160, 8, 2048, 2),            # four pieces in two slots
    ('fp8', 8, 2500, 6016, 8, 1024, 2), ('fp8', 8, 2400, 7168, 8, 1024, 2),            # six and seven in two: every slot refilled two or three times
    ('fp8', 8, 2500, 8192, 8, 1024, 1),                                                # eight in one
    ('fp8', 6, 600, 16384, 16, 2048, 2), ('fp8', 1, 600, 16352, 16, 2048, 5),          # eight in two and in five
    ('fp8', 16, 2368, 8192, 16, 1024, 3), ('fp8', 9, 600, 8160, 16, 1024, 7),          # two column sides: eight in three and in seven
    ('fp8', 14, 4000, 4096, 8, 1024, 2), ('fp8', 16, 4096, 4096, 8, 1024, 1),          # four in two and in one
    ('fp4', 16, 2368, 8192, 8, 2048, 3), ('fp4', 8, 3000, 7168, 8, 2048, 2), ('fp4', 16, 2400, 4096, 8, 2048, 1),
    ('fp8', 5, 520, 1536, 8, 2048, 1), ('fp8', 3, 520, 2048, 8, 2048, 1),              # a piece that is not full, one that is
]


@pytest.mark.parametrize('kind,m,n,k,warps,piece,slots', RINGS)
def test_slots_that_are_filled_again(kind, m, n, k, warps, piece, slots):
    t = _layout(kind, m, n, k)
    assert (t.warps, t.piece, t.slots) == (warps, piece, slots)
    seed_all(m + n + k)
    b, sfb, b_ref = uniform_fp4(n, k, (1, 32), False) if kind == 'fp4' else uniform_fp8((n, k), (1, 32))
    b, sfb = b.cuda(), deep_gemm.transform_sf_into_required_layout(sfb.cuda(), n, k, (1, 32))
    sides = [uniform_fp8((m, k), (1, 32)) for _ in range(3)]
    d = [torch.full((m + 1, n), float('nan'), dtype=torch.float32, device='cuda') for _ in sides]
    for (a, sfa, _), out in zip(sides, d):                                              # (one behind the other, other rows of A each time)
        deep_gemm.fp8_fp4_gemm_nt((a.cuda(), sfa.cuda()), (b, sfb), out[:m], recipe_a=(1, 32), recipe_b=(1, 32))
    assert deep_gemm.device_status() == 0
    for (_, _, a_ref), out in zip(sides, d):
        _check(out[:m], a_ref, b_ref)
        assert torch.isnan(out[m]).all()


def _operands(kind, m, n, k, seed):
    """E4M3 (E2M1) codes of magnitude 1 to 3 with random signs, so that no sum is empty; their values in 64 bits."""
    gen = torch.Generator().manual_seed(seed)
    draw = lambda *s: torch.randint(0, 4, s, generator=gen)  # noqa: E731
    table8 = torch.tensor([0x38, 0x3c, 0xb8, 0x40], dtype=torch.uint8)                  # 1, 1.5, -1, 2
    table4, values = torch.tensor([2, 3, 10, 4]), torch.tensor([1.0, 1.5, -1.0, 2.0], dtype=torch.float64)
    ca, cb = draw(m, k), draw(n, k)
    a = table8[ca].cuda().view(torch.float8_e4m3fn)
    if kind == 'fp4':
        codes = table4[cb]
        b = (codes[:, 0::2] | (codes[:, 1::2] << 4)).to(torch.uint8).view(torch.int8).cuda()
    else:
        b = table8[cb].cuda().view(torch.float8_e4m3fn)
    return a, b, values[ca], values[cb]


def _packed(e):
    e = torch.nn.functional.pad(e, (0, e.size(1) % 2), value=0)
    return (e[:, 0::2] | (e[:, 1::2] << 8)).to(torch.int16).cuda().t().contiguous().t()


FAR = [('fp8', 16, 520, 4096), ('fp8', 16, 2368, 8192), ('fp8', 9, 512, 7200), ('fp8', 1, 520, 16384), ('fp8', 6, 600, 16352), ('fp8', 8, 2500, 6016),
       ('fp8', 8, 512, 7168), ('fp4', 16, 600, 4096), ('fp4', 8, 3000, 7168), ('fp4', 12, 1031, 8160)]


@pytest.mark.parametrize('kind,m,n,k', FAR)
def test_scales_far_apart_over_several_pieces(kind, m, n, k):
    """Per block of K, the scales of A and B lie at opposite ends of their range, in either order: every product is an ordinary number although neither factor is."""
    a, b, av, bv = _operands(kind, m, n, k, m + k)
    blocks = k // 32
    gen = torch.Generator().manual_seed(n)
    far = torch.randint(70, 125, (1, blocks), generator=gen) * (1 - 2 * torch.randint(0, 2, (1, blocks), generator=gen))
    ea = 127 + far + torch.randint(-2, 3, (m, blocks), generator=gen)
    eb = 127 - far + torch.randint(-2, 3, (n, blocks), generator=gen)
    d = torch.zeros((m, n), dtype=torch.float32, device='cuda')
    deep_gemm.fp8_fp4_gemm_nt((a, _packed(ea)), (b, _packed(eb)), d)
    assert deep_gemm.device_status() == 0
    spread = lambda e, v: v * torch.exp2((e - 127).double()).repeat_interleave(32, 1)  # noqa: E731
    _check(d, spread(ea, av), spread(eb, bv))


@pytest.mark.parametrize('kind,m,n,k', FAR)
@pytest.mark.parametrize('byte', [0, 255])
@pytest.mark.parametrize('side', ['a', 'b'])
def test_one_scale_far_from_one(kind, m, n, k, side, byte):
    """One scale byte at an end of its range, all others 1, in the last row of A or of a CTA's sixteen rows of B, at the first and at the last block of K: 0 is 2^-127 (the
    row's other blocks are zeros, so that nothing hides its product), 255 is NaN in that row and nowhere else."""
    a, b, av, bv = _operands(kind, m, n, k, m + n + k)
    row = m - 1 if side == 'a' else 16 * ((n - 1) // 16) - 1
    blocks = k // 32
    for block in (0, blocks - 1):
        ea, eb = torch.full((m, blocks), 127), torch.full((n, blocks), 127)
        x, v, e = (a, av, ea) if side == 'a' else (b, bv, eb)
        x, v = x.clone(), v.clone()
        e[row, block] = byte
        if byte == 0:
            per = 16 if (kind == 'fp4' and side == 'b') else 32                         # bytes of a block
            codes, keep = x.view(torch.uint8)[row], torch.arange(x.size(1), device='cuda') // per == block
            codes[~keep] = 0
            v[row] = torch.where(torch.arange(k) // 32 == block, v[row] * 2.0 ** -127, 0.0)
        d = torch.zeros((m, n), dtype=torch.float32, device='cuda')
        lhs, rhs = (x, b) if side == 'a' else (a, x)
        deep_gemm.fp8_fp4_gemm_nt((lhs, _packed(ea)), (rhs, _packed(eb)), d)
        d = d.cpu().double()
        hit = torch.zeros((m, n), dtype=torch.bool)
        if side == 'a':
            hit[row] = True
        else:
            hit[:, row] = True
        exact = (v if side == 'a' else av) @ (bv if side == 'a' else v).t()
        if byte == 255:
            assert torch.isnan(d[hit]).all() and not torch.isnan(d[~hit]).any()
        else:
            assert (d[hit] == exact[hit]).all()                                         # (32 small whole multiples of 2^-129: exact in FP32)
            assert (d[hit] != 0).float().mean() > 0.5
        assert (d[~hit] == exact[~hit]).all()                                           # (sums of multiples of 1/4 below 2^17: exact)
    assert deep_gemm.device_status() == 0


@pytest.mark.parametrize('m,n,k', [(1, 4752, 2272), (2, 4753, 2080), (5, 4800, 3072), (8, 4767, 2112), (6, 5000, 2816), (7, 12289, 2400), (3, 9999, 3040)])
def test_three_ctas_on_an_sm(m, n, k):
    """Three small pieces, a slot each: a last piece of one block, of an odd number of blocks and a whole one; a last CTA with one row of B and with fifteen."""
    t = _layout('fp8', m, n, k)
    assert (t.warps, t.piece, t.slots, t.max_k) == (8, 1024, 3, 3072)
    seed_all(m + n + k)
    (a, sfa, a_ref), (b, sfb, b_ref) = uniform_fp8((m, k), (1, 32)), uniform_fp8((n, k), (1, 32))
    d = torch.full((m + 1, n), float('nan'), dtype=torch.float32, device='cuda')
    for _ in range(2):
        deep_gemm.fp8_gemm_nt((a.cuda(), sfa.cuda()), (b.cuda(), sfb.cuda()), d[:m], recipe_a=(1, 32), recipe_b=(1, 32))
    assert deep_gemm.device_status() == 0
    _check(d[:m], a_ref, b_ref)
    assert torch.isnan(d[m]).all()


@pytest.mark.parametrize('m,n,k', [(4, 2368, 7680), (1, 3072, 6144), (16, 1031, 8160), (8, 2400, 4128)])
def test_fp32_scales_with_a_long_k_of_e2m1(m, n, k):
    """Behind the relayout a CTA asks for an even share of an SM; both host layers say so to the library and give the same bits."""
    seed_all(m + n + k)
    (a, sfa, a_ref), (b, sfb, b_ref) = uniform_fp8((m, k), (1, 32)), uniform_fp4(n, k, (1, 32), False)
    out = []
    for host in (deep_gemm, deep_gemm._api):
        d = torch.full((m + 1, n), float('nan'), dtype=torch.float32, device='cuda')
        host.fp8_fp4_gemm_nt((a.cuda(), sfa.cuda()), (b.cuda(), sfb.cuda()), d[:m], recipe_a=(1, 32), recipe_b=(1, 32))
        _check(d[:m], a_ref, b_ref)
        assert torch.isnan(d[m]).all()
        out.append(d[:m].cpu())
    assert deep_gemm.device_status() == 0
    assert torch.equal(*out)
