"""The rule and the tiles of the kernel for a few rows, asked of the library without a GPU."""

import ctypes

import pytest

from deep_gemm import _lib as L


def _desc(kind, m, n, k):
    return L.GemmDesc(m=m, n=n, k=k, a_dtype=L.E4M3, b_dtype=L.E2M1X2 if kind == 'fp4' else L.E4M3, d_dtype=L.BF16)


def _takes(kind, m, n, k):
    return L.lib().dg_gemm_reads_any_scales(ctypes.byref(_desc(kind, m, n, k))) == 1


def _layout(kind, m, n, k):
    out = L.FewRowsLayout()
    assert L.lib().dg_gemm_few_rows_layout(ctypes.byref(_desc(kind, m, n, k)), ctypes.byref(out)) == 0, L.last_error()
    return out


@pytest.mark.parametrize('kind', ['fp8', 'fp4'])
def test_everything_that_is_taken_fits(kind):
    """Rows and K inside the instantiation, shared memory inside the 227 KB of a CTA, a piece inside the count of one barrier (2^20 - 1 bytes)."""
    taken = 0
    for m in range(1, 17):
        for k in range(32, 16385, 224 if m in (1, 8, 16) else 736):
            for n in (1, 16, 512, 1024, 2048, 2368, 2369, 2560, 2912, 4096, 4736, 4737, 8192, 9472, 13312, 24576):
                if not _takes(kind, m, n, k):
                    continue
                t = _layout(kind, m, n, k)
                taken += 1
                assert m <= t.rows and k <= t.max_k and t.slots >= 1, (m, n, k)
                assert t.dynamic_smem + t.static_smem <= 227 * 1024 and t.dynamic_smem <= 208 * 1024, (m, n, k)
                assert t.slots == 1 or (t.slots - 1) * t.piece < k, (m, n, k)              # (no slot that no piece goes to)
                assert 16 * t.piece < 2 ** 20 and m * k < 2 ** 20
    assert taken > 2000


def test_a_layout_is_refused_where_the_kernel_does_not_run():
    out = L.FewRowsLayout()
    for desc in (_desc('fp8', 17, 512, 512), _desc('fp8', 1, 512, 528), _desc('fp8', 1, 65536, 4096), _desc('fp4', 1, 512, 16384)):
        assert L.lib().dg_gemm_few_rows_layout(ctypes.byref(desc), ctypes.byref(out)) != 0 and 'not a problem of a few rows' in L.last_error()


@pytest.mark.parametrize('m,last_k', [(1, 3072), (4, 3072), (5, 3072), (6, 2816), (7, 2400), (8, 2112)])
def test_three_ctas_share_an_sm_where_there_are_more_than_two_for_it(m, last_k):
    """E4M3, K just above one piece of 2048: 228 KB of an SM, 1 KB of each CTA's share reserved; every piece has a slot. Up to two CTAs per SM keep the large pieces."""
    for k in (2080, 2112, 2400, 2816, 3072):
        if k > last_k:
            continue
        for n in (4752, 9472):
            t = _layout('fp8', m, n, k)
            assert 3 * (t.dynamic_smem + t.static_smem + 1024) <= 228 * 1024 and t.slots * t.piece >= k, (m, n, k)
        assert _layout('fp8', m, 4736, k).piece == 2048


@pytest.mark.parametrize('kind,m,k,last', [
    ('fp8', 4, 64, 24576), ('fp8', 4, 128, 23680), ('fp8', 4, 160, 24576), ('fp8', 4, 1024, 24576), ('fp8', 1, 2048, 24576), ('fp8', 4, 2080, 21312), ('fp8', 5, 3072, 16384),
    ('fp8', 7, 2560, 14208), ('fp8', 4, 4096, 12288), ('fp8', 4, 4128, 8192), ('fp8', 7, 4128, 11840), ('fp8', 7, 7168, 7021), ('fp8', 1, 8192, 8192), ('fp8', 1, 16384, 2368),
    ('fp8', 6, 16384, 2368), ('fp8', 8, 128, 12288), ('fp8', 8, 160, 12288), ('fp8', 8, 2048, 12288), ('fp8', 8, 7168, 4096), ('fp8', 8, 8192, 2560),
    ('fp8', 16, 1024, 8192), ('fp8', 16, 3072, 6144), ('fp8', 16, 4096, 4096), ('fp8', 9, 8192, 2368),
    ('fp4', 7, 2048, 16384), ('fp4', 7, 4096, 8192), ('fp4', 7, 8192, 4096), ('fp4', 8, 7680, 3072), ('fp4', 8, 7712, 3072), ('fp4', 8, 7808, 2368), ('fp4', 8, 8192, 2368),
    ('fp4', 12, 256, 3072), ('fp4', 16, 96, 3072), ('fp4', 16, 288, 3072), ('fp4', 16, 8192, 2368)])
def test_the_widest_b_of_a_few_rows(kind, m, k, last):
    """Both sides of the limits on N, which lie where the tensor-core kernel becomes the faster one. (K of 16384 has a lower limit too.)"""
    assert _takes(kind, m, last, k) and not _takes(kind, m, (last + 8) // 8 * 8, k) and not _takes(kind, m, last + 12288, k)
    assert _takes(kind, m, 511, k) == (k <= 4096 or (m <= 8 and k <= 8192))


def test_whole_tiles_of_sixteen_rows():
    """E2M1, 16 rows, K of one or two K blocks: more CTAs than SMs are worthwhile only where the other kernel's tiles are not whole."""
    for k in (128, 256):
        assert _takes('fp4', 16, 2368, k) and not _takes('fp4', 16, 2400, k) and _takes('fp4', 16, 2416, k) and not _takes('fp4', 16, 3072, k) and _takes('fp4', 15, 3072, k)


def test_scales_of_b_that_the_other_kernel_needs_relaid():
    """N no multiple of 8: wider than where whole columns of 16 bytes end."""
    assert _takes('fp8', 7, 17500, 2560) and not _takes('fp8', 7, 17504, 2560)
    assert _takes('fp8', 4, 24570, 128) and not _takes('fp8', 4, 24576, 128)
    assert _takes('fp4', 8, 3001, 8192) and not _takes('fp4', 8, 3000, 8192)


def test_what_the_rule_refuses():
    """Rows, K and types outside it; what a tensor map or an epilogue asks of the tensor-core kernel."""
    for kind, m, n, k in (('fp8', 17, 512, 512), ('fp8', 1, 512, 16416), ('fp8', 7, 512, 16384), ('fp8', 9, 2368, 8224), ('fp4', 1, 512, 8224), ('fp8', 1, 512, 48)):
        assert not _takes(kind, m, n, k)
    for field, value in (('accumulate', 1), ('major_a', 1), ('major_b', 1), ('num_sms', 20), ('epilogue', 3), ('gemm_type', 1)):
        desc = _desc('fp8', 16, 512, 512)
        assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 1
        setattr(desc, field, value)
        assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 0


@pytest.mark.parametrize('kind,m,n,k', [
    ('fp4', 8, 2369, 7168), ('fp4', 4, 3072, 7680), ('fp4', 3, 2376, 6784), ('fp4', 6, 2376, 6272), ('fp4', 1, 256, 7296), ('fp4', 4, 10240, 128), ('fp8', 4, 4737, 7296), ('fp8', 6, 4737, 6272), ('fp8', 6, 767, 16384)])
def test_sizes_that_only_scales_read_in_place_make_worthwhile(kind, m, n, k):
    """Packed scales take the kernel for a few rows, FP32 ones (relaid in front of either kernel) the tensor-core kernel."""
    desc = _desc(kind, m, n, k)
    assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 1
    desc.reserved0 = 1
    assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 0


@pytest.mark.parametrize('kind,m,n,k', [
    ('fp4', 8, 2368, 8192), ('fp4', 1, 257, 7680), ('fp4', 1, 256, 7168), ('fp4', 4, 4096, 6144), ('fp4', 4, 10240, 384), ('fp4', 4, 10000, 128), ('fp4', 4, 3072, 7200), ('fp4', 1, 4096, 7168), ('fp4', 5, 4096, 6656),
    ('fp8', 4, 4736, 8192), ('fp8', 4, 8192, 7200), ('fp8', 5, 6000, 7168), ('fp8', 3, 8192, 8192), ('fp8', 7, 7168, 6144), ('fp8', 6, 768, 16384), ('fp8', 4, 20480, 2080),
    ('fp8', 4, 24576, 2048), ('fp8', 1, 2112, 7168), ('fp8', 16, 2112, 7168), ('fp8', 8, 2912, 7200)])
def test_sizes_that_fp32_scales_keep(kind, m, n, k):
    desc = _desc(kind, m, n, k)
    desc.reserved0 = 1
    assert L.lib().dg_gemm_reads_any_scales(ctypes.byref(desc)) == 1


@pytest.mark.parametrize('m,n,k,share', [(4, 2368, 7680, 1), (1, 1024, 4128, 1), (16, 2368, 8192, 1), (1, 3072, 6144, 2), (2, 4096, 5632, 2)])
def test_an_even_share_of_the_sms_behind_a_relayout(m, n, k, share):
    """E2M1 with a long K: as many CTAs fit an SM as are needed to hold them all, and not one more (228 KB, 1 KB of each CTA's share reserved)."""
    desc, out = _desc('fp4', m, n, k), L.FewRowsLayout()
    desc.reserved0 = 1
    assert L.lib().dg_gemm_few_rows_layout(ctypes.byref(desc), ctypes.byref(out)) == 0
    size = out.dynamic_smem + out.static_smem + 1024
    assert share * size <= 228 * 1024 < (share + 1) * size and out.dynamic_smem <= 208 * 1024
    assert out.dynamic_smem >= _layout('fp4', m, n, k).dynamic_smem
