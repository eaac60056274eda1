"""The entry points look at sizes and strides of permuted operands without making tensors of them: shapes, messages and the layout of
re-laid scales on meta tensors (no GPU), through both host layers where both have the call."""

import pytest
import torch

import deep_gemm
from deep_gemm import _api


def _meta(*shape, dtype=torch.float8_e4m3fn):
    return torch.empty(shape, dtype=dtype, device='meta')


def _scales(mn, k, *lead):
    return _meta(*lead, -(-k // 64), mn, dtype=torch.int16).transpose(-2, -1)


@pytest.mark.parametrize('host', [deep_gemm, _api])
def test_every_spelling_takes_its_operands_and_refuses_others(host):
    m, n, k = 64, 256, 384
    a, b = (_meta(m, k), _scales(m, k)), (_meta(n, k), _scales(n, k))
    at, bt = [(x.t().contiguous(), s.t()) for x, s in (a, b)]
    d = _meta(m, n, dtype=torch.bfloat16)
    for name, lhs, rhs in (('nt', a, b), ('nn', a, bt), ('tn', at, bt), ('tt', at, b)):
        gemm = getattr(host, f'fp8_fp4_gemm_{name}')
        gemm(lhs, rhs, d)
        gemm(lhs, rhs, d, d)                                                            # accumulated
        with pytest.raises(RuntimeError, match="Conflicting shape dimension 'n': tensor #2 annotation=\"mn\" axis=1 gives 255"):
            gemm(lhs, rhs, _meta(m, 255, dtype=torch.bfloat16))
        with pytest.raises(RuntimeError, match='SF rows: expected 64, got 63' if name[0] == 'n' else 'SF rows: expected 64, got 63'):
            gemm((lhs[0], _scales(m - 1, k) if name[0] == 'n' else _scales(m - 1, k).t()), rhs, d)
    with pytest.raises((IndexError, RuntimeError)):
        host.fp8_fp4_gemm_nn(a, (bt[0][0], bt[1]), d)                                   # one dimension: nothing to transpose
    with pytest.raises(RuntimeError, match='Shape mismatch: tensor #0, annotation="mk"'):
        host.fp8_fp4_gemm_nt((a[0][None], a[1]), b, d)


@pytest.mark.parametrize('host', [deep_gemm, _api])
def test_einsum_forms_with_permuted_operands(host):
    t, h, r, dd = 96, 4, 256, 128
    a = (_meta(t, h, r), _scales(t, r, h).permute(1, 0, 2))
    b = (_meta(h, dd, r), _scales(dd, r, h))
    out = (_meta(t, h, dd), _meta(h * dd // 64, t, dtype=torch.int16).t())
    host.fp8_einsum('bhr,hdr->bhd', a, b, out)
    host.fp8_einsum('bhr,hdr->bhd', a, b, _meta(t, h, dd, dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match='only the forward expression accepts'):
        host.fp8_einsum('bhd,hdr->bhr', (_meta(t, h, dd), _scales(t, dd, h).permute(1, 0, 2)), b, out)
    with pytest.raises(RuntimeError, match='Unsupported einsum expression'):
        host.fp8_einsum('bhd,hdr', a, b, out)
    with pytest.raises(RuntimeError):
        host.fp8_einsum('bhr,hdr->bhd', (a[0][0], a[1]), b, out)                        # two dimensions where three are permuted
    x, w = _meta(t, h, r, dtype=torch.bfloat16), _meta(h, dd, r, dtype=torch.bfloat16)
    host.einsum('bhr,hdr->bhd', x, w, _meta(t, h, dd, dtype=torch.bfloat16))
    host.einsum('bhd,hdr->bhr', _meta(t, h, dd, dtype=torch.bfloat16), w, _meta(t, h, r, dtype=torch.bfloat16))
    host.einsum('bhd,bhr->hdr', _meta(t, h, dd, dtype=torch.bfloat16), x, _meta(h, dd, r, dtype=torch.bfloat16))


@pytest.mark.parametrize('host', [deep_gemm, _api])
@pytest.mark.parametrize('lead,num_groups', [((), None), ((3,), 3)])
@pytest.mark.parametrize('mn,k', [(40, 384), (37, 200), (1, 64)])
def test_the_layout_of_relaid_scales(host, lead, num_groups, mn, k):
    """Result [.., MN, ceil(K / 64)], MN-major, groups one after the other; what has that layout already is handed back as it is."""
    sf = _meta(*lead, mn, -(-k // 32), dtype=torch.float32)
    out = host.transform_sf_into_required_layout(sf, mn, k, (1, 32), num_groups)
    cols = -(-k // 64)
    assert out.shape == (*lead, mn, cols) and out.dtype == torch.int16
    assert out.stride()[-2:] == (1, mn) and (not lead or out.stride(0) == mn * cols)
    ready = _scales(mn, k, *lead)
    assert host.transform_sf_into_required_layout(ready, mn, k, (1, 32), num_groups) is ready
