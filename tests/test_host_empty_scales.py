"""Scales without rows or columns on meta tensors (no GPU), through both host layers."""

import pytest
import torch

import deep_gemm
from deep_gemm import _api


@pytest.mark.parametrize('host', [deep_gemm, _api])
@pytest.mark.parametrize('groups,mn,k', [(None, 0, 256), (None, 0, 32), (3, 64, 0), (3, 0, 96), (0, 16, 512), (None, 8, 0), (2, 0, 0)])
def test_strides_of_empty_results(host, groups, mn, k):
    """What has no elements is laid out as torch lays out the [.., ceil(K / 64), MN] storage seen transposed, where an empty dimension counts as one."""
    lead = () if groups is None else (groups,)
    sf = torch.empty((*lead, mn, -(-k // 32)), dtype=torch.float32, device='meta')
    out = host.transform_sf_into_required_layout(sf, mn, k, (1, 32), groups)
    like = torch.empty((*lead, -(-k // 64), mn), dtype=torch.int16, device='meta').transpose(-2, -1)
    assert out.shape == like.shape and out.stride() == like.stride() and out.dtype == torch.int16
