"""The entry points that allocate their outputs natively return what the out= forms write, in the same layout."""
import pytest
import torch

import torch_dist_ext_b200 as tdx
from torch_dist_ext_b200.ops import attention, gemm
from torch_dist_ext_b200.utils.config import OUT_FP8_BLOCK128, OUT_FP8_TOKEN, OUT_SAME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (5, 640, 1024), (128, 19200, 128)])      # 19200: more tiles than SMs
@pytest.mark.parametrize("out_dtype", [None, torch.float32])
def test_linear(m, n, k, out_dtype):
    a = torch.randn(m, k, device="cuda", dtype=torch.float16)
    w = torch.randn(n, k, device="cuda", dtype=torch.float16) * 0.1
    got = gemm.linear(a, w, out_dtype=out_dtype)
    out = torch.empty(m, n, device="cuda", dtype=out_dtype or torch.float16)
    assert gemm.linear(a, w, out, out_dtype=out_dtype) is out
    assert got.dtype == out.dtype and got.is_contiguous() and torch.equal(got, out)
    assert not gemm.linear(a.requires_grad_(), w).requires_grad


def test_attention():
    qkv = torch.randn(3, 12 * 128, device="cuda", dtype=torch.bfloat16)
    q = qkv[:, : 8 * 128].view(3, 8, 128)                    # a view with a longer row pitch
    k, v = (torch.randn(3, 300, 2, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    lens = torch.tensor([300, 1, 129], device="cuda", dtype=torch.int32)
    out = torch.empty(3, 8, 128, device="cuda", dtype=torch.bfloat16)
    got = attention.decode_attention(q, k, v, lens, 300)
    assert got.is_contiguous() and torch.equal(got, attention.decode_attention(q, k, v, lens, 300, out))
    kp = qkv[:, 8 * 128: 9 * 128].view(3, 1, 128)
    got = attention.prefill_attention(q, kp, kp)
    assert got.is_contiguous() and torch.equal(got, attention.prefill_attention(q, kp, kp, out))


@pytest.mark.parametrize("mode", [OUT_SAME, OUT_FP8_TOKEN, OUT_FP8_BLOCK128])
@pytest.mark.parametrize("want_residual", [True, False])
def test_fused_norm(mode, want_residual):
    tdx.setup_env(0, 1, max_size_in_bytes=4 << 20)
    x = torch.randn(2, 3, 512, device="cuda", dtype=torch.bfloat16)
    gamma = torch.ones(512, device="cuda", dtype=torch.bfloat16)
    norm, res, scales = tdx.fused_allreduce_rms(x, x, gamma, 1e-6, out_mode=mode, want_residual=want_residual)
    e_norm, e_res, e_scales = tdx.reference.fused_allreduce_rms_reference([x.view(6, 512)], x.view(6, 512), gamma, 1e-6, mode)
    assert norm.shape == x.shape and norm.dtype == e_norm.dtype and (res is None) == (not want_residual)
    assert (norm.view(6, 512).float() - e_norm.float()).abs().max() <= e_norm.float().abs().max() * 2.0 ** -3    # an e4m3 step
    if want_residual:
        assert torch.equal(res.view(6, 512), e_res)
    assert (scales is None) == (mode == OUT_SAME) and (scales is None or scales.shape == e_scales.shape)
    tdx.teardown_env()
