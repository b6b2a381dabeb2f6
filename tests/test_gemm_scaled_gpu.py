"""The block-scaled e4m3 GEMM (gemm_scaled.cu) at the edges of its tiles, rounds and pieces, against 64-bit PyTorch math."""
import pytest
import torch

from torch_dist_ext_b200 import _lib
from torch_dist_ext_b200.ops import gemm, quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 256, 128),          # one row, one K block
    (33, 384, 256),         # one and a half tiles of weights
    (64, 7168, 8192),       # decode: tiles in pieces of K
    (17, 5376, 8192),       # four pieces whose warps add up rows 2 w, 2 w + 1 (+ 16): one row more for half the lanes
    (49, 3840, 4096),       # the same with eight pieces, 32 rows apart
    (128, 38144, 512),      # decode: 149 tiles, one more than the multiprocessors
    (129, 256, 1024),       # the smallest pair: one row in the second CTA
    (257, 1280, 8192),      # ragged rows, fewer tiles than pairs
    (300, 640, 384),        # half a tile of weights at the end
    (2048, 7168, 2048),     # three full rounds and two tiles over
    (4100, 1280, 1024),     # ragged rows over a full round
])
def test_block_scaled_matches_64_bit(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a_q, a_s = quant.quant_fp8(torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16), block_scaled=True)
    w_q, w_s = gemm.quantize_weight_block128(torch.randn(n, k, device="cuda", generator=g) * 0.05)
    a = (a_q.double().view(m, k // 128, 128) * a_s.double()[..., None]).view(m, k)
    w = (w_q.double().view(n // 128, 128, k // 128, 128) * w_s.double()[:, None, :, None]).view(n, k)
    want = a @ w.t()
    scale = want.abs().max()
    for out_dtype in (torch.bfloat16, torch.float32):
        torch.full((20 << 20,), float("nan"), device="cuda")     # freed at once: the scratch may hold anything
        outs = [gemm.linear_fp8_blockscaled(a_q, a_s, w_q, w_s, out_dtype=out_dtype) for _ in range(2)]
        torch.cuda.synchronize()
        assert gemm.pipeline_status() == 0
        assert torch.equal(outs[0], outs[1]), "the sum must not depend on which piece arrives last"
        # half a rounding step of the output type (2^-9 for bf16) of the largest value; fp32: one rounding per K block
        # and sum, 2^-24 each, with a margin of 8
        bound = scale * (2.0 ** -8 if out_dtype == torch.bfloat16 else (k // 128 + 8) * 2.0 ** -21)
        assert (outs[0].double() - want).abs().max() <= bound


def _operands(m, n, k, seed):
    """e4m3 rows and weights (any row counts) with their scales, and the product in 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a_q, a_s = quant.quant_fp8(torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16), block_scaled=True)
    rows = -(-n // 128) * 128
    w_q, w_s = gemm.quantize_weight_block128(torch.randn(rows, k, device="cuda", generator=g) * 0.05)
    a = (a_q.double().view(m, k // 128, 128) * a_s.double()[..., None]).view(m, k)
    w = (w_q.double().view(rows // 128, 128, k // 128, 128) * w_s.double()[:, None, :, None]).view(rows, k)[:n]
    return a_q, a_s, w_q[:n], w_s, a @ w.t()


def _bound(want, k, out_dtype):
    return want.abs().max() * {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: (k // 128 + 8) * 2.0 ** -21}[out_dtype]      # as above


@pytest.mark.parametrize("m,n,k", [
    (1, 200, 1024), (17, 1000, 2048), (33, 384, 256), (64, 1279, 4096),        # pieces in clusters; rows of weights that end inside a tile
    (129, 256, 1024), (257, 1280, 8192), (300, 640, 384), (200, 1001, 8192),   # pairs, pieces through memory
    (128, 38030, 512), (2048, 7100, 1024),                                     # whole tiles
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_any_weight_rows(m, n, k, out_dtype):
    """The kernel of gemm_scaled.cu itself, also where products this small run on the swapped one: stores with and without
    bounds checks, in every type."""
    a_q, a_s, w_q, w_s, want = _operands(m, n, k, m + n + k)
    ops, status = _lib.ops(), gemm._workspace(a_q.device)[2]
    outs = [ops.gemm_scaled_call(a_q, w_q, out_dtype, a_s, w_s, status) for _ in range(2)]
    torch.cuda.synchronize()
    assert gemm.pipeline_status() == 0 and torch.equal(outs[0], outs[1])
    assert (outs[0].double() - want).abs().max() <= _bound(want, k, out_dtype)


@pytest.mark.parametrize("m,n,k", [(64, 7168, 1024), (300, 6400, 2048), (16, 1280, 8192), (129, 1280, 8192), (256, 1152, 2048), (700, 300, 4096)])
def test_out_strides_and_types(m, n, k):
    """Through the entry point, on either side of the line between the two kernels: ``out=``, rows of wider buffers as
    operands, every output type."""
    a_q, a_s, w_q, w_s, want = _operands(m, n, k, m + n)
    wide_a = torch.zeros(m, k + 128, device="cuda", dtype=torch.uint8)
    wide_w = torch.zeros(n, k + 256, device="cuda", dtype=torch.uint8)
    wide_a[:, 128:] = a_q.view(torch.uint8)
    wide_w[:, :k] = w_q.view(torch.uint8)
    a_v, w_v = wide_a.view(torch.float8_e4m3fn)[:, 128:], wide_w.view(torch.float8_e4m3fn)[:, :k]
    for out_dtype in (torch.bfloat16, torch.float16, torch.float32):
        got = gemm.linear_fp8_blockscaled(a_q, a_s, w_q, w_s, out_dtype=out_dtype)
        out = torch.full((m, n), float("nan"), device="cuda", dtype=out_dtype)
        assert gemm.linear_fp8_blockscaled(a_v, a_s, w_v, w_s, out) is out
        assert torch.equal(got, out) and (got.double() - want).abs().max() <= _bound(want, k, out_dtype)
    assert gemm.linear_fp8_blockscaled(a_q, a_s, w_q, w_s, out_dtype=None).dtype == torch.get_default_dtype()
    assert gemm.pipeline_status() == 0
