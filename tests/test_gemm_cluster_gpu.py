"""GEMMs whose K splits meet inside a cluster: uneven splits, ragged rows and columns, every output type, against 64-bit
PyTorch math; and splits of more tiles than the device holds clusters, which meet in global memory, with the rotary and silu
epilogues (those of a cluster are in test_gemm_epilogues_gpu.py)."""
import pytest
import torch

from torch_dist_ext_b200.ops import gemm, rope

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 128, 128),       # two K blocks, two splits
    (3, 130, 576),       # nine K blocks over eight splits; two rows in the second tile
    (17, 768, 4096),     # six tiles of eight splits
    (64, 4096, 1792),    # 28 K blocks over four splits
    (100, 3584, 4096),   # ragged columns of a 128-wide tile
    (128, 9472, 128),    # 74 tiles, as many as there are clusters of two
    (33, 9600, 256),     # 75 tiles: no room for clusters, one split
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_cluster_splits_match_64_bit(m, n, k, out_dtype):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    want = a.double() @ w.double().t()
    outs = [gemm.linear(a, w, out_dtype=out_dtype) for _ in range(2)]
    torch.cuda.synchronize()
    assert gemm.pipeline_status() == 0
    assert torch.equal(outs[0], outs[1]), "the splits are added in a fixed order"
    # bf16: half a rounding step (2^-9) of the largest value, doubled; fp32: 2^-24 per addition along K, with a margin of 4
    bound = want.abs().max() * (2.0 ** -8 if out_dtype == torch.bfloat16 else k * 2.0 ** -22)
    assert (outs[0].double() - want).abs().max() <= bound
    ws, counters, _ = gemm._workspace(a.device)
    assert float(ws.abs().max()) == 0.0 and int(counters.abs().sum()) == 0


@pytest.mark.parametrize("m,n,k", [
    (256, 256, 1024),     # one tile in pieces
    (300, 1280, 4096),    # ragged rows: ten tiles of four pieces
    (257, 4352, 2048),    # 34 tiles: too many for clusters of eight CTAs
    (700, 3584, 1792),    # 42 tiles, whole
    (260, 263, 4160),     # ragged both ways, uneven pieces, unaligned output rows
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_pieces_of_a_pair_tile_match_64_bit(m, n, k, out_dtype):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    want = a.double() @ w.double().t()
    outs = [gemm.linear(a, w, out_dtype=out_dtype) for _ in range(2)]
    torch.cuda.synchronize()
    assert gemm.pipeline_status() == 0 and torch.equal(outs[0], outs[1])
    # as above
    bound = want.abs().max() * (2.0 ** -8 if out_dtype == torch.bfloat16 else k * 2.0 ** -22)
    assert (outs[0].double() - want).abs().max() <= bound


@pytest.mark.parametrize("m,n,k", [
    (129, 200, 4096),    # a 256-wide tile of which 200 columns are there, one row in the second row tile
    (300, 64, 2048),     # 64-wide
    (512, 192, 8192),
    (200, 130, 6400),   # output rows that are no multiple of four values: stored one by one
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_splits_of_tall_products(m, n, k, out_dtype):
    """More than 128 rows of a weight with fewer than 256: the activations are on the 128-row side and columns contiguous."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    dtype = torch.float16 if out_dtype == torch.float16 else torch.bfloat16
    a = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(dtype)
    want = a.double() @ w.double().t()
    outs = [gemm.linear(a, w, out_dtype=out_dtype) for _ in range(2)]
    torch.cuda.synchronize()
    assert gemm.pipeline_status() == 0 and torch.equal(outs[0], outs[1])
    bound = want.abs().max() * (k * 2.0 ** -22 if out_dtype == torch.float32 else 2.0 ** -8)      # as above
    assert (outs[0].double() - want).abs().max() <= bound
    # an output that starts in the middle of a wider buffer, two values off a 16-byte boundary
    wide = torch.zeros(m * n + 2, device="cuda", dtype=out_dtype)
    gemm.linear(a, w, wide[2:].view(m, n), out_dtype=out_dtype)
    assert torch.equal(wide[2:].view(m, n), outs[0]) and not wide[:2].any()


@pytest.mark.parametrize("m,n,k", [
    (16, 128, 16384),    # one tile of sixteen splits
    (33, 512, 14336),    # four
    (5, 640, 14400),     # five, 225 K blocks: fifteen splits of fifteen
    (128, 250, 8192),    # two, ragged rows
    (17, 1024, 14336),   # eight tiles: no room for sixteen
    (160, 64, 14336),    # the activations on the 128-row side
    (256, 200, 8192),
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_few_tiles_and_a_long_k(m, n, k, out_dtype):
    """Clusters of up to sixteen splits, which share nothing with a call on another stream: both at a time."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = [torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2)]
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    want = [x.double() @ w.double().t() for x in a]
    streams = [torch.cuda.Stream() for _ in a]
    torch.cuda.synchronize()
    outs = [[], []]
    for _ in range(4):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[i].append(gemm.linear(a[i], w, out_dtype=out_dtype))
    torch.cuda.synchronize()
    assert gemm.pipeline_status() == 0
    for i in range(2):
        assert all(torch.equal(outs[i][0], o) for o in outs[i]), "the splits are added in a fixed order"
        bound = want[i].abs().max() * (k * 2.0 ** -22 if out_dtype == torch.float32 else 2.0 ** -8)      # as above
        assert (outs[i][0].double() - want[i]).abs().max() <= bound


def _scratch_is_zero(device):
    ws, counters, _ = gemm._workspace(device)
    return float(ws.abs().max()) == 0.0 and int(counters.abs().sum()) == 0


@pytest.mark.parametrize("m,n,k,splits", [(1, 10240, 1024, 4), (33, 10101, 512, 3), (128, 9728, 640, 5)])
def test_splits_meet_in_memory(m, n, k, splits):
    """More than 74 tiles, cut along K all the same: fp32 additions into scratch, and the split that arrives last finishes the
    tile and leaves the scratch zeroed for the second call."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    want = a.double() @ w.double().t()
    for out_dtype in (torch.bfloat16, torch.float32):
        for _ in range(2):
            out = gemm.linear(a, w, out_dtype=out_dtype, splits=splits)
            bound = want.abs().max() * (2.0 ** -8 if out_dtype == torch.bfloat16 else k * 2.0 ** -22)      # as above
            assert (out.double() - want).abs().max() <= bound
            assert _scratch_is_zero(a.device) and gemm.pipeline_status() == 0


@pytest.mark.parametrize("m", [1, 17, 100])
def test_rotary_epilogue_in_memory(m):
    q_heads, kv_heads, k, seq = 64, 8, 512, 40          # 80 tiles
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn((q_heads + 2 * kv_heads) * 128, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    positions = torch.randint(0, seq, (m,), device="cuda", generator=g)
    cos_sin = rope.build_cos_sin_cache(seq, 128, 5e5, "cuda")
    want = (a.double() @ w.double().t()).view(m, -1, 128)
    cos, sin = cos_sin[positions].double()[:, None, :64], cos_sin[positions].double()[:, None, 64:]
    x = want[:, :q_heads + kv_heads].clone()
    want[:, :q_heads + kv_heads] = torch.cat([x[..., :64] * cos - x[..., 64:] * sin, x[..., 64:] * cos + x[..., :64] * sin], -1)
    bound = want.abs().max() * 2.0 ** -7                # a rounding step of bf16 of the largest value
    rows = torch.arange(m, device="cuda")
    for _ in range(2):
        k_cache = torch.zeros(m + 2, seq, kv_heads, 128, dtype=torch.bfloat16, device="cuda")
        v_cache = torch.zeros_like(k_cache)
        out = gemm.linear_rope_kv(a, w, positions, cos_sin, k_cache, v_cache, q_heads, kv_heads)
        assert (out.view(m, -1, 128).double() - want).abs().max() <= bound
        assert (k_cache[rows, positions].double() - want[:, q_heads:q_heads + kv_heads]).abs().max() <= bound
        assert (v_cache[rows, positions].double() - want[:, q_heads + kv_heads:]).abs().max() <= bound
        k_cache[rows, positions] = 0
        v_cache[rows, positions] = 0
        assert not k_cache.any() and not v_cache.any()
        assert _scratch_is_zero(a.device) and gemm.pipeline_status() == 0


@pytest.mark.parametrize("m", [1, 17, 100])
def test_silu_epilogue_in_memory(m):
    ffn, k = 64 * 80, 512
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * ffn, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    gu = a.double() @ w.double().t()
    want = torch.nn.functional.silu(gu[:, :ffn]) * gu[:, ffn:]
    for _ in range(2):
        out = gemm.linear_silu_mul(a, w)
        assert (out.double() - want).abs().max() <= want.abs().max() * 2.0 ** -7      # as above
        assert _scratch_is_zero(a.device) and gemm.pipeline_status() == 0
