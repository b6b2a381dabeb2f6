"""Decode GEMMs whose K splits meet inside a cluster: uneven splits, ragged rows and columns, every output type and the
pair epilogues, against 64-bit PyTorch math; and the same call with its splits meeting in global memory."""
import pytest
import torch

from torch_dist_ext_b200.ops import gemm

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
