"""Host-side launch planning of the GEMM and of decode attention (pure Python, no GPU)."""
import pytest
import torch

from torch_dist_ext_b200.ops import attention, gemm

SMS = 148


@pytest.mark.parametrize("m", [1, 16, 64, 128])
@pytest.mark.parametrize("n,k", [(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (768, 4096), (512, 1792)])
def test_decode_shapes_run_swapped_and_fill_the_sms(m, n, k):
    swap, bn, splits = gemm.plan(m, n, k)
    assert swap, "up to 128 tokens the weights take the 128-row side of the tile"
    assert bn in (16, 32, 64, 128) and bn >= min(m, 128)
    tiles = -(-n // 128) * -(-m // bn)
    kblocks = k // 64
    assert 1 <= splits <= max(1, kblocks // 2)
    if tiles >= SMS:
        assert splits == 1
    else:
        assert tiles * splits <= SMS            # one wave
        assert splits == max(1, min(kblocks // 2, SMS // tiles))


@pytest.mark.parametrize("m,n,k", [(2048, 28672, 4096), (8192, 4096, 14336), (256, 256, 64), (300, 520, 512)])
def test_prefill_shapes_run_unswapped_with_wide_tiles(m, n, k):
    swap, bn, splits = gemm.plan(m, n, k)
    assert not swap and bn in (128, 256)
    if (m // 128) * (n // 256) >= SMS:
        assert bn == 256 and splits == 1


def test_block_scaled_plan_keeps_the_epilogue_in_registers():
    for m in (1, 16, 64, 2048):
        swap, bn, splits = gemm.plan(m, 28672, 8192, elem_size=1, scaled=True)
        assert swap and bn <= 64, "the promoting epilogue holds one fp32 accumulator per column"
        assert splits >= 1


@pytest.mark.parametrize("batch,kv_heads,max_len", [(1, 8, 2048), (16, 8, 2048), (64, 8, 2048), (64, 1, 2048), (1, 1, 64),
                                                     (256, 8, 4096), (3, 2, 100000)])
def test_attention_splits_fit_one_wave_and_keep_128_positions(batch, kv_heads, max_len):
    s = attention.pick_splits(batch, kv_heads, max_len)
    assert s >= 1
    assert s <= max(1, -(-max_len // 128))                       # at least 128 positions per split
    assert s == 1 or batch * kv_heads * s <= 2 * SMS             # two CTAs per SM, one wave
    t = attention.pick_splits(batch, kv_heads, max_len, ctas_per_sm=1)
    assert 1 <= t <= max(1, -(-max_len // 128))
    assert t == 1 or batch * kv_heads * t <= SMS                 # the tensor-core kernel holds one CTA per SM


def test_tensor_core_attention_splits_follow_the_measured_costs():
    pick = lambda b, h, n: attention.pick_splits(b, h, n, ctas_per_sm=1)
    assert pick(1, 1, 2048) == 8                                 # 16 chunks: 8 x 2, not 16 x 1 (merge grows with the splits)
    assert pick(16, 1, 2048) == 4                                # not 9: 9 splits leave 2 chunks to most CTAs, like 8
    assert pick(64, 1, 2048) == 1                                # a third of the SMs already busy: the merge costs more
    assert pick(16, 8, 2048) == 1
    assert pick(1, 1, 128) == 1
    assert pick(3, 2, 100000) > 8                                # long contexts still spread over the SMs


def test_splits_that_merge_in_a_cluster_are_cheaper():
    held = {2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 7: 15, 8: 15}    # clusters that a B200 holds at a time
    pick = lambda b, h, n, c: attention.pick_splits(b, h, n, ctas_per_sm=1, clusters=c)
    assert pick(16, 1, 2048, None) == 4 and pick(16, 1, 2048, held) == 6          # 16 x 6 CTAs; eight splits would not fit
    assert pick(64, 1, 2048, None) == 1 and pick(64, 1, 2048, held) == 2
    assert pick(1, 1, 2000, held) == 8
    for b, h, n in [(1, 1, 128), (7, 2, 300), (3, 8, 5000), (16, 8, 2048), (40, 1, 777), (150, 1, 2048), (2, 1, 100000)]:
        s = pick(b, h, n, held)
        assert s >= 1 and (s == 1 or (b * h * s <= SMS and s <= -(-n // 128)))


def test_fused_decode_epilogues_need_the_weights_on_the_wide_side_and_a_split():
    assert gemm.fused_epilogue_fits(1, 4096) and gemm.fused_epilogue_fits(128, 4096)
    assert not gemm.fused_epilogue_fits(129, 4096)                 # the tokens take the 128-row side
    assert gemm.fused_epilogue_fits(2048, 8192, 1, scaled=True)    # block-scaled operands always run weights-wide
    assert not gemm.fused_epilogue_fits(16, 64)                    # one 128-byte K block: no split, no finalizer
    assert gemm.fused_epilogue_fits(16, 128) and not gemm.fused_epilogue_fits(16, 128, 1, scaled=True)


@pytest.mark.parametrize("bn", [16, 32, 64, 128, 256])
def test_pair_finalizer_threads_cover_every_row_pair_and_column_once(bn):
    """The finalizer's work split (gemm_tcgen05.cu: PairShape, pair_finalize): epilogue warp w has TMEM quarter
    q = w % 4; row pair r = (q % 2) * 32 + lane, column half = q // 2, walked in steps of min(16, bn / 2) columns."""
    half_cols = bn // 2
    width = min(16, half_cols)
    steps = half_cols // width
    seen = {}
    for warp in range(2, 6):
        q = warp % 4
        for lane in range(32):
            r, half = (q % 2) * 32 + lane, q // 2
            for s in range(steps):
                for j in range(width):
                    c = half * half_cols + s * width + j
                    for row in (r, r + 64):
                        assert (row, c) not in seen
                        seen[(row, c)] = (warp, lane)
    assert len(seen) == 128 * bn


@pytest.mark.parametrize("m,n,k", [(200, 28672, 8192), (200, 57344, 8192), (200, 19200, 4096), (2048, 4096, 14336), (300, 520, 512)])
def test_calls_on_cta_pairs_share_no_scratch(m, n, k, monkeypatch):
    """Two calls may run on two streams at a time: a product whose last tiles are cut along K gets slices and counters of its
    own, of the size that its plan asks for."""
    calls = []

    class Ops:
        def gemm_tn_pair(self, a, w, out, sx, sy, status, ws, counters):
            calls.append((ws, counters))

        def __getattr__(self, name):
            return getattr(torch.ops.torch_dist_ext, name)

    monkeypatch.setattr(gemm._lib, "ops", Ops)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(gemm, "_workspace", lambda device: (None, torch.zeros(4096, dtype=torch.int32), None))
    a, w = torch.empty(m, k, dtype=torch.bfloat16), torch.empty(1, k, dtype=torch.bfloat16).expand(n, k)
    gemm.linear(a, w)
    gemm.linear(a, w)
    tiles = -(-m // 256) * -(-n // 256)
    tail = tiles % (SMS // 2) if tiles > SMS // 2 else 0
    floats, words = torch.ops.torch_dist_ext.gemm_pair_scratch(m, n, k, 2, SMS)
    assert (floats, words) == (0, 0) or (words == 2 * tail and floats in [tail * parts * 65536 for parts in (2, 3, 4)])
    assert (floats > 0) == (n > 4096)
    (ws0, c0), (ws1, c1) = calls
    if floats == 0:
        assert ws0 is None and c0 is None
    else:
        assert ws0.numel() == floats and c0.numel() == words and int(c0.abs().sum()) == 0
        assert ws0.data_ptr() != ws1.data_ptr() and c0.data_ptr() != c1.data_ptr()


@pytest.mark.parametrize("m,n,default,persistent,walks", [
    (64, 28672, True, None, True), (64, 28672, False, None, False),     # TDX_GEMM_PERSIST=0: one tile per CTA
    (64, 28672, False, True, True), (64, 28672, True, False, False),    # an explicit choice of the call
    (1, 18945, True, None, True), (1, 18944, True, None, False), (129, 200, True, None, False),
])
def test_the_persistent_kernel_can_be_turned_off(m, n, default, persistent, walks, monkeypatch):
    taken = []

    class Ops:
        class linear_decode:
            default = staticmethod(lambda *args: taken.append("tiles"))

        def gemm_tn(self, *args):
            taken.append("tiles")

        def gemm_tn_persistent(self, *args):
            taken.append("walk")

    monkeypatch.setattr(gemm._lib, "ops", Ops)
    monkeypatch.setattr(gemm, "_PERSIST_DEFAULT", default)
    monkeypatch.setattr(gemm, "_workspace", lambda device: (None, None, None))
    a, w = torch.empty(m, 64, dtype=torch.bfloat16), torch.empty(1, 64, dtype=torch.bfloat16).expand(n, 64)
    gemm.linear(a, w, persistent=persistent)
    gemm.linear(a, w, torch.empty(m, n, dtype=torch.bfloat16), persistent=persistent)
    assert taken == ["walk" if walks else "tiles"] * 2


@pytest.mark.parametrize("m,n,k", [(64, 7168, 1024), (2, 256, 4096)])
def test_block_scaled_output_type_may_be_none(m, n, k, monkeypatch):
    """``out_dtype=None`` means torch's default type, for the kernel that allocates its output natively and for the other."""
    made = []

    class Ops:
        class gemm_scaled_call:
            default = staticmethod(lambda a, w, out_dtype, *rest: made.append(out_dtype))

        def gemm_tn(self, w, a, out, *rest):
            made.append(out.dtype)

    monkeypatch.setattr(gemm._lib, "ops", Ops)
    monkeypatch.setattr(gemm, "_workspace", lambda device: (None, None, None))
    a, w = torch.empty(m, k, dtype=torch.float8_e4m3fn), torch.empty(n, k, dtype=torch.float8_e4m3fn)
    gemm.linear_fp8_blockscaled(a, torch.empty(m, k // 128), w, torch.empty(n // 128, k // 128), out_dtype=None)
    assert made == [torch.float32]


def test_remembered_splits_follow_the_value_of_max_len(monkeypatch):
    """Split counts are remembered by their sizes. A length held in a tensor counts by its value, not by the tensor."""
    seen = []

    class Ops:
        class attention_decode_call:
            default = staticmethod(lambda q, k, v, lens, part, nsplit, *rest: seen.append(nsplit))

    monkeypatch.setattr(attention._lib, "ops", Ops)
    monkeypatch.setattr(attention, "_resident_clusters", lambda device: {})
    monkeypatch.setattr(attention, "_partial", lambda device, floats: None)
    monkeypatch.setattr(gemm, "_workspace", lambda device: (None, None, None))
    q, cache, length = torch.empty(1, 8, 128), torch.empty(1, 1, 1, 128).expand(1, 8192, 1, 128), torch.tensor(128)
    for n in (128, 8192):
        length.fill_(n)
        attention.decode_attention(q, cache, cache, None, length)
        attention.decode_attention(q, cache, cache, None, n)
    assert seen[0] == seen[1] == 1 and seen[2] == seen[3] > 8


@pytest.mark.parametrize("m,n,k,few", [
    (1, 8192, 1024, True), (16, 8320, 1024, False), (17, 5120, 8192, True), (32, 5248, 8192, False),
    (33, 2560, 8192, True), (64, 2688, 8192, False), (65, 1280, 4096, True), (128, 1408, 4096, False),
    (129, 1280, 1024, True), (129, 1792, 1024, False), (256, 4736, 4096, True), (257, 4736, 4096, False),
    (192, 2688, 8192, True), (192, 2816, 8192, False), (512, 640, 14336, True), (512, 768, 14336, False),
])
def test_few_tiles_of_a_block_scaled_product(m, n, k, few):
    assert gemm._few_scaled_tiles(m, n, k) == few
    if few and m > 128:      # its K pieces are resident, or it has none: they never meet in the scratch of the device
        tiles = -(-n // 128) * -(-m // 64)
        _, bn, splits = gemm.plan(m, n, k, 1, scaled=True)
        assert bn == 64 and (tiles <= SMS // 2 or splits == 1)
