"""How the block-scaled GEMM divides its work: every K block of every tile is done exactly once, and the scratch
has a slice for every piece."""
import pytest

from torch_dist_ext_b200 import _lib


def _work(workers, full_rounds, parts, per, ntiles, kb):
    """next_work of gemm_scaled.cu for every worker: (worker, tile, kb0, kb1)."""
    out = []
    for w in range(workers):
        n = 0
        while n < full_rounds or parts == 1:
            if w + n * workers >= ntiles:
                break
            out.append((w, w + n * workers, 0, kb))
            n += 1
        t = full_rounds * workers + w // parts
        if parts > 1 and t < ntiles:
            out.append((w, t, w % parts * per, min(kb, w % parts * per + per)))
    return out


@pytest.mark.parametrize("sms", [148, 132, 20])
@pytest.mark.parametrize("m", [1, 64, 128, 129, 300, 2048, 8192])
@pytest.mark.parametrize("n", [128, 1280, 7168, 8192, 28672])
@pytest.mark.parametrize("kb", [1, 2, 8, 28, 64, 224])
def test_every_block_once(sms, m, n, kb):
    ctas, workers, full, parts, per, slices, counters = _lib.ops().gemm_scaled_plan(m, n, kb, sms, sms // 2, sms // 5, sms // 10)
    assert ctas == (2 if m > 128 else 1) and workers * ctas <= sms
    tiles = -(-m // (128 * ctas)) * -(-n // 256)
    assert parts == 1 or (tiles - full * (sms // ctas)) * parts <= sms // ctas
    done = {}
    for w, t, a, b in _work(workers, full, parts, per, tiles, kb):
        assert 0 <= t < tiles and 0 <= a < b <= kb
        for i in range(a, b):
            assert (t, i) not in done
            done[t, i] = w
        if ctas == 2 and (a, b) != (0, kb):
            assert (w * ctas + ctas) * 128 * 256 <= slices and (t - full * workers) * ctas + ctas <= counters
    assert len(done) == tiles * kb
    if ctas == 1:      # pieces of a decode tile are the CTAs of one cluster, and there are no full rounds before them
        assert parts in (1, 2, 4, 8) and (parts == 1 or (full == 0 and workers == tiles * parts)) and slices == 0
