"""How the attention backward hands out its work: every pair of (query head, query tile) that a K/V tile meets goes to one CTA, and the
cast adds exactly the parts that were written (host rule and index arithmetic of the kernels, without a GPU)."""
import random

import pytest

from context_parallelism_b200 import _native as nv


def _visible_tiles(nq, k0, k_off, causal):
    return nq - (min(nq, max(0, k_off + k0) // 128) if causal else 0)


@pytest.mark.parametrize("seed", range(40))
def test_parts_cover_the_sweep(seed):
    r = random.Random(seed)
    Hkv, G, B, D = r.choice([1, 2, 3]), r.choice([1, 2, 4]), r.choice([1, 2]), r.choice([64, 128])
    Tq, Tk = r.randint(1, 3000), r.randint(1, 3000)
    causal, k_off = r.random() < 0.7, r.choice([0, 0, 5, 128, 700])
    rule = nv.lib().cpb_flash_bwd_chunk(B, Tq, Tk, G * Hkv, Hkv, D, int(causal), k_off, 1)
    nq, n_kt = -(-Tq // 128), -(-Tk // 128)
    pairs = G * nq
    assert 0 <= rule <= pairs
    for chunk in {rule, 1, 2, r.randint(1, pairs + 3)} - {0}:
        parts = -(-pairs // chunk)
        done, written = {}, {}
        tiles = lambda c: sum(G * _visible_tiles(nq, kt * 128, k_off, causal) > c * chunk for kt in range(n_kt)) if causal else n_kt  # noqa: E731
        for i in range(Hkv * B * sum(tiles(c) for c in range(parts))):    # bwd_work()
            c = 0
            while i >= tiles(c) * Hkv * B:
                i, c = i - tiles(c) * Hkv * B, c + 1
            kt, hkv, b, it0 = i // (Hkv * B), i % Hkv, (i // Hkv) % B, c * chunk
            seen = _visible_tiles(nq, kt * 128, k_off, causal)
            assert it0 < seen * G
            written[kt, hkv, b] = written.get((kt, hkv, b), 0) + 1
            assert it0 // chunk == written[kt, hkv, b] - 1            # part numbers without gaps
            for it in range(it0, min(it0 + chunk, seen * G)):
                key = kt, hkv, b, it // seen, nq - seen + it % seen
                assert key not in done
                done[key] = True
        for kt in range(n_kt):
            seen = _visible_tiles(nq, kt * 128, k_off, causal)
            tile_parts = -(-(G * max(0, nq - max(0, k_off + kt * 128) // 128)) // chunk) if causal else parts
            for hkv in range(Hkv):
                for b in range(B):
                    assert written.get((kt, hkv, b), 0) == tile_parts
                    assert sum(k[:3] == (kt, hkv, b) for k in done) == seen * G if n_kt * Hkv * B < 12 else True
        assert len(done) == Hkv * B * G * sum(_visible_tiles(nq, kt * 128, k_off, causal) for kt in range(n_kt))


def test_tiles_with_a_part():
    """bwd_tiles() of the kernels is a count: the tiles that have a part are the first ones, and their number has a closed form."""
    r = random.Random(5)
    for _ in range(3000):
        nq, n_kt, G, chunk, k_off = r.randint(1, 40), r.randint(1, 40), r.randint(1, 6), r.randint(1, 60), r.choice([0, 1, 127, 128, 300, 6000])
        for c in range(-(-G * nq // chunk) + 1):
            want = [G * _visible_tiles(nq, kt * 128, k_off, True) > c * chunk for kt in range(n_kt)]
            last = nq - 1 - c * chunk // G
            end = 128 * last + 127 - k_off
            assert want == sorted(want, reverse=True) and sum(want) == (0 if last < 0 or end < 0 else min(n_kt, end // 128 + 1))


def test_rule_leaves_long_even_sweeps_alone():
    f = nv.lib().cpb_flash_bwd_chunk
    assert f(1, 131072, 131072, 32, 8, 64, 1, 0, 1) == 0 and f(1, 32768, 32768, 32, 8, 128, 1, 0, 1) == 0
    assert 0 < f(2, 4096, 4096, 6, 2, 64, 1, 0, 1) < 96               # 128 CTAs, the longest of 96 pairs
    assert f(1, 0, 5, 2, 1, 64, 1, 0, 1) == 0 and f(1, 5, 5, 2, 0, 64, 1, 0, 1) == 0
