"""How the attention backward hands out its work: every pair of (query head, query tile) that a K/V tile meets goes to one CTA, and the
cast adds exactly the parts that were written (host rule and index arithmetic of the kernels, without a GPU)."""
import heapq
import random
import time

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


def _rule(B, Tq, Tk, Hq, Hkv, D, causal, k_off, local, sms):
    """cpb_flash_bwd_chunk() with every hand-out followed to its end."""
    nq, n_kt, G, hb = -(-Tq // 128), -(-Tk // 128), Hq // Hkv, Hkv * B
    if n_kt * hb > 16 * sms:
        return 0
    tile, start_end = (1.25, 11.0) if D == 64 else (1.9, 13.0)
    hidden = [(k_off + k * 128) // 128 if local else nq * k // n_kt for k in range(n_kt)]
    lens = [G * (nq - (min(nq, max(0, h)) if causal else 0)) for h in hidden]

    def finish(items):
        done, end = [0.0] * sms, 0.0
        for pairs in items:
            end = max(end, t := done[0] + start_end + pairs * tile)
            heapq.heapreplace(done, t)
        return end
    best, chunk = finish(n for _ in range(hb) for n in lens) * 0.97, 0
    for parts in range(1, 25):
        c = -(-G * nq // parts)
        if parts > 1 and c < 2:
            break
        written = sum(-(-n // c) if local else parts for n in lens)
        t = finish(min(n - at, c) for at in range(0, G * nq, c) for n in lens if n > at for _ in range(hb)) + (0.5 + written * hb * 128 * D * 2 * 8 / 4e6)
        if t < best:
            best, chunk = t, c
    return chunk


def test_rule_follows_only_what_can_win_and_finds_the_same():
    r = random.Random(11)
    f, sms = nv.lib().cpb_flash_bwd_chunk, 148                      # 148 without a GPU
    shapes = [(1, 32749, 32749, 4, 1, 128, 1, 0, 1), (2, 1000, 1000, 6, 2, 64, 1, 0, 1), (1, 8192, 16384, 8, 2, 64, 1, 0, 0), (1, 9000, 9000, 4, 1, 64, 0, 0, 1)]
    for _ in range(60):
        Hkv, T = r.choice([1, 2, 4]), int(2 ** r.uniform(0, 13.5))
        shapes.append((r.choice([1, 2]), T, r.choice([T, 2 * T]), r.choice([1, 2, 4]) * Hkv, Hkv, r.choice([64, 128]), r.randint(0, 1), r.choice([0, 0, 300]), r.randint(0, 1)))
    assert [f(*s) for s in shapes] == [_rule(*s, sms) for s in shapes]


@pytest.mark.parametrize("D", [64, 128])
def test_rule_takes_little_host_time(D):
    """A new shape is planned in front of its first launch: 25 hand-outs of 2048 CTAs took 15 ms."""
    f, took = nv.lib().cpb_flash_bwd_chunk, []
    for i in range(9):
        t = time.perf_counter()
        f(1, 32768 - i, 32768 - i, 32, 8, D, 1, 0, 1)
        took.append(time.perf_counter() - t)
    assert min(took) < 4e-3
