"""The packed walk of the persistent kernels (causal calls of a few rounds): every item once, each block's longest first, and never worse than the
fixed order it replaces."""
import ctypes as C
import threading
import time

import pytest

from delta_matching_b200 import _lib

CTAS = 148


def _plan(heads, nblk, ctas=CTAS):
    first, items = (C.c_int32 * (ctas + 1))(), (C.c_int32 * (heads * nblk))()
    if not _lib.lib().dm_walk_plan(heads, nblk, ctas, first, items):
        return None
    assert first[0] == 0 and first[ctas] == heads * nblk
    return [list(items[first[c]:first[c + 1]]) for c in range(ctas)]


def _cost(i, heads, nblk):
    return nblk - i // heads + 2                             # its tiles, and two for what an item costs besides


def _snake(heads, nblk, ctas=CTAS):
    n = heads * nblk
    walk = [[r * ctas + (ctas - 1 - c if r & 1 else c) for r in range((n + ctas - 1) // ctas)] for c in range(ctas)]
    return [[i for i in w if i < n] for w in walk]


def _most(walk, heads, nblk):
    return max(sum(_cost(i, heads, nblk) for i in w) for w in walk)


# the fewest and the most items that are packed; one head of many blocks; many heads of two and three; other numbers of blocks to share among
@pytest.mark.parametrize("heads,nblk,ctas", [(9, 33, 148), (99, 3, 148), (50, 16, 148), (160, 5, 148), (1, 512, 148), (1, 781, 148), (329, 2, 148),
                                             (21, 22, 148), (16, 28, 148), (16, 30, 148), (100, 8, 148), (11, 61, 148), (1, 800, 160), (355, 2, 160),
                                             (107, 3, 160), (1, 11, 5), (38, 2, 5)])
def test_packed_walk(heads, nblk, ctas):
    plan, snake = _plan(heads, nblk, ctas), _snake(heads, nblk, ctas)
    assert plan is not None
    assert sorted(i for w in plan for i in w) == list(range(heads * nblk))
    assert all(w and w == sorted(w) for w in plan)                 # rank-major: longest first
    assert _most(plan, heads, nblk) < 0.97 * _most(snake, heads, nblk)


# where the mean block is above the load that a packing has to come down to; where every packing found is; more items or blocks than the lists hold
@pytest.mark.parametrize("heads,nblk,ctas", [(48, 6, 148), (32, 16, 148), (1, 800, 148), (2, 400, 148), (7, 9, 5), (1, 3, 2), (160, 5, 160),
                                             (149, 1, 148), (75, 2, 148), (1, 801, 148), (9, 89, 148), (21, 22, 161)])
def test_fixed_order(heads, nblk, ctas):
    assert _plan(heads, nblk, ctas) is None


def test_where_it_is_used():
    assert all(_plan(h, n) for h, n in ((21, 22), (1, 512), (8, 44), (16, 28)))
    assert _plan(8, 4) is None                               # one round
    assert _plan(128, 32) is None                            # many rounds: the fixed order is as good
    assert _plan(149, 1) is None                             # lengths that do not differ
    worst = max(sum(_cost(i, 1, 512) for i in w) for w in _plan(1, 512))
    assert worst <= 1.01 * sum(_cost(i, 1, 512) for i in range(512)) / CTAS


def _seconds_a_call(shapes):
    """Of the entry point alone, over all shapes in turn; the best of several rounds."""
    f, first, items = _lib.lib().dm_walk_plan, (C.c_int32 * (CTAS + 1))(), (C.c_int32 * 800)()
    best = 1.0
    for _ in range(6):
        t = time.perf_counter()
        for heads, nblk in shapes:
            f(heads, nblk, CTAS, first, items)
        best = min(best, (time.perf_counter() - t) / len(shapes))
    return best


def test_programs_of_many_lengths():
    """Some dozens of shapes in turn are all kept, those with a plan beside those without, and a shape that is not kept costs about as much as a
    launch: 1 and 5 to 10 us here, 200 to 600 where a fill scans every size for every block.  The limits leave an order for a busy machine."""
    long = [(1, n) for n in range(300, 360)]
    assert _seconds_a_call(long) < 20e-6
    assert _seconds_a_call([s for n in range(60) for s in (long[n], (128 + n, 2))]) < 20e-6
    assert _seconds_a_call([(1, n) for n in range(260, 400)]) < 80e-6


def test_threads():
    shapes = [(1, n) for n in range(250, 420, 2)] + [(h, n) for h in (2, 7, 8, 16, 21, 34) for n in range(150 // h + 1, 150 // h + 20, 2)]
    want, got = [_plan(*s) for s in shapes], {}
    assert sum(w is not None for w in want) > 64 and None in want           # more with a plan than are kept, and some without

    def ask(i):
        order = list(range(i, len(shapes))) + list(range(i))
        got[i] = all([_plan(*shapes[j]) == want[j] for j in order])

    threads = [threading.Thread(target=ask, args=(17 * i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 4 and all(got.values())


# one group of one head; groups of four and seven query heads, batches, the stale delta; items of 1 to 88 tiles (dV in two windows)
@pytest.mark.gpu
@pytest.mark.parametrize("B,N,H,Hk,mode", [(1, 512, 75, 75, "matched"), (1, 1536, 34, 34, "matched"), (1, 2816, 21, 21, "matched"),
                                           (1, 5632, 8, 8, "matched"), (2, 3584, 8, 2, "matched"), (2, 3584, 8, 2, "stale"),
                                           (3, 2816, 7, 1, "stale"), (5, 11264, 1, 1, "stale"), (5, 11264, 1, 1, "matched")])
def test_packed_calls_give_the_bits_of_calls_in_the_fixed_order(B, N, H, Hk, mode):
    import torch
    from delta_matching_b200 import dm_attn_func
    rep, nblk = H // Hk, N // 128
    assert _plan(B * H, nblk)
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v, do = (torch.randn(B, N, h, 128, generator=g, device="cuda", dtype=torch.bfloat16) for h in (H, Hk, Hk, H))

    def run(b, lo, hi):                                      # KV groups lo .. hi - 1 of some sequences
        x = [t[b, :, lo * r:hi * r].contiguous().requires_grad_() for t, r in ((q, rep), (k, 1), (v, 1))]
        o = dm_attn_func(*x, causal=True, mode=mode)
        return (o.detach(), *torch.autograd.grad(o, x, do[b, :, lo * rep:hi * rep].contiguous()))

    whole, step = run(slice(0, B), 0, Hk), max(1, CTAS // (nblk * rep))      # groups whose items are one round, or one group
    assert _plan(step * rep, nblk) is None
    for b in range(B):
        for lo in range(0, Hk, step):
            hi = min(Hk, lo + step)
            for a, c, r in zip(whole, run(slice(b, b + 1), lo, hi), (rep, rep, 1, 1)):
                assert torch.equal(a[b:b + 1, :, lo * r:hi * r], c)
