"""The choice of tiles of the one-rank GEMM launches (csrc/gemm_local.cu), on the host alone: the estimate is that of the
longest unit when the tiles are dealt out one by one as the kernel does it, and making the choice takes no longer for a
launch of many tiles than for one of few."""
import ctypes as C
import random
import time

import pytest

from rtp_b200.ops import _lib


def plan(jobs, n_sm=148, policy=-1):
    f = _lib.lib().rtp_lint_local_plan
    f.argtypes = [C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int), C.POINTER(C.c_longlong)]
    arr = (C.c_int * (4 * len(jobs)))(*[int(v) for j in jobs for v in j])
    out = (C.c_longlong * 64)()
    return f, (n_sm, policy, len(jobs), arr, out)


def backward(M, i, o):
    return [(o, i, M, 1), (M, i, o, 0)]      # dW with the column sums of dy, dx


@pytest.mark.parametrize("policy", [-1, 0, 1])
def test_estimate_is_the_longest_unit(policy):
    rng = random.Random(policy)
    few = 0
    for _ in range(300):
        jobs = [(rng.randint(1, 6000), 8 * rng.randint(1, 400), rng.randint(1, 9000), rng.random() < 0.4)
                for _ in range(rng.choice([1, 1, 2, 2, 3, 8]))]
        n_sm = rng.choice([148, 148, 132, 7])
        f, args = plan(jobs, n_sm, policy)
        n = f(*args)
        out = args[4]
        assert n == len(jobs) + sum(bool(j[3]) for j in jobs)
        units, tiles = out[1], [(out[3 + 2 * q], out[4 + 2 * q]) for q in range(n)]
        assert [c for c, _ in tiles] == sorted((c for c, _ in tiles), reverse=True)
        total = sum(k for _, k in tiles)
        if total > 8 * units:
            assert out[0] == sum(c * k for c, k in tiles) // units + tiles[0][0] // 2 + out[2]
            continue
        few += 1
        load, t = [0] * units, 0
        for cost, count in tiles:
            for _ in range(count):
                r, u = divmod(t, units)
                load[units - 1 - u if r & 1 else u] += cost
                t += 1
        assert out[0] == max(load) + out[2]
    assert few > 50


@pytest.mark.parametrize("tokens,i,o", [(1, 2048, 2048), (8, 2048, 8192), (100, 2048, 8192), (64, 4096, 4096)])
def test_weight_gradients_of_few_tokens_take_wide_tiles(tokens, i, o):
    """A tile of one or two k-blocks takes as long as its epilogue, which a narrower tile hardly shortens."""
    f, args = plan(backward(tokens, i, o))
    n = f(*args)
    most = max(args[4][4 + 2 * q] for q in range(n))
    assert most <= (o // 128) * (i // 128)


def test_choice_is_as_quick_for_many_tiles():
    def took(jobs):
        f, args = plan(jobs)
        best = 1.0
        for _ in range(400):
            t = time.perf_counter()
            f(*args)
            best = min(best, time.perf_counter() - t)
        return best
    small = took(backward(256, 256, 256))
    for M, i, o in [(1024, 2048, 2048), (16384, 256, 256), (36864, 288, 64), (4096, 2048, 2048)]:
        assert took(backward(M, i, o)) < 2 * small + 5e-7, (M, i, o)
