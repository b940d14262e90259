"""Plans whose C blocks are all at most 8 x 8 or 16 x 16 (a warp for each) at the edges of that path, bit for bit against
the oracle (the kernel does the oracle's fma chain, so the bound is zero)."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu

# expression, extents and number of blocks per mode: one element; every row, column and contracted extent
# around a step of four and of sixteen; both modes fastest; several modes an index; modes apart; 255 and 256
# C blocks, and the 316 that blocks of 9 and more need at K 15; a contracted extent of 65, and 17 rows, take the
# general kernel
CASES = [
    ("ik, kj -> ij", {"i": ([1], 16), "k": ([1], 5), "j": ([1], 16)}),
    ("ik, kj -> ij", {"i": ([1, 7, 8], 17), "k": ([1, 3, 4, 5, 8], 9), "j": ([1, 2, 7, 8], 16)}),
    ("ki, jk -> ji", {"i": ([1, 7, 8], 17), "k": ([1, 3, 4, 5, 33], 9), "j": ([1, 2, 7, 8], 16)}),
    ("ik, kj -> ij", {"i": ([8], 16), "k": ([63, 64], 4), "j": ([5], 16)}),
    ("ik, kj -> ij", {"i": ([8], 16), "k": ([64, 65], 4), "j": ([5], 16)}),
    ("ik, kj -> ij", {"i": ([9, 8], 18), "k": ([5], 4), "j": ([5], 18)}),
    ("ik, kj -> ij", {"i": ([1, 9, 15, 16], 20), "k": ([1, 13, 15], 5), "j": ([7, 8, 9, 16], 19)}),
    ("ki, jk -> ji", {"i": ([16], 25), "k": ([15, 16, 17, 33, 64], 5), "j": ([2, 16], 25)}),
    ("ik, kj -> ij", {"i": ([9], 15), "k": ([15], 3), "j": ([16], 21)}),
    ("ik, kj -> ij", {"i": ([9, 17], 25), "k": ([15], 3), "j": ([16], 25)}),
    ("ik, kj -> ij", {"i": ([3], 15), "k": ([5], 4), "j": ([6], 17)}),
    ("ijl, lkm -> kimj", {"i": ([1, 2], 5), "j": ([2, 4], 4), "l": ([3, 6], 4), "k": ([2, 3], 4), "m": ([1, 2], 4)}),
    ("ilj, kl -> jik", {"i": ([1, 2], 6), "j": ([2, 4], 6), "l": ([3, 6], 4), "k": ([5, 8], 8)}),
    ("kil, ljk -> ji", {"k": ([2, 5], 3), "i": ([6, 8], 16), "l": ([3, 7], 3), "j": ([4, 8], 17)}),
]


@pytest.mark.parametrize("expr,modes", CASES)
@pytest.mark.parametrize("mode", [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64])
def test_small_blocks(ctx, expr, modes, mode):
    import torch
    rng = np.random.default_rng(31)
    sizes = {c: list(map(int, rng.choice(e, n))) for c, (e, n) in modes.items()}
    ta, tb, tc = expr.replace(" ", "").replace("->", ",").split(",")
    some = lambda occ: lambda c: rng.random(len(c[0])) < occ  # noqa: E731
    A, B = (W.build_tensor(rng, [sizes[c] for c in s], some(0.7), None, "normal") for s in (ta, tb))
    C0 = W.build_tensor(rng, [sizes[c] for c in tc], some(0.8), None, "normal")
    a, b = dev(ctx, A), dev(ctx, B)
    for alpha, beta, eps in ((1.0, 0.0, 0.0), (-0.75, 0.5, 0.0), (1.5, 1.0, 1.0), (0.0, -2.0, 0.0), (1.0, -0.0, 0.0)):
        c = dev(ctx, C0)
        sht.contract(ctx, expr, alpha, a, b, beta, c, eps, mode=mode)
        want = oracle.contract(expr, alpha, host(A), host(B), beta, host(C0), eps=eps)
        assert np.array_equal(c.get_sparse_info()[0], want.C.ids)
        assert bits_equal(c.download(), want.C.data), (alpha, beta)
    c = dev(ctx, C0)
    plan = sht.Plan(ctx, expr, a, b, c, mode=mode)
    s = torch.cuda.Stream()
    for graph in (False, True):
        plan.execute(1.0, 0.0, stream=s, graph=graph)
        s.synchronize()
        want = oracle.contract(expr, 1.0, host(A), host(B), 0.0, host(C0))
        assert bits_equal(c.download(), want.C.data)
    plan.close()


def test_values_past_a_block_do_not_spread(ctx):
    # infinities and NaN in neighbouring blocks and rows stay with the elements that they belong to
    rng = np.random.default_rng(32)
    si, sk, sj = [3, 5] * 10, [2, 5, 3], [6, 1] * 10
    full = lambda c: np.ones(len(c[0]), bool)  # noqa: E731
    A, B = W.build_tensor(rng, [si, sk], full, None, "normal"), W.build_tensor(rng, [sk, sj], full, None, "normal")
    A.data[rng.integers(0, A.data.size, 20)] = np.inf
    B.data[rng.integers(0, B.data.size, 20)] = np.nan
    Ch = W.empty_tensor([si, sj])
    c = dev(ctx, Ch)
    sht.contract(ctx, "ik, kj -> ij", 1.0, dev(ctx, A), dev(ctx, B), 0.0, c)
    want = oracle.contract("ik, kj -> ij", 1.0, host(A), host(B), 0.0, host(Ch)).C.data
    got = c.download()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(want).any() and np.isfinite(want).any()
    ok = ~np.isnan(want)
    assert bits_equal(got[ok], want[ok])
