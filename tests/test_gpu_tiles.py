"""The FP64 tile kernel at the edges of its tiles, chunks and 16-byte copies, bit for bit against the
oracle (the kernel does the oracle's fma chain, so the bound is zero)."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu
MODES = [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64]


def dev(ctx, h):
    t = sht.Tensor(ctx, h.block_sizes)
    t.reserve(h.index_lists() if len(h.ids) else [[] for _ in h.block_sizes])
    return t.upload(h.data) if h.nnz else t


def host(t):
    return oracle.HostTensor(t.block_sizes, t.ids, t.offsets, t.data)


def check(ctx, expr, sizes, mode, alpha, beta, occ=0.7, seed=1):
    rng = np.random.default_rng(seed)
    ta, tb, tc = expr.replace(" ", "").replace("->", ",").split(",")
    keep = lambda c: rng.random(len(c[0])) < occ  # noqa: E731
    A = W.build_tensor(rng, [sizes[c] for c in ta], keep, None, "normal")
    B = W.build_tensor(rng, [sizes[c] for c in tb], keep, None, "normal")
    Ch = W.build_tensor(rng, [sizes[c] for c in tc], keep, None, "normal")
    a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, Ch)
    sht.contract(ctx, expr, alpha, a, b, beta, c, mode=mode)
    want = oracle.contract(expr, alpha, host(A), host(B), beta, host(Ch))
    assert np.array_equal(c.get_sparse_info()[0], want.C.ids)
    assert bits_equal(c.download(), want.C.data)


# rows fastest / k fastest for either operand; the last two gather (contracted or free modes apart)
EXPRS = ["ik, jk -> ij", "ki, kj -> ij", "ik, kj -> ji", "ki, jk -> ij", "kil, ljk -> ji", "ikj, km -> imj"]


@pytest.mark.parametrize("expr", EXPRS)
@pytest.mark.parametrize("mode", MODES)
def test_tile_and_chunk_edges(ctx, expr, mode):
    # row, column and contracted extents on both sides of 8, 32 and 64; blocks start at odd elements
    three = len(expr.split(",")[0].strip()) == 3
    rows = [1, 9, 13] if three else [1, 7, 31, 32, 33, 63, 64, 65, 129]
    ks = [1, 3, 5] if three else [1, 4, 5, 31, 32, 33, 67]
    sizes = {"i": rows, "j": rows[::-1], "k": ks, "l": [2, 7], "m": [5, 64, 3]}
    check(ctx, expr, sizes, mode, 1.0, 0.0)
    check(ctx, expr, sizes, mode, -0.75, 0.5, seed=2)


@pytest.mark.parametrize("mode", MODES)
def test_many_pairs_per_block(ctx, mode):
    # one C block fed by more pairs than the pair ring or a warp's batch holds
    check(ctx, "ik, kj -> ij", {"i": [40], "j": [17], "k": [3] * 90}, mode, 1.0, 1.0, occ=1.0)


@pytest.mark.parametrize("mode", MODES)
def test_special_values_propagate(ctx, mode):
    rng = np.random.default_rng(3)
    sizes = {"i": [33, 5], "j": [9, 20], "k": [6, 35]}
    A = W.build_tensor(rng, [sizes["i"], sizes["k"]], lambda c: np.ones(len(c[0]), bool), None, "normal")
    B = W.build_tensor(rng, [sizes["k"], sizes["j"]], lambda c: np.ones(len(c[0]), bool), None, "normal")
    A.data[[0, 50, 333]] = [np.inf, -0.0, np.nan]
    B.data[[3, 70]] = [-np.inf, 0.0]
    C = W.empty_tensor([sizes["i"], sizes["j"]])
    a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, C)
    sht.contract(ctx, "ik, kj -> ij", 1.0, a, b, 0.0, c, mode=mode)
    want = oracle.contract("ik, kj -> ij", 1.0, host(A), host(B), 0.0, host(C)).C.data
    got = c.download()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert bits_equal(np.nan_to_num(got, nan=0.0, posinf=1e300, neginf=-1e300),
                      np.nan_to_num(want, nan=0.0, posinf=1e300, neginf=-1e300))
