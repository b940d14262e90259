"""Plans built from counts (small block grids) against the general path's rules: pair list, result
pattern and work list, through the oracle, at the edges of that path."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu


def tensor(rng, sizes, occ):
    return W.build_tensor(rng, sizes, lambda c: rng.random(len(c[0])) < occ, None, "normal")


# expression, blocks per mode: orders and modes in every position, one cell, a contracted grid at and
# past the path's 512 keys, a C grid past its 2^18 cells (the last two take the general path)
CASES = [
    ("ik, kj -> ij", {"i": 1, "k": 1, "j": 1}, 1.0),
    ("ik, kj -> ij", {"i": 40, "k": 33, "j": 65}, 0.3),
    ("kil, ljk -> ji", {"k": 4, "i": 9, "l": 5, "j": 7}, 0.4),
    ("ijl, lk -> kji", {"i": 6, "j": 7, "l": 8, "k": 9}, 0.3),
    ("abcd, cdij -> abij", {"a": 3, "b": 4, "c": 3, "d": 2, "i": 3, "j": 2}, 0.5),
    ("ik, kj -> ij", {"i": 3, "k": 512, "j": 2}, 0.6),
    ("ik, kj -> ij", {"i": 3, "k": 513, "j": 2}, 0.6),
    ("ik, kj -> ij", {"i": 520, "k": 2, "j": 520}, 0.02),
]


@pytest.mark.parametrize("expr,blocks,occ", CASES)
@pytest.mark.parametrize("mode", [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64, sht.Mode.SPLIT])
@pytest.mark.parametrize("eps", [0.0, 1.0])
def test_pairs_pattern_values(ctx, expr, blocks, occ, mode, eps):
    rng = np.random.default_rng(41)
    sizes = {c: list(map(int, rng.integers(1, 4, n))) for c, n in blocks.items()}
    ta, tb, tc = expr.replace(" ", "").replace("->", ",").split(",")
    A, B = tensor(rng, [sizes[c] for c in ta], occ), tensor(rng, [sizes[c] for c in tb], occ)
    C0 = tensor(rng, [sizes[c] for c in tc], 0.1)
    for Ch, beta in ((W.empty_tensor(C0.block_sizes), 0.0), (C0, -0.5), (C0, 0.0)):
        a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, Ch)
        plan = sht.Plan(ctx, expr, a, b, c, eps, mode=mode)
        want = oracle.contract(expr, 1.0, host(A), host(B), beta, host(Ch), eps=eps)
        assert np.array_equal(plan.pairs(), want.pairs)
        ids, offs, _ = c.get_sparse_info()
        assert np.array_equal(ids, want.C.ids) and np.array_equal(offs, want.C.offsets)
        assert plan.report()["flops"] == pytest.approx(want.flops, rel=1e-12)
        if not len(Ch.ids):
            assert not c.download().any()  # a plan's new blocks start zero-filled
        plan.execute(1.0, beta)
        d = dev(ctx, Ch)
        rep = sht.contract(ctx, expr, 1.0, a, b, beta, d, eps, mode=mode)
        assert rep["npairs"] == len(want.pairs) and rep["nblocks_c"] == len(want.C.ids)
        for t in (c, d):
            assert np.array_equal(t.get_sparse_info()[0], want.C.ids)
            got = t.download()
            if mode == sht.Mode.SPLIT:
                assert np.linalg.norm(got - want.C.data) <= 1e-12 * max(np.linalg.norm(want.C.data), 1e-300)
            else:
                assert bits_equal(got, want.C.data)


def test_growth_orders_after_earlier_work(ctx):
    # a second product adds blocks to C while the first may still be running, on another stream; the
    # host index of the grown C is read back afterwards
    import torch
    rng = np.random.default_rng(5)
    sizes = {c: [32] * 6 for c in "ijk"}
    A1, B = tensor(rng, [sizes["i"], sizes["k"]], 0.3), tensor(rng, [sizes["k"], sizes["j"]], 0.4)
    A2 = tensor(rng, [sizes["i"], sizes["k"]], 0.5)
    a1, a2, b = dev(ctx, A1), dev(ctx, A2), dev(ctx, B)
    Ch = W.empty_tensor([sizes["i"], sizes["j"]])
    w1 = oracle.contract("ik, kj -> ij", 1.0, host(A1), host(B), 0.0, host(Ch))
    w2 = oracle.contract("ik, kj -> ij", 2.0, host(A2), host(B), 1.0, w1.C)
    assert len(w2.C.ids) > len(w1.C.ids) > 0
    s = torch.cuda.Stream()
    for mode in (sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64):
        for _ in range(5):
            c = dev(ctx, Ch)
            sht.contract(ctx, "ik, kj -> ij", 1.0, a1, b, 0.0, c, mode=mode, stream=s)
            sht.contract(ctx, "ik, kj -> ij", 2.0, a2, b, 1.0, c, mode=mode, stream=s)
            s.synchronize()
            assert np.array_equal(c.get_sparse_info()[0], w2.C.ids)
            assert bits_equal(c.download(), w2.C.data)
