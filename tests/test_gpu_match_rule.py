"""Plans by counting and by sorting, on both sides of the rule that chooses between them, against the oracle."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu


# many pairs of few C blocks and of many; a C that exists already is planned by sorting from fewer on
@pytest.mark.parametrize("n,k", [((60, 60), 250), ((70, 70), 300), ((400, 400), 2)])
@pytest.mark.parametrize("mode", [sht.Mode.PLAIN_FP64, sht.Mode.SPLIT])
def test_both_sides(ctx, n, k, mode):
    rng = np.random.default_rng(12)
    si, sj, sk = (list(map(int, rng.integers(1, 3, x))) for x in (*n, k))
    full = lambda c: np.ones(len(c[0]), bool)  # noqa: E731
    A, B = (W.build_tensor(rng, s, full, None, "normal") for s in ([si, sk], [sk, sj]))
    Ch = W.empty_tensor([si, sj])
    want = oracle.contract("ik, kj -> ij", 1.0, host(A), host(B), 0.0, host(Ch))
    a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, Ch)
    for turn in range(2):  # into a new C, then into one that holds the pattern
        rep = sht.contract(ctx, "ik, kj -> ij", 1.0, a, b, 0.0, c, mode=mode)
        assert rep["npairs"] == len(want.pairs) and rep["flops"] == pytest.approx(want.flops, rel=1e-12)
        ids, offs, _ = c.get_sparse_info()
        assert np.array_equal(ids, want.C.ids) and np.array_equal(offs, want.C.offsets)
        got = c.download()
        if mode == sht.Mode.SPLIT:
            assert np.linalg.norm(got - want.C.data) <= 1e-12 * np.linalg.norm(want.C.data)
        else:
            assert bits_equal(got, want.C.data)
    plan = sht.Plan(ctx, "ik, kj -> ij", a, b, c, mode=mode)
    assert np.array_equal(plan.pairs(), want.pairs)
    plan.close()
