"""Operands whose free or contracted modes lie apart or in another order: copied into the order that the
tile kernel reads, or gathered by it; bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu
MODES = [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64]

# both operands, A only, B only; free modes apart; contracted modes apart, in another order, not the
# fastest first
EXPRS = ["kil, ljk -> ji", "ikjl, lkm -> imj", "kli, lkj -> ij", "akb, kc -> abc", "abdc, cdij -> abij", "iPa, Pjb -> ijab"]


def case(expr, occ, seed=1, odd=False):
    rng = np.random.default_rng(seed)
    ta, tb, tc = expr.replace(" ", "").replace("->", ",").split(",")
    four = max(len(ta), len(tb)) > 3
    pick = [1, 2, 5] if odd else [2, 5, 9] if four else [3, 8, 17]
    sizes = {c: list(map(int, rng.choice(pick, 3 if four else 4))) for c in ta + tb}
    some = lambda c: rng.random(len(c[0])) < occ  # noqa: E731
    return tuple(W.build_tensor(rng, [sizes[c] for c in s], some, None, "normal") for s in (ta, tb, tc))


@pytest.mark.parametrize("expr", EXPRS)
@pytest.mark.parametrize("mode", MODES)
def test_contract_and_plan(ctx, expr, mode):
    # many pairs per block (copied operands) and few (gathered ones), every alpha and beta kind; the plan is
    # executed again after the operands' values changed
    for occ, odd in ((0.6, False), (0.2, False), (0.6, True)):
        A, B, C0 = case(expr, occ, odd=odd)
        a, b = dev(ctx, A), dev(ctx, B)
        for alpha, beta in ((1.0, 0.0), (-0.75, 0.5), (0.0, 2.0)):
            c = dev(ctx, C0)
            sht.contract(ctx, expr, alpha, a, b, beta, c, mode=mode)
            want = oracle.contract(expr, alpha, host(A), host(B), beta, host(C0))
            assert np.array_equal(c.get_sparse_info()[0], want.C.ids)
            assert bits_equal(c.download(), want.C.data)
        c = dev(ctx, C0)
        plan = sht.Plan(ctx, expr, a, b, c, mode=mode)
        if mode == sht.Mode.BATCHED_FP64:
            plan.autotune()
        for turn in range(2):
            plan.execute(1.0, 0.0)
            want = oracle.contract(expr, 1.0, host(A), host(B), 0.0, host(C0))
            assert bits_equal(c.download(), want.C.data)
            A.data[:] = A.data[::-1].copy()
            B.data *= -0.5
            if len(A.ids):
                a.upload(A.data)
            if len(B.ids):
                b.upload(B.data)
        plan.close()


@pytest.mark.parametrize("mode", MODES)
def test_graph_replay_takes_new_values(ctx, mode):
    import torch
    A, B, C0 = case("kil, ljk -> ji", 0.6)
    a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, C0)
    plan = sht.Plan(ctx, "kil, ljk -> ji", a, b, c, mode=mode)
    s = torch.cuda.Stream()
    for _ in range(2):
        plan.execute(1.0, 0.0, stream=s, graph=True)
        s.synchronize()
        want = oracle.contract("kil, ljk -> ji", 1.0, host(A), host(B), 0.0, host(C0))
        assert bits_equal(c.download(), want.C.data)
        A.data *= 3.0
        a.upload(A.data)
    plan.close()


@pytest.mark.parametrize("mode", MODES)
def test_without_memory_for_the_copies(mode):
    # the pool has room for the plan and not for the operands' copies (1.2 MB and 1.2 MB)
    expr = "kil, ljk -> ji"
    rng = np.random.default_rng(3)
    n = [20] * 3
    A = W.build_tensor(rng, [n, n, n], lambda c: rng.random(len(c[0])) < 0.7, None, "normal")
    B = W.build_tensor(rng, [n, n, n], lambda c: rng.random(len(c[0])) < 0.7, None, "normal")
    C0 = W.build_tensor(rng, [n, n], lambda c: np.ones(len(c[0]), bool), None, "normal")
    want = oracle.contract(expr, 1.0, host(A), host(B), 0.5, host(C0))
    ctx = sht.Context(16 << 20)
    a, b = dev(ctx, A), dev(ctx, B)
    for free in (300 << 10, 1500 << 10, 8 << 20):
        c = dev(ctx, C0)
        hold = ctx.allocate(ctx.get_free_mem() - free)
        sht.contract(ctx, expr, 1.0, a, b, 0.5, c, mode=mode)
        assert bits_equal(c.download(), want.C.data)
        ctx.free(hold)
    del a, b, c
    ctx.close()


def test_served_together_with_linear_requests(ctx):
    jobs = []
    for n, expr in enumerate(["kil, ljk -> ji", "ik, kj -> ij", "abdc, cdij -> abij", "iPa, Pjb -> ijab"]):
        A, B, C0 = case(expr, 0.5, seed=n + 5)
        jobs.append((expr, A, B, C0, dev(ctx, A), dev(ctx, B), dev(ctx, C0), 0.0 if n == 3 else 1.5))
    with sht.Server(ctx) as srv:
        ids = [srv.submit(e, alpha, a, b, 0.5, c) for e, _, _, _, a, b, c, alpha in jobs]
        for i in ids:
            srv.wait(i, 60)
    for e, A, B, C0, _, _, c, alpha in jobs:
        want = oracle.contract(e, alpha, host(A), host(B), 0.5, host(C0))
        assert bits_equal(c.download(), want.C.data)


def test_operand_reserved_larger_after_the_plan(ctx):
    # the plan's copy of the operand has the size of its pattern at creation
    A, B, C0 = case("kil, ljk -> ji", 0.6)
    a, b, c = dev(ctx, A), dev(ctx, B), dev(ctx, C0)
    plan = sht.Plan(ctx, "kil, ljk -> ji", a, b, c)
    a.reserve_all()
    with pytest.raises(sht.ShtError) as ei:
        plan.execute(1.0, 0.0)
    assert ei.value.status == sht.Status.ERR_STATE
    plan.close()
