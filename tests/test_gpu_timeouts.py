"""Bounded waits of the FP64 tile kernel: with a limit of one poll they run out, the call that follows
reports it once, and the context works on."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu

FP64 = [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64]


@pytest.fixture
def one_poll(ctx):
    ctx.stream_sync()
    ctx.set_wait_limit(1)
    yield ctx
    ctx.set_wait_limit(0)
    try:
        ctx.stream_sync()
    except sht.ShtError:
        pass  # a failed test leaves none of its errors behind


def timeout(call, *args, **kw):
    with pytest.raises(sht.ShtError) as ei:
        call(*args, **kw)
    assert ei.value.status == sht.Status.ERR_TIMEOUT
    return str(ei.value)


def long_waits(ctx):
    # one C block of 16 pairs, each of which takes its tile a hundred chunks: the roles that run ahead wait for
    # far longer than a poll
    rng = np.random.default_rng(3)
    A = W.build_tensor(rng, [[64], [3200] * 16], lambda c: np.ones(len(c[0]), bool), None, "normal")
    B = W.build_tensor(rng, [[3200] * 16, [64]], lambda c: np.ones(len(c[0]), bool), None, "normal")
    Ch = W.empty_tensor([[64], [64]])
    want = oracle.contract(EXPR, 1.0, host(A), host(B), 0.0, host(Ch))
    return dev(ctx, A), dev(ctx, B), dev(ctx, Ch), want.C.data


EXPR = "ik, kj -> ij"


@pytest.mark.parametrize("mode", FP64)
def test_contract_times_out_and_recovers(one_poll, mode):
    ctx = one_poll
    A, B, C, want = long_waits(ctx)
    sht.contract(ctx, EXPR, 1.0, A, B, 0.0, C, mode=mode)
    assert "split" not in timeout(ctx.stream_sync)
    ctx.stream_sync()  # reported once
    ctx.set_wait_limit(0)
    sht.contract(ctx, EXPR, 1.0, A, B, 0.0, C, mode=mode)
    assert bits_equal(C.download(), want)


def test_plan_and_graph_report_an_earlier_timeout(one_poll):
    import torch
    ctx = one_poll
    A, B, C, want = long_waits(ctx)
    plan = sht.Plan(ctx, EXPR, A, B, C, mode=sht.Mode.BATCHED_FP64)
    s = torch.cuda.Stream()
    for graph in (False, True):
        plan.execute(1.0, 0.0, stream=s)
        s.synchronize()
        timeout(plan.execute, 1.0, 0.0, stream=s, graph=graph)
    ctx.set_wait_limit(0)
    plan.execute(1.0, 0.0, stream=s, graph=True)
    s.synchronize()
    ctx.stream_sync()
    assert bits_equal(C.download(), want)


def test_stack_of_large_blocks_times_out_and_recovers(one_poll):
    # eight ops per resident CTA, each sixteen chunks long: tiles are claimed far ahead of their turn
    import torch
    ctx = one_poll
    n, m, K = 8 * 296, 64, 512
    k = sht.Kernel(ctx, EXPR, [m, K], [K, m], [m, m])
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = (torch.rand(n * m * K, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    c = torch.zeros(n * m * m, dtype=torch.float64, device="cuda")
    k.call(a, b, c, n)
    torch.cuda.synchronize()
    timeout(k.call, a, b, c, n)
    ctx.set_wait_limit(0)
    k.call(a, b, c, n)
    torch.cuda.synchronize()
    want = torch.bmm(b.view(n, m, K), a.view(n, K, m)).reshape(-1)
    # 512 products and sums on either side, each rounded once, all terms below 1
    assert (c - want).abs().max().item() <= 2 * K * K * 2.0 ** -53


def test_served_request_times_out(one_poll):
    ctx = one_poll
    A, B, C, want = long_waits(ctx)
    with sht.Server(ctx) as srv:
        msg = timeout(srv.wait, srv.submit(EXPR, 1.0, A, B, 0.0, C), 60)
        assert "tensor cores" not in msg
        ctx.set_wait_limit(0)
        srv.wait(srv.submit(EXPR, 1.0, A, B, 0.0, C), 60)
    assert bits_equal(C.download(), want)
