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


@pytest.mark.parametrize("mode", FP64)
def test_contract_times_out_and_recovers(one_poll, mode):
    ctx = one_poll
    w = W.c1(seed=14, scale=0.25, occupancy=0.4)
    A, B, C = dev(ctx, w.A), dev(ctx, w.B), dev(ctx, w.C)
    sht.contract(ctx, w.expr, 1.0, A, B, 0.0, C, mode=mode)
    assert "split" not in timeout(ctx.stream_sync)
    ctx.stream_sync()  # reported once
    ctx.set_wait_limit(0)
    sht.contract(ctx, w.expr, 1.0, A, B, 0.0, C, mode=mode)
    want = oracle.contract(w.expr, 1.0, host(w.A), host(w.B), 0.0, host(w.C))
    assert bits_equal(C.download(), want.C.data)


def test_plan_and_graph_report_an_earlier_timeout(one_poll):
    import torch
    ctx = one_poll
    w = W.c1(seed=14, scale=0.25, occupancy=0.4)
    A, B, C = dev(ctx, w.A), dev(ctx, w.B), dev(ctx, w.C)
    plan = sht.Plan(ctx, w.expr, A, B, C, mode=sht.Mode.BATCHED_FP64)
    s = torch.cuda.Stream()
    for graph in (False, True):
        plan.execute(1.0, 0.0, stream=s)
        s.synchronize()
        timeout(plan.execute, 1.0, 0.0, stream=s, graph=graph)
    ctx.set_wait_limit(0)
    plan.execute(1.0, 0.0, stream=s, graph=True)
    s.synchronize()
    ctx.stream_sync()
    want = oracle.contract(w.expr, 1.0, host(w.A), host(w.B), 0.0, host(w.C))
    assert bits_equal(C.download(), want.C.data)


def test_stack_of_large_blocks_times_out_and_recovers(one_poll):
    import torch
    ctx = one_poll
    sa, sb, sc, n = [13, 32, 64], [9, 25, 64], [13, 9, 32, 25], 64
    k = sht.Kernel(ctx, "iaP, jbP -> ijab", sa, sb, sc)
    g = torch.Generator().manual_seed(3)
    a, b = (torch.rand(n * int(np.prod(x)), dtype=torch.float64, generator=g).cuda() for x in (sa, sb))
    c = torch.zeros(n * int(np.prod(sc)), dtype=torch.float64, device="cuda")
    k.call(a, b, c, n)
    torch.cuda.synchronize()
    timeout(k.call, a, b, c, n)
    ctx.set_wait_limit(0)
    k.call(a, b, c, n)
    torch.cuda.synchronize()
    want = torch.einsum("zPai, zPbj -> zbaji", a.view(n, *sa[::-1]), b.view(n, *sb[::-1])).reshape(-1)
    # one rounding per product and sum of 64 terms on either side, all below 1
    assert (c - want).abs().max().item() <= 2 * 64 * 64 * 2.0 ** -53


def test_served_request_times_out(one_poll):
    ctx = one_poll
    w = W.c1(seed=14, scale=0.25, occupancy=0.4)
    A, B, C = dev(ctx, w.A), dev(ctx, w.B), dev(ctx, w.C)
    with sht.Server(ctx) as srv:
        msg = timeout(srv.wait, srv.submit(w.expr, 1.0, A, B, 0.0, C), 60)
        assert "tensor cores" not in msg
        ctx.set_wait_limit(0)
        srv.wait(srv.submit(w.expr, 1.0, A, B, 0.0, C), 60)
    want = oracle.contract(w.expr, 1.0, host(w.A), host(w.B), 0.0, host(w.C))
    assert bits_equal(C.download(), want.C.data)
