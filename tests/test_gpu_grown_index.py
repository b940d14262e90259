"""A C whose pattern a contraction grew: its index and its blocks are complete when the call returns,
by an error too, and reading the index back neither races nor waits for the caller's stream."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.bits import bits_equal
from tests.test_gpu_tiles import dev, host

pytestmark = pytest.mark.gpu

EXPR = "ik, kj -> ij"
BUSY = 100_000_000  # cycles that keep a stream busy (50 ms at 2 GHz)


def full(rng, *nblk):
    return W.build_tensor(rng, [[8] * n for n in nblk], lambda c: np.ones(len(c[0]), bool), None, "normal")


def test_growth_is_complete_when_the_call_runs_out_of_memory():
    # A split contraction that adds blocks to C while the caller's stream is busy, in a pool left with a
    # little more memory at each try: some tries grow C and then find no room for their records.
    # Operands: 1024 blocks each, whose slices take 36.7 MB; 16384 pairs, whose records take most of
    # the rest.
    import torch
    rng = np.random.default_rng(7)
    A, B = full(rng, 16, 64), full(rng, 64, 16)
    C0 = W.build_tensor(rng, [[8] * 16, [8] * 16], lambda c: (c[0] + c[1]) % 2 == 0, None, "normal")
    grown = np.zeros((16, 16, 8, 8))
    for (i, j), blk in zip(((int(n) % 16, int(n) // 16) for n in C0.ids), C0.data.reshape(-1, 8, 8)):
        grown[j, i] = blk
    s = torch.cuda.Stream()
    ctx = sht.Context(64 << 20)
    a, b = dev(ctx, A), dev(ctx, B)
    seen = set()
    for free in range(36 << 20, 41 << 20, 64 << 10):
        c = dev(ctx, C0)
        hold = ctx.allocate(ctx.get_free_mem() - free)
        with torch.cuda.stream(s):
            torch.cuda._sleep(BUSY // 4)
        err = None
        try:
            sht.contract(ctx, EXPR, 1.0, a, b, 1.0, c, mode=sht.Mode.SPLIT, stream=s)
        except sht.ShtError as e:
            assert e.status == sht.Status.ERR_OOM
            err = e
        # the caller's stream may still be busy; nothing of C is pending on it after an error
        if err is None:
            s.synchronize()
        ids, offs, rows = c.get_sparse_info()
        got = c.download()
        s.synchronize()
        ctx.free(hold)
        if err is None:
            seen.add("done")
            break
        if len(ids) == len(C0.ids):
            seen.add("unchanged")
            assert np.array_equal(ids, C0.ids) and bits_equal(got, C0.data)
        else:
            seen.add("grown")
            assert np.array_equal(ids, np.arange(256)) and np.array_equal(offs, 64 * np.arange(256))
            assert np.array_equal(rows, 16 * np.arange(16))
            assert bits_equal(got, grown.reshape(-1))
    assert "grown" in seen and "done" in seen, seen
    del a, b, c
    ctx.close()


def test_split_growth_orders_after_earlier_work(ctx):
    # the second product moves C's blocks while the first may still write them
    import torch
    rng = np.random.default_rng(6)
    sizes = [[32] * 6, [32] * 6]

    def some(occ):
        return W.build_tensor(rng, sizes, lambda c: rng.random(len(c[0])) < occ, None, "normal")
    A1, A2, B = some(0.3), some(0.5), some(0.4)
    w1 = oracle.contract(EXPR, 1.0, host(A1), host(B), 0.0, host(W.empty_tensor(sizes)))
    w2 = oracle.contract(EXPR, 2.0, host(A2), host(B), 1.0, w1.C)
    assert len(w2.C.ids) > len(w1.C.ids) > 0
    a1, a2, b = dev(ctx, A1), dev(ctx, A2), dev(ctx, B)
    s = torch.cuda.Stream()
    for _ in range(5):
        c = dev(ctx, W.empty_tensor(sizes))
        with torch.cuda.stream(s):
            torch.cuda._sleep(BUSY // 50)
        sht.contract(ctx, EXPR, 1.0, a1, b, 0.0, c, mode=sht.Mode.SPLIT, stream=s)
        sht.contract(ctx, EXPR, 2.0, a2, b, 1.0, c, mode=sht.Mode.SPLIT, stream=s)
        s.synchronize()
        assert np.array_equal(c.get_sparse_info()[0], w2.C.ids)
        assert np.linalg.norm(c.download() - w2.C.data) <= 1e-12 * np.linalg.norm(w2.C.data)


def test_server_and_owner_read_a_grown_index_at_once(ctx):
    # a grown tensor is submitted as an operand, and its owner reads its index while the server's loop
    # reads the same index back for planning
    rng = np.random.default_rng(8)
    n, k = [2] * 100, [3]
    A = W.build_tensor(rng, [n, k], lambda c: np.ones(len(c[0]), bool), None, "normal")
    B = W.build_tensor(rng, [k, n], lambda c: np.ones(len(c[0]), bool), None, "normal")
    V = W.build_tensor(rng, [n, k], lambda c: np.ones(len(c[0]), bool), None, "normal")
    a, b, v = dev(ctx, A), dev(ctx, B), dev(ctx, V)
    w1 = oracle.contract(EXPR, 1.0, host(A), host(B), 0.0, host(W.empty_tensor([n, n])))
    w2 = oracle.contract(EXPR, 1.0, oracle.HostTensor([n, n], w1.C.ids, w1.C.offsets, w1.C.data), host(V), 0.0,
                         host(W.empty_tensor([n, k])))
    ds = [dev(ctx, W.empty_tensor([n, n])) for _ in range(40)]
    for d in ds:
        sht.contract(ctx, EXPR, 1.0, a, b, 0.0, d)
    ctx.stream_sync()
    with sht.Server(ctx) as srv:
        for d in ds:
            e = dev(ctx, W.empty_tensor([n, k]))
            rid = srv.submit(EXPR, 1.0, d, v, 0.0, e)
            ids, offs, _ = d.get_sparse_info()
            assert np.array_equal(ids, w1.C.ids) and np.array_equal(offs, w1.C.offsets)
            srv.wait(rid, 60)
            assert bits_equal(e.download(), w2.C.data)


@pytest.mark.parametrize("mode", [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64])
def test_grown_operand_does_not_wait_for_the_stream(ctx, mode):
    # D = A B grows D; E = D A is then planned and queued while the stream is still busy
    import torch
    rng = np.random.default_rng(9)
    A = full(rng, 6, 6)
    a = dev(ctx, A)
    w1 = oracle.contract(EXPR, 1.0, host(A), host(A), 0.0, host(W.empty_tensor(A.block_sizes)))
    w2 = oracle.contract(EXPR, 1.0, oracle.HostTensor(A.block_sizes, w1.C.ids, w1.C.offsets, w1.C.data), host(A), 0.0,
                         host(W.empty_tensor(A.block_sizes)))
    s = torch.cuda.Stream()
    for cycles in (1000, 4 * BUSY):  # the first turn loads the kernels
        d, e = dev(ctx, W.empty_tensor(A.block_sizes)), dev(ctx, W.empty_tensor(A.block_sizes))
        sht.contract(ctx, EXPR, 1.0, a, a, 0.0, d, mode=mode, stream=s)
        s.synchronize()
        with torch.cuda.stream(s):
            torch.cuda._sleep(cycles)
        sht.contract(ctx, EXPR, 1.0, d, a, 0.0, e, mode=mode, stream=s)
        busy = not s.query()
        s.synchronize()
        assert bits_equal(e.download(), w2.C.data)
    assert busy
