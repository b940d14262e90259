"""A burst whose results do not all fit the pool: requests that find no memory while finished
ones still hold it are planned again as their callers free the results, and a request that can
never fit fails."""
import time

import numpy as np
import pytest

import shtensor_b200 as sht
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu

NB, BS = 20, 100  # C: 20 x 20 blocks of 100 x 100 doubles, 32 MB


def panels(ctx, seed):
    rng = np.random.default_rng(seed)
    wide, one = np.full(NB, BS, np.int32), np.full(1, BS, np.int32)
    A, B = sht.Tensor(ctx, [wide, one]), sht.Tensor(ctx, [one, wide])
    A.reserve([np.arange(NB), np.zeros(NB, np.int64)])
    B.reserve([np.zeros(NB, np.int64), np.arange(NB)])
    A.upload(rng.standard_normal(NB * BS * BS))
    B.upload(rng.standard_normal(NB * BS * BS))
    return A, B, lambda: sht.Tensor(ctx, [wide, wide])


def test_burst_larger_than_the_pool_waits_for_its_callers():
    ctx = sht.Context(256 << 20)
    A, B, make = panels(ctx, 3)
    want = make()
    sht.contract(ctx, "ij, jk -> ik", 1.0, A, B, 0.0, want, mode=sht.Mode.PLAIN_FP64)
    bits = want.download()
    del want
    with sht.Server(ctx) as srv:
        cs = [make() for _ in range(16)]  # 512 MB of results
        rids = [srv.submit("ij, jk -> ik", 1.0, A, B, 0.0, C) for C in cs]
        time.sleep(0.4)  # the first results fill the pool before any is collected
        for i, rid in enumerate(rids):
            srv.wait(rid, 60)
            assert bits_equal(cs[i].download(), bits)
            cs[i] = None
        st = srv.stats()
    assert st["completed"] == 16 and st["failed"] == 0
    assert st["deferrals"] > 0
    del A, B
    ctx.close()


def test_a_result_larger_than_the_pool_fails():
    ctx = sht.Context(24 << 20)
    A, B, make = panels(ctx, 4)
    C = make()
    with sht.Server(ctx) as srv:
        rid = srv.submit("ij, jk -> ik", 1.0, A, B, 0.0, C)
        with pytest.raises(sht.ShtError) as ei:
            srv.wait(rid, 60)
        assert ei.value.status == sht.Status.ERR_OOM
    del ei, A, B, C
    ctx.close()
