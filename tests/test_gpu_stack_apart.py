"""Kernel<double>::call on blocks whose modes lie apart, at the sizes where its kernels change over; bit for
bit against the oracle."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu

# A and B of an op on both sides of 24 KB (3072 doubles), of two ops' buffers (100 KB) and of one's (200 KB);
# C blocks of several tiles, which few ops leave to the tile kernel
STACKS = [("kil, ljk -> ji", (12, 13, 10), (10, 12, 12)), ("kil, ljk -> ji", (12, 13, 10), (10, 13, 12)),
          ("kil, ljk -> ji", (20, 16, 20), (20, 16, 20)), ("kil, ljk -> ji", (20, 16, 20), (20, 17, 20)),
          ("kil, ljk -> ji", (32, 20, 20), (20, 20, 32)), ("kil, ljk -> ji", (32, 20, 20), (20, 21, 32)),
          ("iPa, jPb -> ijab", (9, 15, 25), (8, 15, 10)), ("abcd, dcij -> abij", (10, 9, 8, 6), (6, 8, 9, 7))]


@pytest.mark.parametrize("expr,sa,sb", STACKS)
@pytest.mark.parametrize("ops,shift", [(1, 0), (3, 1), (311, 0)])
def test_stack(ctx, expr, sa, sb, ops, shift):
    import torch
    x, y, o = (s.strip() for s in expr.replace("->", ",").split(","))
    ext = dict(zip(x, sa)) | dict(zip(y, sb))
    sc = [ext[q] for q in o]
    rng = np.random.default_rng(ops)
    na, nb, nc = (int(np.prod(s)) for s in (sa, sb, sc))
    ha, hb, hc = (rng.standard_normal(ops * n) for n in (na, nb, nc))

    def on_device(v):  # starting `shift` elements into an allocation
        t = torch.full((v.size + shift + 8,), float("nan"), dtype=torch.float64, device="cuda")
        t[shift:shift + v.size] = torch.from_numpy(v).cuda()
        return t

    for alpha, beta in ((1.0, 0.0), (-1.25, 0.5)):
        tc = on_device(hc)
        sht.Kernel(ctx, expr, list(sa), list(sb), sc, alpha, beta).call(on_device(ha)[shift:], on_device(hb)[shift:],
                                                                        tc[shift:], ops)
        got = tc.cpu().numpy()
        assert np.isnan(got[:shift]).all() and np.isnan(got[shift + hc.size:]).all()
        for op in {0, ops // 2, ops - 1}:
            one = lambda h, n: h[op * n:(op + 1) * n].copy()  # noqa: E731
            want = oracle.kernel_xmm(expr, list(sa), list(sb), sc, alpha, beta, one(ha, na), one(hb, nb), one(hc, nc), 1)
            assert bits_equal(got[shift + op * nc:shift + (op + 1) * nc], want)


@pytest.mark.parametrize("ops", [148, 149, 296, 300, 444, 445])
def test_fp32_shapes_around_a_few_ops_per_sm(ctx, ops):
    # the shape and the warps change with the ops for each SM (148 of them)
    import torch
    for sa, sb in (((30, 60), (60, 30)), ((63, 51), (51, 10)), ((64, 16), (16, 64))):
        rng = np.random.default_rng(ops)
        a, b = (rng.standard_normal(ops * s[0] * s[1]).astype(np.float32) for s in (sa, sb))
        sc = [sa[0], sb[1]]
        c = torch.empty(ops * sc[0] * sc[1], dtype=torch.float32, device="cuda")
        sht.Kernel(ctx, "ik, kj -> ij", list(sa), list(sb), sc, dtype=np.float32).call(
            torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c, ops)
        want = oracle.kernel_xmm("ik, kj -> ij", list(sa), list(sb), sc, 1.0, 0.0, a, b,
                                 np.zeros(c.numel(), np.float32), ops)
        assert bits_equal(c.cpu().numpy(), want)
