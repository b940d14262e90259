"""Kernel::call of a few products whose C blocks are far larger than A and B; bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu

# C blocks that are shared among CTAs: outer products, one group more than a CTA's warps take (64 x 65), groups
# that the CTAs do not divide, FP64 products above 100 KB with one buffer
STACKS = [("ik, kj -> ij", (143, 5), (5, 288)), ("ik, kj -> ji", (248, 4), (4, 196)), ("ik, kj -> ij", (64, 3), (3, 65)),
          ("ik, kj -> ij", (301, 1), (1, 299)), ("Pia, Pjb -> abij", (4, 29, 26), (4, 28, 20)),
          ("iaP, jbP -> ijab", (13, 29, 2), (12, 25, 2)), ("iPa, jPb -> ijab", (9, 40, 18), (8, 40, 10))]


@pytest.mark.parametrize("expr,sa,sb", STACKS)
@pytest.mark.parametrize("ops,shift", [(1, 0), (22, 1), (147, 0), (148, 0), (297, 0)])
@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_stack(ctx, expr, sa, sb, ops, shift, dt):
    import torch
    x, y, o = (s.strip() for s in expr.replace("->", ",").split(","))
    ext = dict(zip(x, sa)) | dict(zip(y, sb))
    sc = [ext[q] for q in o]
    rng = np.random.default_rng(ops)
    na, nb, nc = (int(np.prod(s)) for s in (sa, sb, sc))
    ha, hb, hc = (rng.standard_normal(ops * n).astype(dt) for n in (na, nb, nc))

    def on_device(v):  # starting `shift` elements into an allocation
        h = np.full(v.size + shift + 8, np.nan, dt)
        h[shift:shift + v.size] = v
        return torch.from_numpy(h).cuda()

    for alpha, beta in ((1.0, 0.0), (-1.25, 0.5)):
        tc = on_device(hc)
        sht.Kernel(ctx, expr, list(sa), list(sb), sc, alpha, beta, dtype=dt).call(
            on_device(ha)[shift:], on_device(hb)[shift:], tc[shift:], ops)
        got = tc.cpu().numpy()
        assert np.isnan(got[:shift]).all() and np.isnan(got[shift + hc.size:]).all()
        for op in {0, ops // 2, ops - 1}:
            one = lambda h, n: h[op * n:(op + 1) * n].copy()  # noqa: E731
            want = oracle.kernel_xmm(expr, list(sa), list(sb), sc, alpha, beta, one(ha, na), one(hb, nb), one(hc, nc), 1)
            assert bits_equal(got[shift + op * nc:shift + (op + 1) * nc], want)
