"""Kernel::call on blocks whose rows and columns both lie across C's order; bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu

# A and B of an op on both sides of 24 KB (3072 doubles), of two ops' buffers (100 KB) and of one's (200 KB);
# rows or columns of several modes in another order than C's
STACKS = [("Pia, Pjb -> abij", (8, 12, 16), (8, 12, 16)), ("Pia, Pjb -> abij", (8, 12, 16), (8, 13, 16)),
          ("Pai, Pbj -> ijab", (16, 20, 20), (16, 20, 20)), ("Pai, Pbj -> ijab", (16, 20, 20), (16, 21, 20)),
          ("Pia, Pjb -> abij", (32, 20, 20), (32, 20, 20)), ("Pia, Pjb -> abij", (32, 20, 20), (32, 21, 20)),
          ("ijk, kl -> jil", (9, 7, 12), (12, 11)), ("abcP, Pd -> cdba", (5, 3, 7, 9), (9, 10)),
          ("ijk, kl -> jli", (1, 17, 5), (5, 1))]


@pytest.mark.parametrize("expr,sa,sb", STACKS)
@pytest.mark.parametrize("ops,shift", [(1, 0), (5, 1), (149, 0)])
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
