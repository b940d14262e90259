"""Kernel<T>::call at the edges of its kernels' tiles and of the shapes each takes, bit for bit against
the oracle (the same fma chain per element, so the bound is zero)."""
import numpy as np
import pytest

import oracle
import shtensor_b200 as sht
from tests.bits import bits_equal

pytestmark = pytest.mark.gpu

SHAPES = [
    # one element, one fragment and its neighbours, groups of 32 x 16 and their neighbours
    ("ik, kj -> ij", [1, 1], [1, 1], 3),
    ("ik, kj -> ij", [8, 4], [4, 8], 5),
    ("ik, kj -> ij", [9, 5], [5, 7], 301),
    ("ik, kj -> ji", [33, 7], [7, 17], 40),
    ("ki, jk -> ij", [6, 31], [16, 6], 1000),
    ("kil, ljk -> ji", [3, 5, 7], [7, 9, 3], 77),
    ("ikl, lkmj -> mij", [5, 6, 7], [7, 6, 3, 4], 20),
    ("ijl, lk -> ijk", [13, 9, 11], [11, 15], 700),
    # both blocks just within, and just beyond, what a CTA stages (24 KB in FP64, in FP32)
    ("ik, kj -> ij", [48, 32], [32, 48], 9),
    ("ik, kj -> ij", [48, 33], [33, 48], 9),
    ("ik, kj -> ij", [64, 48], [48, 64], 3),
    ("ki, kj -> ij", [49, 65], [49, 66], 3),
    # large blocks: tiles of 64 x 64 and remainders
    ("iaP, jbP -> ijab", [13, 32, 64], [9, 25, 64], 2),
    ("kil, ljk -> ji", [9, 70, 8], [8, 65, 9], 2),
]


@pytest.mark.parametrize("expr,sa,sb,nops", SHAPES)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("alpha,beta,shift", [(1.0, 0.0, 0), (-0.75, 0.5, 1), (0.0, 2.0, 3)])
def test_shapes_bit_exact(ctx, expr, sa, sb, nops, dtype, alpha, beta, shift):
    import torch
    left, out = expr.replace(" ", "").split("->")
    x, y = left.split(",")
    ext = dict(zip(x, sa)) | dict(zip(y, sb))
    sc = [ext[c] for c in out]
    rng = np.random.default_rng(17)
    a, b, c = (rng.uniform(-1, 1, nops * int(np.prod(s))).astype(dtype) for s in (sa, sb, sc))
    want = oracle.kernel_xmm(expr, sa, sb, sc, alpha, beta, a, b, c.copy(), nops)
    k = sht.Kernel(ctx, expr, sa, sb, sc, alpha, beta, dtype=dtype)

    def on_device(v):  # starting `shift` elements into an allocation
        t = torch.full((v.size + shift + 8,), float("nan"), dtype=torch.from_numpy(v[:1]).dtype, device="cuda")
        t[shift:shift + v.size] = torch.from_numpy(v).cuda()
        return t

    ta, tb, tc = on_device(a), on_device(b), on_device(c)
    k.call(ta[shift:], tb[shift:], tc[shift:], nops)
    got = tc.cpu().numpy()
    assert bits_equal(got[shift:shift + c.size], want)
    assert np.isnan(got[:shift]).all() and np.isnan(got[shift + c.size:]).all()  # nothing written outside
