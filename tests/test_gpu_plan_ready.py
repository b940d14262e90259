"""A plan's lists are complete when its creation returns, whichever stream executes it."""
import numpy as np
import pytest

import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.test_gpu_tiles import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [sht.Mode.PLAIN_FP64, sht.Mode.BATCHED_FP64, sht.Mode.SPLIT])
def test_creation_returns_with_its_stream_idle(ctx, mode):
    # 540 x 540 C blocks: past the grids that are planned from counts, and enough work-list items that
    # the kernels after the last read-back take longer than the return to the caller
    import torch
    rng = np.random.default_rng(2)
    n, k = [2] * 540, [2, 3]
    A = W.build_tensor(rng, [n, k], lambda c: np.ones(len(c[0]), bool), None, "normal")
    B = W.build_tensor(rng, [k, n], lambda c: np.ones(len(c[0]), bool), None, "normal")
    a, b = dev(ctx, A), dev(ctx, B)
    s = torch.cuda.Stream()
    for _ in range(3):
        c = dev(ctx, W.empty_tensor([n, n]))
        plan = sht.Plan(ctx, "ik, kj -> ij", a, b, c, mode=mode, stream=s)
        assert s.query()
        assert plan.report()["npairs"] == 2 * 540 * 540
        plan.close()
