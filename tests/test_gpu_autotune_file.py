"""The autotuner's file: choices made for another set of tile shapes are not taken over."""
import numpy as np
import pytest

import shtensor_b200 as sht
from shtensor_b200 import workloads as W
from tests.test_gpu_tiles import dev

pytestmark = pytest.mark.gpu


def test_choices_for_other_shapes_are_tuned_again(tmp_path):
    import torch
    rng = np.random.default_rng(4)
    n = [64] * 4
    A = W.build_tensor(rng, [n, n], lambda c: np.ones(len(c[0]), bool), None, "normal")
    gpu = torch.cuda.get_device_name().replace(" ", "_")
    path = tmp_path / "tuned.txt"
    old = f"{gpu} 6,6,6 3\n"  # 128 x 16 tiles when it was written
    path.write_text(old)
    texts = []
    for _ in range(2):
        ctx = sht.Context(64 << 20)
        a, b, c = dev(ctx, A), dev(ctx, A), dev(ctx, W.empty_tensor([n, n]))
        plan = sht.Plan(ctx, "ik, kj -> ij", a, b, c, mode=sht.Mode.BATCHED_FP64)
        plan.autotune(str(path))
        texts.append(path.read_text())
        plan.close()
        del a, b, c
        ctx.close()
    assert texts[0].startswith(old) and len(texts[0].splitlines()) == 2  # tuned, and written beside it
    assert texts[1] == texts[0]  # and read the next time
