"""A PDE filter where the device has memory for one right-hand side's workspace (64
bytes a node) but not for two: created all the same, with the same results."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_filter_with_memory_for_one_right_hand_side(gpu):
    from topopt_in_petsc_transient_gb300 import Filter
    n = (160, 96, 96)
    nel, nn = int(np.prod(n)), 161 * 97 * 97
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(nel, dtype=torch.float64, device="cuda", generator=g)
    df, dg = -x ** 4, torch.full((nel,), 1.0 / nel, dtype=torch.float64, device="cuda")

    def gradients():
        f = Filter(*n, 2, 2.0)
        a, b = df.clone(), dg.clone()
        torch.cuda.synchronize()
        f.Gradients(x, x, a, 1, b, False, 1.0, 0.5)
        return a, b
    ref = gradients()
    torch.cuda.empty_cache()
    outs = [torch.empty(nel, dtype=torch.float64, device="cuda") for _ in range(6)]  # room for the clones
    del outs
    # staging buffers (5 columns), half of the pair's workspace and 48 MB stay free
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (64 * nn + 5 * 8 * nel + (48 << 20)), dtype=torch.uint8, device="cuda")
    try:
        got = gradients()
    finally:
        del hold
        torch.cuda.empty_cache()
    for a, b in zip(ref, got):
        assert torch.equal(a, b)
