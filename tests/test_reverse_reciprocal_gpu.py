"""The reverse sweep's reciprocal keeps the accuracy of two Newton steps: before the last
rounding its relative error is 2^-80, so that a result differs from the correctly rounded
1 / x only where 1 / x lies within 2^-27 ulp of a rounding boundary (one operand in 2^26)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_reverse_reciprocal_is_almost_always_correctly_rounded(gpu_lib):
    from mosscap_b200 import capi
    rng = np.random.default_rng(3)
    n = 1 << 20
    x = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-300, 301, n) * rng.choice([-1.0, 1.0], n)
    xt = torch.tensor(x, device="cuda")
    out = torch.empty_like(xt)
    capi.check(gpu_lib.mc_debug_reverse_reciprocal(ctypes.c_void_p(xt.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                                   n, None), "mc_debug_reverse_reciprocal")
    torch.cuda.synchronize()
    wrong = int((out.cpu().numpy() != 1.0 / x).sum())
    assert wrong <= 4, wrong  # 2^20 / 2^26 expected
