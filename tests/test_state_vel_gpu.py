"""state_vel on full rfft2 arrays, and the comparison of forcings behind it."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
import oracle as O
from ecs_mhd_2d_b200 import context
from ecs_mhd_2d_b200.synthetic import initial_condition
from conftest import rel_l2


# The derivative is a sum of products of transforms of n points: about 4 log2(n) roundings
# of the largest terms (2^-53 or 2^-24 each), times the cancellation between them (below
# 100 for these states).
@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 4e-13), (torch.float32, 2e-4)])
@pytest.mark.parametrize("n,B,diss", [(64, 1, True), (64, 5, False), (128, 1, False), (128, 3, True), (256, 2, True)])
def test_state_vel_matches_oracle(cuda, n, B, diss, dtype, tol):
    fields = np.stack([initial_condition(i, n) for i in range(B)])
    pd = E.make_param_dict(n, 1 / 40, 1 / 50, forcing="kolmogorov+", data_type=dtype)
    opd = O.make_param_dict(n, 1 / 40, 1 / 50, forcing="kolmogorov+")
    f = np.fft.rfft2(fields)
    f[..., 1::7, n // 2] = 1.0   # outside the box: not read
    got = E.state_vel(torch.as_tensor(f, device="cuda").to(context.complex_of(dtype)), pd, diss).cpu().numpy()
    box = np.abs(np.fft.fftfreq(n, 1 / n))[:, None] < n / 3
    box = box & (np.arange(n // 2 + 1) < n / 3)[None]
    assert not got[..., ~box].any()
    for b in range(B):
        want = O.state_vel(np.where(box, f[b], 0), opd, diss)
        assert rel_l2(got[b], np.where(box, want, 0)) < tol, b


def test_same_physics_compares_every_bit():
    n = 64
    a = E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+")
    same, other, zero = dict(a), dict(a), dict(a)
    same["forcing"] = a["forcing"].clone()
    other["forcing"] = a["forcing"].clone()
    other["forcing"][3, 5] = torch.nextafter(other["forcing"][3, 5], torch.tensor(9.0, dtype=torch.float64))
    zero["forcing"] = a["forcing"].clone()
    zero["forcing"][0, 0] = 0.0
    minus = dict(zero, forcing=zero["forcing"].clone())
    minus["forcing"][0, 0] = -0.0
    assert context.same_physics([a, same, dict(a)])
    assert not context.same_physics([a, same, other])
    assert not context.same_physics([zero, minus])
    assert not context.same_physics([a, dict(a, nu=0.5)])
    assert not context.same_physics([a, dict(a, forcing=None)])
    assert context.same_physics([dict(a, forcing=None), dict(a, forcing=None)])
