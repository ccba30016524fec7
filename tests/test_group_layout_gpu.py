"""Tangent column passes in the group layout (two transforms per warp; FP64 at n = 128,
batches from ECS_GROUP_MINB on) against the warp layout, which every other size, type and
batch uses, and against the oracle's torch twin.

Tolerance against the warp layout: a transform of 128 points rounds to about
log2(128) 2^-53 = 8e-16 of its norm in either layout; a JVP of at most 40 stages runs two
transforms per direction and stage, so the two differ by at most 160 x 2 x 8e-16 = 2.6e-13
of the result if every rounding adds up: 3e-13.  Against the oracle: 1e-12, as in
test_jvp_gpu."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200 import context
from ecs_mhd_2d_b200.synthetic import initial_condition
from conftest import rel_l2
from test_jvp_gpu import TOL, TOL_43, oracle_jvp
import oracle as O

pytestmark = pytest.mark.gpu
N = 128
MODES = [
    ("Lawson_RK4", dict(num_checkpoints=1, ministeps=6, shift_reflect_ny=1, rot=False)),
    ("Lawson_RK43", dict(shift_reflect_ny=1, rot=True, adaptive_dict={"atol": 1e-5, "checkpoints": 2, "max_steps_per_checkpoint": 16})),
]


def _jvp(monkeypatch, minb, mode, kw, B):
    monkeypatch.setenv("ECS_GROUP_MINB", str(minb))
    monkeypatch.setenv("ECS_CHAIN_MAXB", "0")   # one launch per pass
    context.clear_cache()
    try:
        pd = E.make_param_dict(N, 1 / 40, 1 / 40, forcing="kolmogorov+", **kw)
        rng = np.random.default_rng(5)
        prim = {"fields": initial_condition(3, N), "T": 0.04, "sx": 0.3}
        du = np.stack([0.1 * initial_condition(30 + i, N) + 0.01 * rng.standard_normal((2, N, N)) for i in range(B)])
        dT, dsx = np.linspace(-0.9, 1.2, B), np.linspace(0.5, -0.4, B)
        obj = E.Objective(pd, mode)
        out = obj.jvp(dict(prim, fields=torch.as_tensor(prim["fields"], device="cuda")),
                      {"fields": torch.as_tensor(du, device="cuda"), "T": torch.tensor(dT), "sx": torch.tensor(dsx)})
        return {k: v.detach().cpu().numpy() for k, v in out.items()}, prim, du, dT, dsx
    finally:
        monkeypatch.undo()
        context.clear_cache()


@pytest.mark.parametrize("mode,kw", MODES)
@pytest.mark.parametrize("B", [1, 2, 16, 17])   # odd and even; the smallest batch of the layout and the next
def test_group_layout(cuda, monkeypatch, mode, kw, B):
    want, *_ = _jvp(monkeypatch, 1000, mode, kw, B)
    got, prim, du, dT, dsx = _jvp(monkeypatch, 1, mode, kw, B)
    for b in range(B):
        assert rel_l2(got["fields"][b], want["fields"][b]) < 3e-13, b
    b, tol = B - 1, TOL_43 if mode == "Lawson_RK43" else TOL
    pdt = O.make_param_dict(N, 1 / 40, 1 / 40, forcing="kolmogorov+", xp=O.TORCH, **kw)
    exact = oracle_jvp(prim["fields"], prim["T"], prim["sx"], du[b], dT[b], dsx[b], pdt, mode)
    assert rel_l2(got["fields"][b], exact["fields"]) < tol
    assert abs(float(got["T"][b]) - float(exact["T"])) <= tol * max(abs(float(exact["T"])), 1e-30) + 1e-18
