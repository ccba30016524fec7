"""Adaptive solves of more candidates than clusters that run at once: the default route
(k_rk43_chain in up to two rounds of clusters, then launches per stage) equals the
launches per stage bit for bit, statistics included."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200 import context
from ecs_mhd_2d_b200.synthetic import initial_condition

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, n, B, chain):
    if not chain:
        monkeypatch.setenv("ECS_RK43CHAIN_MAXB", "0")
    context.clear_cache()
    try:
        pd = E.make_param_dict(n, 1 / 50, 1 / 50, forcing="kolmogorov+", shift_reflect_ny=1, rot=False,
                               adaptive_dict={"atol": 1e-6, "checkpoints": 4, "max_steps_per_checkpoint": 16})
        fields = torch.as_tensor(np.stack([initial_condition(i, n) for i in range(B)]), device="cuda")
        T = torch.linspace(0.02, 0.3, B, dtype=torch.float64)   # from few to many attempts
        out = E.objective_RPO({"fields": fields, "T": T, "sx": 0.2}, pd, "Lawson_RK43")
        return out["fields"].cpu().clone()
    finally:
        monkeypatch.undo()
        context.clear_cache()


# either side of one and of two rounds of 8- and 16-warp clusters of a B200
@pytest.mark.parametrize("n,B", [(64, 16), (64, 27), (64, 37), (64, 64), (128, 8), (128, 13), (128, 28), (128, 29)])
def test_rounds_equal_launch_per_stage(cuda, monkeypatch, n, B):
    assert torch.equal(_solve(monkeypatch, n, B, True), _solve(monkeypatch, n, B, False))
