"""A state's steps, objective, transpose product and TDRK4 / RK4 tangent carry the same bits
in a batch of any size: chains of either cluster shape, one or two rounds of them, and
launches per pass with either row tile (only the tangents of one Lawson-RK4 or adaptive
linearisation change layout with the batch, in FP64 at n = 128)."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200.synthetic import initial_condition

pytestmark = pytest.mark.gpu
BATCHES = (1, 9, 17, 40, 80)


def _fields(n, dtype, B):
    return torch.as_tensor(np.stack([initial_condition(b, n) for b in range(B)]), dtype=dtype, device="cuda")


def _first(out):
    return {k: torch.as_tensor(v).cpu()[0] for k, v in out.items()}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [64, 128])
def test_first_of_a_batch(cuda, n, dtype):
    pd = E.make_param_dict(n, 1 / 40, 1 / 45, forcing="kolmogorov+", data_type=dtype, num_checkpoints=1, ministeps=3, steps=3,
                           shift_reflect_ny=1, rot=True)
    pda = E.make_param_dict(n, 1 / 40, 1 / 45, forcing="kolmogorov+", data_type=dtype, shift_reflect_ny=0, rot=False,
                            adaptive_dict={"atol": 1e-6 if dtype == torch.float64 else 1e-3, "checkpoints": 1,
                                           "max_steps_per_checkpoint": 16})
    x = {"fields": _fields(n, dtype, 1)[0], "T": 0.01, "sx": 0.2}
    objs = {mode: E.Objective(pd, mode) for mode in ("Lawson_RK4", "TDRK4", "RK4", "Lawson_RK6")}
    want = {}
    for B in BATCHES:
        f = _fields(n, dtype, B)
        T, sx = torch.full((B,), 0.02, dtype=torch.float64), torch.full((B,), 0.1, dtype=torch.float64)
        got = {mode: {"f": E.integrate(torch.fft.rfft2(f[:1]).repeat(B, 1, 1, 1), 0.01, 3, pd, mode)[0].cpu()} for mode in objs}
        got["adaptive"] = _first(E.objective_RPO({"fields": f, "T": T, "sx": sx}, pda, "Lawson_RK43"))
        v = {"fields": f, "T": T, "sx": sx}
        for mode, obj in objs.items():
            got["vjp " + mode] = _first(E.vjp(obj, x)[1](v)[0])
            if mode != "Lawson_RK4":
                got["jvp " + mode] = _first(obj.jvp(x, v))
        for name, out in got.items():
            for k, t in out.items():
                if B == BATCHES[0]:
                    want[name, k] = t
                else:
                    assert torch.equal(t, want[name, k]), (name, k, B)
