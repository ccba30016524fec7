"""The cluster-resident chains are what the default route launches in their batch ranges
(an equality of two routes says nothing if both are the same one), and the control blocks
that an adaptive chain leaves (every CTA decides on a copy, the first writes it back) carry
the statistics of the launches per stage for every candidate."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200 import context
from ecs_mhd_2d_b200.synthetic import initial_condition

pytestmark = pytest.mark.gpu


def _counted(monkeypatch, n, pd, run, env):
    """(result, launches) of run() by a context made with `env`."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    context.clear_cache()
    try:
        run()   # buffers, graphs
        ctx = context.get_context(pd, n, torch.float64)
        before = ctx.lib.ecs_launch_count(ctx.handle)
        out = run()
        return out, ctx.lib.ecs_launch_count(ctx.handle) - before
    finally:
        monkeypatch.undo()
        context.clear_cache()


# one and two rounds of clusters of either shape on a B200
@pytest.mark.parametrize("n,B", [(64, 1), (64, 27), (64, 64), (128, 7), (128, 13), (128, 28)])
def test_adaptive_statistics(cuda, monkeypatch, n, B):
    pd = E.make_param_dict(n, 1 / 50, 1 / 50, forcing="kolmogorov+", shift_reflect_ny=1, rot=False,
                           adaptive_dict={"atol": 1e-6, "checkpoints": 2, "max_steps_per_checkpoint": 16})
    # from few attempts to more than the cap of 32: completed and not
    T = torch.linspace(0.02, 0.6, B, dtype=torch.float64) if B > 1 else torch.tensor([0.1], dtype=torch.float64)
    x = {"fields": torch.as_tensor(np.stack([initial_condition(i, n) for i in range(B)]), device="cuda"), "T": T, "sx": 0.2}

    def run():
        loss, infos = E.loss_RPO(x, pd, "Lawson_RK43")
        return torch.as_tensor(loss).cpu(), infos

    (got, infos), few = _counted(monkeypatch, n, pd, run, {})
    (want, want_infos), many = _counted(monkeypatch, n, pd, run, {"ECS_RK43CHAIN_MAXB": "0"})
    assert torch.equal(got, want) and infos == want_infos
    assert 4 * few < many, (few, many)


@pytest.mark.parametrize("n,B", [(64, 12), (128, 5)])
@pytest.mark.parametrize("call", ["integrate_Lawson_RK4", "integrate_RK4", "integrate_Lawson_RK6", "integrate_TDRK4",
                                  "vjp_Lawson_RK4", "jvp_TDRK4", "jvp_Lawson_RK43"])
def test_default_route(cuda, monkeypatch, call, n, B):
    kind, mode = call.split("_", 1)
    kw = dict(num_checkpoints=1, ministeps=20, shift_reflect_ny=0, rot=False) if mode != "Lawson_RK43" else \
        dict(shift_reflect_ny=0, rot=False, adaptive_dict={"atol": 1e-5, "checkpoints": 2, "max_steps_per_checkpoint": 16})
    pd = E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", **kw)
    f = np.stack([initial_condition(i, n) for i in range(B)])
    x = {"fields": torch.as_tensor(f[0], device="cuda"), "T": 0.05, "sx": 0.2}
    v = {"fields": torch.as_tensor(f, device="cuda"), "T": torch.full((B,), 0.1, dtype=torch.float64),
         "sx": torch.full((B,), 0.2, dtype=torch.float64)}
    fhat = torch.fft.rfft2(v["fields"]).contiguous()

    def run():
        if kind == "integrate":
            E.integrate(fhat, 0.05, 20, pd, mode)
            return
        obj = E.Objective(pd, mode)
        if kind == "vjp":
            E.vjp(obj, x)[1](v)
        else:
            obj.jvp(x, v)

    off = {"ECS_CHAIN_MAXB": "0", "ECS_RK4CHAIN_MAXB": "0", "ECS_RK43CHAIN_MAXB": "0"}
    few, many = (_counted(monkeypatch, n, pd, run, env)[1] for env in ({}, off))
    assert 2 * few < many, (few, many)


# FP32: more states than clusters that run at once on a B200, fewer than twice that
@pytest.mark.parametrize("n,B", [(64, 48), (128, 24)])
@pytest.mark.parametrize("mode", ["Lawson_RK4", "RK4", "Lawson_RK6", "TDRK4"])
def test_two_rounds_in_fp32(cuda, monkeypatch, mode, n, B):
    pd = E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", data_type=torch.float32)
    f = np.fft.rfft2(np.stack([initial_condition(i, n) for i in range(B)]))
    f = torch.as_tensor(f, device="cuda").to(torch.complex64)
    out = []
    for env in ({}, {"ECS_RK4CHAIN_MAXB": "0"}):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        context.clear_cache()
        try:
            E.integrate(f, 0.02, 18, pd, mode)
            ctx = context.get_context(pd, n, torch.float32)
            before = ctx.lib.ecs_launch_count(ctx.handle)
            got = E.integrate(f, 0.02, 18, pd, mode).cpu()
            out.append((got, ctx.lib.ecs_launch_count(ctx.handle) - before))
        finally:
            monkeypatch.undo()
            context.clear_cache()
    assert torch.equal(out[0][0], out[1][0]) and 2 * out[0][1] < out[1][1], [q[1] for q in out]
