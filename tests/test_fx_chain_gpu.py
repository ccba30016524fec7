"""Cluster-resident steps of RK4, Lawson-RK6 and TDRK4 (k_fx_chain), and the recording
Lawson-RK4 steps of linearisations and batched gradients (k_rk4_chain), their adjoint
(k_adj_chain) and the tangents of TDRK4 steps (k_tdj_chain) equal the launches per pass bit
for bit."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200 import context
from ecs_mhd_2d_b200.synthetic import initial_condition

pytestmark = pytest.mark.gpu


def _both(monkeypatch, run, warps=0):
    out = []
    for chain in (True, False):
        monkeypatch.setenv("ECS_RK4CHAIN_MAXB", "64" if chain else "0")
        if chain and warps:
            monkeypatch.setenv("ECS_CHAIN_WARPS", str(warps))
        context.clear_cache()
        try:
            out.append(run())
        finally:
            monkeypatch.undo()
            context.clear_cache()
    return out


def _equal(a, b):
    if isinstance(a, torch.Tensor):
        assert torch.equal(a, b)
    elif isinstance(a, dict):
        for k in a:
            _equal(a[k], b[k])
    else:
        assert len(a) == len(b)
        for x, y in zip(a, b):
            _equal(x, y)


# 1 state, an odd batch, and more states than clusters that run at once; 1 step, and more than a graph's 16
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("mode", ["RK4", "Lawson_RK6", "TDRK4"])
@pytest.mark.parametrize("n,B,steps,warps", [(64, 1, 1, 8), (64, 3, 18, 16), (64, 40, 2, 0), (128, 1, 17, 8), (128, 3, 2, 16), (128, 17, 1, 0)])
def test_integrate(cuda, monkeypatch, mode, n, B, steps, warps, dtype):
    pd = E.make_param_dict(n, 1 / 40, 1 / 50, forcing="kolmogorov+", data_type=dtype)
    f = np.fft.rfft2(np.stack([initial_condition(i, n) for i in range(B)]))
    f = torch.as_tensor(f, device="cuda").to(context.complex_of(dtype))
    a, b = _both(monkeypatch, lambda: E.integrate(f, steps * 0.2 / n, steps, pd, mode).cpu(), warps)
    _equal(a, b)


@pytest.mark.parametrize("mode", ["RK4", "Lawson_RK4", "Lawson_RK6", "TDRK4"])
@pytest.mark.parametrize("n", [64, 128])
def test_recorded_steps(cuda, monkeypatch, mode, n):
    """The trajectory record, through the tangent and the transpose products on it."""
    kw = dict(num_checkpoints=1, ministeps=7, steps=7, shift_reflect_ny=1, rot=False)
    pd = E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", **kw)
    x = {"fields": torch.as_tensor(initial_condition(2, n), device="cuda"), "T": 0.05, "sx": 0.2}
    v = torch.as_tensor(initial_condition(9, n), device="cuda")

    def run():
        obj = E.Objective(pd, mode)
        out = obj.jvp(x, {"fields": v, "T": 0.3, "sx": -0.1})
        return {k: torch.as_tensor(q).cpu() for k, q in out.items()}

    _equal(*_both(monkeypatch, run))


@pytest.mark.parametrize("n,B", [(64, 5), (128, 2)])
def test_batched_gradient(cuda, monkeypatch, n, B):
    pds = [E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", num_checkpoints=1 + b % 3, ministeps=8,
                             shift_reflect_ny=b, rot=False) for b in range(B)]
    xs = [{"fields": torch.as_tensor(initial_condition(b, n), device="cuda"), "T": 0.03 + 0.01 * b, "sx": 0.1 * b}
          for b in range(B)]

    def run():
        return [(torch.as_tensor(l).cpu(), {k: torch.as_tensor(q).cpu() for k, q in g.items()})
                for l, g in E.loss_grad_multi(xs, pds)]

    _equal(*_both(monkeypatch, run))


# whole record, segments that do not divide the steps, chunks of two regenerated steps; one and several cotangents
@pytest.mark.parametrize("mode", ["Lawson_RK4", "TDRK4"])
@pytest.mark.parametrize("n,B,ckpt,items", [(64, 1, 0, 0), (64, 3, 4, 8), (128, 1, 5, 0), (128, 10, 0, 8)])
def test_products(cuda, monkeypatch, n, B, ckpt, items, mode):
    kw = dict(num_checkpoints=1, ministeps=11, shift_reflect_ny=1, rot=True)
    pd = E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", **kw)
    if ckpt and mode == "Lawson_RK4":
        pd["ckpt_every"] = ckpt
    x = {"fields": torch.as_tensor(initial_condition(2, n), device="cuda"), "T": 0.05, "sx": 0.2}
    ct = {"fields": torch.as_tensor(np.stack([initial_condition(40 + b, n) for b in range(B)]), device="cuda"),
          "T": torch.linspace(0.4, -0.2, B, dtype=torch.float64), "sx": torch.linspace(-0.3, 0.1, B, dtype=torch.float64)}

    def run():
        if items:
            monkeypatch.setenv("ECS_REGEN_ITEMS", str(items))
        obj = E.Objective(pd, mode)
        _, jacT = E.vjp(obj, x)
        return [{k: torch.as_tensor(q).cpu() for k, q in out.items()} for out in (jacT(ct)[0], obj.jvp(x, ct))]

    _equal(*_both(monkeypatch, run))
