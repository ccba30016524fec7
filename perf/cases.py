"""Performance cases: the calls a user of this package makes, through its public
entry points, over the sizes of its own configurations and benchmark (grid sides
64, 128 and 256; one state to batches of 64; FP64 and FP32).

  listed()          the named cases
  draw(rng)         one more case of the same ranges
  prepare(case, s)  the inputs (and handles) a program holds before the call, on the GPU
  run(state)        one pass through the public entry points, with its outputs
  work(case)        bytes and floating-point operations of one pass
  exact(case, s)    the same outputs from plain torch in 64 bits

A case's "kind" names the call:
  rhs        state_vel of a spectral state
  step       timestepping.integrate: fixed-step time stepping (DNS, forward maps)
  objective  objective_RPO: one forward shooting
  matvec     Objective.jvp at a kept linearisation (GMRES, Floquet blocks)
  linjvp     Objective.linearize_jvp: primal solve and a batch of tangents in one call
  vjp        the transpose product at a kept linearisation
  grad       loss_and_grad: the adjoint-descent gradient
  gradmulti  loss_grad_multi: several candidates' gradients in one sweep (serving)
  jvpmulti   jvp_multi: several candidates' matvecs in one sweep (serving)
  newton     one Newton step: objective, linearisation, GMRES on A^T A
"""

import math

import numpy as np
import torch

import ecs_mhd_2d_b200 as ecs
from ecs_mhd_2d_b200 import linalg, utils
from ecs_mhd_2d_b200.context import Context

# Adaptive solves: attempts per unit of T at atol 1e-8, mean over seeds at the horizons used here (180 to 320).
ATTEMPTS_PER_T = 250.0


def listed():
    return [
        # the smallest call: one right-hand side of the test-size grid
        dict(name="rhs_n64", kind="rhs", n=64, dtype="f64", batch=1, diss=True),
        # forward integration of 8 candidates (64^2, dt = 0.005, 1024 steps, Re = 40)
        dict(name="step_rk4_n64_b8", kind="step", mode="Lawson_RK4", n=64, dtype="f64", batch=8, steps=1024,
             dt=0.005, re=40.0),
        # forward integration of one candidate: a latency-bound chain of right-hand sides
        dict(name="step_rk4_n128_b1", kind="step", mode="Lawson_RK4", n=128, dtype="f64", batch=1, steps=256,
             dt=0.00375, re=40.0),
        # batched single-precision forward maps of the mixed-precision path
        dict(name="step_rk4_n256_f32_b64", kind="step", mode="Lawson_RK4", n=256, dtype="f32", batch=64, steps=64,
             dt=0.00225, re=50.0),
        # DNS data generation: one trajectory with the sixth-order stepper
        dict(name="dns_rk6_n128_b1", kind="step", mode="Lawson_RK6", n=128, dtype="f64", batch=1, steps=256,
             dt=1 / 256, re=40.0),
        # one adaptive forward shooting (a line-search evaluation)
        dict(name="objective_rk43_n128_b1", kind="objective", mode="Lawson_RK43", n=128, dtype="f64", batch=1,
             T=0.5, atol=1e-8, re=50.0),
        # one Arnoldi step's matvec at a kept adaptive linearisation (sequential GMRES)
        dict(name="matvec_rk43_n128_b1", kind="matvec", mode="Lawson_RK43", n=128, dtype="f64", batch=1, T=0.5,
             atol=1e-8, re=50.0),
        # the benchmark's step on a quarter of its horizon: linearisation and 64 tangents
        dict(name="linjvp_rk43_n128_b64", kind="linjvp", mode="Lawson_RK43", n=128, dtype="f64", batch=64, T=1.15,
             atol=1e-8, re=50.0),
        # a single-precision batch of tangents at a kept linearisation (mixed-precision Krylov block)
        dict(name="matvec_rk4_n256_f32_b32", kind="matvec", mode="Lawson_RK4", n=256, dtype="f32", batch=32,
             steps=64, dt=0.00225, re=50.0),
        # the adjoint-descent gradient, checkpoints every 32 steps
        dict(name="grad_rk4_n128", kind="grad", mode="Lawson_RK4", n=128, dtype="f64", batch=1, steps=256,
             dt=0.0039, re=40.0, ckpt=32),
        # a server's gradients of 8 candidates with their own horizons, one sweep
        dict(name="gradmulti_rk4_n64_b8", kind="gradmulti", mode="Lawson_RK4", n=64, dtype="f64", batch=8, steps=128,
             dt=0.005, re=40.0),
        # one Newton-GMRES step with the transpose as preconditioner (the reference's defaults)
        dict(name="newton_tdrk4_n64", kind="newton", mode="TDRK4", n=64, dtype="f64", batch=1, steps=32, dt=0.005,
             re=40.0, inner=4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    top = 0.8 * work(next(c for c in listed() if c["name"] == "linjvp_rk43_n128_b64"))["flops"]
    while True:
        kind = rng.choice(["rhs", "step", "step", "step", "objective", "objective", "matvec", "matvec", "linjvp",
                           "vjp", "grad", "grad", "gradmulti", "jvpmulti", "newton"])
        n = rng.choice([64, 128, 128, 256])
        re = round(rng.uniform(40.0, 50.0), 2)
        dtype = rng.choice(["f64", "f64", "f32"])
        c = dict(kind=kind, n=n, dtype=dtype, batch=_log_int(rng, 1, 64), re=re)
        fixed = dict(steps=_log_int(rng, 16, 512), dt=round(rng.uniform(0.3, 0.6) / n, 6))
        adaptive = dict(T=round(rng.uniform(0.1, 0.8), 4), atol=rng.choice([1e-8, 1e-7, 1e-6]), dtype="f64")
        if kind == "rhs":
            c.update(diss=rng.random() < 0.5)
            c.pop("re")
        elif kind == "step":
            c.update(fixed, mode=rng.choice(["Lawson_RK4", "Lawson_RK4", "Lawson_RK6", "RK4", "TDRK4"]))
        elif kind in ("objective", "matvec", "linjvp", "vjp"):
            c["mode"] = rng.choice(["Lawson_RK4", "Lawson_RK43", "Lawson_RK43", "TDRK4"])
            c.update(adaptive if c["mode"] == "Lawson_RK43" else fixed)
            if kind == "vjp":
                c["batch"] = _log_int(rng, 1, 8)
                c["steps" if "steps" in c else "T"] = min(c["steps"], 128) if "steps" in c else min(c["T"], 0.2)
        elif kind == "grad":
            c.update(fixed, mode="Lawson_RK4", batch=1, steps=_log_int(rng, 32, 256), ckpt=rng.choice([0, 24, 32]))
        elif kind in ("gradmulti", "jvpmulti"):
            c.update(fixed, mode="Lawson_RK4", batch=rng.randint(2, 12), steps=32 * rng.randint(1, 4), dtype="f64",
                     n=rng.choice([64, 128]))
        else:
            c.update(fixed, mode=rng.choice(["TDRK4", "Lawson_RK4"]), batch=1, steps=_log_int(rng, 16, 64),
                     dtype="f64", n=rng.choice([64, 128]), inner=rng.randint(3, 6))
        w = work(c)["flops"]
        states = 1 if kind in ("matvec", "linjvp", "vjp") else c["batch"]
        if kind in ("vjp", "grad", "gradmulti") and states * c.get("steps", 100) * n * n > 12e6:
            continue   # the 64-bit check keeps a reverse-mode graph of this size
        if w <= top:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dt(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _params(case):
    """param_dict of a case (the benchmark's physics: Kolmogorov forcing, mean field 0.1 along y)."""
    re = case.get("re", 40.0)
    kw = dict(shift_reflect_ny=0, rot=False)
    if "steps" in case:
        ms = 32 if case["steps"] % 32 == 0 else case["steps"]
        kw.update(num_checkpoints=case["steps"] // ms, ministeps=ms, steps=case["steps"])
    if "atol" in case:
        kw["adaptive_dict"] = {"atol": case["atol"], "checkpoints": 32, "max_steps_per_checkpoint": 32}
    if case.get("ckpt"):
        kw["ckpt_every"] = case["ckpt"]
    return ecs.make_param_dict(case["n"], 1 / re, 1 / re, forcing="kolmogorov+", data_type=_dt(case), **kw)


def _horizon(case, b=0):
    return case["T"] if "T" in case else case["dt"] * _steps(case, b)


def _steps(case, b):
    """Steps of candidate b: the multi-candidate sweeps mix horizons."""
    if case["kind"] in ("gradmulti", "jvpmulti"):
        return max(32, case["steps"] - 32 * (b % 2))
    return case["steps"]


def _states(case, seed, count):
    """`count` seeded random states [count, 2, n, n] with |k|^-2 spectra."""
    f = np.stack([ecs.initial_condition(1000 * seed + b, case["n"], amp=2.0) for b in range(count)])
    return torch.as_tensor(f, dtype=_dt(case), device="cuda")


def _tangents(case, seed, count):
    """`count` seeded unit-norm tangents as a batched input dict."""
    g = torch.Generator(device="cuda").manual_seed(7919 + seed)
    n = case["n"]
    v = torch.randn((count, 2 * n * n + 2), generator=g, dtype=torch.float64, device="cuda")
    v = v / torch.linalg.norm(v, dim=1, keepdim=True)
    return {"fields": v[:, 1:-1].reshape(count, 2, n, n).to(_dt(case)).contiguous(), "T": v[:, 0].contiguous(),
            "sx": v[:, -1].contiguous()}


def _spectral(case, seed):
    n = case["n"]
    mask = ecs.construct_domain(n, _dt(case))["mask"]
    return (torch.fft.rfft2(_states(case, seed, case["batch"])) * mask).contiguous()


def _input(case, seed, b=0):
    f = _states(case, seed + 31 * b, 1)[0]
    return {"fields": f, "T": _horizon(case, b), "sx": 0.12 - 0.01 * b}


def _multi(case, seed):
    B = case["batch"]
    xs = [_input(case, seed, b) for b in range(B)]
    pds = []
    for b in range(B):
        pd = dict(_params(case))
        pd.update(num_checkpoints=_steps(case, b) // 32, ministeps=32, shift_reflect_ny=b % 3, rot=b % 4 == 3)
        pds.append(pd)
    return xs, pds


def _one(d):
    return {k: v[0] for k, v in d.items()}


def prepare(case, seed):
    kind, n, B = case["kind"], case["n"], case["batch"]
    s = {"case": case, "kind": kind}
    if kind in ("rhs", "step"):
        s.update(pd=_params(case), f=_spectral(case, seed))
    elif kind == "objective":
        s["pd"] = _params(case)
        f = _states(case, seed, B)
        T = torch.full((B,), _horizon(case), dtype=torch.float64, device="cuda")
        sx = torch.full((B,), 0.12, dtype=torch.float64, device="cuda")
        s["x"] = {"fields": f, "T": T, "sx": sx} if B > 1 else {"fields": f[0], "T": _horizon(case), "sx": 0.12}
    elif kind in ("matvec", "vjp"):
        # a solver holds its own linearisation: one context per base point
        pd = _params(case)
        ctx = Context(n, _dt(case), pd["nu"], pd["eta"], pd["b0"], pd["forcing"].double().cpu().numpy(), max_batch=B)
        obj = ecs.Objective(pd, case["mode"], ctx=ctx)
        x, v = _input(case, seed), _tangents(case, seed, B)
        obj.linearize(x, batch=B)
        s.update(obj=obj, x=x, v=v if B > 1 else _one(v))
        if kind == "vjp":
            s["jacT"] = ecs.vjp(obj, x)[1]
    elif kind == "linjvp":
        v = _tangents(case, seed, B)
        s.update(obj=ecs.Objective(_params(case), case["mode"]), x=_input(case, seed), v=v if B > 1 else _one(v))
    elif kind in ("grad", "newton"):
        s.update(pd=_params(case), x=_input(case, seed))
    else:
        s["x"], s["pds"] = _multi(case, seed)
        if kind == "jvpmulti":
            v = _tangents(case, seed, B)
            s["v"] = [{k: t[b] for k, t in v.items()} for b in range(B)]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _newton_step(pd, mode, x, inner):
    """The step of one Newton-GMRES update (objective, linearisation, GMRES with
    the transpose as left preconditioner)."""
    obj = ecs.Objective(pd, mode)
    n = x["fields"].shape[-1]
    f = obj(x)
    b = utils.flatten(f)

    def A(v):
        return utils.flatten(obj.jvp(x, utils.unflatten(v, n)))

    _, jacT = ecs.vjp(obj, x)

    def A_T(v):
        t = utils.unflatten(v, n)
        return utils.flatten(jacT({"fields": t["fields"].contiguous(), "T": t["T"], "sx": t["sx"]})[0])

    step, res = linalg.gmres(A, b, inner, 1, [A_T])
    return {"f": f, "step": step, "res": res}


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "rhs":
        return ecs.state_vel(s["f"], s["pd"], case["diss"])
    if kind == "step":
        return ecs.integrate(s["f"], _horizon(case), case["steps"], s["pd"], case["mode"])
    if kind == "objective":
        return ecs.objective_RPO(s["x"], s["pd"], case["mode"])
    if kind == "matvec":
        return s["obj"].jvp(s["x"], s["v"])
    if kind == "linjvp":
        return s["obj"].linearize_jvp(s["x"], s["v"])
    if kind == "vjp":
        return s["jacT"](s["v"])[0]
    if kind == "grad":
        (loss, _), g = ecs.loss_and_grad(s["x"], s["pd"], case["mode"])
        return {"loss": loss, "grad": g}
    if kind == "gradmulti":
        r = ecs.loss_grad_multi(s["x"], s["pds"])
        return {"loss": torch.stack([a for a, _ in r]), **_stack([g for _, g in r])}
    if kind == "jvpmulti":
        vals, jvps = ecs.jvp_multi(s["x"], s["v"], s["pds"])
        return [_stack(vals), _stack(jvps)]
    return _newton_step(s["pd"], case["mode"], s["x"], case["inner"])


def _stack(ds):
    return {k: torch.stack([d[k] for d in ds]) for k in ("fields", "T", "sx")}


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------

# Right-hand sides per step or attempt of each stepper.
RHS = {"Lawson_RK4": 4, "RK4": 4, "Lawson_RK6": 8, "TDRK4": 4, "Lawson_RK43": 4}


def _rhs_flops(n):
    """One right-hand side on the dealiased modes: 7 column transforms per
    retained ky, 4 row transforms per x (5 n log2 n operations each), and the
    products and multipliers."""
    K = (n - 1) // 3 + 1
    M = 2 * K - 1
    return (7 * K + 4 * n) * 5 * n * math.log2(n) + 20 * n * n + 60 * K * M


def _evals(case):
    """Right-hand sides along one trajectory."""
    if case["kind"] == "rhs":
        return 1
    if case["mode"] == "Lawson_RK43":
        return 4 * case["T"] * ATTEMPTS_PER_T * (1e-8 / case["atol"]) ** 0.25
    return RHS[case["mode"]] * case["steps"]


def work(case):
    n, B, kind = case["n"], case["batch"], case["kind"]
    real = 8 if case["dtype"] == "f64" else 4
    one, ev = _rhs_flops(n), _evals(case)
    state = 2 * n * n * real
    spectrum = 2 * n * (n // 2 + 1) * 2 * real
    if kind in ("rhs", "step"):
        return {"bytes": 2 * B * spectrum, "flops": B * ev * one}
    if kind == "objective":
        return {"bytes": 2 * B * state, "flops": B * ev * one}
    # a tangent or cotangent costs one linearised right-hand side each (the
    # two-derivative stepper's second stages linearise twice)
    lin = 1.5 if case["mode"] == "TDRK4" else 1.0
    if kind in ("matvec", "vjp"):
        return {"bytes": 2 * B * state, "flops": B * ev * one * lin}
    if kind == "linjvp":
        return {"bytes": 2 * (B + 1) * state, "flops": (1 + B * lin) * ev * one}
    if kind in ("grad", "gradmulti"):
        return {"bytes": 2 * B * state, "flops": 2 * B * ev * one}
    if kind == "jvpmulti":
        return {"bytes": 4 * B * state, "flops": 2 * B * ev * one}
    m = case["inner"]
    krylov = 4.0 * 2 * n * n * m * (m + 3)
    return {"bytes": (m + 3) * state, "flops": (2 + (2 * m + 2) * lin) * ev * one + krylov}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, from torch's own FFTs and automatic differentiation
# ---------------------------------------------------------------------------

class _Exact:
    """The shooting map of a batch of states, plain torch."""

    def __init__(self, case):
        n, re = case["n"], case.get("re", 40.0)
        k = torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device="cuda")
        kx, ky = k.reshape(-1, 1), k[: n // 2 + 1].reshape(1, -1)
        mask = (kx.abs() < n / 3) & (ky.abs() < n / 3)
        mask[0, 0] = False
        ksq = kx * kx + ky * ky
        ksq[0, 0] = 1
        self.case, self.n, self.mask = case, n, mask
        self.u, self.v = ky / ksq * mask, -kx / ksq * mask
        self.kx, self.ky = kx * mask, ky * mask
        self.ksq = self.kx ** 2 + self.ky ** 2
        self.nu = 1.0 / re   # of both channels
        self.L = -self.ksq * self.nu
        y = torch.arange(n, dtype=torch.float64, device="cuda") / n * 2 * math.pi
        force = (4 * torch.cos(4 * y)).to(_dt(case)).double().expand(n, n)
        self.force = torch.fft.rfft2(force) * mask
        self.hs = None

    def ir(self, f):
        return torch.fft.irfft2(f, s=(self.n, self.n))

    def _phys(self, f):
        return (self.ir(1j * self.kx * f), self.ir(1j * self.ky * f), self.ir(1j * self.u * f),
                self.ir(1j * self.v * f))

    def rhs(self, f, diss):
        fx, fy, u, v = self._phys(f)
        v = torch.stack([v[..., 0, :, :], v[..., 1, :, :] + 0.1], -3)
        adv = u * fx + v * fy
        w = torch.fft.rfft2(adv[..., 1, :, :] - adv[..., 0, :, :]) * self.mask + self.force
        j = self.ksq * torch.fft.rfft2(u[..., 0, :, :] * v[..., 1, :, :] - v[..., 0, :, :] * u[..., 1, :, :])
        out = torch.stack([w, j], -3)
        return out + self.L * f if diss else out

    def lin(self, f, d, diss):
        """rhs'(f) d"""
        fx, fy, u, v = self._phys(f)
        v = torch.stack([v[..., 0, :, :], v[..., 1, :, :] + 0.1], -3)
        dx, dy, du, dv = self._phys(d)
        adv = u * dx + du * fx + v * dy + dv * fy
        w = torch.fft.rfft2(adv[..., 1, :, :] - adv[..., 0, :, :]) * self.mask
        j = self.ksq * torch.fft.rfft2(u[..., 0, :, :] * dv[..., 1, :, :] + du[..., 0, :, :] * v[..., 1, :, :]
                                       - v[..., 0, :, :] * du[..., 1, :, :] - dv[..., 0, :, :] * u[..., 1, :, :])
        out = torch.stack([w, j], -3)
        return out + self.L * d if diss else out

    def advance(self, f, t, steps, mode):
        """t: one horizon per state ([B]) or a number."""
        if isinstance(t, torch.Tensor):
            t = t.reshape(-1, 1, 1, 1)
        if mode == "Lawson_RK43":
            return self.adaptive(f, t)
        h = t / steps
        if mode == "RK4":
            for _ in range(steps):
                k1 = h * self.rhs(f, True)
                k2 = h * self.rhs(f + k1 / 2, True)
                k3 = h * self.rhs(f + k2 / 2, True)
                k4 = h * self.rhs(f + k3, True)
                f = f + k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6
        elif mode == "TDRK4":
            for _ in range(steps):
                k1 = h * self.rhs(f, True)
                a1 = h * self.lin(f, k1, True)
                g = f + k1 / 2 + a1 / 8
                k2 = h * self.rhs(g, True)
                a2 = h * self.lin(g, k2, True)
                f = f + k1 + a1 / 6 + a2 / 3
        elif mode == "Lawson_RK4":
            e = torch.exp(self.L * (h / 2)) * self.mask
            for _ in range(steps):
                k1 = e * (h * self.rhs(f, False))
                f = e * f
                k2 = h * self.rhs(f + k1 / 2, False)
                k3 = e * (h * self.rhs(f + k2 / 2, False))
                f, k1, k2 = e * f, e * k1, e * k2
                k4 = h * self.rhs(f + k3, False)
                f = f + k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6
        else:
            e = torch.exp(self.L * (h / 6)) * self.mask
            for _ in range(steps):
                k = [h * self.rhs(f, False)]

                def turn():
                    k[:] = [e * q for q in k]
                    return e * f

                f = turn()
                k.append(h * self.rhs(f + k[0] / 6, False))
                k.append(h * self.rhs(f + k[0] / 12 + k[1] / 12, False))
                f = turn()
                k.append(h * self.rhs(f - k[1] * 4 / 33 + k[2] * 5 / 11, False))
                f = turn()
                k.append(h * self.rhs(f - k[0] / 4 - k[1] * 29 / 44 + k[2] * 31 / 22, False))
                f = turn()
                k.append(h * self.rhs(f + k[0] * 3 / 11 + k[1] * 8 / 33 - k[2] * 4 / 11 + k[3] / 11 + k[4] * 14 / 33,
                                      False))
                f = turn()
                k.append(h * self.rhs(f - k[0] * 17 / 48 - k[1] * 5 / 12 + k[2] + k[3] - k[4] * 13 / 12
                                      + k[5] * 11 / 16, False))
                f = turn()
                k.append(h * self.rhs(f + k[0] * 20 / 39 + k[1] * 12 / 39 - k[2] * 31 / 39 - k[3] / 39
                                      + k[4] * 34 / 39 - k[5] * 11 / 39 + k[6] * 16 / 39, False))
                f = f + 13 / 200 * (k[0] + k[7]) + 4 / 25 * (k[2] + k[6]) + 11 / 40 * (k[3] + k[5])
        return f

    def plan(self, f, t):
        """Step sizes and accept flags of one state's adaptive solve."""
        with torch.no_grad():
            s, h, plan, x = 0.0, 1e-2, [], f
            k1 = t * self.rhs(x, False)
            while abs(s - 1.0) >= 1e-10 and len(plan) < 1024:
                xf, k4, k5, kr = self.attempt(x, k1, t, h)
                err = float((self.ir(h * (k5 - k4) / 6)).abs().max())
                ok = err < self.case["atol"]
                plan.append((h, ok))
                if ok:
                    x, k1, s = xf, k5, s + h
                else:
                    k1 = kr
                h = h * 0.9 * (self.case["atol"] / err) ** 0.25
                h = h - max(s + h - 1.0, 0.0)
            return plan

    def attempt(self, x, k1, t, h):
        e = torch.exp(t * self.L * h / 2)
        x, k1 = e * x, e * k1
        k2 = t * self.rhs(x + h * k1 / 2, False)
        k3 = t * self.rhs(x + h * k2 / 2, False)
        x, k1, k2, k3 = e * x, e * k1, e * k2, e * k3
        k4 = t * self.rhs(x + h * k3, False)
        xf = x + h * (k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6)
        return xf, k4, t * self.rhs(xf, False), k1

    def adaptive(self, f, t):
        k1 = t * self.rhs(f, False)
        for h, ok in self.hs:
            xf, _, k5, kr = self.attempt(f, k1, t, h)
            f, k1 = (xf, k5) if ok else (f, kr)
        return f

    def objective(self, fields, T, sx, steps, mode, ny=0, rot=False):
        """irfft2(f0 - g Phi_T(f0)) of a batch of states."""
        f0 = torch.fft.rfft2(fields)
        f = self.advance(f0, T, steps, mode)
        f = torch.exp(1j * self.kx * sx.reshape(-1, 1, 1, 1)) * f
        f = torch.exp(1j * self.ky * (ny * 2 * math.pi / 8)) * f
        if ny % 2 == 1:
            f = -torch.roll(torch.flip(f, dims=(-2,)), 1, -2)
        if rot:
            f = torch.conj(f) * torch.tensor([1.0, -1.0], dtype=torch.float64, device="cuda").reshape(2, 1, 1)
        return self.ir(f0 - f)

    def phase(self, fields):
        """The stop-gradient fields of the two phase conditions."""
        f0 = torch.fft.rfft2(fields)
        return self.ir(self.rhs(f0, True)), self.ir(1j * self.kx * f0)

    def jvp(self, x, v, steps, mode, ny=0, rot=False):
        """(objective, tangents) at one base point for a batch of tangents."""
        B = v["fields"].shape[0]
        p = (x["fields"].repeat(B, 1, 1, 1), x["T"].repeat(B), x["sx"].repeat(B))
        fn = lambda f, T, sx: self.objective(f, T, sx, steps, mode, ny, rot)   # noqa: E731
        val, tan = torch.func.jvp(fn, p, (v["fields"], v["T"], v["sx"]))
        vt, vx = self.phase(x["fields"])
        mean = lambda a: (a * v["fields"]).mean(dim=(-1, -2, -3))   # noqa: E731
        return val[:1], {"fields": tan, "T": mean(vt), "sx": mean(vx)}

    def vjp(self, x, v, steps, mode):
        out = []
        args = [x["fields"].clone(), x["T"].clone(), x["sx"].clone()]
        for a in args:
            a.requires_grad_(True)
        val = self.objective(args[0], args[1], args[2], steps, mode)
        vt, vx = self.phase(x["fields"])
        B = v["fields"].shape[0]
        for b in range(B):
            g = torch.autograd.grad(val, args, v["fields"][b:b + 1], retain_graph=b < B - 1)
            gf = g[0] + (v["T"][b] * vt + v["sx"][b] * vx) / (2 * self.n * self.n)
            out.append((gf[0], g[1][0], g[2][0]))
        return {"fields": torch.stack([o[0] for o in out]), "T": torch.stack([o[1] for o in out]),
                "sx": torch.stack([o[2] for o in out])}

    def loss_grad(self, x, steps, mode, ny=0, rot=False):
        args = [x["fields"].clone(), x["T"].clone(), x["sx"].clone()]
        for a in args:
            a.requires_grad_(True)
        loss = (self.objective(args[0], args[1], args[2], steps, mode, ny, rot) ** 2).mean()
        g = torch.autograd.grad(loss, args)
        return loss.detach(), {"fields": g[0][0], "T": g[1][0], "sx": g[2][0]}


def _double(x):
    """A single input dict as 64-bit batch-of-one tensors."""
    one = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda").reshape(1)   # noqa: E731
    return {"fields": x["fields"].double()[None], "T": one(x["T"]), "sx": one(x["sx"])}


def exact(case, seed):
    kind, n, B, mode = case["kind"], case["n"], case["batch"], case.get("mode")
    E = _Exact(case)
    steps = case.get("steps")
    zero = torch.zeros(B, dtype=torch.float64, device="cuda")
    if kind in ("rhs", "step"):
        f = _spectral(case, seed).to(torch.complex128)
        with torch.no_grad():
            return E.rhs(f, case["diss"]) if kind == "rhs" else E.advance(f, _horizon(case), steps, mode)
    if kind == "objective":
        f = _states(case, seed, B).double()
        T, sx = torch.full_like(zero, _horizon(case)), torch.full_like(zero, 0.12)
        with torch.no_grad():
            if mode == "Lawson_RK43":
                if B > 8:
                    return None   # every state has its own step sizes
                out = []
                for b in range(B):
                    E.hs = E.plan(torch.fft.rfft2(f[b:b + 1]), _horizon(case))
                    out.append(E.objective(f[b:b + 1], T[:1], sx[:1], steps, mode))
                val = torch.cat(out)
            else:
                val = E.objective(f, T, sx, steps, mode)
        r = {"fields": val, "T": zero, "sx": zero}
        return r if B > 1 else _one(r)
    if kind in ("gradmulti", "jvpmulti"):
        xs, pds = _multi(case, seed)
        v = _tangents(case, seed, B)
        vals, outs = [], []
        for b in range(B):
            sym = dict(ny=pds[b]["shift_reflect_ny"], rot=pds[b]["rot"])
            if kind == "gradmulti":
                r = E.loss_grad(_double(xs[b]), _steps(case, b), mode, **sym)
            else:
                r = E.jvp(_double(xs[b]), {k: t[b:b + 1].double() for k, t in v.items()}, _steps(case, b), mode, **sym)
            vals.append(r[0])
            outs.append(r[1] if kind == "gradmulti" else _one(r[1]))
        if kind == "gradmulti":
            return {"loss": torch.stack(vals), **_stack(outs)}
        return [{"fields": torch.cat(vals), "T": zero, "sx": zero}, _stack(outs)]
    x = _double(_input(case, seed))
    if mode == "Lawson_RK43":
        E.hs = E.plan(torch.fft.rfft2(x["fields"]), _horizon(case))
    if kind == "grad":
        loss, g = E.loss_grad(x, steps, mode)
        return {"loss": loss, "grad": g}
    if kind == "newton":
        return _newton_exact(E, x, steps, mode, case["inner"])
    v = {k: t.double() for k, t in _tangents(case, seed, B).items()}
    if kind == "vjp":
        r = E.vjp(x, v, steps, mode)
        return r if B > 1 else _one(r)
    with torch.no_grad():
        val, r = E.jvp(x, v, steps, mode)
    r = r if B > 1 else _one(r)
    return r if kind == "matvec" else [{"fields": val[0], "T": zero[0], "sx": zero[0]}, r]


def _newton_exact(E, x, steps, mode, inner):
    """The Newton step with dense Arnoldi in torch."""
    n = E.n
    flat = lambda d: torch.cat([d["T"].reshape(1), d["fields"].reshape(-1), d["sx"].reshape(1)])   # noqa: E731
    batch = lambda q: {"fields": q[1:-1].reshape(1, 2, n, n), "T": q[:1], "sx": q[-1:]}   # noqa: E731
    with torch.no_grad():
        val = E.objective(x["fields"], x["T"], x["sx"], steps, mode)
    z = torch.zeros((), dtype=torch.float64, device="cuda")
    f = {"fields": val[0], "T": z, "sx": z}

    def A(q):
        with torch.no_grad():
            return flat(E.jvp(x, batch(q), steps, mode)[1])

    def A_T(q):
        return flat(E.vjp(x, batch(q), steps, mode))

    b = A_T(flat(f))
    Q, H = [b / torch.linalg.norm(b)], torch.zeros((inner + 1, inner), dtype=torch.float64, device="cuda")
    for k in range(inner):
        w = A_T(A(Q[k]))
        for j in range(k + 1):
            H[j, k] = torch.dot(w, Q[j])
            w = w - H[j, k] * Q[j]
        H[k + 1, k] = torch.linalg.norm(w)
        Q.append(w / H[k + 1, k])
    Qm = torch.stack(Q)
    y = torch.linalg.lstsq(H, (Qm @ b).reshape(-1, 1)).solution.reshape(-1)
    step = Qm[:inner].T @ y
    res = torch.linalg.norm(A_T(A(step)) - b) / torch.linalg.norm(b)
    return {"f": f, "step": step, "res": res}
