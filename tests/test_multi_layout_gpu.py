"""A candidate's objective and JVP from ecs_jvp_multi do not depend on the candidates that
share its sweep (a server puts every queued request into the next one): equal bit for bit
in a sweep of one and of many, either side of the batch from which one linearisation's
tangents use another layout of the column passes (16, FP64 at n = 128)."""
import numpy as np
import pytest
import torch

import ecs_mhd_2d_b200 as E
from ecs_mhd_2d_b200.synthetic import initial_condition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B", [(128, 15), (128, 16), (128, 17), (64, 17)])
def test_sweep_size_does_not_change_a_result(cuda, n, B):
    rng = np.random.default_rng(7)
    xs, vs, pds = [], [], []
    for b in range(B):
        pds.append(E.make_param_dict(n, 1 / 40, 1 / 40, forcing="kolmogorov+", num_checkpoints=1 + b % 2, ministeps=5,
                                     shift_reflect_ny=b % 3, rot=b % 2 == 1))
        xs.append({"fields": torch.as_tensor(initial_condition(b, n), device="cuda"), "T": 0.03 + 0.002 * b, "sx": 0.1})
        vs.append({"fields": torch.as_tensor(rng.standard_normal((2, n, n)), device="cuda"), "T": 0.2, "sx": -0.1 * b})
    many = E.jvp_multi(xs, vs, pds)
    for b in (0, B // 2, B - 1):
        one = E.jvp_multi(xs[b:b + 1], vs[b:b + 1], pds[b:b + 1])
        for got, want in zip(many, one):
            for k in ("fields", "T", "sx"):
                assert torch.equal(torch.as_tensor(got[b][k]), torch.as_tensor(want[0][k])), (b, k)
