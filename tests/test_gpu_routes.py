"""Kernels that a rule on sizes picks, at the sizes where the rule changes and where their tiles and pieces end."""
import numpy as np
import pytest

from onyxia_b200 import backend as be
from onyxia_b200 import ir
from onyxia_b200.ir import HostTensor
from gpu_util import cuda_backend
from test_gpu_lovuzen import rel_err, run_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 8, 9, 32, 33, 65])
def test_f32_products_with_long_sums(rows):
    """Weight rows shared by 1 … 8 warps, four and eight of them per warp; tiles cut along k; a second operand that begins inside a step.
    A sum of k products in pieces is off by at most about (k / 32 + 10) · 2^-24 of the sum of magnitudes; 2e-6 holds with room for k ≤ 7000."""
    r = np.random.default_rng(rows)
    for k, k1, n in ((4100, 0, 52), (6912, 260, 1154), (1152, 0, 2370), (132, 0, 20001)):
        x, w = r.standard_normal((rows, k)).astype(np.float32), r.standard_normal((n, k)).astype(np.float32)
        want, more = x.astype(np.float64) @ w.T.astype(np.float64), {}
        if k1:
            more = {"x1": r.standard_normal((rows, k1)).astype(np.float32), "w1": r.standard_normal((n, k1)).astype(np.float32)}
            want = want + more["x1"].astype(np.float64) @ more["w1"].T.astype(np.float64)
        bias = r.standard_normal(n).astype(np.float32)
        assert rel_err(run_linear(ir.F32, x, w, bias=bias, **more), want + bias) < 2e-6, (k, n)
