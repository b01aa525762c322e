"""llg_linear_combination rounds as it is stated: z = c0 x0, then z = c_k x_k + z
with one rounding per further vector, whichever kernel the vector count picks.
The expected values come from exact rational arithmetic, so the comparison is
bit for bit."""
from fractions import Fraction

import numpy as np
import pytest

import llg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvec", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("aliased", [False, True])
def test_rounding_order(gpu, nvec, aliased):
    import torch
    ng, ny = 37, 5
    n = 3 * ng * ny
    rng = np.random.default_rng(nvec)
    c = rng.uniform(-2.0, 2.0, nvec)
    x = rng.uniform(-1.0, 1.0, (nvec, n))
    want = []
    for i in range(n):
        s = c[0] * x[0, i]
        for k in range(1, nvec):
            s = float(Fraction(c[k]) * Fraction(x[k, i]) + Fraction(s))
        want.append(s)
    ctx = llg.Context(llg.default_params(ng, ny))
    X = [torch.from_numpy(v.copy()).to(gpu) for v in x]
    z = X[0] if aliased else torch.full((n,), float("nan"), dtype=torch.float64, device=gpu)
    ctx.linear_combination(c, X, z)
    assert np.array_equal(z.cpu().numpy(), np.array(want))
