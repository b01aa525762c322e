"""Weights that are not finite, as a diverged training leaves them, show in
every cell of the preconditioner's output and in its norm, also in the tiles
without an active cell, which the fused inference otherwise skips."""
import numpy as np
import pytest

import llg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3.4e38])   # (the last is infinite as BF16)
def test_every_cell_shows_it(gpu, value):
    import torch
    ng, ny = 160, 96
    n = ng * ny
    p = llg.default_params(ng, ny)
    p.precond_kind = llg.PREC_LEARNED
    ctx = llg.Context(p)
    mask = np.zeros((ny, ng))
    mask[:8, :8] = 1.0   # most tiles hold no active cell
    ctx.set_mask(np.tile(mask.ravel(), 3))
    rng = np.random.default_rng(2)
    z, m = (torch.from_numpy(rng.standard_normal(3 * n)).to(gpu) for _ in range(2))
    ewt = torch.full_like(z, 10.0)
    w = (0.05 * rng.standard_normal(llg.LEARNED_NWEIGHTS)).astype(np.float32)
    out = torch.zeros_like(z)
    ctx.learned_set_weights(w)
    assert np.isfinite(ctx.learned_apply(z, m, ewt, 0.02, out)) and bool(torch.isfinite(out).all())
    w[5] = value   # first layer: its channel reaches every output through the second
    ctx.learned_set_weights(w)
    assert np.isnan(ctx.learned_apply(z, m, ewt, 0.02, out)) and bool(torch.isnan(out).all())
    w[5] = 0.01
    ctx.learned_set_weights(w)
    assert np.isfinite(ctx.learned_apply(z, m, ewt, 0.02, out)) and bool(torch.isfinite(out).all())
