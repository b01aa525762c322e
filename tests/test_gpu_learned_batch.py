"""Batch sizes of the training kernels: the batch fills the grid's z dimension
(65,535 patches), whatever the kernels split beside it."""
import numpy as np
import pytest

import llg

pytestmark = pytest.mark.gpu


def _patches(nb, P, seed=11):
    g = np.random.default_rng(seed)
    f = lambda *s: g.standard_normal(s).astype(np.float32)  # noqa: E731
    u = f(nb, 3, P, P)
    return dict(u=u, m=f(nb, 3, P, P), mask=np.ones((nb, P, P), np.float32), ewt=np.abs(f(nb, 3, P, P)) + 0.5,
                x=0.9 * u + 0.1 * f(nb, 3, P, P), gamma=np.full(nb, 0.02, np.float32))


def test_large_batch(gpu):
    """32,768 patches, four repeated: a mean over a power of two as many copies.
    Every FP32 quantity is the small batch's times 2^-13, exactly; only the
    FP64 sums over the copies round, far below FP32's last bit."""
    P, reps = 8, 8192
    w = (0.05 * np.random.default_rng(1).standard_normal(llg.LEARNED_NWEIGHTS)).astype(np.float32)
    s = _patches(4, P)
    loss0, grad0, z0 = llg.learned_loss_grad(w, s["u"], s["m"], s["mask"], s["ewt"], s["x"], s["gamma"])
    b = {k: np.concatenate([v] * reps) for k, v in s.items()}
    loss, grad, z = llg.learned_loss_grad(w, b["u"], b["m"], b["mask"], b["ewt"], b["x"], b["gamma"])
    assert abs(loss - loss0) <= 1e-12 * abs(loss0)
    assert np.array_equal(z.reshape(reps, *z0.shape), np.broadcast_to(z0, (reps,) + z0.shape))
    assert np.abs(grad - grad0).max() <= 2.0 ** -23 * np.abs(grad0).max()


def test_a_refused_launch_fails_its_own_call_only(gpu):
    """65,536 patches exceed the grid's z limit: the call reports the refused
    launch, and the next one, on a context of its own, does not see it."""
    import torch
    ctx = llg.Context(llg.default_params(32, 16))
    y = torch.ones(3 * 32 * 16, dtype=torch.float64, device=gpu)
    f = torch.zeros_like(y)
    w = np.zeros(llg.LEARNED_NWEIGHTS, np.float32)
    b = {k: np.repeat(v, 65536, axis=0) for k, v in _patches(1, 8).items()}
    with pytest.raises(llg.LLGError):
        llg.learned_loss_grad(w, b["u"], b["m"], b["mask"], b["ewt"], b["x"], b["gamma"])
    ctx.rhs(0.0, y, f)
    torch.cuda.synchronize()
