"""Transform lengths with a prime factor above 5 that need many threads: the
plan is made (its set-up kernels transform the tensor in FP64 for both forms)
and its field is the oracle's.

Lengths: 7-smooth rows and columns from 1792 points on, where a seventh of the
length is more than 256 threads; heights above 1024 points, whose set-up takes an
eighth of the length; the longest columns a prime factor leaves within the
thread limits; a length whose three columns of threads pass 768."""
import numpy as np
import pytest

import llg
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng,ny,opened", [(1050, 6, 1), (903, 7, 1), (1400, 8, 1), (8, 910, 1), (6, 1008, 1), (5, 1040, 1),
                                          (4, 1025, 1), (7, 2016, 0), (3, 2057, 0), (5, 2816, 0), (4, 3328, 0), (3584, 4, 0),
                                          (5369, 3, 0), (490, 980, 0)])
@pytest.mark.parametrize("precision", [llg.DEMAG_FP64, llg.DEMAG_MIXED])
def test_field_matches_the_oracle(gpu, oracle_lib, ng, ny, opened, precision):
    import torch
    p = llg.default_params(ng, ny, demag_mode=llg.DEMAG_OPEN if opened else llg.DEMAG_PERIODIC, demag_strength=2.5,
                           demag_precision=precision)
    y = np.random.default_rng(ng + ny).uniform(-1.0, 1.0, 3 * ng * ny)
    want = oracle_lib.Oracle(p).demag(y)
    h = torch.full((3 * ng * ny,), float("nan"), dtype=torch.float64, device=gpu)
    llg.Context(p).demag_apply(torch.from_numpy(y).to(gpu), h)
    # the bounds of the two chains' other field tests
    assert rel_err(h.cpu().numpy(), want) <= (1e-11 if precision == llg.DEMAG_FP64 else 5e-6)


@pytest.mark.parametrize("shape", [lambda n: (8, n), lambda n: (n, 8)], ids=["columns", "rows"])
def test_a_longer_plan_outlives_a_shorter_one(gpu, shape):
    """A kernel's shared-memory limit is process-wide: the plan of a shorter
    transform must not lower it under a longer one's."""
    import torch

    def context(n):
        ng, ny = shape(n)
        ctx = llg.Context(llg.default_params(ng, ny, demag_mode=llg.DEMAG_PERIODIC, demag_strength=1.0,
                                             demag_precision=llg.DEMAG_MIXED))
        y = torch.from_numpy(np.random.default_rng(n).uniform(-1.0, 1.0, 3 * ng * ny)).to(gpu)
        return ctx, y, torch.zeros_like(y)

    lengths = (4000, 3000) if shape(1) == (8, 1) else (8100, 6400)   # all above 48 KB a block
    a = context(lengths[0])
    a[0].demag_apply(a[1], a[2])
    want = a[2].clone()
    b = context(lengths[1])
    b[0].demag_apply(b[1], b[2])
    a[2].zero_()
    a[0].demag_apply(a[1], a[2])
    assert torch.equal(a[2], want)


@pytest.mark.parametrize("n", [32, 48, 64, 96, 192, 384, 768, 1536, 3072])
@pytest.mark.parametrize("opened", [0, 1])
@pytest.mark.parametrize("columns", [0, 1])
def test_constant_plans_of_the_fp64_chain(gpu, oracle_lib, n, opened, columns):
    """Lengths with constant radices that the other tests leave out, in rows and in
    columns: two passes, a fused radix of 12, three middle passes."""
    ng, ny = (n // 2 if opened else n), 5
    if columns:
        ng, ny = ny, ng
    import torch
    p = llg.default_params(ng, ny, demag_mode=llg.DEMAG_OPEN if opened else llg.DEMAG_PERIODIC, demag_strength=2.5)
    y = np.random.default_rng(ng + ny).uniform(-1.0, 1.0, 3 * ng * ny)
    want = oracle_lib.Oracle(p).demag(y)
    h = torch.full((3 * ng * ny,), float("nan"), dtype=torch.float64, device=gpu)
    llg.Context(p).demag_apply(torch.from_numpy(y).to(gpu), h)
    assert rel_err(h.cpu().numpy(), want) <= 1e-11


@pytest.mark.parametrize("ng,ny", [(17, 29), (19, 23), (31, 37), (41, 43), (47, 59), (3 * 29, 2 * 31), (1, 37), (870, 37),
                                   (61, 1054)])
def test_prime_passes_of_the_fp64_chain(gpu, oracle_lib, ng, ny):
    """A group of 16 lanes per butterfly up to 31, of 32 from 37 on: odd numbers of
    butterflies, fewer than a warp's groups, and many per thread block."""
    import torch
    p = llg.default_params(ng, ny, demag_mode=llg.DEMAG_PERIODIC, demag_strength=2.5)
    y = np.random.default_rng(ng + ny).uniform(-1.0, 1.0, 3 * ng * ny)
    want = oracle_lib.Oracle(p).demag(y)
    h = torch.full((3 * ng * ny,), float("nan"), dtype=torch.float64, device=gpu)
    llg.Context(p).demag_apply(torch.from_numpy(y).to(gpu), h)
    assert rel_err(h.cpu().numpy(), want) <= 1e-11
