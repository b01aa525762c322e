"""The FP64 in-place transforms of the demag chain (csrc/dev_fft64.cuh).

On the CPU: every in-register DFT and whole transforms of many lengths, pass
by pass, against a long double DFT (tests/native/fft64_check.cu).  On the GPU:
the chain's field against the oracle's at the lengths where a plan's form
changes: primes that take a warp per butterfly, odd periodic lengths, odd
heights (unaligned row pairs), one-pass lengths, and each length with
constant radices, in rows and in columns.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO, rel_err


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_transforms_on_the_cpu(tmp_path):
    exe = tmp_path / "fft64_check"
    src = os.path.join(REPO, "tests", "native", "fft64_check.cu")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Wno-deprecated-gpu-targets", "-I" + os.path.join(PKG, "csrc"), src, "-o", str(exe)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


# (ng, ny, open): rows of 2 ng and columns of 2 ny when open
SHAPES = [(1, 1, 1), (1, 3, 0), (2, 1, 0), (5, 7, 1), (16, 17, 1), (61, 31, 1), (53, 59, 0), (122, 9, 0), (33, 61, 0),
          (64, 64, 1), (128, 64, 1), (77, 128, 1), (91, 26, 1), (256, 37, 1), (375, 225, 1), (512, 6, 1), (768, 5, 1),
          (1024, 8, 1), (1536, 3, 1), (2048, 2, 1), (6, 256, 1), (3, 512, 1), (4, 1024, 1), (2, 2048, 1), (450, 800, 0),
          (1155, 12, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("ng,ny,opened", SHAPES)
@pytest.mark.parametrize("windowed", [0, 1])
def test_field_matches_the_oracle(gpu, llg_lib, oracle_lib, ng, ny, opened, windowed):
    import torch
    if windowed and ng * ny > 20000:
        pytest.skip("one window check per plan form is enough")
    p = llg_lib.default_params(ng, ny, demag_mode=llg_lib.DEMAG_OPEN if opened else llg_lib.DEMAG_PERIODIC,
                               demag_strength=2.5, windowed=windowed)
    rng = np.random.default_rng(ng * 1000 + ny)
    y = rng.uniform(-1.0, 1.0, 3 * ng * ny)
    ctx, o = llg_lib.Context(p), oracle_lib.Oracle(p)
    yin = y.copy()
    if windowed:
        w = rng.uniform(0.0, 1.0, ng * ny)
        axes = np.tile([1.0, 0.0, 0.0], (ng * ny, 1)).T.ravel().copy()
        ctx.set_window(w, axes, axes)
        yin = y * np.tile(w, 3)
        p0 = llg_lib.default_params(ng, ny, demag_mode=p.demag_mode, demag_strength=2.5)
        o = oracle_lib.Oracle(p0)
    want = o.demag(yin)
    h = torch.full((3 * ng * ny,), float("nan"), dtype=torch.float64, device=gpu)
    ctx.demag_apply(torch.from_numpy(y).to(gpu), h)
    # the chain's bound of the parity tests: device tensor and FFT against the host's
    assert rel_err(h.cpu().numpy(), want) <= 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("ng,ny,opened", [(7, 11, 0), (13, 49, 1), (61, 59, 1), (53, 3, 0), (91, 143, 0), (671, 17, 1),
                                          (16, 1891, 0), (2, 53, 0)])
def test_mixed_field_at_prime_lengths(gpu, llg_lib, oracle_lib, ng, ny, opened):
    """The FP32 chain's generic passes (one output per thread; 7, 11 and 13 in
    registers), in rows and columns, against the oracle's FP64 field."""
    import torch
    p = llg_lib.default_params(ng, ny, demag_mode=llg_lib.DEMAG_OPEN if opened else llg_lib.DEMAG_PERIODIC,
                               demag_strength=2.5, demag_precision=llg_lib.DEMAG_MIXED)
    y = np.random.default_rng(ng + ny).uniform(-1.0, 1.0, 3 * ng * ny)
    want = oracle_lib.Oracle(p).demag(y)
    h = torch.full((3 * ng * ny,), float("nan"), dtype=torch.float64, device=gpu)
    llg_lib.Context(p).demag_apply(torch.from_numpy(y).to(gpu), h)
    assert rel_err(h.cpu().numpy(), want) <= 5e-6   # the mixed chain's stated bound
