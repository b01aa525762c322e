"""On the legacy default stream the kernels of a call are launched behind one
another (csrc/launch.h); on any other stream they run as plain launches or a
graph.  Both have to give the same bits, also where the shares of an in-place
kernel's blocks meet inside a memory sector: odd numbers of cells, odd spectrum
heights, unaligned vectors, neighbouring scalar slots."""
import numpy as np
import pytest

import llg

pytestmark = pytest.mark.gpu

DEMAG = [(llg.DEMAG_OPEN, llg.DEMAG_FP64), (llg.DEMAG_OPEN, llg.DEMAG_MIXED), (llg.DEMAG_OFF, llg.DEMAG_FP64)]


def _context(ng, ny, demag, stream=None):
    mode, prec = demag
    return llg.Context(llg.default_params(ng, ny, demag_mode=mode, demag_strength=2.0 if mode else 0.0,
                                          demag_precision=prec, norm_kind=llg.NORM_REG), stream)


def _state(ng, ny):
    m = np.random.default_rng(ng + ny).normal(size=(3, ng * ny)) * 0.2
    m[0] += 1.0
    return (m / np.sqrt((m * m).sum(axis=0))).ravel()


@pytest.mark.parametrize("demag", DEMAG)
@pytest.mark.parametrize("ng,ny", [(375, 225), (61, 59), (1025, 63), (250, 253)])
@pytest.mark.parametrize("offset", [0, 1])
def test_rhs_and_field(gpu, ng, ny, demag, offset):
    import torch
    n3 = 3 * ng * ny
    y0 = torch.zeros(n3 + offset, dtype=torch.float64, device=gpu)[offset:]   # offset 1: 8 bytes past alignment
    y0.copy_(torch.from_numpy(1.5 * _state(ng, ny)))                          # not normalised yet

    def one(stream, reps):
        ctx = _context(ng, ny, demag, stream)
        out = []
        for _ in range(reps):
            y, f, h = torch.empty(n3 + offset, dtype=torch.float64, device=gpu)[offset:], torch.empty_like(y0), \
                torch.zeros_like(y0)
            y.copy_(y0)
            ctx.rhs(0.0, y, f)
            if demag[0]:
                ctx.demag_apply(y0, h)
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in (y, f, h)])
        return out

    with torch.cuda.stream(torch.cuda.Stream()):
        want = one(torch.cuda.current_stream(), 1)[0]
    for got in one(None, 10):
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("demag", DEMAG)
@pytest.mark.parametrize("gs", [llg.GS_CLASSICAL, llg.GS_MODIFIED])
@pytest.mark.parametrize("ng,ny", [(61, 59), (375, 225)])
def test_integration(gpu, ng, ny, gs, demag):
    import torch
    y0 = torch.from_numpy(_state(ng, ny)).to(gpu)

    def one(stream):
        ctx = _context(ng, ny, demag, stream)
        y = torch.zeros_like(y0)
        ctx.integrator_init(0.0, y0, llg.default_solver_opts(gs_type=gs, mxstep=5000))
        ctx.integrate(0.05, y)
        torch.cuda.synchronize()
        s = ctx.stats()
        return y.cpu().numpy(), [s[k] for k in ("nst", "nni", "nli", "hlast")]

    with torch.cuda.stream(torch.cuda.Stream()):
        want = one(torch.cuda.current_stream())
    assert want[1][2] > 0
    got = one(None)
    assert got[1] == want[1] and np.array_equal(got[0], want[0])
