"""The stencil and block-inverse kernels, which are compiled per problem form
(window, anisotropy), against each other.

The block inverse that the preconditioner set-up stores (read from a
checkpoint) is the one psolve forms from the frozen (m, h): applied to a unit
vector psolve returns a column of it, each entry times one plus zeros.  The
comparison is bit for bit, so a form whose set-up kernel rounds otherwise shows.
"""
import numpy as np
import pytest

import llg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aniso", [llg.ANISO_LINEAR, llg.ANISO_CUBIC])
@pytest.mark.parametrize("shape", ["hole", "polycrystal"])
def test_stored_block_inverse_is_psolves(gpu, shape, aniso):
    import torch
    with torch.cuda.stream(torch.cuda.Stream()):
        _compare(torch, gpu, shape, aniso)


def _compare(torch, gpu, shape, aniso):
    ng, ny = 256, 128
    n = ng * ny
    kw = dict(geometry_kind=llg.GEOM_HOLE_SQUARE, hole_radius_frac_y=0.125) if shape == "hole" else \
        dict(geometry_kind=llg.GEOM_POLYCRYSTAL, num_grains=24, dead_grain_frac=0.1, grain_z_bias=1.0, hole_seed=3)
    geo = llg.build_geometry(llg.default_geom(ng, ny, ic_jitter_eps=0.01, **kw))
    ctx = llg.Context(llg.default_params(ng, ny, demag_mode=llg.DEMAG_OPEN, demag_strength=2.0, norm_kind=llg.NORM_REG,
                                         demag_precision=llg.DEMAG_MIXED, aniso_kind=aniso,
                                         windowed=int(shape == "polycrystal")), torch.cuda.current_stream())
    active = np.ones(n, bool)
    if shape == "hole":
        active = geo["active"] == 1
        ctx.set_mask(np.tile(geo["active"].astype(np.float64), 3))
    else:
        ctx.set_window(geo["w"], geo["msk3"], geo["nsk3"])
    y0 = torch.from_numpy(geo["y0"]).to(gpu)
    ctx.integrator_init(0.0, y0, llg.default_solver_opts(gs_type=llg.GS_CLASSICAL))
    ctx.integrate(0.05, torch.zeros_like(y0))
    # the checkpoint's last five vectors: frozen m, frozen h, three of inverse planes
    stored = ctx.checkpoint()[-3 * 24 * n:].copy().view(np.float64).reshape(3, 3, n)
    r, z = torch.zeros_like(y0), torch.zeros_like(y0)
    for b in range(3):
        r.zero_()
        r[b * n:(b + 1) * n] = 1.0
        ctx.psolve(0.0, r, r, r, z, 0.0)
        column = z.cpu().numpy().reshape(3, n)
        assert np.array_equal(column[:, active], stored[:, b, active]), b
