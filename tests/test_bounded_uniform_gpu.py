"""Bounded cases on uniform blocks, packed: the uniform faces with the
boundaries' passes between (pgb_plain_bounded, csrc/plain_tu.cu) against the
per-block kernels, every boundary kind, at extents where a pass ends inside a
CTA.  The bar is the rounding of the fluxes, as in test_uniform_faces_gpu.py."""

import numpy as np
import pytest

from peregrine_b200 import cases, native

pytestmark = pytest.mark.gpu

KINDS = ["slp-adia-wall", "slp-isot-wall", "sub-in-fvt", "sup-in-fa", "sub-in-ftptt", "sub-in-fmt", "sub-out-fp",
         "sup-out-fn"]
VISCOUS = ["no-slp-adia-wall", "no-slp-isot-wall", "mov-adia-wall", "mov-isot-wall"]


def run(cfg, mesh, prims_of, launch, dt, steps):
    import peregrine_b200 as pg

    mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
    mb.set_prims(prims_of(mb))
    mb.path = launch
    mb.step(dt, steps)
    return mb


def compare(a, b, bar=1e-12):
    for x, y in zip(a.blocks, b.blocks):
        for reg in ("Q", a.regs[-1]):
            got, want = getattr(x, reg).get()[x.mesh.interior], getattr(y, reg).get()[y.mesh.interior]
            scale = np.abs(want).reshape(-1, want.shape[-1]).max(axis=0)
            scale[1:4] = scale[1:4].max()
            err = (np.abs(got - want).reshape(-1, want.shape[-1]).max(axis=0) / np.where(scale > 0, scale, 1.0)).max()
            # dQ is a difference of fluxes some hundred times it
            assert err < (bar if reg == "Q" else 100 * bar), (reg, err)


@pytest.mark.parametrize("kind,simulator", [(k, s) for k in KINDS for s in ("euler", "navier-stokes")] +
                         [(k, "navier-stokes") for k in VISCOUS])
@pytest.mark.parametrize("primary,recon,limiter,ns", [("hllc", "muscl", "koren", 2), ("kepaec", "constant", None, 1)])
def test_every_kind(kind, simulator, primary, recon, limiter, ns):
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config(kind, ns=ns, simulator=simulator, primary=primary, recon=recon, limiter=limiter, seed=3)
        out.append(run(cfg, cases.bc_box_mesh(cells=(14, 13, 13), jostle=0.0),
                       lambda mb: cases.bc_box_prims(mb.metrics, ns, seed=3, speed=60.0), launch, 2e-7, 3))
    compare(*out)


@pytest.mark.parametrize("cells,blocks", [((23, 14, 13), (2, 1, 1)), ((17, 12, 16), (1, 2, 2))])
def test_the_channel(cells, blocks):
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.channel_config()
        out.append(run(cfg, cases.channel_mesh(cells, blocks),
                       lambda mb: cases.bc_box_prims(mb.metrics, 2, seed=1, speed=30.0), launch, 2e-7, 5))
    compare(*out)
