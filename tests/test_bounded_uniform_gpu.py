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


def pg_solver(cfg, mesh):
    import peregrine_b200 as pg

    return pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))


def run(cfg, mesh, prims_of, launch, dt, steps):
    mb = pg_solver(cfg, mesh)
    mb.set_prims(prims_of(mb))
    mb.path = launch
    mb.step(dt, steps)
    return mb


def compare(a, b, bar=1e-12):
    # a's packed steps took the uniform faces: its blocks were found uniform, which only they ask for
    assert a.path == native.PATH_PACKED and all(a.uniform(n) for n in range(len(a.blocks)))
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


@pytest.mark.parametrize("kind", ["no-slp-isot-wall", "mov-adia-wall", "sub-in-fmt", "sub-out-fp"])
@pytest.mark.parametrize("primary,recon,limiter", [("kepaec", "constant", None), ("hllc", "muscl", "vanleer"),
                                                   ("rusanov", "muscl", "superbee"), ("ausmup", "muscl", "mc")])
def test_every_scheme(kind, primary, recon, limiter):
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config(kind, ns=3, simulator="navier-stokes", primary=primary, recon=recon,
                                  limiter=limiter, seed=3)
        out.append(run(cfg, cases.bc_box_mesh(cells=(14, 13, 13), jostle=0.0),
                       lambda mb: cases.bc_box_prims(mb.metrics, 3, seed=3, speed=60.0), launch, 2e-7, 3))
    compare(*out)


@pytest.mark.parametrize("kind", ["no-slp-isot-wall", "sub-in-ftptt", "sub-out-fp"])
@pytest.mark.parametrize("simulator,chemistry", [("euler", False), ("navier-stokes", False), ("navier-stokes", True)])
@pytest.mark.parametrize("primary,recon,limiter", [("kepaec", "constant", None), ("hllc", "muscl", "koren")])
def test_thermally_perfect(kind, simulator, chemistry, primary, recon, limiter):
    """Kinetic-theory transport and the coupled source between the same passes."""
    if simulator == "euler" and kind.startswith("no-slp"):
        kind = "slp-isot-wall"
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config(kind, simulator=simulator, primary=primary, recon=recon, limiter=limiter, eos="tpg",
                                  seed=3, tables=cases.H2O2_TABLES)
        if chemistry:
            cfg["mixture"]["chemistry"], cfg["chem-integration"]["kind"] = "finite-rate", "coupled"
            cfg = cfg.validate()
        out.append(run(cfg, cases.bc_box_mesh(cells=(14, 13, 13), jostle=0.0),
                       lambda mb: cases.bc_box_prims(mb.metrics, 9, seed=3, speed=60.0), launch, 2e-9, 3))
    # T's root carries the fits' rounding, as in test_uniform_faces_gpu.py
    compare(*out, bar=1e-11)


@pytest.mark.parametrize("primary,recon,limiter,ns", [("hllc", "muscl", "koren", 2), ("kepaec", "constant", None, 1)])
def test_each_face_has_its_own_area(primary, recon, limiter, ns):
    """A long block is uniform to some hundreds of eps, its node coordinates' rounding over a spacing; a right-hand
    side off its first cell's areas and volume is off by as much.  With each face's own it is as the per-block path's
    to the fluxes' rounding: six faces of some 10 eps each, their size the row's on this rough field."""
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config("slp-adia-wall", ns=ns, simulator="euler", primary=primary, recon=recon,
                                  limiter=limiter, seed=3)
        mesh = cases.bc_box_mesh(cells=(8, 1500, 7), jostle=0.0, lengths=(0.7, 90.0, 0.7))
        mb = pg_solver(cfg, mesh)
        mb.set_prims(cases.bc_box_prims(mb.metrics, ns, seed=3, speed=200.0))
        mb.path = launch
        mb.rhs()
        out.append(getattr(mb.blocks[0], mb.regs[-1]).get()[mb.blocks[0].mesh.interior])
        if launch == native.PATH_PACKED:
            assert mb.uniform(0)
    got, want = (x.reshape(-1, x.shape[-1]) for x in out)
    scale = np.abs(want).max(axis=0)
    scale[1:4] = scale[1:4].max()
    err = (np.abs(got - want).max(axis=0) / scale).max()
    assert err < 64 * np.finfo(float).eps, err


def test_a_stage_that_scales_its_own_dq(monkeypatch):
    """A table whose first combine writes dQ's register, which the second then reads: what the combines' own passes
    read there is the scaled value."""
    from peregrine_b200 import solver

    def records(name):
        recs = (native.Stage * 1)()
        recs[0].q, recs[0].dq, recs[0].ncombine = 0, 1, 2
        scale, add = recs[0].combine
        scale.out, scale.nterms, scale.step = 1, 1, 1
        scale.reg[0], scale.w[0] = -1, 1.0
        add.out, add.own, add.wout, add.nterms, add.step = 0, 1, 1.0, 1, 0
        add.reg[0], add.w[0] = 1, 0.5
        return recs, 2

    monkeypatch.setattr(solver, "stage_records", records)
    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config("slp-adia-wall", ns=2, primary="hllc", recon="muscl", limiter="koren", seed=3)
        out.append(run(cfg, cases.bc_box_mesh(cells=(14, 13, 13), jostle=0.0),
                       lambda mb: cases.bc_box_prims(mb.metrics, 2, seed=3, speed=60.0), launch, 2e-7, 3))
    compare(*out)
