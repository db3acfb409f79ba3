"""The fused passes' faces on uniform blocks (csrc/uniface.cuh) and the passes
around them (every field's halo in one pass, the divergence and combines a
component a thread) against the per-block path, at extents where a face range
ends inside a CTA, a block is two cells thin, or blocks of one case differ in
form.

The bar: both paths round each flux within a few eps of its own size, the
largest the pressure's in a momentum row and the enthalpy's in the energy row,
some 10 eps each of a face; over three steps of a CFL number below one a row
moves by at most that, 1e-12 of its largest value being some 4000 eps."""

import numpy as np
import pytest

from peregrine_b200 import cases, native
from peregrine_b200.mesher import CubeMesher

pytestmark = pytest.mark.gpu


def pair(cfg_of, mesh_of, prims_of, dt, steps=3):
    import peregrine_b200 as pg

    out = []
    for launch in ("batched", "per-block"):
        cfg, mesh = cfg_of(launch), mesh_of()
        mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
        mb.set_prims(prims_of(mb))
        mb.step(dt, steps)
        out.append(mb)
    return out


def compare(a, b, bar=1e-12):
    assert a.path == native.PATH_BATCHED and b.path == native.PATH_PER_BLOCK
    for x, y in zip(a.blocks, b.blocks):
        got, want = x.Q.get()[x.mesh.interior], y.Q.get()[y.mesh.interior]
        scale = np.abs(want).reshape(-1, want.shape[-1]).max(axis=0)
        scale[1:4] = scale[1:4].max()
        scale[scale == 0.0] = 1.0
        err = (np.abs(got - want).reshape(-1, want.shape[-1]).max(axis=0) / scale).max()
        assert err < bar, err


def box(cells, blocks=(1, 1, 1), lengths=(2 * np.pi,) * 3, jostle=0.0):
    cuts = [[n // b + (1 if m < n - n // b * b else 0) for m in range(b)] for n, b in zip(cells, blocks)]
    return CubeMesher(mbdims=list(blocks), cells=cuts, lengths=list(lengths), periodic=[True] * 3, jostle=jostle)


@pytest.mark.parametrize("cells,blocks", [((13, 17, 11), (1, 1, 1)), ((2, 33, 35), (1, 1, 1)), ((37, 2, 31), (1, 1, 1)),
                                          ((64, 16, 2), (2, 1, 1)), ((19, 16, 21), (2, 2, 3))])
@pytest.mark.parametrize("primary,recon,limiter", [("kepaec", "constant", None), ("hllc", "muscl", "koren"),
                                                   ("hllc", "muscl", "vanleer"), ("rusanov", "muscl", "minmod"),
                                                   ("ausmup", "muscl", "mc")])
def test_calorically_perfect(cells, blocks, primary, recon, limiter):
    for simulator, ns in (("navier-stokes", 3), ("euler", 2)):
        a, b = pair(lambda launch: cases.mixing_config(simulator, "tvd-rk3", primary, recon, limiter, ns, launch),
                    lambda: box(cells, blocks), lambda mb: cases.rough_prims(mb.metrics, ns, seed=3, speed=200.0), 1e-5)
        assert all(a.uniform(n) for n in range(len(a.blocks)))
        compare(a, b)


@pytest.mark.parametrize("cells,blocks", [((13, 17, 11), (1, 1, 1)), ((23, 10, 16), (2, 1, 2))])
@pytest.mark.parametrize("tables,primary,recon,limiter", [("h2o2_gri30", "hllc", "muscl", "koren"),
                                                          ("h2o2_gri30", "kepaec", "constant", None),
                                                          ("h2o2_gri30", "rusanov", "muscl", "superbee")])
def test_thermally_perfect(cells, blocks, tables, primary, recon, limiter):
    def prims(mb):
        MW = mb.mixture.constants()["MW"]
        return cases.reacting_prims(mb.metrics, mb.mixture.spnames, MW, cells[0], seed=5, width=2.0, dT=500.0,
                                    radicals=1e-3)

    a, b = pair(lambda launch: cases.reacting_config("navier-stokes", "tvd-rk3", primary, recon, limiter, True, tables,
                                                     launch),
                lambda: box(cells, blocks, (0.01,) * 3), prims, 2e-8)
    assert all(a.uniform(n) for n in range(len(a.blocks)))
    # T's root carries the fits' rounding, 1e-13 of T, into the pressure, whose
    # difference across a cell drives a momentum a thousandth of its flux
    compare(a, b, 1e-11)


@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("primary,recon,limiter", [("hllc", "muscl", "koren"), ("kepaec", "constant", None),
                                                   ("rusanov", "muscl", "mc")])
def test_uniform_and_curvilinear_blocks_in_one_case(simulator, primary, recon, limiter):
    # a jostled block and its neighbours, whose halos hold its nodes, are read
    # by their metric arrays, the lattice blocks past them are not; the faces
    # between are formed by both
    class One(CubeMesher):
        def _shape(self, blk, ijk):
            self.jostle = 0.1 if ijk[0] == 2 else 0.0
            super()._shape(blk, ijk)

    def mesh():
        return One(mbdims=[5, 1, 1], cells=[[7, 6, 5, 4, 6], [14], [11]], lengths=[2 * np.pi] * 3, periodic=[True] * 3)

    a, b = pair(lambda launch: cases.mixing_config(simulator, "tvd-rk3", primary, recon, limiter, 2, launch),
                mesh, lambda mb: cases.rough_prims(mb.metrics, 2, seed=3, speed=200.0), 1e-5)
    assert [a.uniform(n) for n in range(5)] == [True, False, False, False, True]
    compare(a, b)


def test_each_face_has_its_own_area():
    """As in test_bounded_uniform_gpu.py: a long block's right-hand side off each face's own area."""
    import peregrine_b200 as pg

    out = []
    for launch in ("batched", "per-block"):
        cfg = cases.mixing_config("euler", "tvd-rk3", "hllc", "muscl", "koren", 2, launch)
        mb = pg.get_solver(cfg, box((8, 1500, 7), lengths=(0.7, 90.0, 0.7)), pg.get_backend("cuda", cfg))
        mb.set_prims(cases.bc_box_prims(mb.metrics, 2, seed=3, speed=200.0))
        mb.rhs()
        out.append(getattr(mb.blocks[0], mb.regs[-1]).get()[mb.blocks[0].mesh.interior])
        if launch == "batched":
            assert mb.path == native.PATH_BATCHED and mb.uniform(0)
    got, want = (x.reshape(-1, x.shape[-1]) for x in out)
    scale = np.abs(want).max(axis=0)
    scale[1:4] = scale[1:4].max()
    err = (np.abs(got - want).max(axis=0) / scale).max()
    assert err < 64 * np.finfo(float).eps, err


@pytest.mark.parametrize("still", ["A", "B", "C"])
def test_a_species_that_does_not_diffuse(still):
    """An infinite Lewis number: the species' own coefficient is zero, and the others' are what they were."""
    def cfg_of(launch):
        cfg = cases.mixing_config("navier-stokes", "tvd-rk3", "hllc", "muscl", "koren", 3, launch)
        cfg["mixture"]["species"] = {k: dict(v, lewis=np.inf if k == still else v["lewis"])
                                     for k, v in cfg["mixture"]["species"].items()}
        return cfg.validate()

    a, b = pair(cfg_of, lambda: box((13, 17, 11)), lambda mb: cases.rough_prims(mb.metrics, 3, seed=3, speed=200.0), 1e-5)
    compare(a, b)


@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("primary,recon,limiter", [("kepaec", "constant", None), ("hllc", "muscl", "koren"),
                                                   ("rusanov", "muscl", "superbee"), ("ausmup", "muscl", "vanleer")])
def test_supersonic_faces(simulator, primary, recon, limiter):
    # at this speed faces of both signs are supersonic along every axis, where one side's flux is the face's
    a, b = pair(lambda launch: cases.mixing_config(simulator, "rk2", primary, recon, limiter, 3, launch),
                lambda: box((13, 17, 11)), lambda mb: cases.rough_prims(mb.metrics, 3, seed=3, speed=1500.0), 2e-6)
    assert all(a.uniform(n) for n in range(len(a.blocks)))
    compare(a, b)
    got, want = a.cflmax(), b.cflmax()
    assert all(abs(got[k] - want[k]) < 1e-12 * want[k] for k in want)
