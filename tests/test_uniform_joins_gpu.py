"""The fused passes over joins that are not low face to high face in the
identity orientation, against the per-block path of the same blocks: axes
running backward (negative area vectors; such a block stays uniform), axes
permuted (such a block reads its metric arrays, its neighbour may not), and
faces joined by a rotation, whose halo cells' momentum and velocity are turned
(k_ufaces and k_halo_fields, csrc/uniface.cuh; k_halo_boxes2 from a field
offset, csrc/plain.cuh).  Blocks of 2048 cells or more in all, which is where
these passes run.

The bar is test_uniform_faces_gpu.py's."""

import numpy as np
import pytest

from peregrine_b200 import cases, native
from peregrine_b200.mesher import CubeMesher, fill_node_halos, reorient

pytestmark = pytest.mark.gpu


class Reoriented(CubeMesher):
    """A periodic box of two blocks, the second laid out along other axes."""

    def __init__(self, S, length):
        super().__init__(mbdims=[2, 1, 1], cells=[[14, 13], [12], [15]], lengths=[length] * 3, periodic=[True] * 3)
        self.S = S

    def make_blocks(self, ng):
        blocks = super().make_blocks(ng)
        reorient(blocks, 1, self.S)
        fill_node_halos(blocks)
        return blocks


class Pinwheel(CubeMesher):
    """One block, a quarter of the plane's p4 pattern: its low i and j faces joined by a quarter turn about their
    common edge, its high ones about theirs, k periodic."""

    def __init__(self, n, nk, length, klength=None):
        super().__init__(cells=[[n], [n], [nk]], lengths=[length, length, klength or length * nk / n],
                         periodic=[True] * 3)

    def make_blocks(self, ng):
        blocks = super().make_blocks(ng)
        turn = np.array([[0.0, -1.0, 0.0], [1.0, 0.0, 0.0], [0.0, 0.0, 1.0]])
        for nface in (1, 2, 3, 4):
            face = blocks[0].get_intface(nface)
            face.orient, face.rot = ("513", turn) if nface < 3 else ("243", turn.T)
            face.set_nbrface()
        return blocks


def pair(cfg_of, mesh, prims_of, dt, uniform=None, steps=3):
    import peregrine_b200 as pg

    out = []
    for launch in ("batched", "per-block"):
        cfg = cfg_of(launch)
        mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
        mb.set_prims(prims_of(mb))
        mb.step(dt, steps)
        out.append(mb)
    a, b = out
    assert a.path == native.PATH_BATCHED and b.path == native.PATH_PER_BLOCK and a.batched_form() == 2
    assert [a.uniform(n) for n in range(len(a.blocks))] == uniform
    return a, b


def compare(a, b, bar=1e-12):
    for x, y in zip(a.blocks, b.blocks):
        got, want = x.Q.get()[x.mesh.interior], y.Q.get()[y.mesh.interior]
        scale = np.abs(want).reshape(-1, want.shape[-1]).max(axis=0)
        scale[1:4] = scale[1:4].max()
        err = (np.abs(got - want).reshape(-1, want.shape[-1]).max(axis=0) / scale).max()
        assert err < bar, err


SCHEMES = [("kepaec", "constant", None), ("hllc", "muscl", "koren"), ("rusanov", "muscl", "minmod"),
           ("ausmup", "muscl", "vanleer")]


@pytest.mark.parametrize("S", ["156", "426", "453", "264", "345"])
@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("primary,recon,limiter", SCHEMES)
def test_a_block_laid_out_along_other_axes(S, simulator, primary, recon, limiter):
    a, b = pair(lambda launch: cases.mixing_config(simulator, "tvd-rk3", primary, recon, limiter, 3, launch),
                Reoriented(S, 2 * np.pi), lambda mb: cases.rough_prims(mb.metrics, 3, seed=3, speed=200.0), 1e-5,
                uniform=[True, S in ("156", "426", "453")])
    compare(a, b)
    got, want = a.cflmax(), b.cflmax()
    assert all(abs(got[k] - want[k]) < 1e-12 * want[k] for k in want)


@pytest.mark.parametrize("S", ["156", "264"])
def test_a_reacting_block_laid_out_along_other_axes(S):
    def prims(mb):
        return cases.reacting_prims(mb.metrics, mb.mixture.spnames, mb.mixture.constants()["MW"], 14, seed=5,
                                    width=2.0, dT=500.0, radicals=1e-3)

    a, b = pair(lambda launch: cases.reacting_config(launch=launch), Reoriented(S, 0.01), prims, 2e-8,
                uniform=[True, S == "156"])
    compare(a, b, 1e-11)


@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("primary,recon,limiter", SCHEMES)
def test_faces_joined_by_a_quarter_turn(simulator, primary, recon, limiter):
    a, b = pair(lambda launch: cases.mixing_config(simulator, "tvd-rk3", primary, recon, limiter, 2, launch),
                Pinwheel(15, 13, 2 * np.pi), lambda mb: cases.rough_prims(mb.metrics, 2, seed=3, speed=200.0), 1e-5,
                uniform=[True])
    compare(a, b)


@pytest.mark.parametrize("n,nk", [(16, 12), (41, 2)])
def test_the_double_flux_across_a_quarter_turn(n, nk):
    a, b = pair(lambda launch: cases.mixing_layer_config("pr", "euler-df", "tvd-rk3", launch),
                Pinwheel(n, nk, n * 2e-5), lambda mb: cases.mixing_layer_prims(mb.metrics, n, seed=2), 1e-9,
                uniform=[True])
    compare(a, b)


def bounded(mesh, simulator, primary, recon, limiter):
    """The packed steps of a box whose k faces are walls against the per-block ones."""
    import peregrine_b200 as pg

    out = []
    for launch in (native.PATH_PACKED, native.PATH_PER_BLOCK):
        cfg = cases.bc_box_config("no-slp-isot-wall" if simulator == "navier-stokes" else "slp-adia-wall", ns=2,
                                  simulator=simulator, primary=primary, recon=recon, limiter=limiter, seed=3)
        mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
        mb.set_prims(cases.bc_box_prims(mb.metrics, 2, seed=3, speed=60.0))
        mb.path = launch
        mb.step(2e-7, 3)
        out.append(mb)
    assert all(out[0].uniform(n) for n in range(len(out[0].blocks)))
    compare(*out)


@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("primary,recon,limiter", SCHEMES)
def test_bounded_blocks_joined_by_a_quarter_turn(simulator, primary, recon, limiter):
    mesh = Pinwheel(15, 13, 1.0)
    mesh.periodic[2], mesh.defaultbc = False, "outer"
    bounded(mesh, simulator, primary, recon, limiter)


@pytest.mark.parametrize("S", ["156", "426", "453"])
@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
def test_a_bounded_block_laid_out_along_other_axes(S, simulator):
    mesh = Reoriented(S, 1.0)
    mesh.periodic[2], mesh.defaultbc = False, "outer"
    bounded(mesh, simulator, "hllc", "muscl", "koren")
