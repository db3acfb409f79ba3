"""The double flux's batched stages with p handed from stage to stage
(df_stage, csrc/pgb_host.cu; k_rcellflux_df, csrc/react.cuh) against the
per-block path: thin blocks, whose state is formed on the interior and copied,
and a thick one, formed over the halo too; the integrators' stage counts, with
two, three and four stages p's two fields taken in turn.

The bar is the per-block path's of the other batched tests: rounding, 1e-12 of
each component's largest."""

import numpy as np
import pytest

from peregrine_b200 import cases, native

pytestmark = pytest.mark.gpu


def layer(launch, integrator, mesh):
    import peregrine_b200 as pg

    cfg = cases.mixing_layer_config("pr", "euler-df", integrator, launch)
    mb = pg.get_solver(cfg, cases.mixing_layer_mesh(*mesh), pg.get_backend("cuda", cfg))
    mb.set_prims(cases.mixing_layer_prims(mb.metrics, mesh[1], seed=2))
    return mb


@pytest.mark.parametrize("mesh", [(37, 31, 3, 2), (48, 48, 48, 1)])
@pytest.mark.parametrize("integrator", ["rk1", "rk2", "tvd-rk3", "rk4", "rk34"])
def test_steps_as_the_per_block_path(mesh, integrator):
    a, b = layer("batched", integrator, mesh), layer("per-block", integrator, mesh)
    assert a.path == native.PATH_BATCHED and a.batched_form() == 2
    for mb in (a, b):
        mb.step(1e-9, 3)
    for x, y in zip(a.blocks, b.blocks):
        got, want = x.Q.get()[x.mesh.interior], y.Q.get()[y.mesh.interior]
        scale = np.abs(want).reshape(-1, want.shape[-1]).max(axis=0)
        scale[1:4] = scale[1:4].max()
        assert (np.abs(got - want).reshape(-1, want.shape[-1]).max(axis=0) / scale).max() < 1e-12
        # the state the last stage's right-hand side formed
        for name in ("p", "T"):
            got, want = (mb.sim.iovars.data(blk, [name])[name][x.mesh.interior] for mb, blk in ((a, x), (b, y)))
            assert np.abs(got - want).max() < 1e-9 * np.abs(want).max()


def records(nregs, rows):
    """Stage records of rows (register read, [(out, own weight, [(register, weight)], dQ's weight)]), dQ the last
    register."""
    recs = (native.Stage * len(rows))()
    for rec, (q, combines) in zip(recs, rows):
        rec.q, rec.dq, rec.ncombine = q, nregs - 1, len(combines)
        for cb, (out, own, reads, wdq) in zip(rec.combine, combines):
            cb.out, cb.own, cb.wout, cb.nterms, cb.step = out, int(own != 0.0), own, len(reads) + 1, 1
            for n, (r, w) in enumerate(reads + [(-1, wdq)]):
                cb.reg[n], cb.w[n] = r, w
    return recs, nregs


# tables whose stages do not all read what the stage before wrote: start 0, stages 1 and 2, dQ 3
REREAD = {
    # stage 2 reads the register stage 0 wrote
    "an older stage": [(0, [(1, 0.0, [(0, 1.0)], 0.5)]), (1, [(2, 0.0, [(0, 1.0)], 0.5)]),
                       (1, [(2, 0.5, [(0, 0.5)], 0.25)]), (2, [(0, 0.5, [(2, 0.5)], 0.5)])],
    # stage 1 reads the step's start again, and two stages more follow it
    "the step's start": [(0, [(1, 0.0, [(0, 1.0)], 0.5)]), (0, [(2, 0.0, [(1, 1.0)], 0.25)]),
                         (2, [(1, 0.0, [(0, 0.75), (2, 0.25)], 0.25)]), (1, [(2, 0.0, [(1, 1.0)], 0.25)]),
                         (2, [(0, 0.5, [(2, 0.5)], 0.25)])],
}


@pytest.mark.parametrize("mesh", [(37, 31, 3, 2), (48, 48, 48, 1)])
@pytest.mark.parametrize("table", list(REREAD))
def test_a_table_that_reads_a_register_again(monkeypatch, mesh, table):
    from peregrine_b200 import solver

    monkeypatch.setattr(solver, "stage_records", lambda name: records(4, REREAD[table]))
    a, b = layer("batched", "rk4", mesh), layer("per-block", "rk4", mesh)
    assert a.path == native.PATH_BATCHED and a.batched_form() == 2
    for mb in (a, b):
        mb.step(1e-9, 3)
    for x, y in zip(a.blocks, b.blocks):
        got, want = x.Q.get()[x.mesh.interior], y.Q.get()[y.mesh.interior]
        scale = np.abs(want).reshape(-1, want.shape[-1]).max(axis=0)
        scale[1:4] = scale[1:4].max()
        assert (np.abs(got - want).reshape(-1, want.shape[-1]).max(axis=0) / scale).max() < 1e-12


def test_each_face_has_its_own_area():
    """A long block's right-hand side off each face's own area and each cell's own volume (as in
    test_bounded_uniform_gpu.py): the mass, momentum and species rows as the per-block path's to the rounding of six
    faces, on a pressure whose differences are its own size.  (The energy row sums a plane's theta p, eps rho and kappa,
    tens of times their sum each; its bar is the steps' above.)"""
    import peregrine_b200 as pg

    out = []
    for launch in ("batched", "per-block"):
        cfg = cases.mixing_layer_config("pr", "euler-df", "tvd-rk3", launch)
        mb = pg.get_solver(cfg, cases.mixing_layer_mesh(8, 1500, 7, 1), pg.get_backend("cuda", cfg))
        prims = cases.mixing_layer_prims(mb.metrics, 1500, seed=2)
        for q in prims:
            q[..., 0] *= 1.0 + 0.2 * np.random.default_rng(4).uniform(-1.0, 1.0, q.shape[:-1])
        mb.set_prims(prims)
        mb.rhs()
        out.append(getattr(mb.blocks[0], mb.regs[-1]).get()[mb.blocks[0].mesh.interior])
        if launch == "batched":
            assert mb.path == native.PATH_BATCHED and mb.uniform(0)
    got, want = (x.reshape(-1, x.shape[-1]) for x in out)
    scale = np.abs(want).max(axis=0)
    scale[1:4] = scale[1:4].max()
    err = np.abs(got - want).max(axis=0) / scale
    assert np.delete(err, 4).max() < 64 * np.finfo(float).eps, err
