"""The caller's tile and instance of the uniform stage kernel against the
library's own choice (default_choice, csrc/pgb_host.cu): a set tile runs on the
instance asked for, or the first, whether it is set before the first step or
after the default has chosen another instance."""

import numpy as np
import pytest

from peregrine_b200 import autotune, cases, native

pytestmark = pytest.mark.gpu


def ragged():
    """264 tiles of the first instance for 148 SMs, so that the default takes the 14-wide one."""
    import peregrine_b200 as pg

    cfg = cases.tgv_config("euler", "tvd-rk3", "batched")
    mb = pg.get_solver(cfg, cases.tgv_mesh(64, (2, 2, 1)), pg.get_backend("cuda", cfg))
    mb.set_prims(cases.tgv_prims(mb.mesh_blocks, mb.metrics, seed=1, noise=1e-3))
    return mb


def test_a_set_tile_stays_whenever_it_is_set():
    first, later = ragged(), ragged()
    first.set_tile(0, 24, 7, 5)
    for _ in range(2):
        first.step(1e-4, 1)
    later.step(1e-4, 1)
    default = [later.get_tile(b) for b in range(4)]
    assert all(t[0] <= 14 for t in default), "the default is to choose another instance here"
    later.set_tile(0, 24, 7, 5)
    later.step(1e-4, 1)
    for mb in (first, later):
        assert mb.get_tile(0) == (24, 7, 5)
    assert [first.get_tile(b) for b in range(4)] == [later.get_tile(b) for b in range(4)]
    for x, y in zip(first.blocks, later.blocks):
        assert np.allclose(x.Q.get(), y.Q.get(), rtol=1e-12, atol=1e-9)
    # back to the default, and a tile no instance holds replaced by it
    for mb in (first, later):
        native.call("pgb_set_tile", mb.case, 0, 0, 0, 1)
        mb.step(1e-4, 1)
        assert [mb.get_tile(b) for b in range(4)] == default
        mb.set_tile(1, 32, 32, 5)
        mb.step(1e-4, 1)
        assert [mb.get_tile(b) for b in range(4)] == default


def test_an_instance_asked_for_stays():
    mb = ragged()
    mb.step(1e-4, 1)
    native.call("pgb_set_fused_shape", mb.case, 256, 1, 24)
    mb.set_tile(0, 24, 7, 5)
    mb.step(1e-4, 1)
    assert mb.get_tile(0) == (24, 7, 5)
    assert all(mb.get_tile(b)[0] > 14 for b in range(4))


def test_the_tuner_times_the_stage_kernel_alone():
    import peregrine_b200 as pg

    out = []
    for jostle in (0.0, 0.2):
        cfg = cases.tgv_config("navier-stokes", "rk4", "batched")
        mb = pg.get_solver(cfg, cases.tgv_mesh(24, jostle=jostle), pg.get_backend("cuda", cfg))
        mb.set_prims(cases.tgv_prims(mb.mesh_blocks, mb.metrics, seed=1, noise=1e-3))
        inner = mb.blocks[0].mesh.interior
        before = mb.blocks[0].Q.get()[inner]
        out.append(autotune.tune(mb, 1e-4, steps=1, ksplits=(1, 2)))
        assert np.array_equal(mb.blocks[0].Q.get()[inner], before)
    # a lattice steps by the stage kernel; a grid of general metrics by the passes, which have no tiles
    assert out[0]["candidates"] == 2 * len(autotune.shapes()) and out[1] is None


@pytest.mark.parametrize("simulator", ["euler", "navier-stokes"])
@pytest.mark.parametrize("shape", [(256, 1, 24), (256, 1, 30), (128, 2, 14), (512, 1, 14), (512, 1, 16)])
@pytest.mark.parametrize("cells,kchunk", [((13, 13, 13), 4), ((17, 9, 10), 9), ((23, 15, 7), 1)])
def test_tiles_of_one_plane(simulator, shape, cells, kchunk):
    """The tiles of one plane that k's remainder leaves at a block's top: the planes a tile fetches ahead end with
    the halo, in every instance."""
    import peregrine_b200 as pg
    from peregrine_b200.mesher import CubeMesher

    out = []
    for tiles in (False, True):
        cfg = cases.tgv_config(simulator, "rk4", "batched")
        mesh = CubeMesher(cells=[[c] for c in cells], lengths=[2 * np.pi] * 3, periodic=[True] * 3)
        mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
        mb.set_prims(cases.tgv_prims(mb.mesh_blocks, mb.metrics, seed=1, noise=1e-3))
        if tiles:
            native.call("pgb_set_fused_shape", mb.case, *shape)
            native.call("pgb_set_tile", mb.case, 0, 0, 0, 1)
            mb.step(0.0, 1)
            tw, th, _ = mb.get_tile(0)
            mb.set_tile(0, tw, th, kchunk)
        else:
            mb.step(0.0, 1)
        mb.step(1e-3, 3)
        if tiles:
            assert mb.get_tile(0) == (tw, th, kchunk)
        out.append(mb.blocks[0].Q.get()[mb.blocks[0].mesh.interior].reshape(-1, 5))
    scale = np.abs(out[0]).max(axis=0)
    scale[1:4] = scale[1:4].max()
    assert (np.abs(out[1] - out[0]).max(axis=0) / scale).max() < 1e-12
