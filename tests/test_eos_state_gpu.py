"""pgb_eos_get after steps replayed from a captured graph: refused after the
stage kernel's, which keeps no state array, and given after the packed path's,
whichever path was stepped before."""

import ctypes

import numpy as np
import pytest

from peregrine_b200 import cases, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jostle", [0.0, 0.2])
def test_a_replayed_graph_says_what_it_keeps(jostle):
    import peregrine_b200 as pg

    cfg = cases.tgv_config("navier-stokes", "rk4", "batched")
    mb = pg.get_solver(cfg, cases.tgv_mesh(16, jostle=jostle), pg.get_backend("cuda", cfg))
    prims = cases.tgv_prims(mb.mesh_blocks, mb.metrics, seed=1, noise=1e-3)
    blk = mb.blocks[0]

    def T():
        out = np.empty(np.prod(blk.Q.shape[:3]))
        native.call("pgb_eos_get", mb.case, 0, 1, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), out.size)
        return out.reshape(blk.Q.shape[:3], order="F")[blk.mesh.interior]

    assert mb.graph
    for _ in range(2):  # the first captures the graph, the second replays it
        mb.set_prims(prims)
        before = T()
        mb.step(1e-3, 4)
        with pytest.raises(native.PgbError):
            T()
        mb.path = native.PATH_PACKED
        mb.step(1e-3, 4)
        after = T()
        assert np.abs(after - before).max() > 0.0
        mb.path = native.PATH_BATCHED
