"""What a case does where the device has no room for the passes' arrays
(ensure_scratch, csrc/pgb_host.cu): every call that needs them says so, the
second as the first, and once there is room the case steps as one that always
had it.  Memory is taken up by one allocation of torch's, which leaves room for
some of the arrays and not for all."""

import numpy as np
import pytest

from peregrine_b200 import cases, native

pytestmark = pytest.mark.gpu


def solver(n, launch="batched"):
    import peregrine_b200 as pg

    cfg = cases.mixing_config("navier-stokes", "rk2", "hllc", "muscl", "koren", 3, launch)
    mb = pg.get_solver(cfg, cases.tgv_mesh(n), pg.get_backend("cuda", cfg))
    mb.set_prims(cases.rough_prims(mb.metrics, 3, seed=3, speed=200.0))
    return mb


def fill(leave):
    """All but `leave` bytes of the device's free memory, held until it is let go."""
    import torch

    torch.zeros(1, device="cuda")
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def test_no_room_and_then_room():
    import torch

    solver(16).step(1e-5, 1)  # the kernels are loaded
    want, mb = solver(96), solver(96)
    want.step(1e-5, 2)
    # 1e6 cells: 200 MB of transport and gradients fit, 170 MB of face fluxes do not
    held = fill(256 << 20)
    try:
        for _ in range(2):
            with pytest.raises(native.PgbError):
                mb.step(1e-5, 2)
    finally:
        del held
        torch.cuda.empty_cache()
    mb.step(1e-5, 2)
    assert np.array_equal(mb.blocks[0].Q.get(), want.blocks[0].Q.get())


def curvilinear(n):
    import peregrine_b200 as pg

    cfg = cases.tgv_config("navier-stokes", "rk4", "batched")
    mb = pg.get_solver(cfg, cases.tgv_mesh(n, jostle=0.2), pg.get_backend("cuda", cfg))
    mb.set_prims(cases.tgv_prims(mb.mesh_blocks, mb.metrics, seed=1, noise=1e-3))
    return mb


def test_a_curvilinear_case_keeps_to_its_kernels():
    """A single-species case on a general grid steps by the passes where the device has room for their arrays and by
    the stage kernel where it has not; which is settled by its first step, for graphs and single launches alike."""
    import torch

    curvilinear(16).step(1e-4, 1)
    roomy, tight = curvilinear(96), curvilinear(96)
    roomy.step(1e-4, 2)
    passes = roomy.launches_per_step()
    held = fill(128 << 20)  # 250 MB are wanted
    try:
        tight.step(1e-4, 1)
        stage = tight.launches_per_step()
        assert stage < passes
        roomy.step(1e-4, 1)
        assert roomy.launches_per_step() == passes
    finally:
        del held
        torch.cuda.empty_cache()
    for graph in (True, False):
        tight.graph = graph
        tight.step(1e-4, 2)
        assert tight.launches_per_step() == stage
