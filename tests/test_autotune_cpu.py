"""The tuner's handling of a candidate that fails (peregrine_b200/autotune.py),
on a fake of the library's calls: one the library refuses is passed over, a
device error ends the tuning."""

import numpy as np
import pytest

from peregrine_b200 import autotune, native


class Mb:
    path = native.PATH_BATCHED
    case = None
    mesh_blocks = [type("Block", (), {"cells": (8, 8, 8)})()]

    def __init__(self):
        q = type("Array", (), {"get": lambda s: np.zeros(1), "set": lambda s, v: None})()
        self.blocks = [type("Block", (), {"Q": q})()]

    def get_tile(self, n):
        return 8, 8, 8

    def set_tile(self, n, tw, th, kc):
        pass


def fake(fail):
    def call(name, *args):
        if name == "pgb_fused_shapes":
            for n, v in enumerate((256, 1, 24, 7, 512, 1, 14, 8)):
                args[0][n] = v
            args[2]._obj.value = 2
        elif name == "pgb_case_tiled":
            args[1]._obj.value = 1
        elif name == "pgb_last_step_ms":
            args[1]._obj.value = 1.0
        elif name == "pgb_set_fused_shape" and args[1] == 512:
            raise fail

    return call


def test_a_refused_candidate_is_passed_over_and_a_device_error_is_not(monkeypatch):
    monkeypatch.setattr(native, "call", fake(native.PgbError("no such shape")))
    assert autotune.tune(Mb(), 1.0, ksplits=(1,))["candidates"] == 1
    monkeypatch.setattr(native, "call", fake(native.PgbCudaError("an illegal memory access was encountered")))
    with pytest.raises(native.PgbCudaError):
        autotune.tune(Mb(), 1.0, ksplits=(1,))
