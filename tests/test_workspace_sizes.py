"""The workspace that the fp32 engines ask for (host only): its k-split scratch follows the engine's products, so that a small
engine stays small; a large one is capped at two partial tiles per SM (19.4 MB at 148)."""
import ctypes

import pytest

from cavs_b200 import lib
from cavs_b200.treelstm import Config


def _bytes(engine, *cfg):
    fn = getattr(lib(), f"cavs_{engine}_workspace_bytes")
    fn.restype = ctypes.c_size_t
    return fn(ctypes.byref(Config(*cfg)))


@pytest.mark.parametrize("engine", ["treelstm", "treegru"])
def test_a_small_fp32_engine_has_a_small_workspace(engine):
    # hidden 32, embedding 16: the largest product's partials are 32 splits of [16, 128] or [32, 96] values
    assert 0 < _bytes(engine, 32, 16, 100, 5, 2, 0, 200, 100) < 4e6
