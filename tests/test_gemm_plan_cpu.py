"""Which GEMM kernel a product goes to: host arithmetic of the library, for 148 SMs where there is no GPU."""
import ctypes
import json
import os
import subprocess
import sys

import pytest

from causal_trainer_dev_b200.ops.build import LIB_PATH

pytestmark = pytest.mark.skipif(not LIB_PATH.exists(), reason="the CUDA library is not built")

FEW_TILES = [(512, 512, 8192), (640, 328, 4104), (64, 1536, 8960), (1000, 1536, 17920)]
MANY_TILES = [(4096, 1024, 64), (16384, 4096, 4096), (128, 256, 1024)]

_CHOICE = """
import ctypes, sys
lib = ctypes.CDLL(sys.argv[1])
w, s = ctypes.c_int(), ctypes.c_int()
shapes = [tuple(map(int, a.split(","))) for a in sys.argv[2:]]
print([lib.ctb_gemm_split_choice(*x, ctypes.byref(w), ctypes.byref(s)) for x in shapes])
"""


def _choices(shapes, **env):
    out = subprocess.run([sys.executable, "-c", _CHOICE, str(LIB_PATH), *(",".join(map(str, x)) for x in shapes)],
                         capture_output=True, text=True, check=True, env={**os.environ, **env})
    return json.loads(out.stdout)


def test_few_tiles_and_long_k_go_to_the_cluster_kernel():
    assert _choices(FEW_TILES) == [1] * len(FEW_TILES)
    assert _choices(MANY_TILES) == [0] * len(MANY_TILES)


@pytest.mark.parametrize("switch", ["CTB_GEMM_TM=1", "CTB_GEMM_TM=2", "CTB_GEMM_SPLITK=1", "CTB_GEMM_DYNAMIC_TILES=1"])
def test_a_switch_of_the_persistent_kernel_reaches_every_product(switch):
    name, value = switch.split("=")
    assert _choices(FEW_TILES, **{name: value}) == [0] * len(FEW_TILES)
    assert _choices(FEW_TILES, **{name: ""}) == [1] * len(FEW_TILES)


def test_split_k_mode_of_the_persistent_kernel_reaches_every_product():
    lib = ctypes.CDLL(str(LIB_PATH))
    w, s = ctypes.c_int(), ctypes.c_int()
    before = lib.ctb_gemm_set_split_k(1)
    try:
        assert all(lib.ctb_gemm_split_choice(*x, ctypes.byref(w), ctypes.byref(s)) == 0 for x in FEW_TILES)
    finally:
        lib.ctb_gemm_set_split_k(before)
    assert all(lib.ctb_gemm_split_choice(*x, ctypes.byref(w), ctypes.byref(s)) == 1 for x in FEW_TILES)
