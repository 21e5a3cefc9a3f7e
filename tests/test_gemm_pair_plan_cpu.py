"""The choice of the two-CTA kernel's form: host arithmetic of the library, for 148 SMs where there is no GPU."""
import ctypes
import random
import subprocess
import sys

import pytest

from causal_trainer_dev_b200.ops.build import LIB_PATH

pytestmark = pytest.mark.skipif(not LIB_PATH.exists(), reason="the CUDA library is not built")


def _choice(lib, m, n, k, f32=0, accumulate=0):
    form = (ctypes.c_int * 4)()
    return tuple(form) if lib.ctb_gemm_pair_choice(m, n, k, f32, accumulate, form) else None


def test_every_choice_is_a_plan_that_the_kernel_takes():
    lib = ctypes.CDLL(str(LIB_PATH))
    lib.ctb_gemm_workspace.restype = ctypes.c_long
    rng = random.Random(1)
    taken = split = 0
    for _ in range(2000):
        m, n, k = (int(2 ** rng.uniform(0, 17)) for _ in range(3))
        assert n % 8 == 0 or _choice(lib, m, n, k) is None         # rows that end inside of 16 bytes stay where they were
        n = n + -n % 8
        for f32, accumulate in ((0, 0), (1, 0), (1, 1)):
            plan = _choice(lib, m, n, k, f32, accumulate)
            size = lib.ctb_gemm_workspace(m, n, k, 0, f32, accumulate)
            if plan is None:
                assert size == 0
                continue
            tm, whole, slices, band = plan
            tiles = -(-m // (256 * tm)) * -(-n // 256)
            assert tm in (1, 2) and 0 <= whole <= tiles and 1 <= slices <= 8 and band >= 1
            assert whole == tiles or (not accumulate and slices > 1 and -(-k // 64) >= 4 * slices)
            assert size == (tiles - whole) * slices * 256 * tm * 256 * 4 <= 320 << 20
            taken, split = taken + 1, split + (whole < tiles)
    assert taken > 500 and split > 50


def test_the_choice_does_not_depend_on_the_calls_before_it():
    shapes = [(1000, 1536, 17920), (4096, 4096, 128256), (64, 64, 64), (700, 4096, 14336), (16384, 28672, 4096)]
    code = ("import ctypes, sys\nlib = ctypes.CDLL(sys.argv[1])\nf = (ctypes.c_int * 4)()\n"
            "print([(lib.ctb_gemm_pair_choice(*map(int, a.split(',')), 0, 0, f), *f) if "
            "lib.ctb_gemm_pair_choice(*map(int, a.split(',')), 0, 0, f) else None for a in sys.argv[2:]])")
    run = lambda order: subprocess.run(  # noqa: E731
        [sys.executable, "-c", code, str(LIB_PATH), *(",".join(map(str, s)) for s in order)], capture_output=True, text=True,
        check=True).stdout
    forward, backward = eval(run(shapes)), eval(run(shapes[::-1]))
    assert forward == backward[::-1]
    assert forward[0] is not None and forward[1] is not None and forward[2] is None


def test_the_loss_products_choose_whole_tiles():
    """Their epilogues see whole logits: no K slices.  Both tile heights occur."""
    lib = ctypes.CDLL(str(LIB_PATH))
    rng, form, seen = random.Random(2), (ctypes.c_int * 4)(), set()
    for _ in range(3000):
        rows, vocab, d = rng.randint(1, 4096), 8 * rng.randint(100, 16000), 8 * rng.randint(16, 512)
        for gradients in (0, 1):
            if lib.ctb_ce_pair_choice(rows, vocab, d, gradients, form):
                tm, whole, slices, band = form
                assert whole == -(-rows // (256 * tm)) * -(-vocab // 256) and slices == 1 and band >= 1
                seen.add((gradients, tm))
            else:
                seen.add((gradients, None))
    assert seen == {(g, tm) for g in (0, 1) for tm in (1, 2, None)}


def test_the_mode_switch_turns_the_choice_off_and_on():
    lib = ctypes.CDLL(str(LIB_PATH))
    before = lib.ctb_gemm_set_pair(0)
    try:
        assert _choice(lib, 4096, 4096, 128256) is None
        assert lib.ctb_gemm_set_pair(1) == 0 and _choice(lib, 4096, 4096, 4096)[:3] == (1, 256, 1)
        assert lib.ctb_gemm_set_pair(-1) == 1
    finally:
        lib.ctb_gemm_set_pair(before)
