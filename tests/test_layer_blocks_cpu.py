"""The memory of a layer call: its blocks follow the GEMM switches of the moment, and the library knows how large they are
(host arithmetic of the library, for 148 SMs where there is no GPU)."""
import ctypes

import pytest

from causal_trainer_dev_b200.ops import layer, lib
from causal_trainer_dev_b200.ops.build import LIB_PATH

pytestmark = pytest.mark.skipif(not LIB_PATH.exists(), reason="the CUDA library is not built")

SHAPE = (1, 384, 1536, 12, 2, 128, 8960, 128, 1, 0, 1e-6)      # 384 tokens of a 1.5B layer: products with K slices


@pytest.fixture
def pair_switch():
    set_pair = lib.lib().ctb_gemm_set_pair
    before = set_pair(-1)
    yield set_pair
    set_pair(before)


def test_sizes_follow_the_switches(pair_switch):
    chosen = layer._plan(*SHAPE)[1:]
    pair_switch(0)
    off = layer._plan(*SHAPE)[1:]
    pair_switch(-1)
    again = layer._plan(*SHAPE)[1:]
    assert again == chosen and off[0] == chosen[0]
    assert off[1] < chosen[1] and off[2] < chosen[2]            # no workspace where no product is cut


@pytest.mark.parametrize("kept_short,scratch_short", [(1, 0), (0, 1), (256, 0), (0, 4096)])
def test_a_block_that_is_too_small_is_refused(pair_switch, kept_short, scratch_short):
    pair_switch(0)                                                # the block without workspace: nothing in it is optional
    shape, kept, forward, backward = layer._plan(*SHAPE)
    # the last piece of a block ends inside of its last 256 bytes: the refusal is for what the pieces hold
    zeros = layer._Context(), layer._Weights()
    at = 1 << 20                                                  # (addresses that nothing reads: refused before the first launch)
    L = lib.lib()
    c, w = (ctypes.byref(z) for z in zeros)
    low = lambda n, short: n - (short and 255 + short)          # noqa: E731
    assert L.ctb_layer_forward(ctypes.byref(shape), c, w, at, None, at, low(kept, kept_short), at, low(forward, scratch_short),
                               at, at, None) == 1
    assert "too small" in L.ctb_last_error().decode()
    assert L.ctb_layer_backward(ctypes.byref(shape), c, w, w, 0, at, at, at, at, low(kept, kept_short), at,
                                low(backward, scratch_short), at, None) == 1
    assert "too small" in L.ctb_last_error().decode()
    assert L.ctb_layer_forward(ctypes.byref(shape), c, w, at, None, None, 0, at, forward, at, at, None) == 1


def test_only_the_segments_that_the_library_trains():
    from causal_trainer_dev_b200.models import params
    from causal_trainer_dev_b200.models.config import preset

    for bias in (False, True):
        assert layer.takes(params.layer_layout(preset("tiny", attention_bias=bias), 0))
    entries = [("ln1", (64,)), ("ln2", (64,)), ("qkv_w", (192, 64)), ("o_w", (64, 64)), ("gu_w", (256, 64)), ("down_w", (64, 128))]
    assert layer.takes(params._layout("layer.0", entries))
    assert not layer.takes(params._layout("layer.0", [*entries, ("o_b", (64,))]))       # a bias that it would leave out
    assert not layer.takes(params._layout("layer.0", entries[1:]))
