"""Which form of the chunked Mamba2 scan a step takes, and that a recorded step is replayed only for steps of its forms (host-side
decisions, no GPU)."""
import types

import pytest

from poor_mans_mamba_b200.engine.context import LengthBounds
from poor_mans_mamba_b200.engine.model import Model
from poor_mans_mamba_b200.kernels import ops as K
from poor_mans_mamba_b200.parts.mamba2 import Mamba2Mixer

SMALL, LARGE = (24, 64, 128, 1), (48, 128, 256, 1)


def padded(count, lens):
    lens = list(lens) + [0] * (count - len(lens))
    return LengthBounds(sum(lens), count, lens)


@pytest.mark.parametrize("count,lens", [(8, [2000, 1, 1, 1, 45]), (8, [1997, 1, 1, 1, 1, 1, 46]), (8, [1481, 1, 1, 1, 52]), (2, [900, 124]), (2, [2040, 8])])
def test_padded_steps_with_a_long_portion_take_two_launches(count, lens):
    """One long portion beside a few lone tokens is the usual step of a server: the longest sequence counts, not a mean."""
    assert K.ssd_tc_walk_columns(padded(count, lens), *SMALL, True) == 0


@pytest.mark.parametrize("count,lens,cols", [(8, [280, 281, 200, 342, 300, 133], 64), (8, [400, 390, 300, 1, 1, 1, 187], 64), (2, [37, 219], 64),
                                             (16, [150] * 8, 128), (16, [150] * 13, 0), (2, [500, 12], 64), (8, [505, 1, 1, 1, 1, 1, 2], 64)])
def test_padded_steps_of_short_portions_walk(count, lens, cols):
    assert K.ssd_tc_walk_columns(padded(count, lens), *SMALL, True) == cols


def test_bounds_that_are_not_told_of_a_step_count_as_their_one_long_sequence():
    for total, count in [(256, 2), (512, 4), (1024, 2), (1024, 8), (2048, 4), (2048, 8)]:
        cut = [total - count + 1] + [1] * (count - 1)
        assert K.ssd_tc_walk_columns(LengthBounds(total, count), *SMALL, True) == K.ssd_tc_walk_columns(LengthBounds(total, count, cut), *SMALL, True)


def test_forms_at_the_sizes_that_were_timed():
    walks = lambda lens, shape=SMALL, skip=False: K.ssd_tc_walk_columns(lens, *shape, skip) > 0
    assert walks([37]) and walks([256]) and walks([300]) and not walks([385]) and not walks([500]) and not walks([2048])
    assert walks([280, 281, 200, 342, 300]) and walks([512] * 4) and not walks([1000, 50, 60, 70]) and not walks([1024, 100])
    assert not walks([1000] + [1] * 6, skip=True) and walks([512] + [1] * 31, skip=True)
    assert all(walks([n], LARGE) for n in (100, 512, 1024, 2048))
    assert not walks([100], (24, 64, 80, 1)) and not walks([128] * 16) and not walks([1, 1], skip=True) and not walks([])


def test_a_model_answers_once_for_mixers_of_equal_sizes():
    def layer(heads):
        mixer = types.SimpleNamespace(n_heads=heads, d_head=64, d_state=128, n_groups=1)
        return types.SimpleNamespace(length_choices=lambda: [Mamba2Mixer.length_choice(mixer), None])
    model = types.SimpleNamespace(layers=[layer(24), types.SimpleNamespace(), layer(24), layer(8)], _length_choices=None)
    short, long = padded(8, [280, 281, 200, 342, 300, 133]), padded(8, [1400, 1, 1, 134])
    assert Model.length_choices(model, short) == (64, 64) and len(model._length_choices) == 2
    assert Model.length_choices(model, long) == (0, 0)
    assert Model.length_choices(types.SimpleNamespace(layers=[types.SimpleNamespace()], _length_choices=None), short) == ()
