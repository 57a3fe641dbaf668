"""CPU: how many CTAs of the decode attention for long caches share an SM.  The sequences' lengths are not known when this is chosen, so the grid must not take a wave
more than the other choice of the same registers would."""
import ctypes

import pytest

SMS = 148


def _plan(lib, *args):
    splits, per_sm = ctypes.c_int(), ctypes.c_int()
    lib.zl_decode_attention_plan(*args, ctypes.byref(splits), ctypes.byref(per_sm))
    return splits.value, per_sm.value


@pytest.mark.parametrize("tasks,longest", [(16, 4096), (32, 2048), (24, 3000), (64, 700), (64, 1000), (32, 900), (32, 1500), (8, 8192), (4, 16384), (2, 32768), (48, 1000),
                                           (24, 2048), (100, 1024), (32, 4096), (40, 4096)])
def test_halves_take_no_wave_more_than_four_per_sm(lib, tasks, longest):
    splits, per_sm = _plan(lib, tasks, 32, 8, 128, longest, 0)
    ctas = tasks * 8 * splits
    assert per_sm in (3, 4) and -(-ctas // (per_sm * SMS)) <= -(-ctas // (4 * SMS))


@pytest.mark.parametrize("tasks,longest,per_sm", [(24, 4096, 3), (20, 4096, 3), (40, 4096, 3), (20, 8192, 3), (48, 2048, 3), (100, 1024, 3), (16, 4096, 3), (32, 4096, 4), (128, 1000, 4)])
def test_bf16_leaves_three_only_for_fewer_waves(lib, tasks, longest, per_sm):
    assert _plan(lib, tasks, 32, 8, 128, longest, 1)[1] == per_sm


@pytest.mark.parametrize("tasks,dtype,per_sm", [(64, 0, 5), (96, 0, 5), (64, 1, 4), (96, 1, 5)])
def test_heads_of_64(lib, tasks, dtype, per_sm):
    assert _plan(lib, tasks, 32, 8, 64, 1000, dtype) == (1, per_sm)
