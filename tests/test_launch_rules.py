"""The library's rules of a launch, read from it without a device."""
import ctypes

import pytest

from ibis_b200 import lib
from ibis_b200.params import (FLAG_BEDROCK, FLAG_SUNSHADE_L, FLAG_SUNSHADE_U, FLAG_VMAX_MIX, StepParams)

VARIANTS = [0, FLAG_BEDROCK, FLAG_SUNSHADE_U, FLAG_SUNSHADE_L, FLAG_VMAX_MIX | FLAG_BEDROCK,
            FLAG_SUNSHADE_U | FLAG_SUNSHADE_L | FLAG_VMAX_MIX]


@pytest.mark.parametrize("daily", [0, 1])
@pytest.mark.parametrize("flags", VARIANTS)
def test_an_ensembles_block_is_what_an_sm_holds(flags, daily):
    """Blocks an SM's shared memory does not hold run as the largest that it does; the
    launch counts its grid by those threads, and the tuner times each kernel once."""
    params = StepParams()
    params.flags = flags
    c = params.to_c()
    threads = lambda block: lib.load().ibis_ensemble_block(ctypes.byref(c), daily, block)
    most = 224 if not daily and not flags & ~FLAG_BEDROCK else 192
    for block in range(32, 257, 32):
        assert threads(block) == min(block, most)
    for block in (0, 16, 33, 257, 288, -32):
        assert threads(block) == 0
    assert lib.load().ibis_ensemble_block(None, daily, 64) == 0
