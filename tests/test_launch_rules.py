"""The library's rules of a launch, read from it without a device."""
import ctypes

import pytest

from ibis_b200 import lib
from ibis_b200.params import FLAG_BEDROCK, FLAG_DIAG, FLAG_SUNSHADE_L, FLAG_SUNSHADE_U, FLAG_VMAX_MIX, StepParams

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


@pytest.mark.parametrize("flags", VARIANTS)
def test_the_configuration_that_runs(flags):
    """Two blocks of 128 per SM; one of 224 for more than 128 columns an SM of the canopies
    with a larger record, without diagnostics.  A configuration asked for runs where it is
    compiled, else the default of its form (the ones this canopy and diagnostics have)."""
    rule = lib.load().ibis_launch_config
    large = bool(flags & ~FLAG_BEDROCK)
    split = {c["id"] for c in lib.configs() if c["form"] == "split"}
    for sms in (148, 132):
        for ncell in (0, 1, 128 * sms, 128 * sms + 1, 95333):
            assert rule(-1, flags, ncell, sms) == (6 if large and ncell > 128 * sms else 0)
            assert rule(-1, flags | FLAG_DIAG, ncell, sms) == 0
            for config in range(len(lib.configs())):
                default = 8 if config in split else 0
                assert rule(config, flags | FLAG_DIAG, ncell, sms) == default
                assert rule(config, flags, ncell, sms) == (config if not large or config == 6 else default)
    assert rule(-2, flags, 1, 148) < 0 and rule(12, flags, 1, 148) < 0
    assert rule(0, flags, -1, 148) < 0 and rule(0, flags, 1, 0) < 0


def test_groups_of_host_batches():
    """Hourly forcing: up to eight groups of 1,536 columns or more, whatever a wave is; with
    the chunks set, sixteen above 1.15 waves.  Daily weather: twenty above one wave.
    Groups are whole blocks, and cover the batch in no more groups than wanted."""
    sms, rule = 148, lib.load().ibis_host_group
    for config, flags, block, wave in ((-1, 0, 128, 37888), (6, 0, 224, 33152), (-1, FLAG_SUNSHADE_U, 224, 33152)):
        for ncell in (1, 1535, 3071, 3072, 12289, wave, wave + 1, int(1.15 * wave), int(1.15 * wave) + 1, 95333):
            small = flags and ncell <= 128 * sms                # runs as two blocks of 128
            for daily, chunk, want in ((0, 0, min(ncell // 1536, 8)), (0, 8, 16 if ncell > 1.15 * wave else 1),
                                       (1, 0, 20 if ncell > wave else 1)):
                group = rule(daily, config, flags, ncell, chunk, sms)
                if want > 1:
                    assert group % (128 if small else block) == 0 and -(-ncell // group) <= want
                    assert group < ncell / want + (128 if small else block)
                else:
                    assert group == -(-ncell // 32) * 32
    assert rule(0, 8, 0, 1, 0, sms) < 0 and rule(0, 12, 0, 1, 0, sms) < 0 and rule(0, -1, 0, -1, 0, sms) < 0


@pytest.mark.gpu
def test_columns_report_the_configuration_that_runs(cuda_lib):
    import torch

    from ibis_b200.columns import Columns
    most = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    got = lambda flags, **kw: Columns(most + 1, acc=False, **kw).launch_config(24, flags)
    assert got(FLAG_SUNSHADE_U) == 6 and got(FLAG_SUNSHADE_U, diag=True) == 0
    assert got(0, mode=7) == 7 and got(0, mode=7, diag=True) == 0 and got(0, mode="split", diag=True) == 8
    assert got(FLAG_SUNSHADE_U, mode=7) == 0 and got(FLAG_SUNSHADE_U, mode=10) == 8
    assert got(FLAG_SUNSHADE_U, dtype=torch.float64) == 0
