"""Inputs that are not finite show where the float64 kernels show them: the FP32 step's
shortcuts (no radiation at night, no snow block where there is no snow, no methane from
frozen soil) leave no such value unnoticed.
"""
import numpy as np
import pytest
import torch

from ibis_b200 import layout as L
from ibis_b200 import synth
from ibis_b200.columns import Columns

pytestmark = pytest.mark.gpu

NCELL = 160


def _run(dtype, hour, group, field, k, value):
    """One hour with ``value`` in one input of every column: (state, sums) per column not finite."""
    rng = np.random.Generator(np.random.PCG64(17))
    lat = rng.uniform(-50.0, 50.0, size=NCELL)
    stat = synth.make_columns(rng, NCELL, 0.5)
    forc = synth.make_forcing(rng, lat, 1, start_doy=172, start_hour=hour)
    prog = synth.make_initial(rng, stat, {n: v[0] for n, v in forc.items()})
    cols = Columns.from_host(prog, stat, dtype=dtype, acc=True)
    f = cols.forcing(forc)
    plane = L.OFF[group][field][0] + k
    if group == "FORC":
        f[:, plane, :NCELL] = value
    else:
        cols.prog[plane, :NCELL] = value
    cols.run(f, synth.StepParams())
    bad = lambda t: ~torch.isfinite(t[:, :NCELL]).all(0)
    state, sums = bad(cols.prog), bad(cols.acc[:L.N_ACC])
    assert cols.nonfinite()[0] == bool(state.any())
    return state, sums


def _shows_as_in_float64(hour, group, field, k, value):
    (s32, a32), (s64, a64) = (_run(dt, hour, group, field, k, value) for dt in (torch.float32, torch.float64))
    assert bool(a64.all() | s64.all())
    assert torch.equal(s32, s64) and torch.equal(a32, a64)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("field", ["solad", "solai"])
def test_visible_light_at_night(cuda_lib, field, value):
    _shows_as_in_float64(0, "FORC", field, 0, value)


@pytest.mark.parametrize("field,k", [("tsoi", 1), ("tsoi", 5), ("wisoi", 3), ("tsoi_deep", 0)])
def test_soil_state_in_the_methane_sum(cuda_lib, field, k):
    _shows_as_in_float64(12, "PROG", field, k, float("nan"))


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("field,k", [("tsno", 0), ("tsno", 1), ("tsno", 2), ("tlsub", 0)])
def test_snow_temperatures_of_bare_columns(cuda_lib, field, k, value):
    _shows_as_in_float64(12, "PROG", field, k, value)


@pytest.mark.parametrize("field", ["t12", "t34"])
def test_canopy_air_where_it_rains_or_snows(cuda_lib, field):
    """An infinite air temperature shows where precipitation is mixed with the canopy's; the
    dry columns' is solved anew."""
    (s32, a32), (s64, a64) = (_run(dt, 12, "PROG", field, 0, float("inf")) for dt in (torch.float32, torch.float64))
    assert bool(s64.any()) and not bool(s64.all())
    assert torch.equal(s32, s64) and torch.equal(a32, a64)
