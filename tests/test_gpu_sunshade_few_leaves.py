"""Sunlit and shaded leaves of a canopy with hardly any: the smoothed minimum of two rates
keeps its root off zero by 1e-15, which beside a canopy of 1e-6 leaf area is 1e-4 to 1e-3
of the rates.  FP32 forms the rates per leaf area and scales that guard with them, so its
gross assimilation is float64's.

The bound: thirty single-precision operations to a rate, in three passes, with the
intercellular CO2 between them -- some hundred roundings of 6e-8 with unit gains, 6e-6;
5e-5 leaves room for gains.  Rates under 1e-12 mol m-2 s-1 are not compared, nor the upper
canopy's below a leaf area of 1e-2: over the stems it then stands on, its light is a
difference that float32 does not hold (a tenth off at 1e-6, with the guard or without).
"""
import numpy as np
import pytest
import torch

from ibis_b200 import synth
from ibis_b200.columns import Columns
from ibis_b200.params import FLAG_SUNSHADE_L, FLAG_SUNSHADE_U, FLAG_VMAX_MIX

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [FLAG_SUNSHADE_U | FLAG_SUNSHADE_L, FLAG_SUNSHADE_U, FLAG_SUNSHADE_L,
                                   FLAG_SUNSHADE_U | FLAG_SUNSHADE_L | FLAG_VMAX_MIX])
@pytest.mark.parametrize("lai", [0.0, 1e-6, 1e-4, 1e-2, 0.5])
def test_gross_assimilation_of_few_leaves(cuda_lib, lai, flags):
    rng = np.random.Generator(np.random.PCG64(29))
    n = 128
    lat = rng.uniform(-40.0, 40.0, size=n)
    stat = synth.make_columns(rng, n, 0.5)
    stat["lai"][:] = lai
    forc = synth.make_forcing(rng, lat, 1, start_doy=172, start_hour=12)
    prog = synth.make_initial(rng, stat, {k: v[0] for k, v in forc.items()})
    f32 = lambda d: {k: np.asarray(v, np.float32).astype(np.float64) for k, v in d.items()}
    params = synth.StepParams(co2conc=390e-6)
    params.flags |= flags
    got = []
    for dtype in (torch.float32, torch.float64):
        cols = Columns.from_host(f32(prog), f32(stat), dtype=dtype, acc=True, diag=True)
        cols.run(cols.forcing(f32(forc)), params)
        assert not cols.nonfinite()[0]
        got.append(cols.diag_host())
    for k in ("ag_lower",) if 0.0 < lai < 1e-2 else ("ag_upper", "ag_lower"):
        a, b = got[0][k], got[1][k]
        assert np.isfinite(a).all()
        m = np.abs(b) > 1e-12
        assert lai == 0.0 or m.any()
        assert (np.abs(a - b)[m] <= 5e-5 * np.abs(b)[m]).all(), k
