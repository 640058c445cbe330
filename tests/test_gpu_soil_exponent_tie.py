"""The soil-water solve rounds an interface's Clapp-Hornberger exponent to a whole number.
Layers of one soil whose exponent is a half-integer (4.5 is a texture class's) lie on the
tie for every pair of layer thicknesses: FP32 takes the side float64 takes.

On the other side of the tie the top layer is off by 6e-3 in an hour; the bounds are those
the FP32 step is held to for one hour (soil water 1e-5, temperatures 5 mK).
"""
import numpy as np
import pytest
import torch

from ibis_b200 import synth
from ibis_b200.columns import Columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fused", "split"])
@pytest.mark.parametrize("bex", [4.5, 5.5, 8.5])
def test_one_soils_exponent_on_the_tie(cuda_lib, bex, mode):
    wl = synth.make_workload(64, 1, seed=17)
    f32 = lambda d: {k: np.asarray(v, np.float32).astype(np.float64) for k, v in d.items()}
    stat, prog, forc = f32(wl.stat), f32(wl.prog), f32(wl.forc)
    stat["bex"][:] = bex
    prog["wsoi"][:] = np.float32(0.93)
    prog["wisoi"][:] = 0.0
    rng = np.random.default_rng(5)
    for _ in range(24):
        params = wl.params.copy()
        params.hsoi = params.hsoi * rng.uniform(0.75, 1.3, size=params.hsoi.shape)
        out = []
        for dtype in (torch.float32, torch.float64):
            cols = Columns.from_host(prog, stat, dtype=dtype, acc=True,
                                     mode=mode if dtype == torch.float32 else "fused")
            cols.run(cols.forcing(forc), params)
            out.append(cols.prog_host())
        np.testing.assert_allclose(out[0]["wsoi"], out[1]["wsoi"], rtol=0, atol=1e-5)
        np.testing.assert_allclose(out[0]["tsoi"], out[1]["tsoi"], rtol=0, atol=5e-3)
