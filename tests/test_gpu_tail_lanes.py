"""The last warp of a batch that is not a whole number of them: each column's state and
sums are bit for bit what the same column gets in a batch of whole warps, with and without
compensation, and the planes' padding is nobody's.

Lanes past the batch's end either leave at once or repeat the last column writing nothing;
a store of theirs would go to the last column's sums.
"""
import numpy as np
import pytest
import torch

from ibis_b200 import synth
from ibis_b200.columns import Columns
from ibis_b200.params import FLAG_ETPARTS, FLAG_KAHAN, FLAG_NEEPARTS, FLAG_SOIL_MEANS

pytestmark = pytest.mark.gpu

WHOLE = 1024
HOURS = 4


@pytest.fixture(scope="module")
def workload():
    return synth.make_workload(WHOLE, HOURS, seed=31)


def _run(wl, ncell, flags, dtype, diag, mode):
    cut = lambda d: {k: v[:ncell] for k, v in d.items()}
    params = wl.params.copy()
    params.flags = flags
    cols = Columns.from_host(cut(wl.prog), cut(wl.stat), dtype=dtype, acc=True, diag=diag, mode=mode)
    cols.acc[:, ncell:] = 7.0
    cols.run(cols.forcing({k: v[:, :ncell] for k, v in wl.forc.items()}), params)
    torch.cuda.synchronize()
    assert bool((cols.acc[:, ncell:] == 7.0).all()) and not cols.nonfinite()[0]
    return cols


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("dtype,diag,mode", [(torch.float64, False, "fused"), (torch.float64, True, "fused"),
                                             (torch.float32, False, "fused"), (torch.float32, True, "fused"),
                                             (torch.float32, False, 3), (torch.float32, False, 6)])
def test_a_partial_warps_columns_are_a_whole_ones(cuda_lib, workload, dtype, diag, mode, kahan):
    flags = workload.params.flags | FLAG_SOIL_MEANS | FLAG_ETPARTS | FLAG_NEEPARTS
    flags = flags | FLAG_KAHAN if kahan else flags & ~FLAG_KAHAN
    whole = _run(workload, WHOLE, flags, dtype, diag, mode)
    for ncell in (1, 33, 63, 129, 1009):
        part = _run(workload, ncell, flags, dtype, diag, mode)
        assert torch.equal(part.prog[:, :ncell], whole.prog[:, :ncell])
        assert torch.equal(part.acc[:, :ncell], whole.acc[:, :ncell])
        if diag:
            assert np.array_equal(part.diag[:, :ncell].cpu().numpy(), whole.diag[:, :ncell].cpu().numpy(),
                                  equal_nan=True)
