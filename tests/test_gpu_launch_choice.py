"""The library's choice of a launch configuration, and the shapes where the blocks of
each can go wrong: batches of less than a warp, of partial warps and blocks, on both
sides of the sizes where the choice changes.

A column's step does not depend on its batch, so each batch is compared with one run
of configuration 6 over the most columns: the same step code compiled for another
block size, which may contract other multiply-adds; temperatures then differ by a few
float32 ulps an hour (5e-5 K each), bounded here by 5 mK over at most five hours (the
bound the FP32 step is held to against float64 for one hour), contents and sums by
1e-4 and 1e-3 of their size.
"""
import numpy as np
import pytest
import torch

from ibis_b200 import ensemble as E
from ibis_b200 import synth
from ibis_b200.columns import AUTO_FUSED, AUTO_LARGE, Columns
from ibis_b200.params import FLAG_COEFM_MIX, FLAG_GPP_CAPACITY, FLAG_SUNSHADE_L, FLAG_SUNSHADE_U, FLAG_VMAX_MIX

pytestmark = pytest.mark.gpu

MOST = 33153
HOURS = 5


@pytest.fixture(scope="module")
def reference(cuda_lib):
    wl = synth.make_workload(MOST, HOURS, seed=77, edge_cases=True)
    out = {}
    for nstep in (1, HOURS):
        cols = Columns.from_host(wl.prog, wl.stat, acc=True, mode=6)
        cols.run(cols.forcing(wl.forc, 0, nstep), wl.params)
        out[nstep] = (cols.prog_host(), cols.acc_host())
    return wl, out


def _head(wl, n):
    cut = lambda d: {k: v[:n] for k, v in d.items()}
    return cut(wl.prog), cut(wl.stat), {k: v[:, :n] for k, v in wl.forc.items()}


@pytest.mark.parametrize("diag", [False, True])
@pytest.mark.parametrize("nstep", [1, HOURS])
@pytest.mark.parametrize("ncell", [1, 31, 33, 127, 129, 255, 18945, MOST])
def test_batches_of_every_shape_step_as_one(reference, ncell, nstep, diag):
    wl, out = reference
    prog, stat, forc = _head(wl, ncell)
    cols = Columns.from_host(prog, stat, acc=True, diag=diag)
    cols.prog[:, ncell:] = 7.0                       # the padding of each plane is nobody's
    cols.acc[:, ncell:] = 7.0
    cols.run(cols.forcing(forc, 0, nstep), wl.params)
    torch.cuda.synchronize()
    assert bool((cols.prog[:, ncell:] == 7.0).all()) and bool((cols.acc[:, ncell:] == 7.0).all())
    assert not cols.nonfinite()[0]
    p, a = cols.prog_host(), cols.acc_host()
    p0, a0 = out[nstep]
    for k in ("tsoi", "tg", "tu", "ts", "tl", "t12", "t34", "tsno", "ti"):
        np.testing.assert_allclose(p[k], p0[k][:ncell], rtol=0, atol=5e-3, err_msg=k)
    for k in ("wsoi", "wisoi", "fi"):
        np.testing.assert_allclose(p[k], p0[k][:ncell], rtol=0, atol=1e-4, err_msg=k)
    for k, w in a0.items():
        if k.endswith("_mean"):
            continue
        scale = max(float(np.abs(w).max()), 1e-30)
        assert float(np.abs(a[k] - w[:ncell]).max()) <= 1e-3 * scale, k


def test_the_choice_follows_the_batch_and_the_canopy(cuda_lib):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cfg = lambda n, flags: Columns(n, acc=False).launch_config(24, flags)
    assert cfg(1, 0) == cfg(128 * sms + 1, 0) == AUTO_FUSED == 0
    for flags in (FLAG_SUNSHADE_U, FLAG_SUNSHADE_L, FLAG_VMAX_MIX):
        assert cfg(128 * sms, flags) == AUTO_FUSED and cfg(128 * sms + 1, flags) == AUTO_LARGE == 6


@pytest.mark.parametrize("flags", [FLAG_SUNSHADE_U, FLAG_SUNSHADE_U | FLAG_SUNSHADE_L | FLAG_VMAX_MIX])
def test_large_records_step_as_small_ones(cuda_lib, flags):
    """The canopy variants on both sides of their choice (18,944 and 18,945 columns on
    148 SMs): the first 500 columns of each batch, and of the other configuration."""
    wl = synth.make_workload(18945, 3, seed=21)
    wl.params.flags |= flags
    got = []
    for n, mode in ((500, "fused"), (18944, "fused"), (18945, "fused"), (500, 6), (500, 0)):
        prog, stat, forc = _head(wl, n)
        cols = Columns.from_host(prog, stat, acc=True, mode=mode)
        cols.run(cols.forcing(forc), wl.params)
        got.append((cols.prog_host(), cols.acc_host()))
    for p, a in got[1:]:
        for k in ("tsoi", "tg", "tu", "tl", "ti"):
            np.testing.assert_allclose(p[k][:500], got[0][0][k], rtol=0, atol=5e-3, err_msg=k)
        for k in ("aynpp", "aygpptot", "adaet", "afsena", "ch4"):
            w = got[0][1][k]
            assert float(np.abs(a[k][:500] - w).max()) <= 1e-3 * float(np.abs(w).max()), k


@pytest.mark.parametrize("daily", [False, True])
def test_every_ensemble_block_runs_with_every_switch(cuda_lib, daily):
    """The largest block accepted needs more shared memory than an SM has with the
    sunlit/shaded canopies, the IBIS 3.0 switches and daily weather together: it
    runs in the largest that fits.  The same kernel in blocks of 32 gives the same bits."""
    spec = E.make_ensemble(5, 13, site_hours=np.full(5, 24), seed=3, daily=daily)
    spec.params.flags |= FLAG_SUNSHADE_U | FLAG_SUNSHADE_L | FLAG_VMAX_MIX
    ens = E.Ensemble(spec)
    out = []
    for block in (32, 256):
        assert ens.occupancy(block) > 0
        ens.reset()
        ens.run(block=block)
        torch.cuda.synchronize()
        assert not any(ens.nonfinite()[:2])
        out.append((ens.prog.clone(), ens.acc.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("flags", [0, FLAG_SUNSHADE_U, FLAG_SUNSHADE_U | FLAG_SUNSHADE_L])
@pytest.mark.parametrize("ncell", [1, 33, 1500])
def test_the_plain_float64_kernel_gives_the_full_ones_bits(cuda_lib, ncell, flags):
    """Without diagnostics and IBIS 3.0 switches float64 columns run a kernel that has
    neither: operation for operation the same step, so not a bit may differ."""
    wl = synth.make_workload(ncell, 4, seed=5, edge_cases=ncell > 1000)
    wl.params.flags |= flags
    out = []
    for diag in (False, True):
        cols = Columns.from_host(wl.prog, wl.stat, acc=True, diag=diag, dtype=torch.float64)
        cols.run(cols.forcing(wl.forc), wl.params)
        out.append((cols.prog_host(), cols.acc_host()))
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("block", [64, 160, 256])
def test_a_run_does_not_depend_on_its_block_or_order(cuda_lib, block):
    """Runs of 0 to 7 hours, in the queue in no order: warps of a block that finish,
    draw and run out of items at different hours, whole items of runs without an hour,
    a year that ends inside the records.  Bit for bit as in blocks of one warp."""
    spec = E.make_ensemble(7, 47, site_hours=np.full(7, 7), seed=9)
    ens = E.Ensemble(spec, year_steps=5)
    gen = torch.Generator().manual_seed(4)
    hours = torch.randint(0, 8, (ens.nrun,), generator=gen, dtype=torch.int32)
    hours[64:128] = 0
    ens.run_nstep.copy_(hours)
    out = []
    for b, order in ((32, torch.arange(ens.nrun)), (block, torch.arange(ens.nrun)),
                     (block, torch.randperm(ens.nrun, generator=gen))):
        ens.order.copy_(order.to(torch.int32))
        ens.reset()
        ens.run(block=b)
        torch.cuda.synchronize()
        assert not any(ens.nonfinite()[:2])
        out.append((ens.prog[:, :ens.nrun].clone(), ens.acc[:, :ens.nrun].clone(), ens.yearly.clone()))
    assert bool((out[0][1][:, 64:128] == 0).all())
    assert bool((out[0][2] != 0).any())
    for got in out[1:]:
        assert all(torch.equal(x, y) for x, y in zip(got, out[0]))


@pytest.mark.parametrize("mode", [0, 6, "split"])
@pytest.mark.parametrize("flags", [FLAG_GPP_CAPACITY, FLAG_VMAX_MIX | FLAG_COEFM_MIX,
                                   FLAG_GPP_CAPACITY | FLAG_VMAX_MIX | FLAG_SUNSHADE_U | FLAG_SUNSHADE_L])
def test_a_launch_of_hours_is_as_many_launches_of_one(cuda_lib, flags, mode):
    """What an IBIS 3.0 launch forms once of the parameters and static planes serves each
    of its hours: the same kernel launched hour by hour forms it anew, to the same bits."""
    wl = synth.make_workload(700, 4, seed=13, edge_cases=True)
    wl.params.flags |= flags
    out = []
    for hours in (4, 1):
        cols = Columns.from_host(wl.prog, wl.stat, acc=True, mode=mode)
        for h in range(0, 4, hours):
            cols.run(cols.forcing(wl.forc, h, h + hours), wl.params)
        out.append((cols.prog_host(), cols.acc_host()))
    for a, b in zip(*out):
        for k in a:
            if not k.endswith("_mean"):
                assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("flags", [0, FLAG_SUNSHADE_U | FLAG_VMAX_MIX])
@pytest.mark.parametrize("ncell,nstep", [(31, 3), (3071, 12), (3072, 11), (3072, 12), (12289, 2), (20000, 13)])
def test_the_librarys_groups_of_host_batches_equal_one_launch(cuda_lib, ncell, nstep, flags):
    """On both sides of the sizes where a batch from host memory is cut into groups, and
    its groups' hours into pieces: the same kernel over the same columns, bit for bit."""
    wl = synth.make_workload(ncell, nstep, seed=8)
    wl.params.flags |= flags
    ref = Columns.from_host(wl.prog, wl.stat, acc=True)
    ref.run(ref.forcing(wl.forc), wl.params)
    cols = Columns.from_host(wl.prog, wl.stat, acc=True)
    h_forc = torch.from_numpy(synth.forcing_planes(wl.forc, cols.ld)).pin_memory()
    h_prog = torch.zeros_like(cols.prog, device="cpu").pin_memory()
    cols.run_host(h_forc, wl.params, host_prog=h_prog)
    torch.cuda.synchronize()
    assert torch.equal(cols.prog, ref.prog) and torch.equal(cols.acc, ref.acc)
    assert torch.equal(h_prog[:, :ncell], ref.prog[:, :ncell].cpu())
