"""StepParams.to_c against the parameters field by field: after assignments, writes
into the arrays, and every kind of copy (each has a record of its own)."""
import copy
import pickle

import numpy as np
import pytest

from ibis_b200.params import PARAM_FIELDS, StepParams


def _same(p):
    c = p.to_c()
    assert c.flags == p.flags
    for name, n, _ in PARAM_FIELDS:
        got = getattr(c, name)
        np.testing.assert_array_equal(np.asarray(got[:] if n > 1 else got), np.asarray(getattr(p, name)), err_msg=name)


@pytest.mark.parametrize("how", ["itself", "copy", "copy.copy", "deepcopy", "pickle"])
def test_record_follows_the_parameters(how):
    rng = np.random.default_rng(1)
    p = StepParams(co2conc=390.0e-6)
    for name, n, _ in PARAM_FIELDS:
        setattr(p, name, rng.normal(size=n) if n > 1 else float(rng.normal()))
    p.vmax_pft[3] = 7.0
    other = {"itself": lambda: p, "copy": p.copy, "copy.copy": lambda: copy.copy(p),
             "deepcopy": lambda: copy.deepcopy(p), "pickle": lambda: pickle.loads(pickle.dumps(p))}[how]()
    _same(other)
    before = bytes(p.to_c())
    other.dtime = 1800.0
    other.flags = 0
    other.coefm = np.arange(5.0)
    _same(other)
    assert how == "itself" or bytes(p.to_c()) == before
    _same(p)
