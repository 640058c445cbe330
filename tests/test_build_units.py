"""Every CUDA source of the package is a unit of its build."""
import os

from ibis_b200 import build


def test_every_source_is_built():
    on_disk = {f for f in os.listdir(build.CSRC) if f.endswith(".cu")}
    assert on_disk == set(build.UNITS)
