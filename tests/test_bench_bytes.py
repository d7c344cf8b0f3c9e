"""The bytes that bench.py charges a bond: those of the form that the force kernel runs in."""
import pytest

import bench


class FakeDev:
    def __init__(self, tiles=(0, 0, 0), mapping=(1, 128, 5), esc=False):
        self._t, self._m, self.esc = tiles, mapping, esc

    def tile_info(self):
        return self._t

    def mapping(self):
        return self._m


@pytest.mark.parametrize("dev,prec,mat,phase,bytes_,bound,classes", [
    (FakeDev((1400, 122, 3)), "fp32", "OSB", "phase_b", 3.125, "issue", True),
    (FakeDev((1600, 0, 3)), "fp32", "OSB", "phase_b", 18.125, "issue", False),      # jittered
    (FakeDev((1400, 122, 1)), "fp32", "CW", "phase_b", 20.125, "hbm", False),       # ZEMWan
    (FakeDev((1400, 122, 0), (1, 128, 2)), "fp32", "OSB", "phase_a", 20.125, "hbm", False),
    (FakeDev((0, 0, 0), (8, 128, 0)), "fp32", "BB", "phase_a", 20.125, "hbm", False),
    (FakeDev(esc=True), "fp32", "BB", "phase_a", 24.125, "hbm", False),
    (FakeDev((1400, 0, 3)), "fp64", "OSB", "phase_b", 10.125, "issue", False),
    (FakeDev((0, 0, 0), (4, 128, 0)), "fp64", "BB", "phase_a", 12.125, "hbm", False),
    (FakeDev((1400, 0, 0), (0, 128, 0)), "fp64", "OSB", "phase_a", 36.125, "hbm", False),
    (FakeDev(), "fp64", "C", "phase_b", 36.125, "hbm", False),
    (FakeDev(esc=True), "fp64", "OSB", "phase_b", 20.125, "hbm", False),
])
def test_bytes_of_the_form_that_runs(dev, prec, mat, phase, bytes_, bound, classes):
    assert bench.bond_stream(dev, prec, mat, phase) == (bytes_, bound, classes)
