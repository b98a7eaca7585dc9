"""The benchmark's own arithmetic: bytes per update and traffic belong to the kernel that ran."""
import sys
from types import SimpleNamespace

import pytest

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench   # noqa: E402


@pytest.mark.parametrize("launches,steps,stages,want", [(1, 100, 4, ("k_yee_resident", 100)), (1, 1, 4, ("k_yee_resident", 1)),
                                                        (501 + 16, 1000, 4, ("k_yee_pair", 2)), (1032, 1000, 4, ("k_yee_step_bulk", 1)),
                                                        (2, 1, 4, ("k_yee_step_bulk", 1)), (1032, 1000, 0, ("k_yee_step", 1))])
def test_kernel_of_a_run(launches, steps, stages, want):
    s = SimpleNamespace(last_launches=lambda: launches, kernel=lambda: (stages, stages > 0))
    assert bench.kernel_of(s, steps) == want


def test_bytes_per_update():
    assert bench.bytes_per_update("k_yee_pair", True, 2) == 24.5
    assert bench.bytes_per_update("k_yee_pair", False, 2) == 26
    assert bench.bytes_per_update("k_yee_resident", True, 100) == 0.52
    assert bench.bytes_per_update("k_yee_step_bulk", True, 1) == 49 and bench.bytes_per_update("k_yee_step", False, 1) == 64
    r = [SimpleNamespace(nx=10, ny=4, nz=2, steps=n) for n in (1, 6, 7)]
    assert bench.served_bytes(r) == 49 * 80 * (1 + 3 + 4)


def test_traffic_only_from_a_profile_of_the_same_kernel():
    assert bench.traffic_per_cell("k_yee_resident", True) is None
    assert bench.traffic_per_cell("k_yee_pair", False) is None
    two, one, register = (bench.traffic_per_cell(*k) for k in (("k_yee_pair", True), ("k_yee_step_bulk", True), ("k_yee_step", False)))
    assert 24.5 < two < one < register < 100
