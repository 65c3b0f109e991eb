"""The f32 sample positions of the correlations (grid_offset) and the division by a constant
(div_by), host-compiled, against the f64 arithmetic they stand in for: bit for bit on random
patches and dividends, ties and their neighbours among them."""
import ctypes as C

import pytest

from chiaro_b200 import runtime


@pytest.fixture(scope="module")
def hc():
    return runtime.load_hostcheck()


@pytest.mark.parametrize("seed", [1, 2])
def test_one_f32_addition_gives_the_f64_coordinate(hc, seed):
    accepted = C.c_uint64()
    assert hc.chiaro_hc_grid_offset_mismatches(1_000_000, seed, C.byref(accepted)) == 0
    assert accepted.value > 300_000


@pytest.mark.parametrize("seed", [1, 2])
def test_division_by_a_constant_rounds_as_the_division(hc, seed):
    assert hc.chiaro_hc_div_by_mismatches(2_000_000, seed) == 0
