"""Which mosaic calls take the kernel with the footprint in registers (no GPU)."""
import pytest


@pytest.mark.parametrize("args,want", [
    ((6, 32, 32, 7, 4, 2), True), ((6, 48, 48, 11, 4, 4), True), ((6, 52, 52, 12, 4, 2), False),
    ((6, 32, 32, 7, 4, 5), False), ((600, 8, 8, 3, 20, 1), False),
    # one-cell windows at every offset: the kernel's 31-bit row numbers
    (((2**31 - 2) // 4, 2, 2, 1, 1, 1), True), ((2**31 // 4, 2, 2, 1, 1, 1), False)])
def test_route(args, want):
    from astroviper_b200 import _kernels as K
    assert K.mosaic_runs_ok(*args) is want


@pytest.mark.parametrize("args,want", [
    # a mosaic's few functions, whatever the samples
    ((6, 7, 4, 500, 2), True), ((6, 7, 4, 1_000_000, 2), True), ((6, 11, 20, 1404, 4), True),
    # a table of a million rows: only for many samples
    ((2400, 7, 20, 28_080, 1), False), ((2400, 11, 20, 1404, 2), False),
    ((2400, 7, 20, 10_000_000, 2), True)])
def test_tap_table_against_samples(args, want):
    from astroviper_b200 import _kernels as K
    assert K._mosaic_taps_pay(*args) is want
