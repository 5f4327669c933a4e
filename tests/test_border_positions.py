"""findBoarder over positions (oacc_segment_tree.cpp:420-460) with the zero
slot first: a value at one position from 2 on is found there, whatever the
slot compares as, so the engines skip the search.  The search itself, step by
step, for every array size up to 1,025."""
import pytest


def compare(epc, z, m, lo, hi, at_zero):
    if m < 0 or m >= epc:
        return 2
    if m == z:
        return at_zero
    t = m + 1 if m < z else m
    return -1 if t < lo else (0 if t < hi else 1)


def search(epc, z, lo, hi, at_zero):
    low, high = 0, epc
    while low < high:
        m = low + (high - low) // 2
        c = compare(epc, z, m, lo, hi, at_zero)
        if c == 0:
            if compare(epc, z, m - 1, lo, hi, at_zero) != 0:
                low = high = m
            else:
                high = m - 1
        elif c == -1:
            low = m + 1
        else:
            high = m - 1
    return high if compare(epc, z, high, lo, hi, at_zero) == 0 else -1


@pytest.mark.parametrize("k", range(1, 11))
def test_single_position_is_found_where_it_is(k):
    epc = 2 ** k + 1
    for lo in range(2, epc):
        for at_zero in (-1, 0, 1):
            assert search(epc, 0, lo, lo + 1, at_zero) == lo
