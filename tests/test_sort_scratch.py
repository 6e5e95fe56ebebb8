"""The no-allocation sort's scratch, restated on the host (no GPU): a pass takes
its tiles' numbers from a counter in the scratch and publishes a tile's digit
counts at (pass * tiles + number) * buckets behind the head.  Calls that overlap on
the scratch draw from one counter, so a number may reach the sum of both calls'
tiles; such a tile returns, and every number below the call's own tiles stays
inside the scratch at every count and key width."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apic-fluid-simulation_gb300", "csrc")
MAX_KEYS, HEAD, THREADS = 1 << 20, 3072 + 32, 512
SORT_WORDS = HEAD + 2 * 256 * 1024
COUNTS = [1, 512, 1024, 1025, 65536, 65537, 131072, 262144, 262145, 500000, MAX_KEYS]


def tiles(n):
    items = 2 if n <= 65536 else 4 if n <= 262144 else 8
    return -(-n // (items * THREADS))


def digit(bits):
    """(passes, digit width) of apic_morton_sort_noalloc."""
    if bits == 0:
        return 0, 0
    width = -(-bits // -(-bits // 10)) if bits <= 20 else 8
    return -(-bits // width), width


def end_of_state(n, bits, number):
    passes, width = digit(bits)
    return HEAD + (((passes - 1) * tiles(n) + number + 1) << width)


@pytest.mark.parametrize("bits", range(1, 33))
def test_numbers_inside(bits):
    for n in COUNTS:
        assert end_of_state(n, bits, tiles(n) - 1) <= SORT_WORDS, (n, bits)


def test_numbers_of_overlapping_calls():
    """Without the return a number could lie past the scratch; with it, none does."""
    past = 0
    for bits in (16, 20, 24, 32):
        for a in COUNTS:
            for b in COUNTS:
                for number in (tiles(a) - 1, tiles(a), tiles(a) + tiles(b) - 1):
                    returns = number >= tiles(a)
                    inside = end_of_state(a, bits, number) <= SORT_WORDS
                    assert returns or inside
                    past += not inside
    assert past > 0
    # the kernel's return comes before its first use of the number
    src = open(os.path.join(CSRC, "sort.cu")).read()
    kernel = src[src.index("k_sort_pass(const uint32_t*"):]
    assert re.search(r"tile = s_tile, ntiles = gridDim\.x;\s*(//[^\n]*\s*)*if \(tile >= ntiles\) return;", kernel)
