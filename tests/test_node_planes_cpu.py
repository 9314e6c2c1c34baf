"""Arithmetic contract of the 8-wide node's two-plane words (CPU).

A word holds the planes a (even child) and b (odd child), each 0..255 quanta from the node origin:
0x43800000 | a << 15 | 0x5C00 | b << 2.  The traversal reads a from the word as a float and b from the
absolute value of its low half, and the collapse picks the bytes for those readings, one quantum outside
the child's box on either side.
"""
import numpy as np
import pytest


def word(a, b):
    return (np.uint32(0x43800000) | (a.astype(np.uint32) << 15) | np.uint32(0x5C00) | (b.astype(np.uint32) << 2))


def read(w):
    even = w.view(np.float32).astype(np.float64)
    odd = np.abs((w & 0xFFFF).astype(np.uint16).view(np.float16).astype(np.float64))
    return even - 256.0, odd - 256.0


def test_every_pair_of_bytes_reads_back():
    a, b = (x.ravel() for x in np.meshgrid(np.arange(256), np.arange(256), indexing="ij"))
    even, odd = read(word(a, b))
    np.testing.assert_array_equal(odd, b)
    n = even - a
    assert n.min() == 0.71875 and n.max() < 0.75
    # an empty slot (lo 255, hi 0) stays empty whatever its neighbour holds
    assert even[a == 255].min() > even[a == 0].max()


@pytest.mark.parametrize("even", [True, False])
def test_child_box_stays_one_quantum_inside_its_planes(even):
    """The bytes the collapse stores for box sides x (in quanta, 2 <= x <= 253: the origin lies two quanta
    below the node box, which spans at most 250) read back at least one quantum outside."""
    rng = np.random.default_rng(3)
    x = np.concatenate([np.arange(2, 254), rng.uniform(2, 253, 20_000), np.nextafter(np.arange(2, 253), 1e9)])
    other = rng.integers(0, 256, x.size)
    lo = np.floor(x - (1.75 if even else 1.0))
    hi = np.ceil(x + (1.0 - 0.71875 if even else 1.0))
    assert lo.min() >= 0 and hi.max() <= 255
    for q, side in ((lo, "lo"), (hi, "hi")):
        v = read(word(q, other) if even else word(other, q))[0 if even else 1]
        if side == "lo":
            assert np.all(v <= x - 1.0) and np.all(v > x - 2.1)
        else:
            assert np.all(v >= x + 1.0) and np.all(v < x + 2.1)


def test_spread_of_child_bits_to_triangle_bits():
    """Eight child bits to 24 triangle bits (three per child) by multiplies and masks."""
    for m in range(256):
        x = (m * 0x101) & 0x00F00F
        x = (x * 0x11) & 0x0C30C3
        x = (x * 0x5) & 0x249249
        assert x * 7 == sum(7 << (3 * s) for s in range(8) if m >> s & 1)


@pytest.mark.parametrize("octant", range(8))
def test_next_child_is_the_one_farthest_from_the_octant(octant):
    pick = [0x0F if octant & 4 else 0xF0, 0x33 if octant & 2 else 0xCC, 0x55 if octant & 1 else 0xAA]
    for m in range(1, 256):
        c = m
        for p in pick:
            c = c & p or c
        assert c == 1 << max((s for s in range(8) if m >> s & 1), key=lambda s: s ^ octant)
