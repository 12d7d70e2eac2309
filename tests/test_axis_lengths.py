"""The list of axis lengths that have kernels of their own (axis_lengths.h)."""
import os
import re

from gpu_fft_b200 import build

SOURCE = open(os.path.join(build.CSRC, "axis_lengths.h")).read()
PARTS = {int(i): [tuple(map(int, t)) for t in re.findall(r"X\((\d+), (\d+), (\d+)\)", body)]
         for i, body in re.findall(r"#define GPUFFT_AXIS_LENGTHS_(\d+)\(X\)((?:.*\\\n)*.*)\n", SOURCE)}


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def test_every_length_once():
    lengths = [a * b * c for part in PARTS.values() for a, b, c in part]
    assert sorted(lengths) == [n for n in range(16, 1025) if _smooth(n)]


def test_parts_are_small():
    """A plan loads the whole part that a length is in: no more than four lengths."""
    assert all(1 <= len(part) <= 4 for part in PARTS.values())


def test_every_part_is_compiled_in_both_precisions():
    made = {tuple(int(d.split("=")[1]) for d in defs) for _, _, defs in build.PARTS}
    assert made == {(d, i) for d in (0, 1) for i in PARTS}
    assert len({obj for _, obj, _ in build.PARTS}) == len(build.PARTS)
