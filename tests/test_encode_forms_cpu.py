"""The forms of input that the chromosome encoding takes: machine numbers as
floats, placements as a list of mappings, part numbers that no type matches."""
import random

import numpy as np
import pytest

from brkga_fft2_b200 import abi
from brkga_fft2_b200.initial import encode

TYPES = np.array([4, 7, 9])
GENE_TYPE = np.array([0, 1, 0, 2, 1, 0])
PARTS = np.array([4, 7, 4, 9, 7, 4])
MACHINE = np.array([0, 1, 0, 1, 0, 1], np.int32)
BINS = [0, 1, 1, 0, 0, 0]


def _place():
    place = np.zeros(6, abi.PLACEMENT_DTYPE)
    place["gene"] = [3, 1, 0, 2, 4, 5]
    place["bin"] = BINS
    return place


def _encode(machine, place, parts):
    return encode(machine, place, parts, TYPES, GENE_TYPE, 2, [0.5], random.Random(5))


REF = _encode(MACHINE, _place(), PARTS)


@pytest.mark.parametrize("machine", [MACHINE.astype(np.float64), MACHINE.astype(np.float32), list(map(int, MACHINE)),
                                     [float(m) for m in MACHINE], MACHINE.astype(np.int64)])
def test_machine_numbers(machine):
    np.testing.assert_array_equal(_encode(machine, _place(), PARTS), REF)


def test_placements_as_mappings():
    rows = [{"gene": int(p["gene"]), "bin": int(p["bin"])} for p in _place()]
    np.testing.assert_array_equal(_encode(MACHINE, rows, PARTS), REF)


@pytest.mark.parametrize("parts", [PARTS.astype(np.float64), PARTS.tolist()])
def test_part_numbers(parts):
    np.testing.assert_array_equal(_encode(MACHINE, _place(), parts), REF)


def test_part_numbers_that_match_no_type_stay_zero():
    """A part number between two types is no type's: the gene gets no key."""
    parts = PARTS.astype(np.float64)
    parts[3] = 9.5
    got = _encode(MACHINE, _place(), parts)
    assert got[3] == 0.0 and got[3 + 6] == 0.0
