"""The sorting and selection networks of the 5x5 and 7x7 median, read from the
kernel's tables and run on every 0-1 input they can meet, which proves them for
all inputs (0-1 principle): sorts on all 0-1 words, selections on all matrices
whose rows and columns are sorted."""
import itertools
import os
import re

import numpy as np
import pytest

import __graft_entry__ as ge


def _struct(name, n):
    with open(os.path.join(ge.PKG_DIR, "csrc", "median.cu"), encoding="utf-8") as f:
        return re.search(r"struct %s<%d> \{(.*?)\n\};" % (name, n), f.read(), re.S).group(1)


def _number(body, name):
    return int(re.search(r"\b%s = (\d+)" % name, body).group(1))


def _pairs(body, name):
    text = re.search(r"int8_t %s\[\w+\]\[2\] = \{(.*?)\};" % name, body, re.S).group(1)
    return [tuple(int(v) for v in p) for p in re.findall(r"\{(\d+), (\d+)\}", text)]


def _run(wires, exchanges):
    for lo, hi in exchanges:
        a, b = np.minimum(wires[lo], wires[hi]), np.maximum(wires[lo], wires[hi])
        wires[lo], wires[hi] = a, b
    return wires


@pytest.mark.parametrize("n", [4, 6])
def test_sorting_networks(n):
    body = _struct("SortNet", n)
    exchanges = _pairs(body, "ab")
    assert len(exchanges) == _number(body, "n")
    words = np.array(list(itertools.product((0, 1), repeat=n)))
    assert np.array_equal(np.array(_run(list(words.T), exchanges)).T, np.sort(words, axis=1))


@pytest.mark.parametrize("k,patterns", [(5, 252), (7, 3432)])
def test_selection_networks(k, patterns):
    body = _struct("FinalNet", k)
    at, exchanges = _pairs(body, "at"), _pairs(body, "ab")
    assert len(at) == _number(body, "wires") and len(exchanges) == _number(body, "n")
    # Rows and columns ascending: the number of ones grows from row to row.
    ones = np.array(list(itertools.combinations_with_replacement(range(k + 1), k)))
    assert len(ones) == patterns
    matrices = (np.arange(k) >= k - ones[:, :, None]).astype(np.int8)
    wires = _run([matrices[:, i, j] for i, j in at], exchanges)
    median = (ones.sum(axis=1) > k * k // 2).astype(np.int8)
    assert np.array_equal(wires[_number(body, "out")], median)
