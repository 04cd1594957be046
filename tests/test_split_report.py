"""What get_split and get_batch_split report, and the splits the autotuner tries
(no GPU needed: host-side state of the library)."""
from __future__ import annotations

import os
import re

import pytest

from conftest import ROOT, load_recipe

WIDE = open(os.path.join(ROOT, "bigint_b200", "csrc", "wide_kernels.cu")).read()


@pytest.fixture(scope="module")
def bb():
    load_recipe("bigint_b200/build.py").build()
    import bigint_b200

    return bigint_b200


def built_in(name):
    """The wide-digit transforms' column lengths by points, the last first."""
    body = re.search(name + r"\[.*?\] = \{(.*?)\};", WIDE, re.S).group(1)
    return [int(x) for x in body.split(",")][::-1]


@pytest.mark.parametrize("log_n", range(5, 27))
def test_reports_what_runs(bb, log_n):
    bb.set_split(log_n, 0)
    bb.set_batch_split(log_n, 0)
    single, batch = bb.get_split(log_n), bb.get_batch_split(log_n)
    if log_n >= 14:  # half as many points, 2^25 the most
        assert single == built_in("kWideColumn")[26 - log_n]
        assert batch == built_in("kWideBatchColumn")[26 - log_n]
    else:
        three = max(2, (log_n - 1) // 2)
        assert single == (three if log_n < 9 else 0)
        assert batch == three
    try:  # no transform of this length has columns of 2^2 and rows of 2^10 to 2^14
        if 14 <= log_n <= 17:
            bb.set_split(log_n, 2)
            bb.set_batch_split(log_n, 2)
            assert (bb.get_split(log_n), bb.get_batch_split(log_n)) == (single, batch)
    finally:
        bb.set_split(log_n, 0)
        bb.set_batch_split(log_n, 0)


@pytest.mark.parametrize("log_n", range(10, 26))
def test_autotuner_tries_splits_that_run(bb, log_n):
    tune = load_recipe("bigint_b200/autotune.py")
    splits = tune.valid_splits(log_n)
    assert bb.get_batch_split(log_n) in splits
    try:
        for l2 in splits:
            bb.set_batch_split(log_n, l2)
            assert bb.get_batch_split(log_n) == l2
            if log_n >= tune.FIRST_SPLIT:
                bb.set_split(log_n, l2)
                assert bb.get_split(log_n) == l2
    finally:
        bb.set_split(log_n, 0)
        bb.set_batch_split(log_n, 0)
