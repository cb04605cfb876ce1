"""The picker's measured table is of the library's present kernels: classes timed
again give the table's times, variant by variant."""
import json

import numpy as np
import pytest

from nvshmem_b200 import picker as P

pytestmark = pytest.mark.gpu


def test_table_is_of_these_kernels():
    d = np.load(P.DATA)
    n = 48
    classes = P.sample_classes(seed=2024, n=800, patterns=P.TRAIN_PATTERNS)[:n]
    again = P.measure(classes, 10_000, reps=5)
    assert np.array_equal(np.stack([P.features(**c) for c in classes]), d["train_x"][:n])
    assert json.loads(str(d["meta"]))["variants"] == P.VARIANT_NAMES
    ratio = np.nanmedian(again / d["train_t"][:n], axis=0)
    print(dict(zip(P.VARIANT_NAMES, np.round(ratio, 2))))
    # a variant's time over all classes; boxes and runs differ by some percent
    assert np.all((ratio > 0.75) & (ratio < 1.33)), ratio
