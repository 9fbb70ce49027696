"""The stress and energy record: the mixed form's FP64 evaluation against the FP64 form, and
the reduction over chunks and systems against sums of its own per-system parts."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# less than a window, grids under three cells a side, window edges and the switches of the
# window size (4096, 65536), lists longer than a mask word (a dense box and a wide padding)
@pytest.mark.parametrize("n,phi,aor,contacts,pad,cap", [
    (2, 0.05, 1.0, 1, 0.1, 0), (9, 0.8, 1.0, 1, 0.1, 0), (33, 0.8, 1.0, 2, 0.1, 0),
    (1025, 0.85, 1.0, 1, 0.1, 0), (4097, 0.85, 0.5, 2, 0.2, 0), (65537, 0.84, 1.0, 1, 0.1, 0),
    (3000, 0.85, 0.2, 1, 4.0, 200)])
def test_mixed_record_equals_fp64(n, phi, aor, contacts, pad, cap):
    """1e-9 of the largest component: the state's representation (48 bits) is all that
    differs."""
    from spherocyls_gb300 import SpherocylBox, generate_packing

    L, x, y, p, R, A = generate_packing(n, phi, aor, seed=11)
    got = [SpherocylBox(L, x, y, p, A, R, pad, precision=f, contacts=contacts,
                        max_nbrs=cap).calc_se() for f in ("mixed", "fp64")]
    assert np.abs(got[0] - got[1]).max() <= 1e-9 * np.abs(got[1]).max()


@pytest.mark.parametrize("sizes", [[1024, 1025, 2], [300] * 40, [50000, 64, 9000]])
def test_records_of_a_batch_equal_single_records(sizes):
    from spherocyls_gb300 import BoxBatch, SpherocylBox, generate_packing

    packs = [generate_packing(n, 0.8, 0.5, seed=k % 7) for k, n in enumerate(sizes)]
    cat = lambda k: np.concatenate([q[k] for q in packs])  # noqa: E731
    b = BoxBatch(sizes, [q[0] for q in packs], cat(1), cat(2), cat(3), cat(5), cat(4), 0.1)
    for _ in range(2):  # (the counters of finished chunks are back at zero)
        got = b.calc_se()
        for k in {0, 1, len(sizes) - 1}:
            q = packs[k]
            one = SpherocylBox(q[0], q[1], q[2], q[3], q[5], q[4], 0.1).calc_se()
            assert np.array_equal(got[k], one)
