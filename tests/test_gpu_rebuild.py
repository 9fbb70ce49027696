"""The rebuild kernel: batches of which some systems are rebuilt at a step.

Systems do not see each other, so each system of a batch must advance bit for bit as it
does alone, whichever of its fellows are rebuilt with it.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(n, seed):
    from spherocyls_gb300 import generate_packing

    return generate_packing(n, 0.84, 0.7, seed=seed)


def _run(packs, rates, precision, steps, **kw):
    from spherocyls_gb300 import BoxBatch

    cat = lambda k: np.concatenate([p[k] for p in packs])  # noqa: E731
    b = BoxBatch([len(p[1]) for p in packs], [p[0] for p in packs], cat(1), cat(2), cat(3), cat(5),
                 cat(4), 0.15, precision=precision, **kw)
    for s, r in enumerate(rates):
        b.set_strain_rate(r, sys=s)
    b.set_step(0.02)
    b.strain_steps(steps)
    out = np.array(b.state())
    got = []
    p0 = 0
    for p in packs:
        got.append(out[:, p0:p0 + len(p[1])])
        p0 += len(p[1])
    return got


# windows of 128 slots shared by several systems; more systems than a block lists (1024);
# few and many particles to rebuild at once (eight threads a slot or one); one large system
# among small ones
@pytest.mark.parametrize("sizes", [
    [6, 8, 126, 128, 255, 40], [50] * 1100, [3000] * 30, [60000, 30, 500, 77]])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_systems_of_a_batch_advance_as_alone(precision, sizes):
    packs = [_pack(n, 7 + k % 5) for k, n in enumerate(sizes)]
    rates = [10.0 ** -(1 + k % 4) for k in range(len(sizes))]
    got = _run(packs, rates, precision, 30)
    for k in sorted({0, 1, 2, 3, len(sizes) - 1}):
        alone = _run([packs[k]], [rates[k]], precision, 30)[0]
        assert np.array_equal(got[k], alone)
