"""Several handles stepped from their own threads on one GPU: each has the bits it has alone.
Every step carries a cooperative rebuild kernel, whose blocks have to be resident together
beside whatever the other handles run."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sc(library):
    import spherocyls_gb300

    return spherocyls_gb300


def _run(sc, pack, precision, out, k):
    L, x, y, p, R, A = pack
    with sc.SpherocylBox(L, x, y, p, A, R, 0.2, precision=precision) as b:
        b.set_strain_rate(0.05)
        b.set_step(0.02)
        se = b.strain_steps(60, se_every=10)
        b.find_neighbors()
        b.fire_minimize(1e-30, 60)
        out[k] = (np.array(b.state()), se)


@pytest.mark.parametrize("sizes", [(1000, 1000), (30000, 30000), (200, 4000, 60000, 9000)])
def test_handles_in_threads(sc, sizes):
    jobs = [(sc.generate_packing(n, 0.85, 1.0, seed=n + k), prec)
            for k, n in enumerate(sizes) for prec in ("fp64", "mixed")]
    alone, beside = {}, {}
    for k, (pack, prec) in enumerate(jobs):
        _run(sc, pack, prec, alone, k)
    threads = [threading.Thread(target=_run, args=(sc, pack, prec, beside, k))
               for k, (pack, prec) in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert sorted(beside) == sorted(alone)
    for k in alone:
        assert np.array_equal(alone[k][0], beside[k][0]), k
        assert np.array_equal(alone[k][1], beside[k][1]), k
