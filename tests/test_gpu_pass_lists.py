"""Force pass of the mixed form at the ends of its lists: it reads two entries of a list
before it knows the list's length, so capacities of one and two, and particles without
neighbours, have to give what a roomy list gives."""
import numpy as np
import pytest

import spherocyls_gb300 as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 2, 3])
@pytest.mark.parametrize("n", [2, 127, 128, 129, 1000])
def test_capacity_of_a_few(cap, n):
    # touching pairs far from one another, a lone particle last when n is odd
    k = np.arange(n)
    side = int(np.ceil(np.sqrt((n + 1) // 2)))
    L = 8.0 * max(side, 3)
    x = 8.0 * (k // 2 % side) + 2.0 + 0.8 * (k % 2)
    y = 8.0 * (k // 2 // side) + 3.0 + 0.1 * (k % 2)
    phi = 0.3 * np.sin(k)
    R, A = np.full(n, 0.5), np.full(n, 0.4)
    out = []
    for c in (cap, 64):
        b = sc.SpherocylBox(L, x, y, phi, A, R, 0.2, precision="mixed", max_nbrs=c)
        b.set_strain_rate(1e-3)
        b.set_step(0.01)
        b.calc_forces()
        first = b.forces()
        b.strain_steps(5)
        out.append([np.asarray(a) for a in (*first, *b.state()[:3])])
    for a, r in zip(*out):
        assert np.array_equal(a, r)
    assert np.abs(out[0][0][:2]).max() > 0.05
