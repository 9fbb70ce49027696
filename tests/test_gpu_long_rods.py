"""Rods thousands of radii long: FP32 shaft vectors are off by more than a contact's overlap
at their ends, and the screens have to allow for it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(ratio, k):
    """k systems of two rods, the end of one a hair (overlap 3e-5 to 6e-4 of the contact
    distance) inside the side of the other."""
    rng = np.random.default_rng(int(ratio))
    L = 8.0 * (ratio + 2.0)
    x, y, p = np.empty(2 * k), np.empty(2 * k), np.empty(2 * k)
    for i in range(k):
        th = rng.uniform(-np.pi, np.pi)
        u = np.array([np.cos(th), np.sin(th)])
        n = np.array([-u[1], u[0]])
        a = th + rng.uniform(0.3, np.pi - 0.3)
        v = np.array([np.cos(a), np.sin(a)])  # away from the first rod
        c = rng.uniform(0.3 * L, 0.7 * L, 2)
        end = c + rng.uniform(-0.8, 0.8) * ratio * u + 2.0 * (1 - 10 ** rng.uniform(-4.5, -3.2)) * n
        q = end + ratio * v
        order = [2 * i, 2 * i + 1] if i % 2 else [2 * i + 1, 2 * i]
        x[order], y[order], p[order] = (c[0], q[0]), (c[1], q[1]), (th, a)
    return L, x, y, p


@pytest.mark.parametrize("ratio", [10.0, 300.0, 3000.0, 30000.0])
@pytest.mark.parametrize("contacts", [1, 2])
def test_contacts_of_long_rods(oracle_built, library, ratio, contacts):
    from spherocyls_gb300 import BoxBatch

    k = 64
    L, x, y, p = _pairs(ratio, k)
    R, A = np.ones(2 * k), np.full(2 * k, ratio)
    want, energy = [], []
    for i in range(k):
        s = slice(2 * i, 2 * i + 2)
        ob = oracle_built.OracleBox(L, x[s], y[s], p[s], A[s], R[s], 0.5, two_point=contacts == 2)
        ob.find_neighbors()
        ob.calc_se()
        energy.append(ob.se()[0])
        ob.calc_forces()
        want.append(np.array(ob.forces()))
    want, energy = np.concatenate(want, axis=1), np.array(energy)
    assert (np.abs(want[0]) > 0).all()
    # overlaps are differences of lengths of the rods' size: their rounding bounds the forces
    tol = 1e-15 * 50 * ratio
    b = BoxBatch([2] * k, [L] * k, x, y, p, A, R, 0.5, contacts=contacts)
    b.calc_forces()
    assert np.abs(np.array(b.forces())[:2] - want[:2]).max() <= tol
    e = b.calc_se()[:, 0]
    assert np.abs(np.sqrt(e) - np.sqrt(energy)).max() <= tol
    b.close()
    # the mixed form's record: its state is the FP64 one to about 2^-48
    m = BoxBatch([2] * k, [L] * k, x, y, p, A, R, 0.5, precision="mixed", contacts=contacts)
    e = m.calc_se()[:, 0]
    assert np.abs(np.sqrt(e) - np.sqrt(energy)).max() <= tol + 2.0 ** -46 * 8 * ratio
    m.close()
