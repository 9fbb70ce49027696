"""The FP64 pass through its pair buffers against the one-kernel pass.

Both run the same IEEE operations in the same order, so every result is equal bit for
bit.  A list capacity above one mask word (64) selects the one-kernel pass.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _boxes(n, phi, aor, contacts, gamma, seed=5, pad=0.1):
    from spherocyls_gb300 import SpherocylBox, generate_packing

    L, x, y, p, R, A = generate_packing(n, min(phi, 0.5 if phi > 1 else phi), aor, seed=seed)
    if phi > 1:  # denser than any packing: the generated one shrunk
        f = np.sqrt(0.5 / phi)
        L, x, y = L * f, x * f, y * f
    got = []
    for cap in (64, 65):
        b = SpherocylBox(L, x, y, p, A, R, pad, contacts=contacts, max_nbrs=cap)
        b.set_strain_rate(1e-3)
        b.set_step(0.02)
        if gamma:
            b.set_gamma(gamma)
        got.append(b)
    return got


# one window and less, the window edges (8, 32, 128), grids under three cells a side, the
# switches of the kernels' shapes (4096, 8192, 65536), windows with more contacts than they keep (3.5)
@pytest.mark.parametrize("n,phi,aor,contacts,gamma", [
    (2, 0.05, 1.0, 1, 0.0), (9, 0.8, 1.0, 1, 0.3), (32, 0.8, 1.0, 2, 0.0), (33, 0.7, 1.5, 1, 0.05),
    (1000, 0.9, 0.3, 2, -0.2), (4097, 0.84, 1.0, 2, 0.1),
    (8192, 0.84, 1.0, 1, 0.1), (8201, 0.84, 1.0, 1, 0.1), (65536, 0.84, 1.0, 1, 0.1), (65537, 0.84, 1.0, 1, 0.1),
    (2048, 3.5, 0.05, 1, 0.0), (2048, 3.5, 0.05, 2, 0.2), (9000, 3.5, 0.05, 2, 0.2), (70000, 3.5, 0.05, 1, 0.0)])
def test_pair_buffers_give_the_same_bits(n, phi, aor, contacts, gamma):
    a, b = _boxes(n, phi, aor, contacts, gamma)
    assert np.array_equal(a.calc_se(), b.calc_se())
    for u, v in zip(a.forces(), b.forces()):
        assert np.array_equal(u, v)
    k = 20 if phi < 1 else 2
    assert np.array_equal(a.strain_steps(k, se_every=k // 2), b.strain_steps(k, se_every=k // 2))
    a.set_resize_rate(1e-4)
    b.set_resize_rate(1e-4)
    a.resize_steps(3)
    b.resize_steps(3)
    a.pure_strain_steps(3)
    b.pure_strain_steps(3)
    for u, v in zip(a.state(), b.state()):
        assert np.array_equal(u, v)
    if n <= 2048 and phi < 1:
        for h in (a, b):
            h.fire_minimize(1e-14, 20)
            h.cg_minimize(5)
        for u, v in zip(a.state(), b.state()):
            assert np.array_equal(u, v)


def test_lists_hold_the_same_pairs():
    a, b = _boxes(777, 0.85, 1.0, 1, 0.2)
    assert np.array_equal(a.pairs(), b.pairs())


@pytest.mark.parametrize("n,phi,aor,gamma,pad", [
    (40, 0.8, 1.0, 0.0, 0.0), (500, 0.85, 1.0, 0.45, 0.1), (500, 0.85, 1.0, -0.3, 0.1),
    (5000, 0.84, 1.5, 0.3, 0.2), (70000, 0.84, 0.3, 0.1, 0.3)])
def test_list_equals_the_oracles(oracle_built, n, phi, aor, gamma, pad):
    """The FP32-decided list is the reference's (check_neighbors,
    src/cpp/spherocyl_box.cpp:303-318), pair for pair."""
    from spherocyls_gb300 import generate_packing

    a, _ = _boxes(n, phi, aor, 1, gamma, pad=pad)
    L, x, y, p, R, A = generate_packing(n, phi, aor, seed=5)
    ob = oracle_built.OracleBox(L, x, y, p, A, R, pad, gamma=gamma)
    ob.find_neighbors()
    ref = ob.pairs()
    assert np.array_equal(a.pairs(), ref[np.lexsort((ref[:, 1], ref[:, 0]))])


@pytest.mark.parametrize("shape", [0.0, 1e-170, 1e-80, 0.02])
def test_shapes_at_the_end_of_the_range(oracle_built, shape):
    """Half shafts of zero (discs) and so short that the reciprocal of their square leaves
    the range of the shared quotients, against the oracle: 1e-12 of the RMS force, the
    bound of the FP64 form's forces."""
    from spherocyls_gb300 import SpherocylBox, generate_packing

    L, x, y, p, R, A = generate_packing(600, 0.85, 0.05, seed=9)
    A = np.full_like(A, shape)
    b = SpherocylBox(L, x, y, p, A, R, 0.1)
    b.calc_forces()
    ob = oracle_built.OracleBox(L, x, y, p, A, R, 0.1)
    ob.find_neighbors()
    ob.calc_forces()
    f = ob.forces()
    rms = np.sqrt(np.mean([f[0] ** 2, f[1] ** 2]))
    for u, v in zip(b.forces(), f):
        assert np.abs(u - v).max() <= 1e-12 * rms
