"""Discs (half shafts of zero) among rods, with the lower and with the higher particle index.

The reference's one-point rule takes the lower index as its "p" and finds a disc's contact
with a rod anywhere along the rod when the rod is p, and at the rod's -1 end alone when the
disc is (its 0/0, clamped); the two-point rule finds it anywhere.  Both sides of a pair have
to agree on it: every contact has its reaction."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the passes' bounds against the oracle: the FP64 form's forces to 1e-12 of the RMS force, the
# mixed form's to 1e-4 of it
TOL = {"fp64": 1e-12, "mixed": 1e-4}


@pytest.fixture(scope="module")
def sc(library):
    import spherocyls_gb300

    return spherocyls_gb300


def _pack(sc, n, order):
    """Every third particle a disc (spread over the indices, the lower or the higher half)."""
    L, x, y, p, R, A = sc.generate_packing(n, 0.85, 2.0, seed=n)
    k = np.arange(n)
    disc = {"mixed": k % 3 == 0, "low": k < n // 3, "high": k >= n - n // 3}[order]
    A = np.where(disc, 0.0, A)
    return L, x, y, p, R, A


def _oracle(orc, pack, pad, contacts):
    L, x, y, p, R, A = pack
    b = orc.OracleBox(L, x, y, p, A, R, pad, two_point=contacts == 2)
    b.find_neighbors()
    b.calc_forces()
    return np.array(b.forces())


def _check(forces, want, tol):
    rms = np.sqrt(np.mean(want[:2] ** 2))
    assert np.abs(forces - want).max() <= tol * rms
    # every reaction is there: the forces of all particles sum to nothing
    assert np.abs(forces[:2].sum(axis=1)).max() <= tol * rms * forces.shape[1]


CASES = [("fp64", 1, {}), ("fp64", 1, dict(max_nbrs=80)), ("fp64", 2, {}), ("mixed", 2, {}),
         ("mixed", 2, dict(pass_kind="tile")), ("mixed", 1, {}),
         ("mixed", 1, dict(pass_kind="tile")), ("mixed", 1, dict(pass_kind="tile", tile_target=16))]


@pytest.mark.parametrize("order", ["mixed", "low", "high"])
@pytest.mark.parametrize("precision,contacts,kw", CASES)
def test_forces_of_discs_among_rods(sc, oracle_built, precision, contacts, kw, order):
    pack = _pack(sc, 600, order)
    L, x, y, p, R, A = pack
    want = _oracle(oracle_built, pack, 0.3, contacts)
    with sc.SpherocylBox(L, x, y, p, A, R, 0.3, precision=precision, contacts=contacts,
                         **kw) as b:
        b.calc_forces()
        _check(np.array(b.forces()), want, TOL[precision])


def _shapes(sc, order):
    pack = _pack(sc, 600, "mixed" if order in ("all", "short") else order)
    if order in ("all", "short"):  # discs alone; shafts whose squares' products underflow
        pack = (*pack[:5], np.full_like(pack[5], 0.0 if order == "all" else 1e-80))
    return pack


@pytest.mark.parametrize("contacts", [1, 2])
@pytest.mark.parametrize("order", ["mixed", "low", "high", "all", "short"])
def test_minimiser_forces_of_discs(sc, oracle_built, order, contacts):
    """The minimiser's form of the FP64 pair code (shared reciprocals): the largest force of
    the first FIRE iteration, to 1e-9."""
    pack = _shapes(sc, order)
    L, x, y, p, R, A = pack
    want = _oracle(oracle_built, pack, 0.3, contacts)
    inertia = oracle_built.OracleBox(L, x, y, p, A, R, 0.3).consts()[0]
    big = np.sqrt(np.maximum(want[0] ** 2 + want[1] ** 2, want[2] ** 2 / inertia).max())
    with sc.SpherocylBox(L, x, y, p, A, R, 0.3, contacts=contacts) as b:
        _, fm, _ = b.fire_minimize(1e-30, 1, dt0=1e-9, dt_max=1e-9)
    assert abs(fm[0] - big) <= 1e-9 * big


@pytest.mark.parametrize("contacts", [1, 2])
@pytest.mark.parametrize("order", ["mixed", "low", "high", "all"])
def test_mixed_stress_of_discs(sc, order, contacts):
    """The mixed form's FP64 stress record against the FP64 form's, to 1e-9."""
    L, x, y, p, R, A = _shapes(sc, order)
    se = []
    for precision in ("fp64", "mixed"):
        with sc.SpherocylBox(L, x, y, p, A, R, 0.3, precision=precision, contacts=contacts) as b:
            se.append(np.array(b.calc_se()).ravel())
    assert np.abs(se[1] - se[0]).max() <= 1e-9 * np.abs(se[0]).max()


def test_persistent_steps_of_discs(sc):
    """The persistent kernel against the graph path, bit for bit."""
    L, x, y, p, R, A = _pack(sc, 600, "mixed")
    out = []
    for persist in (False, True):
        with sc.SpherocylBox(L, x, y, p, A, R, 0.3, precision="mixed",
                             persist_steps=persist) as b:
            b.set_strain_rate(1e-2)
            b.set_step(0.02)
            b.strain_steps(60)
            out.append(np.array(b.state()))
    assert np.array_equal(out[0], out[1])
