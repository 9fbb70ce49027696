"""The mixed form in other units: lengths from 1e-18 to 1e18, where FP32 products of lengths
come near the ends of their range, against the FP64 form at the same scale (1e-4 of the RMS
force, the mixed form's bound)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sc(library):
    import spherocyls_gb300

    return spherocyls_gb300


@pytest.mark.parametrize("scale", [1e-18, 1e-17, 1e-13, 1e-6, 1e18])
@pytest.mark.parametrize("contacts", [1, 2])
@pytest.mark.parametrize("kw", [dict(), dict(pass_kind="tile"), dict(persist_steps=True)])
def test_forces_in_other_units(sc, scale, contacts, kw):
    # (at lengths below the lists' absolute margins every candidate is listed, more than the
    # tile pass has room for in a dense packing)
    L, x, y, p, R, A = sc.generate_packing(4096, 0.3 if kw.get("pass_kind") else 0.85, 1.5,
                                           seed=61)
    L, x, y, R, A = (v * scale for v in (L, x, y, R, A))
    out = {}
    for precision, k in (("fp64", {}), ("mixed", kw)):
        with sc.SpherocylBox(L, x, y, p, A, R, 0.3 * scale, precision=precision,
                             contacts=contacts, max_nbrs=160, **k) as b:
            b.calc_forces()
            f = np.array(b.forces())
            f[:2] *= scale
            out[precision] = f
            fmax = b.fire_minimize(1e-30, 1, dt0=1e-30, dt_max=1e-30)[1][0] * scale
            assert np.isfinite(fmax) and fmax > 0
            out[precision + "fire"] = fmax
    rms = np.sqrt(np.mean(out["fp64"][:2] ** 2))
    assert np.abs(out["mixed"] - out["fp64"]).max() <= 1e-4 * rms
    assert abs(out["mixedfire"] - out["fp64fire"]) <= 1e-4 * out["fp64fire"]


@pytest.mark.parametrize("n,phi", [(8, 0.5), (16, 0.7), (24, 0.7)])
def test_small_grids_keep_their_bits(sc, n, phi):
    """Boxes under three cells a side run the variant that scales, with a unit of 1: the
    persistent kernel, which does not scale, gives the same bits."""
    L, x, y, p, R, A = sc.generate_packing(n, phi, 1.0, seed=n)
    out = []
    for persist in (False, True):
        with sc.SpherocylBox(L, x, y, p, A, R, 0.2, precision="mixed",
                             persist_steps=persist) as b:
            b.set_strain_rate(1e-2)
            b.set_step(0.02)
            b.strain_steps(60)
            out.append(np.array(b.state()))
            cols = b.box()["cols"]
    assert cols < 3
    assert np.array_equal(out[0], out[1])
