"""A grid barrier that times out leaves its status word, and nothing is rebuilt or advanced
on what that launch left behind: the calls report the time-out, the lists and the state stay.
The status is set from the host here; no wait runs out."""
from __future__ import annotations

import numpy as np
import pytest

import handle_probe

pytestmark = pytest.mark.gpu

BARRIER_TIMEOUT = 8  # ST_BARRIER_TIMEOUT


@pytest.fixture(scope="module")
def sc(library):
    import spherocyls_gb300

    return spherocyls_gb300


@pytest.fixture(scope="module")
def probe(library, tmp_path_factory):
    return handle_probe.load(tmp_path_factory.mktemp("probe"))


def _box(sc, n, **kw):
    L, x, y, p, R, A = sc.generate_packing(n, 0.85, 1.0, seed=n)
    b = sc.SpherocylBox(L, x, y, p, A, R, 0.2, **kw)
    b.set_strain_rate(1e-3)
    b.set_step(0.02)
    b.strain_steps(5)
    return b


@pytest.mark.parametrize("kw", [dict(precision="fp64"), dict(precision="mixed"),
                                dict(precision="mixed", pass_kind="tile")])
def test_no_rebuild_after_a_timeout(sc, probe, kw):
    from spherocyls_gb300 import _lib

    b = _box(sc, 1000, **kw)
    n = b.counters()["rebuilds"]
    assert probe.probe_or_status(b.h, BARRIER_TIMEOUT) == 0
    with pytest.raises(sc.ScError) as ei:
        b.find_neighbors()
    assert ei.value.status == _lib.SC_E_TIMEOUT
    assert b.counters()["rebuilds"] == n
    b.close()


@pytest.mark.parametrize("call", ["steps", "fire"])
def test_persistent_kernels_stop_after_a_timeout(sc, probe, call):
    from spherocyls_gb300 import _lib

    b = _box(sc, 1000, precision="mixed", persist_steps=True)
    b.fire_minimize(1e-3, 1)
    s0 = np.array(b.state())
    assert probe.probe_or_status(b.h, BARRIER_TIMEOUT) == 0
    with pytest.raises(sc.ScError) as ei:
        b.strain_steps(20) if call == "steps" else b.fire_minimize(1e-3, 20)
    assert ei.value.status == _lib.SC_E_TIMEOUT
    assert np.array_equal(np.array(b.state()), s0)
    b.close()
