"""The FP64 form's pair results and reciprocals are taken where there is memory for them and
given back to an allocation that finds none: a handle has the same bits with them, without
them, and where they go on the way."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import handle_probe

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sc(library):
    import spherocyls_gb300

    return spherocyls_gb300


@pytest.fixture(scope="module")
def probe(library, tmp_path_factory):
    return handle_probe.load(tmp_path_factory.mktemp("probe"))


def _protocols(b, between=lambda: None):
    """Every FP64 path of the passes, the rebuild and the minimisers."""
    out = []
    b.set_strain_rate(0.05)
    b.set_resize_rate(1e-3)
    b.set_step(0.02)
    for call in (lambda: b.strain_steps(60, se_every=7), lambda: b.strain_steps(40),
                 lambda: b.resize_steps(20, se_every=20), lambda: b.calc_se(),
                 lambda: b.gd_minimize(10), lambda: b.fire_minimize(1e-30, 110),
                 lambda: b.cg_minimize(12), lambda: b.pure_strain_steps(10), b.find_neighbors,
                 b.calc_forces):
        r = call()
        between()
        out += [np.asarray(v, dtype=float) for v in (r if isinstance(r, tuple) else (r,))
                if v is not None]
        out.append(np.array(b.state()))
    out += [np.array(b.forces()), np.array(b.pairs())]
    return out


def _box(sc, contacts, n=1500, **kw):
    L, x, y, p, R, A = sc.generate_packing(n, 0.85, 1.0, seed=12)
    A = np.where(np.arange(n) % 7 == 0, 0.0, A)
    return sc.SpherocylBox(L, x, y, p, A, R, 0.2, contacts=contacts, **kw)


def _same(a, b):
    assert len(a) == len(b)
    for k, (u, v) in enumerate(zip(a, b)):
        assert np.array_equal(u, v, equal_nan=True), k


@pytest.mark.parametrize("contacts", [1, 2])
@pytest.mark.parametrize("kw", [dict(), dict(use_graphs=False), dict(max_nbrs=70)])
def test_the_same_bits_without_them(sc, probe, contacts, kw):
    with _box(sc, contacts, **kw) as b:
        assert probe.probe_extras(b.h) == (1 if "max_nbrs" in kw else 2)
        want = _protocols(b)
    with _box(sc, contacts, **kw) as b:
        assert probe.probe_give_back(b.h) == 0 and probe.probe_extras(b.h) == 0
        assert probe.probe_give_back(b.h) != 0
        _same(_protocols(b), want)


@pytest.mark.parametrize("contacts", [1, 2])
def test_the_same_bits_where_they_go_on_the_way(sc, probe, contacts):
    with _box(sc, contacts) as b:
        want = _protocols(b)
    for call in (0, 3, 5):
        with _box(sc, contacts) as b:
            left = [k == call for k in range(20)]

            def between():
                if left.pop(0):
                    assert probe.probe_give_back(b.h) == 0

            _same(_protocols(b, between), want)
            assert probe.probe_extras(b.h) == 0


def test_a_full_device(sc, probe):
    """2^20 particles where there is room for their state (about 0.6 GB with the runtime's own)
    and some more, but not for the 0.2 GB of extras: created, minimised and stepped."""
    from spherocyls_gb300 import _lib

    n = 1 << 20
    pack = sc.generate_packing_device(n, 0.85, 1.0, seed=5)
    L, x, y, p, R, A = pack

    def run(b):
        b.set_strain_rate(0.05)
        b.set_step(0.02)
        b.strain_steps(3, se_every=1)
        b.fire_minimize(1e-30, 3)
        b.strain_steps(20)
        b.cg_minimize(1)
        return np.array(b.state())

    with sc.SpherocylBox(L, x, y, p, A, R, 0.1) as b:
        want = run(b)
    assert _lib.lib().sc_trim_memory(0) == 0
    # full before the handle is made, and after
    for left, after in ((760 << 20, False), (1200 << 20, False), (8 << 20, True)):
        block = None if after else probe.probe_fill(left)
        try:
            with sc.SpherocylBox(L, x, y, p, A, R, 0.1) as b:
                assert (probe.probe_extras(b.h) == 2) == (left != 760 << 20)
                if after:
                    block = probe.probe_fill(left)
                got = run(b)
                assert (probe.probe_extras(b.h) == 2) == (left == 1200 << 20)
        finally:
            assert block and probe.probe_free(ctypes.c_void_p(block)) == 0
            _lib.lib().sc_trim_memory(0)
        assert np.array_equal(got, want, equal_nan=True)
