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


class _NoMemory:
    """No device memory for the handle while it lasts."""

    def __init__(self, probe, b):
        self.probe, self.b = probe, b

    def __enter__(self):
        from spherocyls_gb300 import _lib

        _lib.lib().sc_trim_memory(0)
        self.block = self.probe.probe_fill(64 << 20)
        assert self.block and self.probe.probe_exhaust(self.b.h) >= 0

    def __exit__(self, *exc):
        from spherocyls_gb300 import _lib

        assert self.probe.probe_release(self.b.h) == 0
        assert self.probe.probe_free(ctypes.c_void_p(self.block)) == 0
        _lib.lib().sc_trim_memory(0)


def _mixed(sc, n=20000, **kw):
    L, x, y, p, R, A = sc.generate_packing(n, 0.6, 1.0, seed=8)
    b = sc.SpherocylBox(L, x, y, p, A, R, 0.2, precision="mixed", **kw)
    b.set_strain_rate(0.05)
    b.set_step(0.02)
    return b


def test_tile_arrays_after_a_refusal(sc, probe):
    """A pass change that finds no memory for all of the tile pass's arrays is an error, and the
    next one gets those that are missing."""
    from spherocyls_gb300 import _lib

    with _mixed(sc) as b, _mixed(sc, pass_kind="tile") as want:
        with _NoMemory(probe, b):
            assert probe.probe_set_pass(b.h, 1, 0, 0.2) == _lib.SC_E_NOMEM
        assert b.options()["pass_kind"] == "auto"  # as it was
        assert probe.probe_set_pass(b.h, 1, 0, 0.2) == 0
        for box in (b, want):
            box.strain_steps(20)
        assert np.array_equal(np.array(b.state()), np.array(want.state()))


def test_step_arrays_after_a_refusal(sc, probe):
    """Steps and records whose windows and tables find no memory are an error; later ones run."""
    from spherocyls_gb300 import _lib

    with _mixed(sc) as b, _mixed(sc) as want:
        with _NoMemory(probe, b):
            with pytest.raises(sc.ScError) as ei:
                b.strain_steps(100, se_every=1)
            assert ei.value.status in (_lib.SC_E_NOMEM, _lib.SC_E_CUDA)
        a, c = (box.strain_steps(100, se_every=1) for box in (b, want))
        assert np.array_equal(a, c) and np.array_equal(np.array(b.state()), np.array(want.state()))


def test_no_cells_after_a_refusal(sc, probe):
    """A grid that outgrows its cell arrays where there is no memory is an error, and so is every
    later call that needs cells; the state can still be read."""
    from spherocyls_gb300 import _lib

    with _mixed(sc, n=200000) as b:
        s0 = np.array(b.state())
        with _NoMemory(probe, b):
            with pytest.raises(sc.ScError) as ei:
                b.affine_scale(2.0)
            assert ei.value.status == _lib.SC_E_NOMEM
        for call in (b.find_neighbors, b.calc_forces, lambda: b.strain_steps(1), b.calc_se):
            with pytest.raises(sc.ScError) as ei:
                call()
            assert ei.value.status == _lib.SC_E_NOMEM
        assert np.abs(np.array(b.state())[:2] - 2.0 * s0[:2]).max() <= 1e-9 * 2.0 * s0[:2].max()
