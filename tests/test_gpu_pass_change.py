"""A handle whose force pass changes rebuilds with kernels of another grid: the list pass
takes blocks of 128 threads up to 4096 particles, the tile pass blocks of 512, and sc_autotune
may take a live handle from one to the other.  Whatever it ran before, a handle then has the
bits of one made with that pass."""
from __future__ import annotations

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


PAD = 0.2
KINDS = {"list": 0, "tile": 1}


def _box(sc, pack, kind, **kw):
    L, x, y, p, R, A = pack
    b = sc.SpherocylBox(L, x, y, p, A, R, PAD, precision="mixed", pass_kind=kind, **kw)
    b.set_strain_rate(0.05)
    b.set_step(0.02)
    return b


def _advance(b):
    """Ten steps, then a forced rebuild; the state and the half neighbour list."""
    b.strain_steps(10)
    b.find_neighbors()
    return np.array(b.state()), np.array(b.pairs())


# below, at and above the size where the list pass changes its block; multiples of 16 and 64
# and none
@pytest.mark.parametrize("n", [500, 1000, 1500, 4000, 4096, 5000])
@pytest.mark.parametrize("first", ["list", "tile"])
def test_pass_changes_keep_the_bits(sc, probe, n, first):
    pack = sc.generate_packing(n, 0.85, 1.0, seed=n)
    kind = first
    live = _box(sc, pack, kind)
    _advance(live)
    for _ in range(4):
        kind = "tile" if kind == "list" else "list"
        assert probe.probe_set_pass(live.h, KINDS[kind], 0, PAD) == 0
        fresh = _box(sc, (pack[0], *live.state(), *pack[4:]), kind)
        fresh.set_gamma(live.box()["gamma"])
        for _ in range(2):
            a, c = _advance(live), _advance(fresh)
            assert np.array_equal(a[0], c[0]) and np.array_equal(a[1], c[1])
        fresh.close()
    live.close()


@pytest.mark.parametrize("n", [1000, 4096])
def test_autotuned_handle_equals_a_fresh_one(sc, n):
    """Made with the tile pass, taken to whatever the autotuner picks, back to work."""
    pack = sc.generate_packing(n, 0.85, 1.0, seed=n + 1)
    live = _box(sc, pack, "tile")
    _advance(live)
    f, _ = live.autotune(5)
    s = np.array(live.state())
    o = live.options()
    L, _, _, _, R, A = pack
    fresh = sc.SpherocylBox(L, *s, A, R, f * PAD, precision="mixed", pass_kind=o["pass_kind"],
                            tile_target=o["tile_target"])
    fresh.set_strain_rate(0.05)
    fresh.set_step(0.02)
    fresh.set_gamma(live.box()["gamma"])
    for _ in range(3):
        a, c = _advance(live), _advance(fresh)
        assert np.array_equal(a[0], c[0]) and np.array_equal(a[1], c[1])
    live.close()
    fresh.close()
