"""A step so long that its predictor takes particles sixty boxes out, where an FP32 coordinate
is off by more than a contact's overlap: the FP64 form still finds what touches there."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(shift, overlap):
    """Discs of diameter D.  k1 pushes i along x; ka and kb push j the same way a little less
    far, so that i, 0.1 short of j, reaches into it by `overlap` at the predictor.  D is 127.5
    FP32 spacings there (x about 1.2e5), so that rounding may take the two apart."""
    L, dt, D = 2000.0, 1.2e6, 127.5 / 128
    i, j = np.array([10.9 + shift, 20.0]), np.array([11.0 + D + shift, 20.0])
    k1 = i - [0.9 * D, 0.0]
    th = np.radians(70.0)
    push = 0.1 / D  # the force on i: (1 - 0.9) / D
    f = (push - (0.1 + overlap) / dt) / (2 * np.cos(th))  # each pusher's force on j
    ka, kb = (j - D * (1.0 - f * D) * np.array([np.cos(th), s * np.sin(th)]) for s in (1, -1))
    x, y = np.array([i, j, k1, ka, kb]).T.copy()
    z = np.zeros(5)
    return L, x, y, z, np.full(5, D / 2), z, dt


@pytest.mark.parametrize("max_nbrs", [0, 80])
@pytest.mark.parametrize("order", [[0, 1, 2, 3, 4], [4, 3, 2, 1, 0]])
def test_contacts_far_outside_the_box(oracle_built, library, order, max_nbrs):
    from spherocyls_gb300 import SpherocylBox

    touched = 0
    for shift in np.linspace(0.0, 0.0078, 12):
        L, x, y, p, R, A, dt = _pack(shift, 0.0015)
        x, y = x[order], y[order]
        ob = oracle_built.OracleBox(L, x, y, p, A, R, 0.5, strain_rate=0.0, step=dt)
        ob.find_neighbors()
        ob.calc_forces()
        ob.run_strain_steps(1)
        with SpherocylBox(L, x, y, p, A, R, 0.5, max_nbrs=max_nbrs) as b:
            b.set_strain_rate(0.0)
            b.set_step(dt)
            b.strain_steps(1)
            got, want = np.array(b.state()), np.array(ob.state())
        # i would have gone on by half of push * dt without the contact
        touched += abs(want[0][order.index(0)] - (x[order.index(0)] + 0.05 * dt)) % L > 1.0
        d = got[:2] - want[:2]
        assert np.abs(d - L * np.round(d / L)).max() <= 1e-6 * L
    assert touched == 12
