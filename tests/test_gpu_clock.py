"""The restart clock (seconds): interval steps and response steps of one handle
add up, and a run continued from a restart carries the same clock, bit for bit,
whatever the interval (0.1 yr has no exact binary form)."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth

pytestmark = pytest.mark.gpu


def model(scheme):
    w = synth.Workload("ck", 8, 10, 0.1, 3, 2, "sawtooth", sle=False, visc3d=False, seed=5)
    p = w.params(vlib.default_params)
    p.scheme = scheme
    m = vlib.Model(p)
    m.set_reference(*w.reference())
    return m, w.ice_at(3)


@pytest.mark.parametrize("scheme", [0, 2])
def test_response_and_interval_steps_add_up(scheme):
    m, ice = model(scheme)
    m.set_dt(7.0 * synth.SEC_PER_YEAR)
    sigma = np.zeros(m.nlm, complex)
    want = 0.0
    for dt in (0.1, 3.0, 50.0):
        m.begin_step()
        m.advance(sigma)
        m.update(ice, dt)
        want += (7.0 + dt) * synth.SEC_PER_YEAR
        # rounding: one sum each of at most 1.7e2 yr in seconds
        assert abs(m.state()[1] - want) <= 8 * np.spacing(want)


@pytest.mark.parametrize("dt", [0.1, 0.7])
def test_clock_survives_a_restart(dt):
    a, ice = model(0)
    b, _ = model(0)
    for _ in range(60):
        tau, t = a.state()
        b.set_state(tau, t)
        for m in (a, b):
            m.update(ice, dt)
        assert a.state()[1] == b.state()[1]
