"""Scalar transport of fields with zeros of both signs: the operator's result bit for bit, the
signs of its zeros included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("u,v", [(12.0, 7.0), (-12.0, 7.0), (12.0, -7.0), (-12.0, -7.0)])
def test_signs_of_zeros(gwm, orc, u, v):
    rng = np.random.default_rng(9)
    q = rng.choice(np.array([0.0, -0.0, 1.0], np.float32), (3, 40, 37), p=[0.45, 0.45, 0.1])
    a = dict(dt=20.0, dx=1000.0, dy=1000.0, periodic_x=True, periodic_y=False, nsteps=1)
    ref = orc.scalar_ssprk3(q, u, v, precision=32, **a).astype(np.float32)
    out = gwm.scalar_ssprk3(q, u_adv=u, v_adv=v, **a)
    np.testing.assert_array_equal(out.view(np.uint32), ref.view(np.uint32))
