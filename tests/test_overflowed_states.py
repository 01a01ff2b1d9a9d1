"""States that have overflowed: the kernels give what the operators' formulas give, not what a
rearranged form of them makes of an infinity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(gwm):
    hill = gwm.build_terrain("cosine_mountain", 20, 18, 1000.0, 1000.0, height=800.0, half_width_x=0.3,
                             half_width_y=0.3)
    grid = gwm.GridSpec(20, 18, 12, dx=1000.0, dy=1000.0, z_top=12000.0, terrain=hill)
    state = gwm.build_case("mountain_wave_background", grid, gwm.CaseParams(rho_surface=1.18, theta_ref=300.0))
    state["rho_theta"][0, 7, 9] = np.float32(1.0e34)  # its pressure overflows
    return grid, state


# The column reference above a cell of infinite pressure: its own density is inf / inf, and the
# level above starts anew from the floor of the pressure (fmaxf takes the number), whichever way
# gravity points.  So only the first two Z faces of the column are touched in one substep.
@pytest.mark.parametrize("rows", [3, 8])
@pytest.mark.parametrize("gravity", [9.81, -9.81])
def test_column_reference_of_an_infinite_pressure(gwm, gravity, rows):
    grid, state = _state(gwm)
    step = gwm.StepConfig(dt=0.1, fast_substeps=1, gravity=gravity)
    with gwm.Model(grid, gwm.MemberSpec(step=step)) as m:
        m.set_tile("fast_substep", rows)
        m.upload(state)
        m.fast_modes()
        w = m.download()["w"]
    assert np.isnan(w[1, 7, 9])
    assert np.isfinite(w[2:, 7, 9]).all()
    w[1, 7, 9] = 0.0
    assert np.isfinite(w).all()
