"""Every tiling of a kernel computes the same values, also where the values leave the range
that a forecast lives in: there the kernels' general forms run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNELS = ("slow_stage", "fast_substep", "tracer_stage")


def _step_with(gwm, grid, spec, state, rows, run=lambda m: m.step(1)):
    with gwm.Model(grid, spec) as m:
        for kernel in KERNELS:
            m.set_tile(kernel, rows)
        m.upload(state)
        run(m)
        return m.download()


# Two neighbouring cells whose p' (theta of 4e5 K: 0.7 of the 2^31 Pa at which a total wraps) or
# theta (1e8 K: 0.75 of the 2^27 K) only together leave the range of a warp's total.
@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("theta", [4.0e5, 1.0e8])
@pytest.mark.parametrize("row", [4, 17])
def test_wild_cells_in_adjacent_rows(gwm, row, theta, fast):
    grid = gwm.GridSpec(96, 48, 12, dx=1000.0, dy=1000.0, z_top=6000.0)
    state = gwm.build_case("moist_sounding", grid, gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=3))
    for j in (row, row + 1):
        state["rho_theta"][5, j, 40] = state["rho"][5, j, 40] * np.float32(theta)
    spec = gwm.MemberSpec(step=gwm.StepConfig(dt=1.0e-4, fast_substeps=3, enable_fast_modes=fast))
    a, b = (_step_with(gwm, grid, spec, state, rows) for rows in (16, 3))
    assert np.isfinite(a["w"]).all()
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


# Tracers in the range that upwind transport's tails leave (residuals of the quotient by one
# reciprocal underflow there), zeros of either sign, and a wind that moves a third of a cell a step.
@pytest.mark.parametrize("low,high", [(-149.0, -130.0), (-125.0, -105.0)])
@pytest.mark.parametrize("terrain", [False, True])
def test_tails_of_tracers(gwm, terrain, low, high):
    nx, ny, nz = 70, 37, 14
    hill = None
    if terrain:
        hill = gwm.build_terrain("cosine_mountain", nx, ny, 1000.0, 1000.0, height=300.0, half_width_x=0.3,
                                 half_width_y=0.3)
    flat = gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz)
    grid = gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz, terrain=hill)
    state = gwm.build_case("moist_sounding", flat, gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=3,
                                                                  relative_humidity=1.01), moist=True)
    rng = np.random.default_rng(2)
    state["u"] = (rng.uniform(50.0, 150.0, state["u"].shape)).astype(np.float32)
    state["u"][:, :, -1] = state["u"][:, :, 0]
    for k in ("qv", "qc", "qr"):
        v = np.exp2(rng.uniform(low, high, state[k].shape))
        v[rng.random(v.shape) < 0.05] = -0.0
        state[k] = v.astype(np.float32)
    state["precip"] = np.zeros((ny, nx))
    spec = gwm.MemberSpec(step=gwm.StepConfig(dt=3.0, fast_substeps=3), moist=True)
    a, b = (_step_with(gwm, grid, spec, state, rows, lambda m: m.advance_passive_tracers_ssprk3()) for rows in (16, 3))
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


# Cells beyond the EOS's series, infinite and not-a-number values and tracers that overflow: the
# kernels' tests for their general forms, each in one cell of an otherwise ordinary state and all
# together.
ODD = {"warm": ("rho_theta", 1.2), "cold": ("rho_theta", 0.8), "dense": ("rho", 40.0), "inf_theta": ("rho_theta", np.inf),
       "nan_u": ("u", np.nan), "inf_w": ("w", np.inf), "huge_v": ("v", 3.0e38), "inf_qr": ("qr", np.inf),
       "huge_qc": ("qc", 3.0e38), "nan_qv": ("qv", np.nan)}


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("odd", [*ODD, "all"])
def test_odd_cells(gwm, odd, terrain, periodic):
    nx, ny, nz = 70, 53, 11
    hill = None
    if terrain:
        hill = gwm.build_terrain("cosine_mountain", nx, ny, 1000.0, 1000.0, height=300.0, half_width_x=0.3,
                                 half_width_y=0.3)
    flat = gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz)
    grid = gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz, terrain=hill, periodic_x=periodic,
                        periodic_y=periodic)
    state = gwm.build_case("moist_sounding", flat, gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=3,
                                                                  relative_humidity=1.01), moist=True)
    rng = np.random.default_rng(8)
    for k in ("qc", "qr"):
        state[k] = (state["rho"] * rng.uniform(0.0, 1e-3, state["rho"].shape)).astype(np.float32)
    for n, name in enumerate(ODD if odd == "all" else [odd]):
        field, value = ODD[name]
        at = (1 + 3 * n % 9, 7 + 4 * n, 13 + 5 * n)  # n <= 9: inside
        if np.isfinite(value) and value < 100.0:
            state[field][at] *= np.float32(value)
        else:
            state[field][at] = np.float32(value)
    state["precip"] = np.zeros((ny, nx))
    spec = gwm.MemberSpec(step=gwm.StepConfig(dt=0.5, fast_substeps=3),
                          rain=gwm.WarmRainConfig(dt=0.5, rain_terminal_velocity=12.0), moist=True)
    a, b = (_step_with(gwm, grid, spec, state, rows) for rows in (16, 3))
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)
