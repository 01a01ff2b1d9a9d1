"""Whole steps at the sizes where warm rain changes how many warps share a column: its level sums
of theta feed the next step.  The rows of a small grid are repeated (a power of two of times, so
that the level means round alike), which leaves every value as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, LOW = 40, 16  # two strips of 32 columns a row


# 32 strips: eight warps a column; 4096: four; 8192: two
@pytest.mark.parametrize("copies", [128, 256])
@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("terrain", [False, True])
def test_steps_of_repeated_rows(gwm, terrain, learned, copies):
    nz = 13
    base = gwm.build_case("moist_sounding", gwm.GridSpec(NX, LOW, nz, dx=3000.0, dy=3000.0, z_top=250.0 * nz),
                          gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=7, relative_humidity=1.02), moist=True)
    rng = np.random.default_rng(4)
    base["qc"] = (base["rho"] * rng.uniform(0.0, 3e-3, base["rho"].shape)).astype(np.float32)
    base["qr"] = (base["rho"] * rng.uniform(0.0, 2e-3, base["rho"].shape)).astype(np.float32)
    base["v"][:, -1] = base["v"][:, 0]
    out = {}
    for n in (1, copies):
        hill = None
        if terrain:
            hill = np.tile(gwm.build_terrain("cosine_mountain", NX, LOW, 3000.0, 3000.0, height=200.0, half_width_x=0.3,
                                             half_width_y=0.3), (n, 1))
        grid = gwm.GridSpec(NX, LOW * n, nz, dx=3000.0, dy=3000.0, z_top=250.0 * nz, terrain=hill)
        state = {}
        for k, f in base.items():
            rows = np.tile(f[:, :LOW], (1, n, 1))
            state[k] = np.concatenate([rows, rows[:, :1]], axis=1) if k == "v" else rows
        spec = gwm.MemberSpec(step=gwm.StepConfig(dt=0.5, fast_substeps=3),
                              rain=gwm.WarmRainConfig(dt=0.5, rain_terminal_velocity=12.0), moist=True)
        with gwm.Model(grid, spec) as m:
            if learned:
                m.set_rain_surrogate()
            m.upload(dict(state, precip=np.zeros((LOW * n, NX))))
            m.step(3)
            out[n] = m.download()
    assert out[1]["precip"].max() > 0
    for k, f in out[1].items():
        big = out[copies][k]
        axis = 0 if f.ndim == 2 else 1
        rows = f if k != "v" else f[:, :LOW]
        got = big if k != "v" else big[:, :LOW * copies]
        np.testing.assert_array_equal(got, np.concatenate([rows] * copies, axis=axis), err_msg=k)
