"""Kernels whose work split depends on the sizes, at the sizes where the split changes:
scalar transport in strips of 29 columns and 32 rows, warm rain with a column's levels shared
by eight, four or two warps, the training gradient in chunks of samples, and the terrain
substep without its density or momentum update."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one cell, a halo that wraps more than once, strip edges and remainders; winds of every sign;
# spacings within and outside the range of the residual quotients
@pytest.mark.parametrize("nx,ny,nz,u,v,px,py,steps,dx", [
    (1, 1, 1, 12.0, 7.0, True, True, 3, 1000.0),
    (2, 3, 2, -12.0, 7.0, True, True, 2, 1000.0),
    (29, 32, 1, 12.0, -7.0, True, False, 5, 1000.0),
    (30, 33, 2, -12.0, -7.0, False, True, 4, 700.0),
    (59, 129, 3, 0.0, 7.0, False, False, 3, 1000.0),
    (257, 5, 2, -12.0, 0.0, True, True, 1, 333.0),
    (61, 40, 2, 12.0, 7.0, False, False, 3, 3.0e6),
])
def test_scalar_strips_match_the_restated_roundings(gwm, orc, nx, ny, nz, u, v, px, py, steps, dx):
    rng = np.random.default_rng(11)
    q = rng.normal(1.0, 0.5, (nz, ny, nx)).astype(np.float32)
    q[rng.random(q.shape) < 0.1] = 0.0
    q[rng.random(q.shape) < 0.05] *= np.float32(1e-30)  # differences below the residual range
    a = dict(dt=0.25 * dx / 12.0, dx=dx, dy=dx, periodic_x=px, periodic_y=py, nsteps=steps)
    ref = orc.scalar_ssprk3(q, u, v, precision=32, **a)  # FP32 with the operator's roundings
    np.testing.assert_array_equal(gwm.scalar_ssprk3(q, u_adv=u, v_adv=v, **a), ref.astype(np.float32))


# 2 strips of 32 columns a row: 16 rows are split over eight warps, 1184 rows (2368 strips)
# over four, 2368 rows over two; fewer levels than warps, remainders, one level
@pytest.mark.parametrize("fallout", [None, "metric", "nominal"])
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("nz", [1, 5, 13, 64])
def test_warm_rain_level_split(gwm, nz, terrain, fallout):
    nx, low = 40, 16
    rng = np.random.default_rng(3)
    base = gwm.build_case("moist_sounding", gwm.GridSpec(nx, low, nz, dx=3000.0, dy=3000.0, z_top=260.0 * nz),
                          gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=7, relative_humidity=1.02), moist=True)
    base["qc"] = (base["rho"] * rng.uniform(0.0, 3e-3, base["rho"].shape)).astype(np.float32)
    base["qr"] = (base["rho"] * rng.uniform(0.0, 2e-3, base["rho"].shape)).astype(np.float32)
    base["qr"][:, ::3] = 0.0
    out = {}
    for copies in (1, 74, 148):
        ny = low * copies
        hill = None
        if terrain:  # heights of the first rows in every copy
            hill = np.tile(gwm.build_terrain("cosine_mountain", nx, low, 3000.0, 3000.0, height=200.0, half_width_x=0.3,
                                             half_width_y=0.3), (copies, 1))
        grid = gwm.GridSpec(nx, ny, nz, dx=3000.0, dy=3000.0, z_top=260.0 * nz, terrain=hill)
        state = {}
        for k, f in base.items():
            rows = np.tile(f[:, :low], (1, copies, 1))
            state[k] = np.concatenate([rows, rows[:, :1]], axis=1) if k == "v" else rows
        rain = gwm.WarmRainConfig(dt=2.0, rain_terminal_velocity=12.0, sedimentation_layer_depth_m=400.0)
        with gwm.Model(grid, gwm.MemberSpec(rain=rain, moist=True)) as m:
            m.upload(dict(state, precip=np.zeros((ny, nx))))
            m.apply_warm_rain_microphysics(fallout)
            out[copies] = m.download(keys=["rho_theta", "qv", "qc", "qr", "precip"])
    assert fallout is None or out[1]["precip"].max() > 0
    for copies in (74, 148):
        for k, f in out[1].items():
            reps = (copies, 1) if f.ndim == 2 else (1, copies, 1)
            np.testing.assert_array_equal(out[copies][k], np.tile(f, reps), err_msg=f"{k}, {copies} copies")


# warm rain against the FP64 oracle where eight warps share few, odd and many levels; bounds of
# the moist step's own comparison
@pytest.mark.parametrize("nz", [3, 9, 50])
def test_warm_rain_level_split_vs_oracle(gwm, orc, nz):
    grid = gwm.GridSpec(33, 5, nz, dx=3000.0, dy=3000.0, z_top=300.0 * nz)
    state = gwm.build_case("moist_sounding", grid, gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=7,
                                                                  relative_humidity=1.02), moist=True)
    state["qr"] = (state["rho"] * np.random.default_rng(5).uniform(0.0, 2e-3, state["rho"].shape)).astype(np.float32)
    with gwm.Model(grid, gwm.MemberSpec(rain=gwm.WarmRainConfig(dt=2.0, rain_terminal_velocity=12.0),
                                        moist=True)) as m:
        m.upload(state)
        m.apply_warm_rain_microphysics("metric")
        out = m.download()
    ref = orc.run(orc.GridSpec(33, 5, nz, dx=3000.0, dy=3000.0, z_top=300.0 * nz), orc.StepSpec(),
                  {k: v.astype(np.float64) for k, v in state.items()}, 1, phases=orc.PHASE_RAIN,
                  rain=orc.RainSpec(dt=2.0, terminal_velocity=12.0), precision=64)
    for k in ("rho_theta", "qv", "qc", "qr", "precip"):
        tol = 1e-5 if k == "rho_theta" else 1e-3
        assert np.abs(out[k] - ref[k]).max() <= tol * max(np.abs(ref[k]).max(), 1e-9), k


# a chunk of 1024 samples and its neighbours, one sample, a remainder of four-lane groups
@pytest.mark.parametrize("n", [1, 31, 1023, 1025, 2048])
def test_training_gradient_chunks(gwm, orc, n):
    from test_surrogate import _random_net
    p, norm = _random_net(5)
    rng = np.random.default_rng(6)
    f32 = lambda a: np.asarray(a).astype(np.float32)
    p, norm, x, y = f32(p), f32(norm), f32(rng.normal(0, 1.5, (n, 7))), f32(rng.normal(0, 1.5, (n, 5)))
    loss, grad = gwm.mlp_loss_grad(p, norm, x, y)
    f64 = lambda a: a.astype(np.float64)
    lo, go = orc.mlp_loss_grad(f64(p), f64(norm), f64(x), f64(y))
    assert abs(loss - lo) <= 1e-5 * lo  # bounds of the 3000-sample comparison
    assert np.abs(grad - go).max() <= 2e-4 * np.abs(go).max()


@pytest.mark.parametrize("momentum,density", [(False, True), (True, False), (False, False)])
def test_terrain_substep_without_momentum_or_density(gwm, momentum, density):
    hill = gwm.build_terrain("cosine_mountain", 45, 37, 1000.0, 1000.0, height=400.0, half_width_x=0.3,
                             half_width_y=0.3)
    grid = gwm.GridSpec(45, 37, 19, dx=1000.0, dy=1000.0, z_top=9500.0, terrain=hill)
    state = gwm.build_case("mountain_wave_background", grid, gwm.CaseParams(rho_surface=1.18, theta_ref=300.0,
                                                                            u_background=10.0))
    step = gwm.StepConfig(dt=1.0, fast_substeps=3, fast_update_horizontal_momentum=momentum,
                          fast_update_density=density)
    out = {}
    with gwm.Model(grid, gwm.MemberSpec(step=step)) as m:
        for rows in (8, 3):
            m.set_tile("fast_substep", rows)
            m.upload(state)
            m.step(2)
            out[rows] = m.download()
    for k in out[3]:
        np.testing.assert_array_equal(out[3][k], out[8][k], err_msg=k)
