"""The stand-alone operators run the TMA-fed kernels by default, whose bounded waits can give
up: the call that ran such a kernel reports it, for every member, and the next call is not
charged with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _member(gwm, terrain, nx=72, ny=40, nz=16):
    hill = None
    if terrain:
        hill = gwm.build_terrain("cosine_mountain", nx, ny, 2000.0, 2000.0, height=300.0, half_width_x=0.3,
                                 half_width_y=0.3)
    flat = gwm.GridSpec(nx, ny, nz, dx=2000.0, dy=2000.0, z_top=8000.0)
    grid = gwm.GridSpec(nx, ny, nz, dx=2000.0, dy=2000.0, z_top=8000.0, terrain=hill)
    state = gwm.build_case("moist_sounding", flat, gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=3,
                                                                  relative_humidity=1.02), moist=True)
    spec = gwm.MemberSpec(step=gwm.StepConfig(dt=1.0, fast_substeps=3),
                          rain=gwm.WarmRainConfig(dt=1.0, rain_terminal_velocity=12.0), moist=True)
    return grid, state, spec


OPERATORS = {"tracers": lambda m: m.advance_passive_tracers_ssprk3(), "fast_modes": lambda m: m.fast_modes()}


@pytest.mark.parametrize("members", [1, 2])
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("op", list(OPERATORS))
def test_operator_reports_a_wait_that_gave_up(gwm, op, terrain, members):
    grid, state, spec = _member(gwm, terrain)
    run = OPERATORS[op]
    out = {}
    for stall in (False, True):
        with gwm.Model([grid] * members, [spec] * members) as m:
            for q in range(members):
                m.upload(state, member=q)
            if stall:
                for q in range(members):
                    m.test_stall_tile_load(plane=2, member=q)
                with pytest.raises(RuntimeError, match="status -5"):
                    run(m)
                for q in range(members):
                    m.upload(state, member=q)
            run(m)
            out[stall] = [m.download(member=q) for q in range(members)]
    for a, b in zip(out[False], out[True]):
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# The first plane that a CTA loads never arrives while the ones above it do: its wait gives up
# in the prologue, and the planes behind it are still accounted for when the CTA leaves.
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("op", ["step", *OPERATORS])
def test_first_plane_of_a_chunk_never_arrives(gwm, op, terrain):
    grid, state, spec = _member(gwm, terrain)
    run = dict(OPERATORS, step=lambda m: m.step(1))[op]
    out = {}
    for stall in (False, True):
        with gwm.Model(grid, spec) as m:
            m.upload(state)
            if stall:
                m.test_stall_tile_load(plane=0)
                with pytest.raises(RuntimeError, match="status -5"):
                    run(m)
                m.upload(state)
            run(m)
            out[stall] = m.download()
    for k in out[False]:
        np.testing.assert_array_equal(out[True][k], out[False][k], err_msg=k)


# Each kernel of a step in turn: k_slow_tma, k_fast_rows (inner and last substep) and
# k_tracer_tma on flat levels, their terrain forms on terrain.
@pytest.mark.parametrize("plane", [0, 3])
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("kernel", ["slow_stage", "fast_substep", "last_substep", "tracer_stage"])
def test_each_kernel_of_a_step_gives_up_and_recovers(gwm, kernel, terrain, plane):
    grid, state, spec = _member(gwm, terrain)
    out = {}
    for stall in (False, True):
        with gwm.Model(grid, spec) as m:
            m.upload(state)
            if stall:
                m.test_stall_tile_load(plane=plane, kernel=kernel)
                with pytest.raises(RuntimeError, match="status -5"):
                    m.step(1)
                m.upload(state)
            m.step(1)
            out[stall] = m.download()
    for k in out[False]:
        np.testing.assert_array_equal(out[True][k], out[False][k], err_msg=k)
