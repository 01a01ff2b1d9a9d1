"""The acoustic tile that a context starts with, and the environment variable that sets it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("text,rows", [(None, 3), ("0", 0), ("3", 3), ("4", 4), ("8", 8), ("16", 16), ("", 3),
                                       ("5", 3), ("tma", 3), ("-8", 3)])
def test_acoustic_tile_of_a_new_context(gwm, monkeypatch, text, rows):
    monkeypatch.delenv("GWM_B200_FAST_TILE_ROWS", raising=False)
    if text is not None:
        monkeypatch.setenv("GWM_B200_FAST_TILE_ROWS", text)
    with gwm.Model(gwm.GridSpec(20, 18, 6), gwm.MemberSpec()) as m:
        assert {k: m.get_tile(k) for k in ("slow_stage", "fast_substep", "tracer_stage")} == {
            "slow_stage": 3, "fast_substep": rows, "tracer_stage": 3}
