"""Fields of the bench line that follow the form the engine ran."""

from __future__ import annotations

from types import SimpleNamespace

import pytest

import bench

C2 = SimpleNamespace(n_tiles=102, schur_tile_updates=144931)   # 1000-atom cube, natural order
SHEET = SimpleNamespace(n_tiles=7, schur_tile_updates=91)


def test_the_engines_plan_summary_serves():
    """The engine's own summary carries what schur_steps reads."""
    from aospectrum_b200.engine import PlanSummary

    fields = {f: 1 for f in PlanSummary.__dataclass_fields__}
    assert bench.schur_steps(PlanSummary(**fields), 64, 2, False) == 2


@pytest.mark.parametrize("info,pencils,depth,pairs,steps", [
    (C2, 64, 2, False, 4), (C2, 8, 2, False, 4), (C2, 7, 2, False, 2), (C2, 64, 2, True, 2),
    (C2, 64, 1, False, 1), (SHEET, 4000, 2, False, 2)])
def test_schur_steps_and_their_capture(info, pencils, depth, pairs, steps):
    assert bench.schur_steps(info, pencils, depth, pairs) == steps
    traffic = bench.schur_traffic_per_unit(steps)
    if steps == 1:
        assert traffic is None
        return
    assert {2: "two_step", 4: "four_step"}[steps] in traffic["source"]
    # a target's 256 KB read and written once per update, operands beside it
    assert traffic["bytes_per_unit"] > 2 * 128 * 128 * 8 / steps
