"""Kerr-family rays where the unguarded and the guarded FP32 step take turns: the
spin axis in view, the horizon of a near-extremal hole, a barely naked singularity,
step budgets that end within a few steps -- against the CPU oracle, with the
parity suite's bars (escape directions at the axis: the FP32 oracle itself is
within 1e-4 rad of the FP64 integration on 98.5 % of such rays)."""
import pytest

import parity
from bhrt import lib, scenes
from bhrt.abi import BH_KERR, BH_KERR_NEWMAN

pytestmark = pytest.mark.gpu

NX, NY = 96, 54

CASES = [
    # name, model, a*, q, distance, elevation, max steps, naked, share of escapes within 1e-4 rad
    ("axis", BH_KERR_NEWMAN, 0.8, 0.3, 12.0, 89.5, 2000, False, 0.98),
    ("near_axis", BH_KERR, 0.9, 0.0, 8.0, 86.0, 2000, False, 0.98),
    ("axis_in_view", BH_KERR, 0.9, 0.0, 20.0, 10.0, 2000, False, 0.98),
    ("near_extremal", BH_KERR_NEWMAN, 0.99, 0.1, 3.0, 20.0, 2000, False, 0.98),
    ("barely_naked", BH_KERR, 1.00001, 0.0, 10.0, 30.0, 2000, True, 0.98),
    ("budget_1", BH_KERR, 0.9, 0.0, 20.0, 10.0, 1, False, 0.98),
    ("budget_2", BH_KERR, 0.9, 0.0, 20.0, 89.0, 2, False, 0.98),
    ("budget_41", BH_KERR_NEWMAN, -0.7, 0.4, 6.0, 60.0, 41, False, 0.98),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("disk", [True, False], ids=["disk", "no_disk"])
def test_step_forms_match_oracle(cuda, oracle, case, disk):
    from bhrt.device import probe_grid
    _, model, a, q, dist, el, steps, naked, share = case
    P = scenes.scene(lib.derive, model, a, q, NX, NY, dist, el, 50.0, disk=disk, allow_naked=naked)
    P.maxSteps = steps
    s = parity.compare_rays(probe_grid(P, NX, NY), oracle.probe_grid(P, NX, NY))
    assert s["cls_mismatch_inner"] == 0, s
    assert s["esc_frac_1e4"] >= share, s


@pytest.mark.parametrize("steps", [24, 37, 2000])
def test_mixed_passages_match_fp64(cuda, steps):
    """FP64 polar passages taken together by a warp's lanes, with step budgets that end
    inside a passage or just after it, against the all-FP64 integration."""
    from bhrt.device import probe_grid
    P = scenes.scene(lib.derive, BH_KERR, 0.9, 0.0, NX, NY, 12.0, 89.5, 50.0)
    P.maxSteps = steps
    got, want = probe_grid(P, NX, NY, precision=1), probe_grid(P, NX, NY, precision=2)
    s = parity.compare_rays(got, want)
    assert s["outcome_mismatch_inner"] == 0, s
    assert s["esc_frac_1e4"] >= 0.98, s
    again = probe_grid(P, NX, NY, precision=1)
    assert again.tobytes() == got.tobytes()
