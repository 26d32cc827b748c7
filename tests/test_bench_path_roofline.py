"""bench.py's roofline of the path kernel on the CPU, with a stand-in context."""
import pytest

import bench

STATS = {"extend_launches": 10, "extend_ms": 5.0, "accumulate_ms": 0.3, "plan_ms": 0.2, "rays": 80_000_000,
         "shadow_rays": 20_000_000, "camera_samples": 40_000_000, "node_visits": 500_000_000, "prim_tests": 300_000_000,
         "shadow_node_visits": 100_000_000, "shadow_prim_tests": 20_000_000}
PEAKS = {"hbm": 6650.0, "l1": 30000.0, "l2": 17500.0, "sms": 148, "sm_mhz": 1965.0}


class FakeCtx:
    def set_tuning(self, **kw):
        pass


@pytest.mark.parametrize("mhz", [1965.0, None])
@pytest.mark.parametrize("profile", [True, False])
def test_levels_of_the_path_kernel(profile, mhz):
    out, kernel_ms, _ = bench.path_roofline(FakeCtx(), lambda: dict(STATS), dict(PEAKS, sm_mhz=mhz), profile)
    prof = bench.path_profile()
    per_s = {"hbm": 40e6 * 16 / 5e-3 / 1e9, "l1": (600e6 * 64 + 320e6 * 48) / 5e-3 / 1e9}
    if profile:
        per_s["l2"] = prof["l2_bytes_per_ray"] * 100e6 / 5e-3 / 1e9
        if mhz:
            per_s["issue"] = prof["warp_inst_per_ray"] * 100e6 / 5e-3 / 1e9
    assert {k: v["achieved"] for k, v in out["levels"].items()} == pytest.approx(per_s)
    fracs = {k: v["frac"] for k, v in out["levels"].items()}
    assert out["bound"] == max(fracs, key=fracs.get) and out["frac"] == fracs[out["bound"]]
    assert (out["traffic"] is None) == (not profile)
    assert sum(kernel_ms.values()) == pytest.approx(5.5) and out["share_of_kernel_time"] == pytest.approx(5.0 / 5.5)
