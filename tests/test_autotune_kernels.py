"""What the autotuner times is what a launch runs: named start blocks (never the library's choice,
which depends on the number of pairs), each launched kernel once, and no ranking of other kernels."""
import pytest

from fast_shepherd_score_b200 import autotune

SIZES = [("esp", 400, 50), ("esp", 40, 50), ("shape", 50, 50), ("shape", 400, 50),
         ("esp_combo", 25, 8), ("esp_combo", 25, 50), ("shape_pharm", 60, 20), ("pharm", 20, 32),
         ("shape", 30, 1)]


@pytest.mark.parametrize("mode,max_fit,starts", SIZES)
def test_start_blocks_are_named(mode, max_fit, starts):
    tiles = autotune.candidates(mode, max_fit, starts, tensor_cores=True)
    assert all(1 <= c["chunks"] <= starts for c in tiles)
    for lanes in {c["lanes_per_pose"] for c in tiles}:
        mine = {c["chunks"] for c in tiles if c["lanes_per_pose"] == lanes}
        # fewest idle slots in CTAs of up to 320 threads, by trying all of them
        def idle(c):
            poses = -(-starts // c)
            return -(-poses * lanes // 32) * 32 // lanes * c - starts
        fit = [c for c in range(1, starts + 1) if -(-starts // c) <= 320 // lanes]
        assert min(fit, key=lambda c: (idle(c), c)) in mine
        for warps in (1, 2, 4):
            assert -(-starts // (warps * 32 // lanes)) in mine


@pytest.mark.parametrize("mode,max_fit,starts", SIZES)
def test_each_kernel_once(mode, max_fit, starts):
    def kernel(c):   # launch_align: from 4 lanes on, up to 16 fit points a lane, 1 and 3 are one
        lanes, var = c["lanes_per_pose"], c.get("kernel_variant", 0)
        spread = lanes >= 4 and max_fit <= 16 * lanes
        if var == 3 and spread and not (mode == "esp" and lanes == 32):
            var = 1
        poses = -(-(-(-starts // c["chunks"]) * lanes) // 32) * 32 // lanes   # of whole warps
        return lanes, -(-starts // poses), c["cta_per_sm"], var, c.get("accumulate", 0)
    tiles = [kernel(c) for c in autotune.candidates(mode, max_fit, starts, tensor_cores=True)]
    assert len(tiles) == len(set(tiles))


def test_key_names_the_kernels(monkeypatch):
    monkeypatch.setattr(autotune, "_device_name", lambda device: "gpu")
    key = lambda: autotune.shape_key("cuda:0", "shape", 50, 50, 30.0, 50, 256, 200)
    before = key()
    monkeypatch.setattr(autotune, "KERNELS", autotune.KERNELS + 1)
    assert key() != before
