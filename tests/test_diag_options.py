"""Options of the diagnostics' command line are taken whatever the command; no GPU."""
import pytest

from bsofi_b200 import _lib, diag


@pytest.mark.parametrize("option", ["--factor-warps=8", "--workers=3", "--chains=2",
                                    "--batch-workers=4"])
def test_option_before_a_command(option, monkeypatch, capsys):
    keys = ["invert_ms", "chain_ms", "leaves", "wait_tile_us", "factor_us", "update_publish_us",
            "to_next_leaf_us", "wait_total_ms", "wait_first_leaf_ms", "wait_p50_us", "wait_p90_us",
            "wait_max_us", "factor_total_ms", "update_total_ms"]
    monkeypatch.setattr(diag, "bsof_timeline", lambda n, L, reps: dict.fromkeys(keys, n + L))
    lib = _lib.load()
    try:
        assert diag.main([option, "bsof-timeline", "64", "4"]) == 0
    finally:
        lib.bsofi_device_set_bsof_workers(0)
        lib.bsofi_device_set_batch_chains(0)
        lib.bsofi_device_set_batch_workers(0)
    assert "n 64 L 4" in capsys.readouterr().out
