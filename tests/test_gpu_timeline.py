"""The BSOF chain's timeline: a leaf starts, is factored, gets the next leaf's
tile and is done, in this order, and the time without the tile is reported as
waiting.  One worker CTA (the chain waits for it) against the plan's count."""
import pytest

from bsofi_b200 import _lib, diag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(64, 6), (256, 3), (300, 3), (641, 2)])
def test_phases_of_a_leaf(cuda_device, n, L):
    lib = _lib.load()
    lib.bsofi_device_set_bsof_workers(1)
    try:
        slow = diag.bsof_timeline(n, L, 2)
    finally:
        lib.bsofi_device_set_bsof_workers(0)
    for r in (slow, diag.bsof_timeline(n, L, 2)):
        assert r["factor_us"] > 0 and r["update_publish_us"] > 0
        assert r["wait_max_us"] >= r["wait_p90_us"] >= r["wait_p50_us"] >= 0
        parts = r["factor_total_ms"] + r["wait_total_ms"] + r["update_total_ms"]
        assert 0 < parts <= r["chain_ms"]
    assert slow["wait_total_ms"] > r["wait_total_ms"]
    assert slow["wait_total_ms"] > 0.2 * slow["chain_ms"]
