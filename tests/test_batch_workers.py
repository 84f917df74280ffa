"""BSOF worker counts of the server's requests: host rule, no GPU."""
import pytest

from bsofi_b200 import _lib


@pytest.mark.parametrize("n,workers", [(1, 10), (64, 10), (223, 10), (224, 12), (256, 12),
                                       (257, 24), (576, 24)])
def test_server_request(n, workers):
    """A request alone waits for its chain, which starves with fewer than 12 from n = 224 on."""
    assert _lib.load().bsofi_batch_workers_for(n) == workers


def test_setting_wins():
    lib = _lib.load()
    lib.bsofi_device_set_batch_workers(5)
    try:
        assert [lib.bsofi_batch_workers_for(n) for n in (64, 256, 400)] == [5, 5, 5]
    finally:
        lib.bsofi_device_set_batch_workers(0)
