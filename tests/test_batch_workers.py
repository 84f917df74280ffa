"""BSOF worker counts of batches and of the server's requests: host rules, no GPU."""
import pytest

from bsofi_b200 import _lib


@pytest.mark.parametrize("n,workers", [(1, 10), (64, 10), (223, 10), (224, 12), (256, 12),
                                       (257, 24), (576, 24)])
def test_server_request(n, workers):
    """A request alone waits for its chain, which starves with fewer than 12 from n = 224 on."""
    assert _lib.load().bsofi_batch_workers_for(n) == workers


@pytest.mark.parametrize("count,streams,workers", [
    (9, 8, [8, 8, 8, 16, 16, 24]), (15, 8, [8, 8, 8, 16, 16, 24]), (7, 6, [8, 8, 8, 16, 16, 24]),
    (13, 12, [8, 8, 8, 16, 16, 24]),  # a short queue: the last large instance runs alone
    (16, 8, [8, 10, 10, 10, 10, 24]), (48, 8, [8, 10, 10, 10, 10, 24]),
    (12, 6, [8, 10, 10, 10, 10, 24]), (24, 12, [8, 10, 10, 10, 10, 24]),
    (48, 4, [8, 8, 8, 8, 12, 24]), (41, 5, [8, 8, 8, 8, 12, 24])])
def test_batch_behind_few_streams(count, streams, workers):
    """Instances that queue want SMs for their products: fewer for the chains."""
    lib = _lib.load()
    assert [lib.bsofi_batch_workers(n, count, streams) for n in (143, 144, 179, 180, 256, 257)] == workers


@pytest.mark.parametrize("count,streams,small,large", [(1, 1, 16, 16), (5, 5, 16, 16), (6, 6, 16, 16),
                                                       (8, 8, 12, 16), (12, 12, 8, 16),
                                                       (13, 13, 10, 10), (48, 16, 10, 10),
                                                       (20, 4, 16, 16), (32, 4, 16, 16),
                                                       (40, 2, 16, 16)])
def test_batch_one_stream_an_instance_or_room_for_all(count, streams, small, large):
    lib = _lib.load()
    assert [lib.bsofi_batch_workers(n, count, streams) for n in (64, 179, 180, 256, 257)] == \
        [small, small, large, large, 24]


def test_setting_wins():
    lib = _lib.load()
    lib.bsofi_device_set_batch_workers(5)
    try:
        assert [lib.bsofi_batch_workers_for(n) for n in (64, 256, 400)] == [5, 5, 5]
        assert lib.bsofi_batch_workers(400, 48, 8) == 5
    finally:
        lib.bsofi_device_set_batch_workers(0)
