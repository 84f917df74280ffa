"""The band kernels of small blocks (BSOI by row bands, BSTRI's recurrence by
column bands) against the launch plans they replace, over every form of input
that both take: odd block sizes, leading dimensions and addresses that break
16-byte alignment, one and several band heights, the first and last sizes of
the rule.

The two routes compute the same products in another order, so the inverses
agree within the forward-error bound of the parity tests; tau and the
factorization are the same kernel's and must be equal.
"""
import numpy as np
import pytest

from bsofi_b200 import api
from bsofi_b200.hubbard import pcyclic_blocks, random_pcyclic
from conftest import inverse_tolerance, rel_fro
from gpu_util import block_residual_colmajor, pcyclic_device

pytestmark = pytest.mark.gpu

# A plan whose two knobs differ from every default of n <= 128.
OTHER_FORMS = [2, 0, 32, 0]


@pytest.fixture(autouse=True)
def _clear_plans():
    api.plan_clear()
    yield
    api.plan_clear()


def _invert(torch, M, n, L, ldd, off, dev):
    N = n * L
    buf = torch.full((N * ldd + 1,), float("nan"), dtype=torch.float64, device=dev)
    A = buf[off:off + N * ldd].view(N, ldd)
    A[:, :N] = torch.from_numpy(np.ascontiguousarray(M.T)).to(dev)
    tau = torch.zeros(N, dtype=torch.float64, device=dev)
    ws = torch.empty(api.workspace_bytes(n, L, ldd), dtype=torch.uint8, device=dev)
    assert api.device_invert(n, L, A.data_ptr(), ldd, tau.data_ptr(), ws.data_ptr()) == 0
    torch.cuda.synchronize()
    return A[:, :N].T.cpu().numpy(), tau.cpu().numpy()


@pytest.mark.parametrize("n,L", [(1, 2), (2, 3), (7, 40), (8, 2), (16, 8), (31, 17), (33, 40),
                                 (64, 3), (64, 20), (65, 12), (100, 21), (127, 5), (128, 14),
                                 (129, 6)])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (2, 1)])
def test_bands_match_the_other_forms(cuda_device, n, L, pad, off):
    import torch
    M = random_pcyclic(n, L, seed=11 * n + L)
    ldd = n * L + pad
    X, tau = _invert(torch, M, n, L, ldd, off, cuda_device)
    assert api.plan_set(n, L, OTHER_FORMS) == 0
    X0, tau0 = _invert(torch, M, n, L, ldd, off, cuda_device)
    np.testing.assert_array_equal(tau, tau0)
    assert rel_fro(X, X0) < inverse_tolerance(M, X0)


@pytest.mark.parametrize("n,L", [(64, 148), (64, 149), (128, 74), (100, 94)])
def test_largest_sizes_of_the_rule(cuda_device, n, L):
    """One band of up to 64 rows per SM of a B200 (N = 9472), and just past it."""
    import torch
    M = random_pcyclic(n, L, seed=n + L)
    diag, sub = pcyclic_blocks(M, n, L)
    N = n * L
    A = pcyclic_device(torch, diag, sub, N, cuda_device)
    tau = torch.zeros(N, dtype=torch.float64, device=cuda_device)
    ws = torch.empty(api.workspace_bytes(n, L, N), dtype=torch.uint8, device=cuda_device)
    assert api.device_invert(n, L, A.data_ptr(), N, tau.data_ptr(), ws.data_ptr()) == 0
    torch.cuda.synchronize()
    assert block_residual_colmajor(torch, diag, sub, A, N) < 1e-13
