"""Device calls on a workspace that is 8-byte aligned only.

The interface asks no more of it than its doubles do, so a caller may cut it
from a buffer of its own at any element.  One size for each form of the
kernels that keep state there (Q_k^T formation up to n = 64, 128, 256, 400 and
640); the inverse agrees with numpy's within the forward-error bound.
"""
import numpy as np
import pytest

from bsofi_b200 import api
from bsofi_b200.hubbard import random_pcyclic
from conftest import inverse_tolerance, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(1, 2), (16, 3), (33, 4), (100, 3), (129, 2), (200, 2), (300, 2),
                                 (402, 2)])
@pytest.mark.parametrize("calls", ["two", "one"])
def test_workspace_at_any_double(cuda_device, n, L, calls):
    import torch
    M = random_pcyclic(n, L, seed=3 * n + L)
    N = n * L
    A = torch.from_numpy(np.ascontiguousarray(M.T)).to(cuda_device)
    tau = torch.zeros(N, dtype=torch.float64, device=cuda_device)
    buf = torch.empty(api.workspace_bytes(n, L, N) // 8 + 2, dtype=torch.float64, device=cuda_device)
    assert buf.data_ptr() % 16 == 0
    args = (n, L, A.data_ptr(), N, tau.data_ptr(), buf[1:].data_ptr())
    if calls == "two":
        assert api.device_bsoftri(*args) == 0
        assert api.device_bsoi(*args) == 0
    else:
        assert api.device_invert(*args) == 0
    torch.cuda.synchronize()
    X0 = np.linalg.inv(M)
    assert rel_fro(A.T.cpu().numpy(), X0) < inverse_tolerance(M, X0)
