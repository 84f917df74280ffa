"""The last sizes that run BSOI by row bands and the first past them.

Bands need one SM each, of at most 64 rows up to n = 112 and 48 above; they end
earlier where tiles are faster.  The launches of the BSOI call tell the route (leaf
factors, Q_k^T and bands; otherwise also a copy before and after the steps).
"""
import numpy as np
import pytest

from bsofi_b200 import api
from gpu_util import block_residual_colmajor, pcyclic_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,most", [(64, None), (65, 9000), (96, 9000), (97, None), (112, None),
                                    (113, 5800), (128, 5800)])
@pytest.mark.parametrize("past", [0, 1])
def test_limit(cuda_device, n, most, past):
    import torch
    if most is None:
        most = 64 * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    L = most // n + past
    N = n * L
    rng = np.random.default_rng(n + past)
    diag = rng.standard_normal((L, n, n)) + np.eye(n)
    sub = rng.standard_normal((L, n, n))
    A = pcyclic_device(torch, diag, sub, N, cuda_device)
    tau = torch.zeros(N, dtype=torch.float64, device=cuda_device)
    ws = torch.empty(api.workspace_bytes(n, L, N), dtype=torch.uint8, device=cuda_device)
    args = (n, L, A.data_ptr(), N, tau.data_ptr(), ws.data_ptr())
    assert api.device_bsoftri(*args) == 0
    assert api.device_bsoi(*args) == 0
    assert (api.last_launches() == 3) == (past == 0)
    torch.cuda.synchronize()
    assert block_residual_colmajor(torch, diag, sub, A, N) < 1e-13
