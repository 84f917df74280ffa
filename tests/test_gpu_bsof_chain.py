"""The BSOF chain kernel at the sizes where it changes form: widest panels of
each configuration and one past it, ragged last leaves, two and three block
rows, columns with nothing to eliminate, and norms outside the range of the
fast reflector arithmetic.

Reference: the oracle's factorization (LAPACK's reflectors and tau are unique).
Tolerances as in test_gpu_parity.py; at a power-of-two scale every quantity
is the unscaled one times a power of two but for roundings, so tau is held to
the same 1e-12.
"""
import numpy as np
import pytest

import oracle
from bsofi_b200 import api
from bsofi_b200.hubbard import assemble_pcyclic, random_pcyclic
from conftest import inverse_tolerance, rel_fro, split_state

pytestmark = pytest.mark.gpu

# (n, L): 64 / 128 / 256 / 416 / 592 / 640 are the largest blocks of the kernel's
# forms; leaves of 16 (8 above 256) columns end evenly, one short and one over;
# odd n with an odd number of blocks has columns of both alignments.
SIZES = [(1, 2), (15, 3), (16, 2), (17, 5), (32, 3), (63, 3), (64, 4), (65, 3), (127, 2), (128, 3),
         (129, 2), (129, 3), (136, 3), (255, 2), (256, 2), (257, 2), (257, 3), (392, 2), (400, 2),
         (401, 2), (401, 3), (416, 2), (417, 2), (592, 2), (593, 3), (640, 2), (641, 2)]


@pytest.mark.parametrize("n,L", SIZES)
def test_chain_vs_oracle(cuda_device, n, L):
    M = random_pcyclic(n, L, seed=7 * n + L)
    A_ref, tau_ref, _ = oracle.port_bsoftri(M, n, L)
    X, state, tau, info = api.invert(M, n, L)
    assert info == 0
    np.testing.assert_allclose(tau, tau_ref, rtol=0, atol=1e-12)
    refl, refl_ref = split_state(state, n, L)[1], split_state(A_ref, n, L)[1]
    np.testing.assert_allclose(refl, refl_ref, rtol=0, atol=1e-10)
    X_ref, _ = oracle.port_bsoi(A_ref, tau_ref, n, L)
    assert rel_fro(X, X_ref) < inverse_tolerance(M, X_ref)


@pytest.mark.parametrize("n,L", [(24, 3), (130, 2)])
def test_nothing_to_eliminate(cuda_device, n, L):
    """Zero coupling blocks under upper triangular diagonal blocks: every
    reflector is the identity (tau = 0, R's diagonal keeps its sign)."""
    rng = np.random.default_rng(n)
    diag = np.triu(rng.standard_normal((L, n, n)), 1)
    diag += np.einsum("k,ij->kij", np.array([-2.0, 3.0, 5.0])[:L], np.eye(n))
    M = assemble_pcyclic(diag, np.zeros((L, n, n)))
    X, state, tau, info = api.invert(M, n, L)
    assert info == 0
    np.testing.assert_array_equal(tau, 0.0)
    assert rel_fro(X, np.linalg.inv(M)) < inverse_tolerance(M, np.linalg.inv(M))


@pytest.mark.parametrize("n,L", [(20, 3), (96, 2), (260, 2)])
@pytest.mark.parametrize("e", [-490, 480])
def test_scaled_input(cuda_device, n, L, e):
    """Squared norms near 2^-970 and 2^+970: outside the fast range, inside
    the doubles."""
    M = random_pcyclic(n, L, seed=n + L)
    X, _, tau, info = api.invert(M, n, L)
    Xs, _, taus, infos = api.invert(np.ldexp(M, e), n, L)
    assert info == 0 and infos == 0
    np.testing.assert_allclose(taus, tau, rtol=0, atol=1e-12)
    assert rel_fro(np.ldexp(Xs, e), X) < inverse_tolerance(M, X)
