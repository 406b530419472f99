"""Krylov spaces larger than one launch's shared memory holds coefficients for."""
import numpy as np
import pytest

import models as M
from conftest import make_model

pytestmark = pytest.mark.gpu


def disordered_chain(L, sz2, J, seed):
    """Open XXX chain in random fields: no symmetry but Sz, every level its own."""
    h = np.random.default_rng(seed).uniform(-1.0, 1.0, L)
    return (M.SPIN, L, M.sector(sz2=sz2), M.heisenberg_terms(L, False, J) + [(h[i], [("Sz", i)]) for i in range(L)]), h


def dense(L, sz2, J, h):
    up = (L + sz2) // 2
    states = [s for s in range(1 << L) if bin(s).count("1") == up]
    at = {s: i for i, s in enumerate(states)}
    A = np.zeros((len(states), len(states)))
    for i, s in enumerate(states):
        z = [0.5 if s >> b & 1 else -0.5 for b in range(L)]
        A[i, i] = sum(J * z[b] * z[b + 1] for b in range(L - 1)) + np.dot(h, z)
        for b in range(L - 1):
            if z[b] != z[b + 1]:
                A[at[s ^ (3 << b)], i] += 0.5 * J
    return A


@pytest.mark.parametrize("steps", [1025, 2100])
def test_lanczos_fp64_past_one_launch_of_coefficients(qk, steps):
    """Full reorthogonalisation against more vectors than one launch takes: a vector left out lets
    copies of the converged end of the spectrum grow back."""
    model, h = disordered_chain(14, 2, 1.0, 3)
    H = qk.MatrixFreeHamiltonian(*make_model(qk, *model))
    values, _ = qk.lanczos_ritz_values(H, steps, steps, seed=1, mixed=False)
    want = np.linalg.eigvalsh(dense(14, 2, 1.0, h))
    assert len(values) == steps and H.dimension == len(want) == 3003
    # FP64 Ritz values of the converged ends: thousands of roundings of 2^-53 on numbers up to ||H|| < 16
    np.testing.assert_allclose(values[:40], want[:40], rtol=0, atol=steps * 2.0 ** -53 * 16)
    np.testing.assert_allclose(values[-40:], want[-40:], rtol=0, atol=steps * 2.0 ** -53 * 16)
