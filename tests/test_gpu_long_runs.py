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


def test_davidson_fp64_wide_basis(qk):
    """256 states in a basis that grows to 768: residual passes narrower than four pairs.

    Three bonds with hops between strongly staggered sites, eleven sites in weak fields: a seed and its
    corrections stay in a block of eight states that no other seed reaches, so the 768-wide projected
    matrix is three-by-three blocks and its diagonalisation cheap."""
    L, J = 17, (1.0, 0.8, 1.2)
    rng = np.random.default_rng(7)
    h = np.concatenate([np.tile([10.0, -10.0], 3), rng.uniform(-0.5, 0.5, 11)])
    terms = [(h[i], [("Sz", i)]) for i in range(L)]
    for b in range(3):
        terms += [(0.5 * J[b], [("Sp", 2 * b), ("Sm", 2 * b + 1)]), (0.5 * J[b], [("Sm", 2 * b), ("Sp", 2 * b + 1)])]
    H = qk.MatrixFreeHamiltonian(*make_model(qk, M.SPIN, L, M.sector(sz2=-1), terms))
    r = qk.davidson_lowest_ex(H, n_eig=256, max_subspace=768, tol=1e-12, max_iter=3, return_vectors=True)
    assert r.iterations == 3
    # ground states of the three bonds (fields +-10) and the 256 lowest arrangements of the other sites
    from itertools import combinations
    rest = np.sort([h[6:][list(c)].sum() - 0.5 * h[6:].sum() for c in combinations(range(11), 5)])[:256]
    want = rest - sum(0.5 * np.sqrt(20.0 ** 2 + j ** 2) for j in J)
    scale = 64 * 2.0 ** -53 * 34  # roundings of numbers up to ||H||
    assert np.all(np.abs(r.eigenvalues - want) <= r.residuals + scale)
    for k in range(0, 256, 5):  # the residuals are those of the vectors handed back
        v = r.eigenvectors[k]
        assert abs(np.linalg.norm(H.apply(v) - r.eigenvalues[k] * v) - r.residuals[k]) <= scale
    assert r.residuals.min() > 1e-9  # not converged yet: the pass had something to compute
