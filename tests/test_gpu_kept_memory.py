"""Device memory that Hamiltonians keep between solver calls."""
import numpy as np
import pytest

import models as M
from conftest import make_model

pytestmark = pytest.mark.gpu

GB2 = 2 << 30


def ham(qk, model):
    return qk.MatrixFreeHamiltonian(*make_model(qk, *model))


def test_fp64_vectors_kept_by_several_hamiltonians(qk):
    """Three runs of 1.1 GB of vectors each, as in a scan that keeps its Hamiltonians: 2 GB are kept over all."""
    hams = [ham(qk, M.heisenberg(22, True, 0, J)) for J in (1.0, 1.1, 1.2)]
    energies = []
    for H in hams:
        energies.append(qk.lanczos_fixed_steps(H, 100, mixed=False).energy)
    assert sum(H.workspace_bytes() for H in hams) <= GB2
    np.testing.assert_allclose(energies, np.array([1.0, 1.1, 1.2]) * energies[0], rtol=1e-6)
    # with the room taken, the others' runs still work, and a release makes room
    v0 = np.ones(hams[2].dimension, dtype=complex)
    v0[0] = 2.0
    qk.continued_fraction_coeffs(hams[2], v0, n_iter=5)
    qk.davidson_lowest_ex(hams[2], n_eig=1, max_subspace=8, max_iter=3)
    assert sum(H.workspace_bytes() for H in hams) <= GB2
    hams[0].workspace_bytes(release=True)
    qk.lanczos_fixed_steps(hams[2], 10, mixed=False)
    kept = hams[2].workspace_bytes()
    assert kept > 0 and kept + hams[1].workspace_bytes() <= GB2
    # a destroyed Hamiltonian's share is free again
    del hams[:2]
    import gc
    gc.collect()
    qk.lanczos_fixed_steps(hams[0], 100, mixed=False)
    assert 100 * hams[0].dimension * 16 <= hams[0].workspace_bytes() <= GB2


def test_three_term_recurrence_keeps_its_few_vectors(qk):
    H = ham(qk, M.heisenberg(16, True))
    v0 = np.random.default_rng(1).standard_normal(H.dimension).astype(complex)
    qk.continued_fraction_coeffs(H, v0, n_iter=20)
    assert 0 < H.workspace_bytes() <= 4 * (16 * H.dimension + 256)


def test_contiguous_workspace_takes_the_place_of_fp64_vectors(qk):
    """The mixed Lanczos and a batch allocate one block; the FP64 vectors kept before it, although larger, go first."""
    H = ham(qk, M.heisenberg(16, True))
    vector = 8 * H.dimension + 256
    qk.lanczos_fixed_steps(H, 80, mixed=False)
    assert H.workspace_bytes() > 80 * 2 * vector
    qk.lanczos_fixed_steps(H, 20, mixed=True)
    assert 20 * (vector - 256) < H.workspace_bytes() <= (20 + 16) * vector
    H.workspace_bytes(release=True)
    qk.lanczos_fixed_steps(H, 80, mixed=False)
    qk.block_lanczos_tridiag([H], 4, 5, mixed=True, start="philox", seed=1)
    # three block vectors of four, and under 2 MB of tables and partial sums
    assert 12 * (vector - 256) < H.workspace_bytes() <= 12 * vector + (2 << 20)
