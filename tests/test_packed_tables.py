"""The packed SpMV's tables against the oracle, on the CPU.

The packed kernel applies H in the reference's order from tables built on the
host (16-bit ranks of merged terms, per-block offsets, straddling tables); the
test walks those tables on the host as the kernel does, every index checked, and
compares with the oracle's rows over the forms a sector and an OpSum can take:
every basis, odd lengths, one block and several, partial last tiles, signs,
complex and many amplitudes, terms that need conditions or leave the sector."""
import ctypes

import numpy as np
import pytest

import models as M
from models import make_model
from oracle_ctypes import OHam, Oracle, available

UNIFORM, SIGNED, CODED, EQUAL, COMPLEX = 0, 1, 2, 4, 8


def packed_apply(qk, model, x):
    basis, site, ops = make_model(qk, *model)
    y = np.full(x.size, np.nan, dtype=np.complex128)
    form = ctypes.c_int()
    dp = lambda a: a.view(np.float64).ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    rc = qk.lib().qkrylov_debug_packed_apply_host(basis._h, site._h, ops._h, dp(x), dp(y), ctypes.byref(form))
    assert rc == qk.SUCCESS, qk.lib().qkrylov_last_error()
    return y, form.value


def random_terms(model, L, seed, count=30):
    """Terms of one to four factors at any sites: long flips, parity strings, conditions, complex amplitudes."""
    rng = np.random.default_rng(seed)
    ops = {M.SPIN: ["Sz", "Sp", "Sm", "Sx", "Sy"], M.FERMION: ["N", "C", "Cdag"],
           M.HUBBARD: ["Nup", "Ndn", "Nupdn", "CUp", "CdagUp", "CDn", "CdagDn"]}[model]
    return [(complex(*rng.normal(size=2)),
             [(ops[rng.integers(len(ops))], int(rng.integers(L))) for _ in range(rng.integers(1, 5))]) for _ in range(count)]


def disordered(L):
    rng = np.random.default_rng(L)
    return [t for i in range(L) for j in range(i) for t in
            ((0.5 * c, [("Sp", i), ("Sm", j)]) for c in [rng.choice([0.7, 1.3, -0.4])])] + [
            t for i in range(L) for j in range(i) for t in [(0.5, [("Sm", i), ("Sp", j)])]]


CASES = {
    "ring2": (M.heisenberg(2, True), UNIFORM | EQUAL),
    "ring4": (M.heisenberg(4, True), UNIFORM | EQUAL),
    "chain9": ((M.SPIN, 9, M.sector(sz2=1), M.heisenberg_terms(9, False)), UNIFORM | EQUAL),
    "ring14_one_block": (M.heisenberg(14, True), UNIFORM | EQUAL),
    "ring16": (M.heisenberg(16, True), UNIFORM | EQUAL),
    "ring17_sz": ((M.SPIN, 17, M.sector(sz2=-3), M.heisenberg_terms(17, True)), UNIFORM | EQUAL),
    "chain18_xxz": ((M.SPIN, 18, M.sector(sz2=2), M.heisenberg_terms(18, False, Jz=0.7)), UNIFORM | EQUAL),
    "ring16_dilute": ((M.SPIN, 16, M.sector(sz2=12), M.heisenberg_terms(16, True)), UNIFORM | EQUAL),
    "polarised": ((M.SPIN, 12, M.sector(sz2=12), M.heisenberg_terms(12, True)), UNIFORM | EQUAL),
    "full_space": ((M.SPIN, 13, M.sector(), M.heisenberg_terms(13, True)), UNIFORM | EQUAL),
    "field": ((M.SPIN, 13, M.sector(), M.xyz_field_terms(13, True)), CODED | COMPLEX),
    "two_couplings": ((M.SPIN, 16, M.sector(sz2=0), M.heisenberg_terms(16, True) + [
        (0.2, [("Sp", i), ("Sm", (i + 2) % 16)]) for i in range(16)] + [
        (0.2, [("Sm", i), ("Sp", (i + 2) % 16)]) for i in range(16)]), CODED),
    "all_pairs": ((M.SPIN, 15, M.sector(sz2=1), disordered(15)), CODED),
    "fermions": ((M.FERMION, 16, M.sector(n=6), M.fermion_chain_terms(16, True)), None),
    "fermions_open": ((M.FERMION, 17, M.sector(n=8), M.fermion_chain_terms(17, False)), UNIFORM | EQUAL),
    "fermions_full": ((M.FERMION, 13, M.sector(), M.fermion_chain_terms(13, True)), None),
    "hubbard7": (M.hubbard(7, True, 3, 4), SIGNED | EQUAL),
    "hubbard8": (M.hubbard(8, True, 4, 4), SIGNED | EQUAL),
    "hubbard_one_species": ((M.HUBBARD, 7, M.sector(nup=3), M.hubbard_terms(7, True)), SIGNED | EQUAL),
    "hubbard_full": ((M.HUBBARD, 6, M.sector(), M.hubbard_terms(6, True)), SIGNED | EQUAL),
    "hubbard1": ((M.HUBBARD, 1, M.sector(nup=1, ndn=0), [(1.0, [("Nup", 0)])]), UNIFORM | EQUAL),
    "hopping_signs": ((M.SPIN, 16, M.sector(sz2=0), [(0.5 * (-1) ** i, [(a, i), (b, (i + 1) % 16)]) for i in range(16)
                                                     for a, b in (("Sp", "Sm"), ("Sm", "Sp"))]), SIGNED | EQUAL),
}
for _s in range(4):
    CASES["random_spin%d" % _s] = ((M.SPIN, 13 + _s % 2, M.sector(sz2=[None, 2, 1, -2][_s]),
                                    random_terms(M.SPIN, 13 + _s % 2, _s)), None)
    CASES["random_fermion%d" % _s] = ((M.FERMION, 14, M.sector(n=6) if _s % 2 else M.sector(),
                                       random_terms(M.FERMION, 14, _s)), None)
    CASES["random_hubbard%d" % _s] = ((M.HUBBARD, 7, [M.sector(), M.sector(nup=3, ndn=2), M.sector(ndn=4), M.sector(nup=7, ndn=0)][_s],
                                       random_terms(M.HUBBARD, 7, _s)), None)


@pytest.mark.parametrize("name", sorted(CASES))
def test_tables_against_oracle(qk, name):
    if not available("qko"):
        pytest.skip("the oracle is not built")
    model, form = CASES[name]
    o = OHam(Oracle("qko"), *model)
    rng = np.random.default_rng(3)
    x = rng.normal(size=o.dim) + 1j * rng.normal(size=o.dim)
    want = o.apply(x) - o.diagonal() * x
    got, f = packed_apply(qk, model, x)
    assert f >= 0 and (form is None or f == form), f
    # two sums of the same <= 64 products, each rounded at 2^-53
    scale = max(1.0, max(abs(t[0]) for t in model[3])) * len(model[3]) * np.abs(x).max()
    np.testing.assert_allclose(got, want, rtol=0, atol=64 * 2.0 ** -53 * scale)


def test_plan_declines(qk):
    """Ranks by search (t-J), states over 32 bits and more amplitudes than codes stay on the other kernels."""
    x = np.zeros(40, dtype=np.complex128)
    assert packed_apply(qk, (M.TJ, 4, M.sector(nup=1, ndn=1), M.tj_terms(4, True)), x[:12])[1] == -1
    assert packed_apply(qk, (M.SPIN, 40, M.sector(sz2=38), M.heisenberg_terms(40, True)), x)[1] == -1
    many = [(1.0 + 0.001 * (i * 18 + j), [("Sp", i), ("Sm", j)]) for i in range(18) for j in range(18) if i != j]
    assert packed_apply(qk, (M.SPIN, 18, M.sector(sz2=16), many), x[:18])[1] == -1


@pytest.mark.parametrize("J", [np.inf, np.nan, 1e39])
def test_plan_declines_amplitudes_that_are_not_finite(qk, J):
    """Empty slots are products with zero, also where the amplitude overflows FP32 only."""
    import math
    for L, n in ((9, 4), (16, 8)):  # one block; outer and straddling entries too
        terms = [(J if i == L - 2 else 1.0, [(a, i), (b, i + 1)]) for i in range(L - 1) for a, b in (("Sp", "Sm"), ("Sm", "Sp"))]
        x = np.zeros(math.comb(L, n), dtype=np.complex128)
        assert packed_apply(qk, (M.SPIN, L, M.sector(sz2=2 * n - L), terms), x)[1] == -1
    terms = [(1e38, t) for _, t in M.heisenberg_terms(9, True) if t[0][0] != "Sz"]
    assert packed_apply(qk, (M.SPIN, 9, M.sector(sz2=1), terms), np.zeros(126, dtype=np.complex128))[1] >= 0
