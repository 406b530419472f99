"""The packed kernels at the sizes and values where they can go wrong: integer sums on extreme
values, both ways to split tiles, block widths and their lanes, one wave of CTAs and more, the
remainders of the 32-byte passes and of the streamed projections."""
import ctypes

import numpy as np
import pytest

import models as M
from conftest import make_model

pytestmark = pytest.mark.gpu


def ham(qk, model):
    return qk.MatrixFreeHamiltonian(*make_model(qk, *model))


def values(kind, n, rng):
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if kind == "spread":  # neighbours up to 2^120 apart, some zero
        x *= 2.0 ** rng.integers(-60, 60, n)
        x[rng.integers(0, n, n // 5)] = 0.0
    elif kind == "tiny":  # near and below the smallest normal number
        x *= 2.0 ** rng.integers(-1080, -1000, n).astype(float)
    elif kind == "huge":
        x *= 2.0 ** 1005
    elif kind == "not finite":
        x[[0, n // 3, n - 1]] = [np.inf, np.nan, complex(0, -np.inf)]
    return x


@pytest.mark.parametrize("kind", ["plain", "spread", "tiny", "huge", "not finite"])
@pytest.mark.parametrize("model", [M.heisenberg(13, True, 1), M.heisenberg(24, True), M.hubbard(8, True, 4, 4)],
                         ids=["ring13", "ring24_whole_tiles", "hubbard8_signs"])
def test_integer_sums_against_the_generic_kernel(qk, model, kind):
    H = ham(qk, model)
    x = values(kind, H.dimension, np.random.default_rng(11))
    y = H.apply(x)
    d = H.diagonal().real
    H.select_kernel(mode=1)
    want = H.apply(x)
    with np.errstate(all="ignore"):
        if kind == "not finite":
            np.testing.assert_array_equal(np.isfinite(y), np.isfinite(want))
            x, y, want = [np.where(np.isfinite(want), a, 0) for a in (np.where(np.isfinite(x), x, 0), y, want)]
    # |H||x| row by row bounds the sums; up to 64 products, each rounded at 2^-53, in either kernel;
    # below the normal numbers one unit of 2^-1074 for each
    a = np.abs(x.real) + np.abs(x.imag)
    s = np.abs(d) * a
    if model[0] == M.HUBBARD:  # signs: neighbours cancel in H |x|, so take the largest
        s = s + 4.0 * model[1] * a.max()
    else:
        s = s + (H.apply(a.astype(np.complex128)).real - d * a)
    assert np.all(np.abs(y - want) <= 64 * 2.0 ** -53 * np.maximum(s, 0) + 128 * 2.0 ** -1074)


BLOCK = {
    "ring12": M.heisenberg(12, True),
    "ring20": M.heisenberg(20, True),  # more than one wave of CTAs at 32 vectors
    "hubbard6": M.hubbard(6, True, 3, 3),
    "field9": (M.SPIN, 9, M.sector(), M.xyz_field_terms(9, True)),
}


@pytest.mark.parametrize("R", [1, 2, 3, 5, 12, 32])
@pytest.mark.parametrize("name", sorted(BLOCK))
def test_block_widths_against_single_vectors(qk, name, R):
    H = ham(qk, BLOCK[name])
    rng = np.random.default_rng(R)
    phi = rng.standard_normal((R, H.dimension)) + 1j * rng.standard_normal((R, H.dimension))
    bound = np.abs(H.diagonal()).max() + 2.0 * BLOCK[name][1]  # of ||H||: a flip of 1 at most on every bond, twice
    for mixed, eps in ((False, 2.0 ** -53), (True, 2.0 ** -24)):
        got, _ = qk.continued_fraction_block(H, list(phi), n_iter=6, mixed=mixed)
        for r in sorted({0, R // 2, R - 1}):
            one = qk.continued_fraction_coeffs(H, phi[r], n_iter=6)
            # six steps of 2^-53 or 2^-24 rounding, each step's error carried on by the next ones
            np.testing.assert_allclose(got[r].alphas[:6], one.alphas[:6], rtol=0, atol=64 * eps * bound)
            np.testing.assert_allclose(got[r].betas[:5], one.betas[:5], rtol=0, atol=64 * eps * bound)


@pytest.mark.parametrize("L", [20, 21])
def test_block_fp64_large_batches(qk, L):
    """32 FP64 vectors on both sides of 2^25 block elements: either engine's first steps are the single vector's."""
    hams = [ham(qk, M.heisenberg(L, True, s)) for s in range(L % 2, L + 1, 2)] * 2
    got = qk.block_lanczos_tridiag(hams, 32, 4, mixed=False, start="philox", seed=5)
    few = qk.block_lanczos_tridiag(hams[:1], 32, 4, mixed=False, start="philox", seed=5)
    for v in (0, 31):
        # four steps of 2^-53 rounding on numbers up to ||H|| <= 0.75 L
        np.testing.assert_allclose(got.alphas[v], few.alphas[v], rtol=0, atol=64 * 2.0 ** -53 * 0.75 * L)
        np.testing.assert_allclose(got.betas[v][:3], few.betas[v][:3], rtol=0, atol=64 * 2.0 ** -53 * 0.75 * L)


# dimensions 4845, 2002, 6435, 3432: every remainder of four, Ritz vectors locked on the way
@pytest.mark.parametrize("L,sz2", [(20, 12), (14, 4), (15, 1), (14, 0)])
def test_lanczos_fp32_remainders(qk, L, sz2):
    H = ham(qk, M.heisenberg(L, True, sz2))
    v0 = np.random.default_rng(L).standard_normal(H.dimension).astype(np.complex128)
    a = qk.lanczos_fixed_steps(H, 80, mixed=True, v0=v0)
    b = qk.lanczos_fixed_steps(H, 80, mixed=False, v0=v0)
    assert abs(a.energy - b.energy) <= 64 * 2.0 ** -24 * 0.75 * L


@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 18) + 255, 300007])
@pytest.mark.parametrize("k,nw", [(1, 3), (15, 3), (16, 4), (17, 4), (33, 3), (5, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_streamed_projections(qk, n, k, nw, shift):
    """Tiles, columns of 16 vectors and their remainders; vectors off the 16-byte grid (shift 1)."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n + k)
    V = [torch.randn(n + 2, dtype=torch.complex64, device="cuda", generator=g)[shift:shift + n] for _ in range(k)]
    W = [torch.randn(n + 2, dtype=torch.complex64, device="cuda", generator=g)[shift:shift + n] for _ in range(nw)]
    ptr = lambda t: (ctypes.c_void_p * len(t))(*[v.data_ptr() for v in t])
    P = np.empty((nw, k), dtype=np.complex128)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = qk.lib().qkrylov_vector_mdot_device_f32(ptr(V), k, ptr(W), nw, n, 2,
                                                 P.view(np.float64).ctypes.data_as(ctypes.POINTER(ctypes.c_double)), stream)
    assert rc == qk.SUCCESS
    for o in range(nw):
        w = W[o].to(torch.complex128)
        for j in range(k):
            v = V[j].to(torch.complex128)
            want = complex(torch.vdot(v, w).cpu())
            # runs of at most 64 products added in FP32, the runs in float pairs
            assert abs(P[o, j] - want) <= 64 * 2.0 ** -24 * float((v.abs() * w.abs()).sum().cpu())


def sparse_values(kind, n, rng):
    x = np.zeros(n, dtype=np.complex128)
    some = rng.integers(0, n, n // 50 + 1)
    if kind == "real":
        x.real = rng.standard_normal(n)
    elif kind == "imaginary":
        x.imag = rng.standard_normal(n)
    elif kind == "unit":
        x[n // 2] = 1.0
    elif kind == "sparse":
        x[some] = rng.standard_normal(len(some)) + 1j * rng.standard_normal(len(some))
    elif kind == "negative zeros":
        x = np.full(n, complex(-0.0, -0.0))
        x[some] = 1.0
    elif kind == "subnormal ones":  # whole rows of one power: 2^-1023, 2^-1043 and 2^-1074 (top bits of the words)
        x.real = rng.standard_normal(n)
        x.imag = np.array([2.0 ** -1023, 2.0 ** -1043, 2.0 ** -1074])[rng.integers(0, 3)] * rng.integers(-1, 2, n)
    elif kind == "subnormal twos":  # two sizes of 2^-1043 and 2^-1023 in one row
        x.real = np.where(rng.integers(0, 2, n) == 1, 2.0 ** -1043, 2.0 ** -1023)
        x.imag = 2.0 ** -1023
    elif kind == "large":
        x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 2.0 ** 1012
    return x


@pytest.mark.parametrize("kind", ["real", "imaginary", "unit", "sparse", "negative zeros", "subnormal ones", "subnormal twos",
                                  "large"])
@pytest.mark.parametrize("model", [M.heisenberg(13, True, 1), M.heisenberg(24, True), M.hubbard(8, True, 4, 4)],
                         ids=["ring13", "ring24_whole_tiles", "hubbard8_signs"])
def test_integer_sums_of_zeros(qk, model, kind):
    H = ham(qk, model)
    x = sparse_values(kind, H.dimension, np.random.default_rng(5))
    y = H.apply(x)
    H.select_kernel(mode=1)
    want = H.apply(x)
    # every row: up to 64 products of numbers up to the largest, each rounded at 2^-53 (or to 2^-1074), in either kernel
    top = 64.0 * max(np.abs(x.real).max(), np.abs(x.imag).max())
    assert np.all(np.abs(y - want) <= 64 * 2.0 ** -53 * top + 128 * 2.0 ** -1074)
    for part, got in ((x.real, y.real), (x.imag, y.imag)):
        if not np.any(part):
            assert not np.any(got)


@pytest.mark.parametrize("kind", ["real", "unit"])
def test_integer_sums_of_zeros_walk_once(qk, kind):
    """A real vector costs an apply what a complex one does (a second walk doubled it)."""
    torch = pytest.importorskip("torch")
    H = ham(qk, M.heisenberg(24, True))
    full = torch.randn(H.dimension, dtype=torch.complex128, device="cuda")
    x = torch.from_numpy(sparse_values(kind, H.dimension, np.random.default_rng(5))).cuda()

    def us(v):
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                H.apply(v)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    us(full)
    assert us(x) <= 1.5 * us(full)


@pytest.mark.parametrize("model", [M.heisenberg(13, True, 1, 1.1 * 2.0 ** -500), M.heisenberg(24, True, 0, 1.1 * 2.0 ** -500),
                                   M.hubbard(8, True, 4, 4, 1.1 * 2.0 ** -500, 2.0 ** -499),
                                   M.heisenberg(13, True, 1, 1.1 * 2.0 ** -950)],
                         ids=["ring13", "ring24_whole_tiles", "hubbard8_signs", "ring13_smaller"])
def test_integer_sums_of_small_couplings(qk, model):
    """Products near the smallest normal number although coupling and vector are far from it."""
    H = ham(qk, model)
    rng = np.random.default_rng(5)
    J = abs(model[3][0][0])
    x = (rng.standard_normal(H.dimension) + 1j * rng.standard_normal(H.dimension)) * (2.0 ** -1000 / J)
    y = H.apply(x)
    H.select_kernel(mode=1)
    want = H.apply(x)
    top = 64.0 * J * max(np.abs(x.real).max(), np.abs(x.imag).max())
    assert top > 0.0
    assert np.all(np.abs(y - want) <= 64 * 2.0 ** -53 * top + 128 * 2.0 ** -1074)
