"""The digit-plane GEMM behind long FP64 products (7 signed base-256 digits per value, kept
digit products summed exactly, one rounding): an integer restatement on the CPU and the
kernel against it, bit for bit, at the edges of its tiles and chunks; rows out of its range."""
import numpy as np
import pytest

S = 7


def digits(x, E):
    """Digits of x under the row exponent E (biased, as the kernel holds it), by integers."""
    if x == 0.0 or abs(x) < 2.0 ** -1022:
        return [0] * S
    m, e = np.frexp(float(x))
    mant, r = int(abs(m) * 2 ** 53), E - (int(e) + 1022) - 2
    N = mant << -r if r <= 0 else (mant + (1 << (r - 1))) >> r if r < 60 else 0
    N = -N if x < 0 else N
    out = []
    for i in range(S - 1, 0, -1):
        d = ((N + 128) & 255) - 128
        out.append(d)
        N = (N - d) >> 8
    return [N] + out[::-1]


def exponent(v):
    big = np.max(np.maximum(np.abs(v.real), np.abs(v.imag)))
    return 0 if big < 2.0 ** -1022 else int(np.frexp(big)[1]) + 1022


def model_entry(a, b, levels=8):
    """sum_k a_k b_k by the kept digit products, as a correctly rounded complex number."""
    Ea, Eb = exponent(a), exponent(b)
    conv = lambda v, E: np.array([digits(t, E) for t in v], dtype=object)  # noqa: E731
    ar, ai, br, bi = conv(a.real, Ea), conv(a.imag, Ea), conv(b.real, Eb), conv(b.imag, Eb)

    def dot(p, q):
        t = 0
        for i in range(S):
            for j in range(min(S, levels - i)):
                t += int(np.dot(p[:, i], q[:, j])) << (8 * (12 - i - j))
        return t

    def value(t):  # units 2^-(8 * 14) of the scaled rows
        n = abs(t)
        sh = max(0, n.bit_length() - 53)
        half = 1 << (sh - 1) if sh else 0
        q, rem = n >> sh, n & ((1 << sh) - 1) if sh else 0
        q += 1 if sh and (rem > half or (rem == half and q & 1)) else 0
        return (-1 if t < 0 else 1) * np.ldexp(float(q), sh - 112 + Ea + Eb - 2042)
    return complex(value(dot(ar, br) - dot(ai, bi)), value(dot(ar, bi) + dot(ai, br)))


def crandn(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


def bound(A, B):
    """Worst case of the kernel: per real k half a unit 2^-56 of each digit expansion times 1/2
    and the dropped levels (below 2^-63), in units of the scaled rows (a power of two at most 4
    times the row maximum), plus the final rounding."""
    K = A.shape[1]
    ra = np.maximum(np.abs(A.real), np.abs(A.imag)).max(1)[:, None]
    rb = np.maximum(np.abs(B.real), np.abs(B.imag)).max(0)[None, :]
    return 2 * K * 1.02 * 2.0 ** -57 * 16 * ra * rb * np.sqrt(2) + 2.0 ** -52 * np.abs(A @ B)


def test_digits_rebuild_the_value_and_stay_in_range():
    rng = np.random.default_rng(1)
    for x in np.concatenate([rng.standard_normal(300) * 10.0 ** rng.uniform(-9, 0, 300), [1.0, -1.0, 0.0]]):
        E = 1023 + 2
        d = digits(x, E)
        assert max(abs(t) for t in d) <= 128
        got = sum(t * 2 ** (8 * (6 - i)) for i, t in enumerate(d))
        assert abs(got - x * 2.0 ** (56 + 1021 - E)) <= 0.5 + 2.0 ** -20
    worst = (0x7F7F7F7F7F7F7C * 2.0 ** -56)  # every digit near its bound
    assert digits(worst, 1021) == [127] * 6 + [124]
    assert 7 * 128 ** 2 * 128 < 2 ** 24 and 4 * 128 ** 2 * 256 <= 2 ** 24  # exact FP32 chunk sums


def test_model_is_closer_to_the_product_than_its_bound():
    rng = np.random.default_rng(2)
    A, B = crandn(rng, (6, 150)), crandn(rng, (150, 5))
    got = np.array([[model_entry(A[i], B[:, j]) for j in range(5)] for i in range(6)])
    assert np.all(np.abs(got - A @ B) <= bound(A, B) + 150 * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))


def contract(ctx, A, B, prec):
    from grafttn import _lib
    return ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                     _lib.PRECISIONS[prec]))


@pytest.mark.gpu
@pytest.mark.parametrize("mkn", [(1, 65, 1), (127, 71, 31), (128, 72, 32), (129, 73, 33), (300, 64 * 2, 95),
                                 (64, 64 * 3 + 1, 161), (1100, 130, 700), (40, 2000, 64), (5, 15000, 3)])
@pytest.mark.parametrize("prec", ["fp64", "fp64e"])
def test_digit_gemm_matches_the_integer_model(ctx, mkn, prec):
    M, K, N = mkn
    rng = np.random.default_rng(M + K + N)
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    A[M // 2] *= 1e-12
    B[:, N // 2] *= 1e9
    got = contract(ctx, A, B, prec)
    assert np.all(np.abs(got - A @ B) <= bound(A, B) * (300 if prec == "fp64e" else 1)
                  + K * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))
    if prec == "fp64e":  # always the digit planes, 7 levels
        for m, n in {(0, 0), (M - 1, N - 1), (M // 2, N // 2), (M - 1, 0)}:
            assert got[m, n] == model_entry(A[m], B[:, n], 7), (m, n)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [600, 1032])
def test_digit_gemm_is_exact_at_the_largest_digits(ctx, K):
    w = 0x7F7F7F7F7F7F7C * 2.0 ** -56
    A = np.full((640, K), w + 1j * w)
    B = np.full((K, 640), w - 1j * w)
    got = contract(ctx, A, B, "fp64")
    assert np.all(got == model_entry(A[0], B[:, 0]))
    rng = np.random.default_rng(K)
    A, B = crandn(rng, (640, K)), crandn(rng, (K, 640))
    got = contract(ctx, A, B, "fp64")
    for m, n in ((0, 0), (639, 639), (127, 31), (128, 32)):
        assert got[m, n] == model_entry(A[m], B[:, n])


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "fp64e"])
def test_rows_without_digits_take_the_fp64_pipe(ctx, prec):
    rng = np.random.default_rng(5)
    M, K, N = 300, 700, 200
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    plain = contract(ctx, A, B, prec)
    big = A.copy()
    big[3] *= 1e200
    big[4] *= 1e-200
    got = contract(ctx, big, B, prec)
    scale = np.abs(big) @ np.abs(B)
    assert np.all(np.abs(got - big @ B) <= K * 2.0 ** -52 * scale)
    bad = A.copy()
    bad[7, 9] = np.inf
    bad[8, 11] = np.nan
    got = contract(ctx, bad, B, prec)
    rows = [i for i in range(M) if i not in (7, 8)]
    assert not np.isfinite(got[7]).any() and np.isnan(got[8]).all()
    assert np.all(np.abs(got[rows] - plain[rows]) <= K * 2.0 ** -52 * (np.abs(A) @ np.abs(B))[rows] * 2)
    badB = B.copy()
    badB[1, 2] = np.inf
    got = contract(ctx, A, badB, prec)
    assert not np.isfinite(got[:, 2]).any() and np.isfinite(got[:, 3:]).all()
    assert np.array_equal(contract(ctx, A, B, prec), plain)  # nothing of it stays


@pytest.mark.gpu
def test_products_read_in_place_match_numpy(ctx):
    """The FP64 kernel without a K-major copy, over its tile sizes and a strided view."""
    rng = np.random.default_rng(6)
    for (a, b, c, n) in [(2, 70, 3, 5), (9, 80, 7, 40), (30, 66, 11, 31), (60, 65, 20, 30)]:
        T, B = crandn(rng, (a, b, c)), crandn(rng, (n, b))
        got = ctx.download(ctx.contract([ctx.upload(T), ctx.upload(B)], [[-1, 1, -3], [-2, 1]], None, None, 0))
        ref = np.einsum("abc,nb->anc", T, B)
        assert np.all(np.abs(got - ref) <= b * 2.0 ** -51 * np.einsum("abc,nb->anc", np.abs(T), np.abs(B)))


@pytest.mark.gpu
@pytest.mark.parametrize("kn", [(1, 1), (3, 8), (25, 9), (50, 10), (64, 17), (64, 48), (10, 300)])
def test_short_contractions_skip_zeros_exactly(ctx, kn):
    """Short FP64 contractions with a mostly zero static: the sums of numpy, and infinities and
    NaN meet the zeros as 0 * inf and 0 * nan do."""
    K, N = kn
    rng = np.random.default_rng(K * N)
    for M in (1, 31, 700):
        T, B = crandn(rng, (M, K)), crandn(rng, (N, K))
        B[rng.random((N, K)) < 0.8] = 0
        B.real[rng.random((N, K)) < 0.3] = 0
        B.imag[rng.random((N, K)) < 0.3] = 0
        got = contract(ctx, T, np.ascontiguousarray(B.T), "fp64")
        assert np.all(np.abs(got - T @ B.T) <= (K + 1) * 2.0 ** -51 * (np.abs(T) @ np.abs(B.T)))
        T[M // 2, K // 2] = np.inf
        T[0, 0] = np.nan
        got = contract(ctx, T, np.ascontiguousarray(B.T), "fp64")
        assert not np.isfinite(got[M // 2]).any() and np.isnan(got[0]).all()
        ok = [i for i in range(M) if i not in (0, M // 2)]
        assert np.isfinite(got[ok]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("mkn", [(7, 511, 3), (7, 512, 3), (100, 5625, 5), (33, 1025, 47), (250, 640, 60), (1, 9000, 1)])
def test_few_outputs_with_a_long_sum(ctx, mkn):
    """The FP64 product in k slices, with remainders in m, n, k and the slices."""
    M, K, N = mkn
    rng = np.random.default_rng(K)
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    got = contract(ctx, A, B, "fp64")
    assert np.all(np.abs(got - A @ B) <= K * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))
