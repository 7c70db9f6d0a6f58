"""The FP64 tensor-core kinetic (boundstate-lanczos_gb300/csrc/bsl_kinetic_tc64.cu)
restated on the CPU: seven 9-bit slices of T and of each plane of v, the classes
k + l <= 6 of their products, and the classes put together in 64-bit integers
and rounded once.  Its error against extended precision must not exceed that of
an FP64 dot product, for planes of every kind of vector the Lanczos loop meets.
"""
import numpy as np
import pytest

S = 7
BIAS = 256 * sum(512 ** k for k in range(S))


def sinc_dvr_t(n, box=0.08):
    d = np.arange(n)[:, None] - np.arange(n)[None, :]
    off = 2.0 / np.where(d == 0, 1, d) ** 2
    dx = box / (n - 1)
    return (0.0635077857002 ** 2 / (2 * 2.01588 * dx * dx)) * np.where(d % 2 == 0, 1.0, -1.0) * np.where(
        d == 0, np.pi ** 2 / 3, off)


def digits(f):
    """Slices (most significant first) of 62-bit fixed-point values."""
    f = [int(x) + BIAS for x in f.ravel()]
    return np.array([[((x >> (9 * k)) & (0x3ff if k == S - 1 else 0x1ff)) - 256 for x in f]
                     for k in range(S - 1, -1, -1)], dtype=np.int64)


def fixed_v(v, e):
    """v 2^(62 - e), truncated towards zero as the kernel's shift does."""
    m, ex = np.frexp(v)
    return np.array([int(np.ldexp(a, 53)) << (b - e + 9) if b - e + 9 >= 0 else
                     (1 if a >= 0 else -1) * (abs(int(np.ldexp(a, 53))) >> -(b - e + 9))
                     for a, b in zip(m.ravel(), ex.ravel().tolist())], dtype=object).reshape(v.shape)


def sliced(T, v):
    """T v of the plane v [q, x] by the kernel's arithmetic."""
    n = len(T)
    et = int(np.frexp(np.abs(T).max())[1])
    e = int(np.frexp(np.abs(v).max())[1])
    b = digits(np.array([int(np.rint(np.longdouble(x) * np.longdouble(2.0) ** (62 - et))) for x in T.ravel()],
                        dtype=object)).reshape(S, n, n)
    a = digits(fixed_v(v, e)).reshape(S, *v.shape)
    assert np.abs(a).max() <= 256 and np.abs(b).max() <= 256
    c = np.zeros((S,) + v.shape, dtype=np.int64)
    for k in range(S):
        for l in range(S - k):
            c[k + l] += b[l] @ a[k]
    f32 = np.float32
    assert np.abs(c[:4]).max() < 2 ** 24
    low = (c[6].astype(f32) * f32(2.0 ** -18) + (c[5].astype(f32) * f32(2.0 ** -9) + c[4].astype(f32)))
    x = (((c[0] * 512 + c[1]) << 18) + (c[2] * 512 + c[3])) * 16384 + np.rint(low * f32(32)).astype(np.int64)
    return np.ldexp(x.astype(np.float64), e + et - 57)


@pytest.mark.parametrize("n", [9, 27, 54, 64])
def test_error_is_not_above_the_fp64_dot_product(n):
    T = sinc_dvr_t(n)
    rng = np.random.default_rng(n)
    g = np.exp(-0.5 * np.linspace(-3, 3, n) ** 2)
    planes = {"normal": rng.standard_normal((n, n)), "uniform": np.full((n, n), 1 / 700.0),
              "gaussian": np.outer(g, g), "decaying": rng.standard_normal((n, n)) * np.outer(g ** 4, g ** 4),
              "one point": np.eye(n)[:, :1] * np.ones((1, n)) * 1e-3, "tiny": rng.standard_normal((n, n)) * 1e-290}
    for name, v in planes.items():
        exact = T.astype(np.longdouble) @ v.astype(np.longdouble)
        plain = np.zeros_like(v)
        for q in range(n):  # serial sums, as a thread of the plain kernel
            plain = plain + T[:, q:q + 1] * v[q:q + 1]
        err = [float(np.sqrt((((x - exact) / np.abs(v).max()) ** 2).mean())) for x in (sliced(T, v), plain)]
        # half an ulp of the result itself is the floor of both
        floor = float(np.sqrt(((exact / np.abs(v).max()) ** 2).mean())) * 2.0 ** -53
        assert err[0] <= max(err[1], floor), (name, err)


@pytest.mark.parametrize("n", [5, 33, 64])
def test_slices_reproduce_t_and_v(n):
    T = sinc_dvr_t(n)
    et = int(np.frexp(T.max())[1])
    b = digits(np.array([int(np.rint(np.longdouble(x) * np.longdouble(2.0) ** (62 - et))) for x in T.ravel()],
                        dtype=object)).reshape(S, n, n)
    for x in b:
        assert np.array_equal(x, x.T)  # a symmetric T stays exactly symmetric
    back = sum(b[l].astype(np.longdouble) * np.longdouble(2.0) ** (et - 8 - 9 * l) for l in range(S))
    assert np.max(np.abs(back - T)) <= np.longdouble(2.0) ** (et - 62)
