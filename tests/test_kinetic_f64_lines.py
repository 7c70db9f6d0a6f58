"""The FP64 tensor-core kinetic (boundstate-lanczos_gb300/csrc/bsl_kinetic_tc64.cu)
restated on the CPU: eight 9-bit slices of T and of each line of v that is
contracted, the classes k + l <= 7 of their products, put together as one
integer and rounded once.  Every element of the result is held to the terms of
its own sum, so a line that is small beside the others of its plane keeps its
accuracy.
"""
import numpy as np
import pytest

S = 8
BIAS = 256 * sum(512 ** k for k in range(S))


def sinc_dvr_t(n, box=0.08):
    d = np.arange(n)[:, None] - np.arange(n)[None, :]
    off = 2.0 / np.where(d == 0, 1, d) ** 2
    dx = box / (n - 1)
    return (0.0635077857002 ** 2 / (2 * 2.01588 * dx * dx)) * np.where(d % 2 == 0, 1.0, -1.0) * np.where(
        d == 0, np.pi ** 2 / 3, off)


def exponent(x):
    """e of a line: |x| < 2^e, never below that of the smallest normal number."""
    m = np.max(np.abs(x))
    return max(int(np.frexp(m)[1]), -1021) if m > 0 else -1021


def fixed(x, e):
    """x 2^(71 - e), truncated towards zero."""
    m, ex = np.frexp(x)
    m, sh = int(np.ldexp(m, 53)), int(ex) - 53 + 71 - e
    return m << sh if sh >= 0 else (1 if m >= 0 else -1) * (abs(m) >> -sh)


def digits(f):
    """Slices (the most significant first) of 71-bit fixed-point values."""
    f = [int(x) + BIAS for x in np.ravel(f)]
    return np.array([[((x >> (9 * k)) & (0x3ff if k == S - 1 else 0x1ff)) - 256 for x in f]
                     for k in range(S - 1, -1, -1)], dtype=np.int64)


def t_digits(T):
    e = exponent(T)
    return e, digits([fixed(x, e) for x in T.ravel()]).reshape(S, *T.shape)


def rounded(x, s):
    """x 2^s of an integer x, rounded once to FP64 (Python's int to float rounds to nearest even)."""
    return np.ldexp(float(x), s)


def sliced(T, v):
    """T v of the lines (columns) of v by the kernel's arithmetic."""
    et, b = t_digits(T)
    out = np.empty_like(v)
    for c in range(v.shape[1]):
        e = exponent(v[:, c])
        a = digits([fixed(x, e) for x in v[:, c]])
        assert np.abs(a).max() <= 256
        cls = np.zeros((S, len(T)), dtype=np.int64)
        for k in range(S):
            for l in range(S - k):
                cls[k + l] += b[l] @ a[k]
        assert np.abs(cls[:7]).max() < 2 ** 24
        cls = cls.astype(np.float32).astype(np.int64)  # the accumulators
        out[:, c] = [rounded(sum(int(x) << (9 * (7 - k)) for k, x in enumerate(cls[:, y])), e + et - 79)
                     for y in range(len(T))]
    return out


def scaled_ints(x):
    """x as integers times 2^-1100 (exact)."""
    return np.array([[int(np.ldexp(m, 53)) << (int(e) - 53 + 1200) if m else 0 for m, e in zip(*np.frexp(r))]
                     for r in x], dtype=object)


def planes(n, rng):
    g = np.exp(-0.5 * np.linspace(-3, 3, n) ** 2)
    tail = np.exp(-25.0 * np.linspace(-1, 1, n) ** 2)  # 1e-11 at the edges, 1e-22 in the corners
    two = rng.standard_normal((n, n))
    two[:, ::2] *= 1e-8
    three = rng.standard_normal((n, n))
    three[:, ::3] *= 1e-20
    one = np.zeros((n, n))
    one[rng.integers(0, n, n), np.arange(n)] = rng.standard_normal(n)
    return {"normal": rng.standard_normal((n, n)), "uniform": np.full((n, n), 1 / 700.0), "gaussian": np.outer(g, g),
            "bound state": np.outer(tail, tail), "columns of 1e-8": two, "columns of 1e-20": three,
            "one point": one, "tiny": rng.standard_normal((n, n)) * 1e-290, "huge": rng.standard_normal((n, n)) * 1e300}


@pytest.mark.parametrize("n", [9, 33, 64])
def test_every_element_is_held_to_its_own_sum(n):
    T = sinc_dvr_t(n)
    Ti = scaled_ints(T)
    for name, v in planes(n, np.random.default_rng(n)).items():
        vi = scaled_ints(v)
        exact, terms = Ti.dot(vi), abs(Ti).dot(abs(vi))
        plain = np.zeros_like(v)
        for q in range(n):  # serial sums, as a thread of the plain kernel
            plain = plain + T[:, q:q + 1] * v[q:q + 1]
        rel = []
        for x in (sliced(T, v), plain):
            off = abs(scaled_ints(x) * (1 << 1200) - exact)
            rel.append(np.array([[float((o << 80) // t) * 2.0 ** -80 if t else float(o) for o, t in zip(*r)]
                                 for r in zip(off, terms)]))
            if len(rel) == 1:
                # one rounding of the element, and the slices: the products left out are
                # 2^-69 of max |T| and the line's largest |v| (rms of 448 products of
                # digits of 148 rms, units of 2^-88), eight times that allowed
                scale = abs(Ti).max() * abs(vi).max(axis=0)
                assert all(o << 66 <= (abs(x) << 13) + s for ro, rx in zip(off, exact)
                           for o, x, s in zip(ro, rx, scale)), name
        assert rel[0].max() <= 2.0 * 2.0 ** -53, name
        # on average over the elements no further off than the FP64 sums, or than one rounding
        rms = [float(np.sqrt((r * r).mean())) for r in rel]
        assert rms[0] <= max(rms[1], 2.0 ** -54), (name, rms)


@pytest.mark.parametrize("n", [5, 33, 64])
def test_slices_reproduce_t(n):
    T = sinc_dvr_t(n)
    e, b = t_digits(T)
    for x in b:
        assert np.array_equal(x, x.T)  # a symmetric T stays exactly symmetric
    back = np.array([[sum(int(b[l, i, q]) << (9 * (S - 1 - l)) for l in range(S)) for q in range(n)] for i in range(n)],
                    dtype=object)
    assert all(np.ldexp(float(x), e - 71) == t and int(float(x)) == x for x, t in zip(back.ravel(), T.ravel()))
    # the class sums that have to be exact: no v can take them past 2^24
    assert 256 * int(np.abs(b[:7]).sum(axis=(0, 2)).max()) <= 15 * 2 ** 20
    assert 256 * int(np.abs(b[:2]).sum(axis=(0, 2)).max()) < 4000000
