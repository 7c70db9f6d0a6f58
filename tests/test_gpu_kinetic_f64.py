"""FP64 H v through the tensor-core kinetic, every element held to the terms of
its own three sums, and the lines of an infinity or a NaN.

One function (l = 0) and waters without charges far away: H v is T v.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package
from test_kinetic_f64_lines import sinc_dvr_t

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bsl():
    return load_package()


def bare(bsl, n):
    p = bsl.HvParams()
    p.nx, p.ny, p.nz = p.pnx, p.pny, p.pnz = n
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = 0.08
    p.l_max, p.theta_points, p.phi_points, p.symmetry = 0, 2, 2, bsl.SYM["Even"]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    return bsl.Hamiltonian.from_cage(p, np.array([[1e7, 0.0, 0.0]]), np.zeros((1, 3)), q_site=np.zeros(3),
                                     precision="fp64")


def kinetic_kernel(bsl, h):
    ms, names = (C.c_double * 5)(), (C.c_char_p * 5)()
    f = bsl.lib().bsl_stage_times
    assert f(C.c_void_p(h.handle.value), 1, C.cast(ms, C.POINTER(C.c_double)), C.cast(names, C.c_void_p)) == 0
    return names[0].decode()


def vectors(n, rng):
    x, y, z = (np.linspace(-1, 1, k) for k in n)
    r2 = z[:, None, None] ** 2 + y[:, None] ** 2 + x ** 2
    normal = rng.standard_normal(r2.shape)
    point = np.zeros(r2.shape)
    point[n[2] // 3, n[1] // 2, n[0] - 1] = 1.0 / 3.0
    columns, rows, planes = normal.copy(), normal.copy(), normal.copy()
    columns[:, :, ::2] *= 1e-20
    rows[:, 1::3] *= 1e-8
    planes[::4] *= 1e-30
    planes[:, :, 1] *= 1e-12
    return {"normal": normal, "bound state": np.exp(-25.0 * r2), "one point": point, "columns": columns, "rows": rows,
            "planes": planes, "tiny": 1e-290 * normal, "subnormal": 1e-310 * normal, "huge": 1e299 * normal}


# a last pair of one plane, 16-row steps with 1, 5 and 16 rows, all 64 points
@pytest.mark.parametrize("n", [(57, 57, 57), (64, 64, 47), (53, 53, 64), (64, 64, 64)])
def test_every_element_is_held_to_its_own_sums(bsl, n):
    h = bare(bsl, n)
    try:
        assert kinetic_kernel(bsl, h) == "k_kin_xy_tc64"
        rng = np.random.default_rng(n[0])
        t = [sinc_dvr_t(k).astype(np.longdouble) for k in n]
        i = np.stack([rng.integers(0, k, 3000) for k in n], 1)
        i[:8] = np.array(np.meshgrid(*[(0, k - 1) for k in n])).reshape(3, -1).T  # the corners
        i[8:72, 0], i[8:72, 1:] = np.arange(64) % n[0], (n[1] // 2, n[2] // 3)
        x, y, z = i.T
        for name, v in vectors(n, rng).items():
            u = np.zeros(v.size)
            h.hv(v.ravel(), u)
            u = u.reshape(v.shape)
            w = v.astype(np.longdouble)
            parts = [t[0][x] * w[z, y, :], t[1][y] * w[z, :, x], t[2][z] * w[:, y, x].T]
            exact, terms = sum(p.sum(1) for p in parts), sum(np.abs(p).sum(1) for p in parts)
            # roundings of the three sums and of the two additions, at most 3 x 2^-53 of the
            # terms; the slices, 2^-66 of max |T| and a line's largest |v|, of which the
            # terms are at least 2^-12.7; one more for the potential's sum
            off = np.abs(u[z, y, x] - exact)
            assert np.all(off <= 5 * 2.0 ** -53 * terms + 8 * 2.0 ** -1074), (name, float(np.max(off / terms) * 2 ** 53))
    finally:
        h.close()


def test_an_infinity_reaches_its_own_lines_only(bsl):
    n = (57, 57, 57)
    h = bare(bsl, n)
    try:
        for bad in (np.inf, -np.inf, np.nan):
            v = np.ones(n[::-1])
            v[11, 7, 5] = bad
            u = np.zeros(v.size)
            h.hv(v.ravel(), u)
            u = u.reshape(v.shape)
            lines = np.zeros(v.shape, dtype=bool)
            lines[11, 7], lines[11, :, 5], lines[:, 7, 5] = True, True, True
            assert np.array_equal(np.isfinite(u), ~lines)
            if not np.isnan(bad):  # T bad has the sign of T; the point itself has -V bad too
                want = np.where(np.arange(57) % 2 == 1, bad, -bad)
                for line, at in ((u[11, 7], 5), (u[11, :, 5], 7), (u[:, 7, 5], 11)):
                    assert np.array_equal(np.delete(line, at), np.delete(want, at))
        v = np.zeros(n[::-1])
        u = np.zeros(v.size)
        h.hv(v.ravel(), u)
        assert np.all(u == 0.0)
    finally:
        h.close()


def check(bsl, h, n, engine, kernel, v):
    """RMS of H v's error over the terms of its sums; each within n roundings of them."""
    h.set_kinetic_engine(engine)
    assert kinetic_kernel(bsl, h) == kernel
    t = [sinc_dvr_t(k).astype(np.longdouble) for k in n]
    i = np.random.default_rng(2).integers(0, n, (4000, 3))
    x, y, z = i.T
    w = v.astype(np.longdouble)
    parts = [t[0][x] * w[z, y, :], t[1][y] * w[z, :, x], t[2][z] * w[:, y, x].T]
    exact, terms = sum(p.sum(1) for p in parts), sum(np.abs(p).sum(1) for p in parts)
    u = np.zeros(v.size)
    h.hv(v.ravel(), u)
    off = np.abs(u.reshape(v.shape)[z, y, x] - exact) / terms
    assert np.max(off) <= sum(n) * 2.0 ** -53
    return float(np.sqrt(np.mean(off ** 2)))


def test_the_cuda_core_engine_selects_the_plain_sums(bsl):
    """In FP64 as well: the same H v from one kernel and the other, and the tensor
    cores' no further off on average, element by element."""
    n = (57, 57, 57)
    h = bare(bsl, n)
    try:
        v = vectors(n, np.random.default_rng(1))["bound state"]
        rms = [check(bsl, h, n, *e, v) for e in (("simt", "k_kin_f64<x,y>"), ("tensor", "k_kin_xy_tc64"))]
        assert rms[1] <= rms[0], rms
    finally:
        h.close()


# planes of 1,190 and of 1,225 points (fewer CTAs than SMs), of 1,980 (160 CTAs), 2,025
# and 4,096 points; 65 points on an axis
@pytest.mark.parametrize("n,kernel", [((34, 35, 5), "k_kin_f64"), ((35, 35, 7), "k_kin_f64<x,y>"),
                                      ((45, 44, 160), "k_kin_f64"), ((45, 45, 160), "k_kin_f64<x,y>"),
                                      ((64, 64, 2), "k_kin_f64<x,y>"), ((9, 65, 3), "k_kin_f64"), ((2, 2, 65), "k_kin_f64")])
def test_plain_sums_in_one_launch_and_in_two(bsl, n, kernel):
    h = bare(bsl, n)
    try:
        check(bsl, h, n, "simt", kernel, np.random.default_rng(4).standard_normal(n[::-1]))
    finally:
        h.close()
