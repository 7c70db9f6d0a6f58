"""Kernels that take one another's place by size and are said to give the same
bits: a grid just below a limit against the same grid with a few planes of
zeros at its end, which is above it.  The spacing is a power of two, so the
kinetic matrices agree, and the potential is zero or one constant everywhere.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
BASES = {9: (2, "All"), 10: (3, "Odd"), 15: (4, "Even"), 16: (3, "All"), 21: (5, "Odd"), 25: (4, "All"),
         28: (6, "Even"), 36: (5, "All")}


@pytest.fixture(scope="module")
def bsl():
    return load_package()


def hamiltonian(bsl, n, nn, precision, water, spacing=1.0 / 1024):
    p = bsl.HvParams()
    p.nx, p.ny, p.nz = p.pnx, p.pny, p.pnz = n
    p.x_max, p.y_max, p.z_max = p.px_max, p.py_max, p.pz_max = [(k - 1) * spacing for k in n]
    p.l_max, p.theta_points, p.phi_points = BASES[nn][0], 4, 3
    p.symmetry = bsl.SYM[BASES[nn][1]]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    return bsl.Hamiltonian.from_cage(p, np.array([water]), np.zeros((1, 3)), q_site=np.zeros(3), precision=precision)


def kinetic_kernel(bsl, h):
    ms, names = (C.c_double * 5)(), (C.c_char_p * 5)()
    f = bsl.lib().bsl_stage_times
    assert f(C.c_void_p(h.handle.value), 1, C.cast(ms, C.POINTER(C.c_double)), C.cast(names, C.c_void_p)) == 0
    return names[0].decode()


def h_v(bsl, n, nn, precision, water, v, engine=None):
    """H v of v (its planes of z, and zeros in the rest of the grid) and the kinetic's kernel."""
    h = hamiltonian(bsl, n, nn, precision, water)
    try:
        if engine:
            h.set_kinetic_engine(engine)
        full = np.zeros((h.basis_size // (n[0] * n[1] * n[2]), n[2], n[1], n[0]))
        full[:, :v.shape[1]] = v
        u = np.zeros(h.basis_size)
        h.hv(full.ravel(), u)
        return u.reshape(full.shape)[:, :v.shape[1]], kinetic_kernel(bsl, h)
    finally:
        h.close()


def full_functions(nn):
    return (BASES[nn][0] + 1) ** 2


FAR = [1e12, 0.0, 0.0]  # V below the smallest FP32 number
NEAR = [0.013, 0.007, 0.011]  # an oxygen inside the box: V at its ceiling at every point


@pytest.mark.parametrize("n,nn", [(16, 15), (16, 21), (16, 16), (16, 9), (11, 28), (6, 10), (13, 36)])
def test_small_grid_kinetic_is_the_tensor_core_kinetic(bsl, n, nn):
    v = np.random.default_rng(nn).standard_normal((full_functions(nn), 16, n, n))
    small = h_v(bsl, (n, n, 16), nn, "mixed", FAR, v)
    large = h_v(bsl, (n, n, 17), nn, "mixed", FAR, v)
    assert small[1] == "k_kin_small" and large[1] in ("k_kin_xyz_tc", "k_kin_xy_tc")
    assert np.array_equal(small[0], large[0]) and np.any(small[0] != 0.0)


@pytest.mark.parametrize("n,nz,more,nn", [(33, 33, 3, 21), (40, 37, 1, 10), (33, 36, 1, 15), (41, 28, 3, 16)])
def test_one_launch_kinetic_is_the_two_launch_kinetic(bsl, n, nz, more, nn):
    v = np.random.default_rng(nn).standard_normal((full_functions(nn), nz, n, n))
    one = h_v(bsl, (n, n, nz), nn, "mixed", FAR, v)
    two = h_v(bsl, (n, n, nz + more), nn, "mixed", FAR, v)
    assert (one[1], two[1]) == ("k_kin_xyz_tc", "k_kin_xy_tc")
    assert np.array_equal(one[0], two[0]) and np.any(one[0] != 0.0)


@pytest.mark.parametrize("nn", sorted(BASES))
def test_block_product_by_rows_is_the_block_product_by_points(bsl, nn):
    """FP64, 25,230 points against 26,912: rows split over warps against a thread a point."""
    v = np.random.default_rng(nn).standard_normal((full_functions(nn), 30, 29, 29))
    rows = h_v(bsl, (29, 29, 30), nn, "fp64", NEAR, v, "simt")
    points = h_v(bsl, (29, 29, 32), nn, "fp64", NEAR, v, "simt")
    assert rows[1] == points[1] == "k_kin_f64"
    assert np.array_equal(rows[0], points[0])
    # the blocks are dense: the coarse quadrature does not keep the functions apart
    assert np.any(rows[0] != h_v(bsl, (29, 29, 30), nn, "fp64", FAR, v, "simt")[0])


@pytest.mark.parametrize("n,more,nn", [((34, 35, 7), 1, 21), ((34, 35, 16), 2, 9)])
def test_plain_kinetic_in_one_launch_is_the_one_in_two(bsl, n, more, nn):
    """The x/y planes of a one-launch grid with a row and a column of zeros more are
    past 1,200 points and take two launches (fewer planes than SMs)."""
    v = np.random.default_rng(nn).standard_normal((full_functions(nn), n[2], n[1], n[0]))
    one = h_v(bsl, n, nn, "fp64", FAR, v, "simt")
    wide = np.zeros(v.shape[:2] + (n[1] + more, n[0] + more))
    wide[:, :, :n[1], :n[0]] = v
    two = h_v(bsl, (n[0] + more, n[1] + more, n[2]), nn, "fp64", FAR, wide, "simt")
    assert (one[1], two[1]) == ("k_kin_f64", "k_kin_f64<x,y>")
    assert np.array_equal(one[0], two[0][:, :, :n[1], :n[0]])
