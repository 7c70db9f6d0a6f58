"""The size-dependent kernels of H v and of the Lanczos iteration against the
oracle and against one another, at the edges of their ranges.

FP64: the kinetic on the tensor cores from 1.6e7 multiply-adds on, the block
product split over rows up to 26,000 points.  Mixed: the kinetic in one launch
up to 16 points per axis, the same bits as the tensor-core kernels'.
"""
import os

import numpy as np
import pytest

from conftest import OracleModel, load_inputs, load_package

pytestmark = pytest.mark.gpu
CALC = "linRotCartSph_NoQuad_ContGrid_Alavi_SPCE"


@pytest.fixture(scope="module")
def bsl():
    return load_package()


def write_case(tmp, n, l_max, sym):
    """An HvInputFile for a box of n = (nx, ny, nz) points and the generated cage."""
    inp = load_inputs()
    cage = os.path.join(tmp, "cage.xyz")
    inp.write_cage_xyz(cage, inp.dodecahedral_cage(1))
    v = inp.hv_fields(n[0], 0.08, l_max, 6, 5, cage, "paths", sym)
    v[2], v[4], v[11], v[13] = n[1], n[2], n[1], n[2]
    hv = os.path.join(tmp, "hv_input.txt")
    inp.write_hv_input(hv, v)
    return hv


# kinetic: plain just below 1.6e7 (23^3 at 15 functions), tensor cores above it, an
# odd number of planes, a last pair of one plane, 16-row steps with 1 and 16 rows,
# 64 points; block product: 26,000 points from below and above, a last warp of
# one point, blocks with and without the row split
@pytest.mark.parametrize("n,l_max,sym", [
    ((23, 23, 23), 4, "Even"), ((25, 25, 23), 5, "Odd"), ((17, 17, 64), 5, "All"), ((33, 33, 25), 3, "Odd"),
    ((64, 64, 7), 5, "Odd"), ((29, 29, 31), 3, "All"), ((13, 11, 9), 2, "All"), ((32, 31, 26), 4, "Even"),
    ((5, 5, 13), 6, "Even"), ((48, 48, 20), 1, "All")])
def test_fp64_hv(bsl, tmp_path, n, l_max, sym):
    hv = write_case(str(tmp_path), n, l_max, sym)
    h = bsl.Hamiltonian(hv, CALC, precision="fp64")
    m = OracleModel(CALC, hv, threads=os.cpu_count() or 8)
    try:
        rng = np.random.default_rng(3)
        z = np.linspace(-3, 3, n[2])[:, None, None] ** 2 + np.linspace(-3, 3, n[1])[:, None] ** 2 + np.linspace(
            -3, 3, n[0]) ** 2
        for v in (rng.standard_normal(h.basis_size), np.tile(np.exp(-z).ravel(), h.basis_size // z.size),
                  1e-200 * rng.standard_normal(h.basis_size)):
            u = np.zeros_like(v)
            h.hv(v, u)
            ref = m.hv(v)
            # a dot product of nx + ny + nz + nn terms, each rounded at 2^-53 of the
            # largest partial sum (max |T| max |v|, up to 3 x its result's size here)
            tol = 2.0 ** -53 * sum(n) * 3
            scale = np.max(np.abs(v)) * max(np.max(np.abs(ref)) / np.max(np.abs(v)), kinetic_scale(n))
            assert np.max(np.abs(u - ref)) <= tol * scale
    finally:
        h.close()
        m.close()


def kinetic_scale(n):
    return sum(0.0635077857002 ** 2 / (2 * 2.01588) * np.pi ** 2 / 3 * ((k - 1) / 0.08) ** 2 for k in n)


def test_fp64_hv_of_non_finite_and_zero_vectors(bsl, tmp_path):
    """An infinity or a NaN reaches every line through its point, a zero vector stays zero."""
    h = bsl.Hamiltonian(write_case(str(tmp_path), (26, 26, 26), 5, "Odd"), CALC, precision="fp64")
    try:
        u = np.zeros(h.basis_size)
        h.hv(np.zeros(h.basis_size), u)
        assert np.all(u == 0.0)
        for bad in (np.inf, np.nan):
            v = np.ones(h.basis_size)
            v[26 * 26 * 11 + 26 * 7 + 5] = bad  # function 0 is l = 5, m = -5
            u = np.zeros(h.basis_size)
            h.hv(v, u)
            w = u[:26 ** 3].reshape(26, 26, 26)
            assert not np.any(np.isfinite(np.concatenate([w[11, 7], w[11, :, 5], w[:, 7, 5]])))
    finally:
        h.close()


def test_fp64_hv_after_a_reported_time_out(bsl, tmp_path):
    """The FP64 tensor-core kinetic leaves when a time-out is recorded; once a run
    has reported it, H v works again."""
    h = bsl.Hamiltonian(write_case(str(tmp_path), (26, 26, 26), 5, "Odd"), CALC, precision="fp64")
    try:
        v = np.random.default_rng(2).standard_normal(h.basis_size)
        ref, u = np.zeros_like(v), np.zeros_like(v)
        h.hv(v, ref)
        h.inject_timeout(2)
        with pytest.raises(bsl.BslError):
            h.lanczos(3)
        h.inject_timeout(0)
        h.hv(v, u)
        assert np.array_equal(u, ref)
    finally:
        h.close()


# one launch: up to 16 points on the CUDA cores (smallest grids, planes of a full and of
# a broken warp count, unequal z, the last size of the range and the first beyond it), up
# to 800,000 coefficients on the tensor cores (z shorter and longer than y, more plane
# pairs than CTAs, the last cube of the range); the first size with two launches
@pytest.mark.parametrize("n,nz,l_max,sym", [(4, 4, 4, "Even"), (5, 16, 5, "Odd"), (11, 6, 3, "Odd"), (7, 9, 3, "All"),
                                            (16, 16, 4, "Even"), (16, 15, 5, "Odd"), (17, 16, 4, "Even"),
                                            (16, 17, 3, "Odd"), (20, 33, 5, "Odd"), (33, 20, 4, "Even"),
                                            (21, 64, 3, "Odd"), (33, 33, 5, "Odd"), (34, 33, 5, "Odd")])
def test_small_grid_kinetic(bsl, tmp_path, n, nz, l_max, sym):
    """Mixed H v with the one-launch kinetic against the FP64 path, and against
    the tensor-core kinetic of three slices: with four slices of v and T it
    differs from FP64 by those slices' truncation only."""
    import ctypes as C
    h = bsl.Hamiltonian(write_case(str(tmp_path), (n, n, nz), l_max, sym), CALC, precision="fp64")
    try:
        v = np.random.default_rng(n).standard_normal(h.basis_size)
        ref, u, u3 = np.zeros_like(v), np.zeros_like(v), np.zeros_like(v)
        h.hv(v, ref)
        h.set_precision("mixed")
        hp = C.c_void_p(h.handle.value)
        assert bsl.lib().bsl_launches_per_iteration(hp) == (3 if bsl.lib().bsl_packed_size(hp) <= 800000 else 4)
        h.hv(v, u)
        # FP32 potential: (nn + 3) roundings of 2^-24 at |V| <= 18 |v|; the kinetic's
        # slices leave 2^-33 of max |T| max |v| per direction
        tol = np.max(np.abs(v)) * (40 * 2.0 ** -24 * 18.0 + 8 * 2.0 ** -33 * kinetic_scale((n, n, nz)))
        assert np.max(np.abs(u - ref)) <= tol
        h.set_kinetic_slices(3)  # the tensor-core kernel
        h.hv(v, u3)
        # the dropped class: four products a_k b_l of |a|, |b| <= 256, n terms each
        drop = 4 * 256 * 256 * 2.0 ** (-16 - 27) * 4 * kinetic_scale((n, n, nz)) * max(n, nz) * np.max(np.abs(v))
        assert np.max(np.abs(u3 - u)) <= 3 * drop
        h.set_kinetic_slices(4)
        # a run and its prefixes: the same bits, the deferred beta included
        a, b, _ = h.lanczos(40)
        for k in (1, 5, 33):
            a2, b2, _ = h.lanczos(k)
            assert np.array_equal(a2, a[:k]) and np.array_equal(b2, b[:k + 1])
    finally:
        h.close()
