"""The size-dependent kernels of H v and of the Lanczos iteration against one
another, at the edges of their ranges.

Mixed: the kinetic in one launch up to 16 points per axis, the same bits as the
tensor-core kernels'.
"""
import os

import numpy as np
import pytest

from conftest import load_inputs, load_package

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


def kinetic_scale(n):
    return sum(0.0635077857002 ** 2 / (2 * 2.01588) * np.pi ** 2 / 3 * ((k - 1) / 0.08) ** 2 for k in n)


# one launch up to 16 points: smallest grids, planes of a full and of a broken warp
# count, unequal z, the last size of the range and the first beyond it
@pytest.mark.parametrize("n,nz,l_max,sym", [(4, 4, 4, "Even"), (5, 16, 5, "Odd"), (11, 6, 3, "Odd"), (7, 9, 3, "All"),
                                            (16, 16, 4, "Even"), (16, 15, 5, "Odd"), (17, 16, 4, "Even"),
                                            (16, 17, 3, "Odd")])
def test_small_grid_kinetic(bsl, tmp_path, n, nz, l_max, sym):
    """Mixed H v with the one-launch kinetic against the FP64 path, and against
    the two-launch kinetic: with three slices of v and T, and with four, it
    differs from FP64 by those slices' truncation only."""
    import ctypes as C
    h = bsl.Hamiltonian(write_case(str(tmp_path), (n, n, nz), l_max, sym), CALC, precision="fp64")
    try:
        v = np.random.default_rng(n).standard_normal(h.basis_size)
        ref, u, u3 = np.zeros_like(v), np.zeros_like(v), np.zeros_like(v)
        h.hv(v, ref)
        h.set_precision("mixed")
        assert bsl.lib().bsl_launches_per_iteration(C.c_void_p(h.handle.value)) == (3 if max(n, nz) <= 16 else 4)
        h.hv(v, u)
        # FP32 potential: (nn + 3) roundings of 2^-24 at |V| <= 18 |v|; the kinetic's
        # slices leave 2^-33 of max |T| max |v| per direction
        tol = np.max(np.abs(v)) * (40 * 2.0 ** -24 * 18.0 + 8 * 2.0 ** -33 * kinetic_scale((n, n, nz)))
        assert np.max(np.abs(u - ref)) <= tol
        h.set_kinetic_slices(3)  # two launches
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
