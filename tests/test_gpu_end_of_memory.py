"""Calls at the end of device memory: bsl_ritz_vectors gives the same vectors, bit
for bit, with a block of single iterations and with nothing beside the vectors;
host H v without room for its staging says so, however often it is called.
"""
import numpy as np
import pytest

from conftest import load_inputs, load_package

pytestmark = pytest.mark.gpu


def hamiltonian(bsl, precision):
    p = bsl.HvParams()
    p.nx = p.ny = p.nz = p.pnx = p.pny = p.pnz = 48
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = 0.08
    p.l_max, p.theta_points, p.phi_points, p.symmetry = 5, 6, 6, bsl.SYM["Odd"]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    waters = load_inputs().dodecahedral_cage(3)
    return bsl.Hamiltonian.from_cage(p, np.array([w[1] for w in waters]), np.array([w[2] for w in waters]),
                                     precision=precision)


def fill_device(torch, keep):
    """Tensors that leave `keep` bytes of the device free, and a few MB."""
    torch.cuda.init()
    held = []
    for step in (2 ** 30, 2 ** 21):
        free = torch.cuda.mem_get_info()[0]
        if free > keep + 2 * step:
            held.append(torch.empty(free - keep - 2 * step, dtype=torch.uint8, device="cuda"))
    return held


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("room", [1.4, 0.3])  # of a vector in the reference layout, beside the vectors
def test_ritz_vectors_at_the_end_of_device_memory(precision, room):
    torch = pytest.importorskip("torch")
    bsl = load_package()
    h = hamiltonian(bsl, precision)
    try:
        rows = np.random.default_rng(1).standard_normal((5, 11))
        rows /= 2 * np.linalg.norm(rows, axis=1)[:, None]
        ref = h.ritz(11, rows)
        vectors, full = 5 * (21 * 48 ** 3 + 1) * 8, 36 * 48 ** 3 * 8
        held = fill_device(torch, vectors + int(room * full))
        try:
            got = h.ritz(11, rows)
        finally:
            del held
            torch.cuda.empty_cache()
        assert np.array_equal(got, ref)
    finally:
        h.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_host_h_v_without_room_for_its_staging(precision):
    torch = pytest.importorskip("torch")
    bsl = load_package()
    h, other = hamiltonian(bsl, precision), hamiltonian(bsl, precision)
    try:
        v = np.random.default_rng(1).standard_normal(h.basis_size)
        ref, u = np.zeros_like(v), np.zeros_like(v)
        other.hv(v, ref)
        held = fill_device(torch, int(1.5 * 36 * 48 ** 3 * 8))  # one of its two vectors
        try:
            for _ in range(3):
                with pytest.raises(bsl.BslError) as ei:
                    h.hv(v, u)
                assert ei.value.code == bsl.ERR_NOMEM
                assert np.all(u == 0.0)
        finally:
            del held
            torch.cuda.empty_cache()
        h.hv(v, u)
        assert np.array_equal(u, ref)
    finally:
        h.close()
        other.close()
