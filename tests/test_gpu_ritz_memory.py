"""bsl_ritz_vectors where the device has little room left: the same vectors, bit
for bit, with a block of single iterations and with nothing beside the vectors.
"""
import numpy as np
import pytest

from conftest import load_inputs, load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("room", [1.4, 0.3])  # of a vector in the reference layout, beside the vectors
def test_ritz_vectors_at_the_end_of_device_memory(precision, room):
    torch = pytest.importorskip("torch")
    bsl = load_package()
    p = bsl.HvParams()
    p.nx = p.ny = p.nz = p.pnx = p.pny = p.pnz = 48
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = 0.08
    p.l_max, p.theta_points, p.phi_points, p.symmetry = 5, 6, 6, bsl.SYM["Odd"]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    waters = load_inputs().dodecahedral_cage(3)
    h = bsl.Hamiltonian.from_cage(p, np.array([w[1] for w in waters]), np.array([w[2] for w in waters]),
                                  precision=precision)
    try:
        rows = np.random.default_rng(1).standard_normal((5, 11))
        rows /= 2 * np.linalg.norm(rows, axis=1)[:, None]
        ref = h.ritz(11, rows)
        vectors, full = 5 * (21 * 48 ** 3 + 1) * 8, 36 * 48 ** 3 * 8
        torch.cuda.init()
        held = []
        keep = vectors + int(room * full)
        try:
            for step in (2 ** 30, 2 ** 21):  # down to a few MB above what is kept
                free = torch.cuda.mem_get_info()[0]
                if free > keep + 2 * step:
                    held.append(torch.empty(free - keep - 2 * step, dtype=torch.uint8, device="cuda"))
            got = h.ritz(11, rows)
        finally:
            del held
            torch.cuda.empty_cache()
        assert np.array_equal(got, ref)
    finally:
        h.close()
