"""The site-by-site kernel of the potential grid (parity with the oracle is in test_gpu_parity.py)."""
import numpy as np
import pytest

from conftest import load_inputs, load_package

pytestmark = pytest.mark.gpu

Q = np.array([0.8476, 0.4238, 0.4238])


@pytest.fixture(scope="module")
def bsl():
    return load_package()


def params(bsl, n, box, l_max, sym, theta, phi):
    p = bsl.HvParams()
    p.nx, p.ny, p.nz = p.pnx, p.pny, p.pnz = n
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = box
    p.l_max, p.theta_points, p.phi_points, p.symmetry = l_max, theta, phi, bsl.SYM[sym]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    return p


def cage(seed):
    waters = load_inputs().dodecahedral_cage(seed)
    return np.array([w[1] for w in waters]), np.array([w[2] for w in waters])


@pytest.mark.parametrize("theta,phi", [(5, 7), (6, 4), (8, 12)])
def test_site_terms_are_the_plain_operations(bsl, theta, phi):
    """The site kernel's root and quotient are the correctly rounded ones: a
    water without charges so far away that its distance leaves the range of the
    fast term makes every thread redo its sums with the plain operations, and
    adds exactly nothing."""
    cm, euler = cage(5)
    far = np.vstack([cm, [[2.0 ** 36, 0.0, 0.0]]]), np.vstack([euler, np.zeros((1, 3))])
    q = np.tile([-Q[0], Q[1], Q[2]], 20)
    p = params(bsl, (13, 12, 11), 0.08, 3, "Odd", theta, phi)
    grids = []
    for c, e, qs in ((cm, euler, q), (*far, np.concatenate([q, np.zeros(3)]))):
        h = bsl.Hamiltonian.from_cage(p, c, e, q_site=qs, precision="mixed")
        grids.append(h.vgrid())
        h.close()
    assert np.array_equal(grids[0][0], grids[1][0]) and np.array_equal(grids[0][1], grids[1][1])
