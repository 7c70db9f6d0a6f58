"""What follows a kernel time-out (injected on the host, as in
test_gpu_failure.py): the words are cleared before the error is returned, so
the next call neither skips its kernels nor reports the error again.
"""
import threading

import numpy as np
import pytest

from conftest import load_inputs, load_package

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bsl():
    return load_package()


def hamiltonian(bsl, n, precision):
    p = bsl.HvParams()
    p.nx = p.ny = p.nz = p.pnx = p.pny = p.pnz = n
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = 0.08
    p.l_max, p.theta_points, p.phi_points, p.symmetry = 5, 6, 6, bsl.SYM["Odd"]
    p.total_mass, p.rotational_constant, p.ceiling_potential = 2.01588, 0.709648713, 18.0
    waters = load_inputs().dodecahedral_cage(3)
    return bsl.Hamiltonian.from_cage(p, np.array([w[1] for w in waters]), np.array([w[2] for w in waters]),
                                     precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_next_call_starts_clean_whatever_the_legacy_stream_holds(bsl, precision):
    """A program that keeps the legacy default stream busy delays whatever is
    queued there; the library's stream does not wait for it."""
    torch = pytest.importorskip("torch")
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    h = hamiltonian(bsl, 30, precision)
    stop, going = threading.Event(), threading.Event()

    def busy():
        held = []
        while not stop.is_set():
            torch.cuda._sleep(20_000_000)  # about 10 ms
            e = torch.cuda.Event()
            e.record()
            held.append(e)
            if len(held) > 2:
                going.set()
                held.pop(0).synchronize()

    try:
        v = np.random.default_rng(2).standard_normal(h.basis_size)
        ref = np.zeros_like(v)
        h.hv(v, ref)
        t = threading.Thread(target=busy)
        t.start()
        try:
            assert going.wait(60)
            for _ in range(5):
                h.inject_timeout(2)
                with pytest.raises(bsl.BslError):
                    h.lanczos(2)
                h.inject_timeout(0)
                u = np.zeros_like(v)
                h.hv(v, u)
                assert np.array_equal(u, ref)
        finally:
            stop.set()
            t.join()
    finally:
        h.close()


@pytest.mark.parametrize("precision,mask", [("fp64", 2), ("mixed", 1), ("mixed", 2), ("mixed", 3)])
def test_device_h_v_is_nan_until_a_call_has_reported(bsl, precision, mask):
    torch = pytest.importorskip("torch")
    h = hamiltonian(bsl, 30, precision)
    try:
        v = torch.randn(21 * 30 ** 3, dtype=torch.float64, device="cuda")
        ref, u = torch.empty_like(v), torch.zeros_like(v)
        s = torch.cuda.current_stream().cuda_stream
        h.hv_device(v.data_ptr(), ref.data_ptr(), s)
        h.inject_timeout(mask)
        h.hv_device(v.data_ptr(), u.data_ptr(), s)
        h.inject_timeout(0)
        assert bool(torch.isnan(u).all())
        u.zero_()
        h.hv_device(v.data_ptr(), u.data_ptr(), s)  # the time-out stands
        assert bool(torch.isnan(u).all())
        w = np.zeros(h.basis_size)
        with pytest.raises(bsl.BslError):
            h.hv(np.ones(h.basis_size), w)
        h.hv_device(v.data_ptr(), u.data_ptr(), s)
        assert torch.equal(u, ref) and bool(torch.isfinite(ref).all())
    finally:
        h.close()
