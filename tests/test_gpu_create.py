"""A context's tables and cleared fields are complete, and ordered before its
kernels, when atus_create returns: contexts made one after another over memory
that earlier ones left full of other values give the same bits."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, STEP_NL, Solver, binfmt

pytestmark = pytest.mark.gpu

DT = 1e-3


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [1 << 14, 1 << 16, 1 << 17])
def test_contexts_made_in_turn_give_the_same_bits(n, precision):
    """16 blocks on 16 contexts of a long 1D axis (its four-step twiddles are
    reordered on the device from an upload) equal the first, and the first a
    numpy split step: two steps are four transforms of a few 2^-53 sqrt(log2 N)
    each and phases up to dt k^2 / 2 = 2e3 with 2^-53 of the argument (complex64:
    2^-24 a rounding), below 1e-11 (2e-5) of the norm."""
    h = binfmt.make_header(1, [n], [-100.0], [100.0])
    x, k = binfmt.x_coords(h, 0), binfmt.k_coords(h, 0)
    psi = np.exp(-0.5 * (x / 8) ** 2) * np.exp(2j * x)
    psi /= np.sqrt(float(h["dx"]) * (np.abs(psi) ** 2).sum())
    V = 0.5 * x * x
    half, full = np.exp(-0.25j * DT * k * k), np.exp(-0.5j * DT * k * k)
    ref = np.fft.ifft(np.fft.fft(psi) * half)
    for f in (full, half):
        ref = ref * np.exp(-1j * DT * (V + 10.0 * np.abs(ref) ** 2))
        ref = np.fft.ifft(np.fft.fft(ref) * f)
    first = None
    for i in range(16):
        s = Solver(h, 1, precision)
        other = Solver(h, 2, precision)  # holds other memory, and leaves values in it
        other.set_psi(0, np.full(n, 3.0 + i))
        s.set_alpha(0, [0.5])
        s.set_psi(0, psi)
        s.set_gs([10.0])
        s.set_potential(0, V)
        s.set_dt(DT)
        s.block(2, STEP_NL)
        got = s.psi(0)
        if first is None:
            first = got
            tol = 1e-11 if precision == PREC_FP64 else 2e-5
            assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)
        np.testing.assert_array_equal(got, first)
        assert not other.psi(1).any()
        s.close()
        other.close()
