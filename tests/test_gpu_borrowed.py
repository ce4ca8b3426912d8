"""Host buffers are the caller's again when a call returns: the pulse amplitudes
of a block may be overwritten at once, also where they are page-locked (the
copy to the device is then asynchronous) and the stream is busy."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, STEP_BRAGG_AD, Laser, Solver, binfmt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(64, 5), (64, 33), (512, 33), (4096, 200), (1 << 16, 3)])
def test_amplitudes_are_taken_before_the_call_returns(n, nk):
    import torch

    h = binfmt.make_header(1, [n], [-8.0], [8.0])
    x = binfmt.x_coords(h, 0)
    psi = np.exp(-0.5 * x * x).astype(np.complex128)
    amp = 0.5 + 0.4 * np.cos(np.arange(nk))
    out = []
    for pinned in (False, True):
        s = Solver(h, 2, PREC_FP64)
        s.set_psi(0, psi)
        for c in range(2):
            s.set_alpha(c, [0.5])
        s.set_gs([1.0, 0.9, 0.9, 1.0])
        s.set_dt(1e-3)
        s.set_laser(Laser.make(Amp=[4.0, 4.0], laser_k=[4.0, 0.0], laser_domh=[8.0, 0.0]))
        s.block(1, STEP_BRAGG_AD, F=np.ones(1))  # kernels loaded: the next calls only queue work
        s.block(2000, STEP_BRAGG_AD)             # tens of milliseconds on the device
        F = torch.empty(nk, dtype=torch.float64, pin_memory=pinned).numpy()
        F[:] = amp
        s.block(nk, STEP_BRAGG_AD, F=F)
        F[:] = 0.0
        out.append([s.psi(c) for c in range(2)])
        s.close()
    np.testing.assert_array_equal(out[1], out[0])
