"""The other routes of a block on a long 1D axis: the numerical two-state step
(it reads the header time), and every pass apart (ATUS_PASS2=0), whose tables
share the four-step order, against the oracle.

Six steps of a few hundred roundings, the coupling never near zero (k x within
+-0.8), stay below 1e-11 of the norm; phases up to dt k^2 / 2 = 2e4 carry 2^-53
of the argument on both sides (2e-12 each)."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, Laser, Solver, binfmt
from oracle.oracle import Laser as OLaser
from oracle.oracle import Oracle
from replay import KIND_BRAGG_AD, KIND_NL, KIND_NUMERICAL_BRAGG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("staged", ["1", "0"])
@pytest.mark.parametrize("n", [1 << 15, 1 << 18])
@pytest.mark.parametrize("kind,ncomp", [(KIND_NL, 1), (KIND_BRAGG_AD, 2), (KIND_NUMERICAL_BRAGG, 2)],
                         ids=["nl", "bragg", "numerical"])
def test_block_matches_oracle(kind, ncomp, n, staged, monkeypatch):
    monkeypatch.setenv("ATUS_PASS2", staged)
    h = binfmt.make_header(1, [n], [-64.0], [64.0])
    x = binfmt.x_coords(h, 0)
    psi = [np.exp(-0.05 * (x - c) ** 2) * np.exp(1j * x) / (1.0 + c) for c in range(ncomp)]
    kw = dict(Amp=[6.0, 5.0], laser_k=[0.0125, 0.0], laser_domh=[2.0, 0.0], phase=[0.1, 0.0], chirp_rate=[0.3, 0.0],
              beta=[0.05, 0, 0], DeltaL=[0.0, 0.5, 0, 0])

    def run(s, make):
        for c in range(ncomp):
            s.set_psi(c, psi[c])
            s.set_alpha(c, [0.5])
        s.set_gs(5.0 - 0.5 * np.arange(ncomp * ncomp))
        if kind == KIND_NL:
            s.set_potential(0, 0.01 * x * x)
        s.set_dt(2e-3)
        for F in (np.array([1.0, 0.5, 0.8]), np.array([0.7, 0.9, 0.6])):
            s.block(3, kind, make(**kw), F)
        return [s.psi(c).copy() for c in range(ncomp)]

    want = run(Oracle(h, ncomp), OLaser.make)
    s = Solver(h, ncomp, PREC_FP64)
    got = run(s, Laser.make)
    s.close()
    norm = np.sqrt(sum(np.linalg.norm(p) ** 2 for p in want))
    assert np.sqrt(sum(np.linalg.norm(p - q) ** 2 for p, q in zip(got, want))) <= 1e-11 * norm
