"""Potential passes of two to four components at every contiguous length they
are register-staged for, against the oracle (the reference's operations in C,
with its own transforms): grids above 8192 points, where the warp-autonomous
and the register-staged passes run.

Both sides take the same forms; the coupling stays within a factor of two of
its peak (k x within +-0.8), so the closed forms keep 13 digits, and three
steps of a few hundred roundings stay below 1e-12 of the norm (complex64
fields: 5e-6), as in test_gpu_multi.py."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, Laser, Solver, binfmt
from oracle.oracle import Laser as OLaser
from oracle.oracle import Oracle
from replay import (KIND_BRAGG_AD, KIND_BRAGG_DS_AD, KIND_DOUBLE_BRAGG_AD, KIND_NL, KIND_NL_IF_2,
                    KIND_NUMERICAL_BRAGG, KIND_NUMERICAL_RAMAN)

pytestmark = pytest.mark.gpu

SHAPES = [(512, 32), (256, 64), (16, 16, 128), (64, 256), (32, 512), (16, 1024), (8, 2048), (4, 4096)]
CASES = {"bragg": (KIND_BRAGG_AD, 2), "numerical2": (KIND_NUMERICAL_BRAGG, 2), "nl2": (KIND_NL, 2),
         "double_bragg": (KIND_DOUBLE_BRAGG_AD, 3), "raman": (KIND_NUMERICAL_RAMAN, 3), "nl3": (KIND_NL, 3),
         "bragg_ds": (KIND_BRAGG_DS_AD, 4), "nl_if_2": (KIND_NL_IF_2, 4)}
KW = dict(Amp=[6.0, 5.0], laser_k=[0.1, 0.0], laser_dk=[0.05, 0.0], laser_domh=[2.0, 0.0], phase=[0.1, 0.0],
          chirp_rate=[0.3, 0.0], beta=[0.4, 0.2, -0.1], DeltaL=[0.0, 0.5, 0.3, 0.2])
KW2 = dict(KW, Amp=[4.0, 0.0], beta=[-0.2, 0, 0])


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("case", CASES)
def test_pass_matches_oracle(shape, case):
    kind, n = CASES[case]
    if n >= 3 and shape[-1] > 2048:
        pytest.skip("three and four components of 4096 points do not fit a tile")
    dim = len(shape)
    h = binfmt.make_header(dim, list(shape), [-8.0] * dim, [8.0] * dim)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(dim)], indexing="ij")
    r2 = sum(x * x for x in X)
    psi = [(1.0 - 0.2 * c) * np.exp(-0.1 * r2) * np.exp(1j * (1 - c) * X[0]) for c in range(n)]
    g = np.fromfunction(lambda i, j: 5.0 - 0.3 * abs(i - j) - 0.1 * (i + j), (n, n))
    F = np.array([1.0, 0.5, 0.8])

    def run(s, make):
        for c in range(n):
            s.set_psi(c, psi[c])
            s.set_alpha(c, [0.5] * dim)
            if kind == KIND_NL and c != 1:
                s.set_potential(c, (1 + c) * 0.3 * r2)
        s.set_gs(g)
        s.set_species2(make(**KW2))
        s.set_dt(2e-3)
        s.block(3, kind, make(**KW), F)
        return [s.psi(c).copy() for c in range(n)]

    want = run(Oracle(h, n), OLaser.make)
    norm = np.sqrt(sum(np.linalg.norm(p) ** 2 for p in want))
    for precision, tol in ((PREC_FP64, 1e-12), (PREC_MIXED, 5e-6)):
        s = Solver(h, n, precision)
        got = run(s, Laser.make)
        s.close()
        diff = np.sqrt(sum(np.linalg.norm(p - q) ** 2 for p, q in zip(got, want)))
        assert diff <= tol * norm, precision
