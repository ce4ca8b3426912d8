"""Three- and four-component potential passes, register-staged, against the
shared-memory tile passes (ATUS_PASS2=0): every step kind, contiguous axes of
32..2048 points, pencil counts that leave a tile partly filled.

Both sides run the same point formulas in FP64 on fields that differ by the
roundings of two radix splits of the same transforms; three steps keep them
within 1e-12 (FP64) and 5e-6 (complex64) of the norm.  Couplings are strong
enough everywhere for the closed forms (which divide by Omega^2) to keep 13
digits."""
import numpy as np
import pytest

from atus2_b200 import (PREC_FP64, PREC_MIXED, STEP_BRAGG_DS_AD, STEP_DOUBLE_BRAGG_AD, STEP_NL, STEP_NL_IF, STEP_NL_IF_2,
                        STEP_NUMERICAL_BRAGG, STEP_NUMERICAL_RAMAN, Laser, Solver, binfmt)

pytestmark = pytest.mark.gpu

SHAPES = [(2, 32), (8, 64), (4, 128), (2, 256), (32, 4, 32), (16, 256), (2, 512), (4, 1024), (2, 2048), (2, 2, 64)]
CASES = {"double_bragg": (STEP_DOUBLE_BRAGG_AD, 3), "nl3": (STEP_NL, 3), "nl4": (STEP_NL, 4), "nl_if": (STEP_NL_IF, 3),
         "nl_if_2": (STEP_NL_IF_2, 4), "bragg_ds": (STEP_BRAGG_DS_AD, 4), "numerical": (STEP_NUMERICAL_BRAGG, 3),
         "raman": (STEP_NUMERICAL_RAMAN, 3)}


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_multi_component_pass_matches_tile_pass(case, shape, precision, monkeypatch):
    kind, ncomp = CASES[case]
    dim = len(shape)
    h = binfmt.make_header(dim, list(shape), [-8.0] * dim, [8.0] * dim)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(dim)], indexing="ij")
    r2 = sum(x * x for x in X)
    psi = [(1.0 - 0.2 * c) * np.exp(-0.1 * r2) * np.exp(1j * (1 - c) * X[0]) for c in range(ncomp)]
    # k x stays within +-0.8: cos(k x - ...) is nowhere near zero
    kw = dict(Amp=[6.0, 5.0], laser_k=[0.1, 0.0], laser_dk=[0.05, 0.0], laser_domh=[2.0, 0.0], phase=[0.1, 0.0],
              chirp_rate=[0.3, 0.0], beta=[0.4, 0.2, -0.1], DeltaL=[0.0, 0.5, 0.3, 0.2])
    out = []
    for staged in (True, False):
        if not staged:
            monkeypatch.setenv("ATUS_PASS2", "0")
        s = Solver(h, ncomp, precision)
        for c in range(ncomp):
            s.set_psi(c, psi[c])
            s.set_alpha(c, [0.5] * dim)
            if kind == STEP_NL and c != 1:
                s.set_potential(c, (1 + c) * 0.3 * r2)
        g = np.fromfunction(lambda i, j: 5.0 - 0.3 * abs(i - j) - 0.1 * (i + j), (ncomp, ncomp))
        s.set_gs(g)
        s.set_species2(Laser.make(**dict(kw, Amp=[4.0, 0.0], beta=[-0.2, 0, 0])))
        s.set_dt(2e-3)
        s.block(3, kind, Laser.make(**kw), np.array([1.0, 0.5, 0.8]))
        out.append([s.psi(c) for c in range(ncomp)])
        s.close()
    norm = np.sqrt(sum(np.linalg.norm(p) ** 2 for p in out[1]))
    diff = np.sqrt(sum(np.linalg.norm(p - q) ** 2 for p, q in zip(*out)))
    assert np.isfinite(norm) and diff <= (1e-12 if precision == PREC_FP64 else 5e-6) * norm
