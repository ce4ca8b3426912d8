"""Two-component potential passes whose components meet in a warp, against the
shared-memory tile passes (ATUS_PASS2=0, a point at a time): every step kind,
contiguous axes of 32..2048 points, pencil counts that leave a warp or a CTA
partly filled, phases small enough for the series and too large for it,
couplings from strong to none.

Both sides do FP64 arithmetic on the same formulas up to the order of a few
products (complex64 fields: FP32 transforms of different radix splits), so
after three steps they agree to 1e-12 (FP64; the eigenvalue form's own
2^-53 |V| / |Omega| reaches 1e-13 where it takes over) and 5e-6 (complex64)
of the norm."""
import numpy as np
import pytest

from atus2_b200 import (PREC_FP64, PREC_MIXED, STEP_BRAGG_AD, STEP_NL, STEP_NL_IF, STEP_NL_IF_2, STEP_NUMERICAL_BRAGG,
                        Laser, Solver, binfmt)

pytestmark = pytest.mark.gpu

SHAPES = [(2, 32), (4, 64), (8, 128), (2, 256), (32, 32, 32), (64, 256), (4, 512), (2, 1024), (2, 2048), (4, 2, 64)]
CASES = {
    "bragg": (STEP_BRAGG_AD, {}),
    "bragg_weak": (STEP_BRAGG_AD, dict(Amp=[1e-9, 0.0])),
    "bragg_off": (STEP_BRAGG_AD, dict(Amp=[0.0, 0.0])),
    "bragg_strong": (STEP_BRAGG_AD, dict(Amp=[80.0, 0.0])),
    "bragg_tilted": (STEP_BRAGG_AD, dict(beta=[40.0, 0, 0], DeltaL=[0.0, 3.0, 0, 0], laser_dk=[0.4, 0.0])),
    "nl": (STEP_NL, {}),
    "nl_far": (STEP_NL, {}),
    "nl_if": (STEP_NL_IF, dict(beta=[2.0, 0, 0], DeltaL=[0.0, 3.0, 0, 0])),
    "nl_if_far": (STEP_NL_IF, dict(beta=[60.0, 0, 0], DeltaL=[0.0, 3.0, 0, 0])),
    "nl_if_2": (STEP_NL_IF_2, dict(beta=[2.0, 0, 0])),
    "numerical": (STEP_NUMERICAL_BRAGG, {}),
}


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_pair_pass_matches_tile_pass(case, shape, precision, monkeypatch):
    kind, over = CASES[case]
    if case == "bragg_weak" and precision == PREC_FP64:
        # the reference's eigenvalue form amplifies the two sides' transform
        # roundings by |V| / |Omega| = 5e9 here: they cannot agree
        pytest.skip("the FP64 eigenvalue form is ill-conditioned at Omega = 1e-9")
    dim = len(shape)
    h = binfmt.make_header(dim, list(shape), [-8.0] * dim, [8.0] * dim)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(dim)], indexing="ij")
    r2 = sum(x * x for x in X)
    psi = [np.exp(-0.1 * r2) * np.exp(1j * X[0]), 0.6 * np.exp(-0.12 * r2) * np.exp(-0.5j * X[-1])]
    kw = dict(Amp=[4.0, 3.0], laser_k=[4.0, 0.0], laser_domh=[16.0, 0.0], phase=[0.3, 0.0])
    kw.update(over)
    V = (40.0 if case == "nl_far" else 0.2) * r2 / 16
    out = []
    for staged in (True, False):
        if not staged:
            monkeypatch.setenv("ATUS_PASS2", "0")
        s = Solver(h, 2, precision)
        for c in range(2):
            s.set_psi(c, psi[c])
            s.set_alpha(c, [0.5] * dim)
        s.set_gs([5.0, 4.5, 4.5, 4.0])
        if kind == STEP_NL:
            s.set_potential(0, V)
            s.set_potential(1, 0.5 * V)
        s.set_species2(Laser.make(beta=[1.0, 0, 0]))
        s.set_dt(2e-3)
        s.block(3, kind, Laser.make(**kw), np.array([1.0, 0.5, 0.8]))
        out.append([s.psi(c) for c in range(2)])
        s.close()
    norm = np.sqrt(sum(np.linalg.norm(p) ** 2 for p in out[1]))
    diff = np.sqrt(sum(np.linalg.norm(p - q) ** 2 for p, q in zip(*out)))
    assert np.isfinite(norm) and diff <= (1e-12 if precision == PREC_FP64 else 5e-6) * norm
