"""Register-staged passes over pencils of 1024..4096 points -- with more tiles
than SMs (the next tile prefetched) and fewer, whole and partly filled ones --
and one-component potential steps with small and large phases, against the
shared-memory tile passes (ATUS_PASS2=0).

Two exact transforms of different radix splits differ by a few 2^-53
sqrt(log2 N) of the norm each: three steps stay below 1e-12 (FP64) and 5e-6
(complex64)."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, STEP_NL, STEP_NL_IF, Laser, Solver, binfmt

pytestmark = pytest.mark.gpu

SHAPES = [(4096, 2), (2, 4096), (4096, 512), (512, 4096), (2048, 1024), (1024, 2048), (256, 1024, 2), (32, 2048, 16),
          (2048, 4), (64, 32), (2, 512)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("case", ["nl", "nl_far", "nl_if", "nl_if_far", "two"])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_long_pencils_match_tile_pass(shape, case, precision, monkeypatch):
    dim = len(shape)
    ncomp = 2 if case == "two" else 1
    kind = STEP_NL if case.startswith("nl") and "if" not in case else STEP_NL_IF
    h = binfmt.make_header(dim, list(shape), [-8.0] * dim, [8.0] * dim)
    X = [binfmt.x_coords(h, a).reshape([-1 if b == a else 1 for b in range(dim)]) for a in range(dim)]
    r2 = sum(x * x for x in X)
    psi = [(1 - 0.3 * c) * np.exp(-0.1 * r2) * np.exp(1j * X[0] - 0.4j * c * X[-1]) for c in range(ncomp)]
    V = (60.0 if case == "nl_far" else 0.3) * r2 / 16
    beta = 60.0 if case == "nl_if_far" else 1.5
    out = []
    for staged in (True, False):
        if not staged:
            monkeypatch.setenv("ATUS_PASS2", "0")
        s = Solver(h, ncomp, precision)
        for c in range(ncomp):
            s.set_psi(c, psi[c])
            s.set_alpha(c, [0.5] * dim)
        s.set_gs(np.full((ncomp, ncomp), 3.0))
        if kind == STEP_NL:
            s.set_potential(0, V)
        s.set_dt(2e-3)
        s.block(3, kind, Laser.make(beta=[beta, 0, 0], DeltaL=[0.2, 0.7, 0, 0]))
        out.append([s.psi(c) for c in range(ncomp)])
        s.close()
    norm = np.sqrt(sum(np.linalg.norm(p) ** 2 for p in out[1]))
    diff = np.sqrt(sum(np.linalg.norm(p - q) ** 2 for p, q in zip(*out)))
    assert np.isfinite(norm) and diff <= (1e-12 if precision == PREC_FP64 else 5e-6) * norm
