"""1D blocks where no cluster of CTAs is used (ATUS_CLUSTER1D=0; the same routes
serve a device that cannot place one): one CTA where the field fits, per-step
or four-step passes where it does not, against a numpy split step.

Bounds as in test_gpu_line1d.py: 33 steps of ~10 roundings stay below 1e-12
(FP64) and 5e-6 (complex64) of the norm."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, STEP_BRAGG_AD, STEP_NL, Laser, Solver, binfmt
from test_gpu_line1d import DT, KW, reference

pytestmark = pytest.mark.gpu

# the longest field that one CTA holds (points), by precision and components
ON_CHIP = {(PREC_FP64, 1): 2048, (PREC_FP64, 2): 1024, (PREC_MIXED, 1): 4096, (PREC_MIXED, 2): 2048}


@pytest.mark.parametrize("n", [256, 512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("case", ["nl1", "bragg"])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_block_without_a_cluster(n, case, precision, monkeypatch):
    monkeypatch.setenv("ATUS_CLUSTER1D", "0")
    nk = 33
    kind, ncomp = (STEP_NL, 1) if case == "nl1" else (STEP_BRAGG_AD, 2)
    L = min(200.0, n * 0.05)
    h = binfmt.make_header(1, [n], [-L / 2], [L / 2])
    x = binfmt.x_coords(h, 0)
    psi = [np.exp(-0.5 * ((x - 0.02 * L * c) / (L / 16)) ** 2) * np.exp(1.5j * x) * (1.0 - 0.4 * c) for c in range(ncomp)]
    norm = np.sqrt(float(h["dx"]) * sum((np.abs(p) ** 2).sum() for p in psi))
    psi = [p / norm for p in psi]
    gs = np.array([[10.0, 9.5], [9.2, 9.8]])[:ncomp, :ncomp]
    V = [0.5 * x * x, 0.0 * x]
    F = 0.6 + 0.4 * np.cos(0.1 * np.arange(nk)) if kind == STEP_BRAGG_AD else np.ones(nk)
    s = Solver(h, ncomp, precision)
    s.set_bragg_stable(True)
    for c in range(ncomp):
        s.set_psi(c, psi[c])
        s.set_alpha(c, [0.5])
    if kind == STEP_NL:
        s.set_potential(0, V[0])
    s.set_gs(gs)
    s.set_dt(DT)
    before = s.launches
    s.block(nk, kind, Laser.make(**KW), F if kind == STEP_BRAGG_AD else None)
    if n <= ON_CHIP[precision, ncomp]:
        assert s.launches - before == 1  # the whole block on chip
    else:
        assert s.launches - before > nk
    ref = reference(h, psi, V, gs, kind, F)
    err = np.sqrt(sum(np.linalg.norm(s.psi(c) - ref[c]) ** 2 for c in range(ncomp)))
    assert err <= (1e-12 if precision == PREC_FP64 else 5e-6) * np.sqrt(sum(np.linalg.norm(r) ** 2 for r in ref))
    s.close()
