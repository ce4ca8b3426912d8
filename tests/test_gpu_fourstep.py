"""Strang blocks on long 1D axes at every pair of view lengths the fused
four-step passes take (128 x 128 .. 4096 x 4096), against a numpy split step.

Two exact FP64 transforms of N points differ by a few 2^-53 sqrt(log2 N) of the
field's norm, and each step multiplies by unit phases whose arguments (up to
dt V = 5, dt k^2 / 2 = 2e5 here) carry 2^-53 of the argument: 5 steps stay
below 1e-9 of the norm for the largest k (2e5 * 2^-53 * 5 = 1e-10).  Mixed
precision: 2^-24 per rounding, a few tens per step: 2e-5."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, STEP_BRAGG_AD, STEP_NL, STEP_NL_IF, Laser, Solver, binfmt

pytestmark = pytest.mark.gpu

DT, NK = 1e-3, 5


def reference(h, psi, V, gs, kind, kw):
    x, k = binfmt.x_coords(h, 0), binfmt.k_coords(h, 0)
    half, full = np.exp(-0.25j * DT * k * k), np.exp(-0.5j * DT * k * k)
    psi = [np.fft.ifft(np.fft.fft(p) * half) for p in psi]
    for j in range(NK):
        rho = [np.abs(p) ** 2 for p in psi]
        ph = [sum(gs[i][m] * rho[m] for m in range(len(psi))) for i in range(len(psi))]
        if kind == STEP_BRAGG_AD:
            t1 = DT * (j + 1)
            W = kw["Amp"][0] * np.cos(kw["laser_k"][0] * x - kw["laser_domh"][0] * t1)
            m, d = 0.5 * (ph[0] + ph[1]), 0.5 * (ph[0] - ph[1])
            r = np.sqrt(d * d + W * W)
            s, c, e = DT * np.sinc(DT * r / np.pi), np.cos(DT * r), np.exp(-1j * DT * m)
            psi = [e * ((c - 1j * s * d) * psi[0] - 1j * s * W * psi[1]),
                   e * ((c + 1j * s * d) * psi[1] - 1j * s * W * psi[0])]
        else:
            own = [V if kind == STEP_NL else kw["beta"][0] * x - kw["DeltaL"][i] for i in range(len(psi))]
            psi = [p * np.exp(-1j * DT * (q + v)) for p, q, v in zip(psi, ph, own)]
        f = half if j == NK - 1 else full
        psi = [np.fft.ifft(np.fft.fft(p) * f) for p in psi]
    return psi


@pytest.mark.parametrize("lg", [14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24])
@pytest.mark.parametrize("case", ["nl", "nl_if", "bragg", "nl_if_mixed", "bragg_mixed", "three"])
def test_long_axis_block(lg, case):
    n = 1 << lg
    if (lg > 20 and case in ("nl_if", "nl_if_mixed", "three")) or (lg > 22 and case != "nl"):
        pytest.skip("covered by the other steps at this size")
    mixed = case.endswith("mixed")
    kind = STEP_NL if case == "nl" else STEP_BRAGG_AD if case.startswith("bragg") else STEP_NL_IF
    ncomp = {"nl": 1, "three": 3}.get(case, 2)
    h = binfmt.make_header(1, [n], [-100.0], [100.0])
    x = binfmt.x_coords(h, 0)
    rng = np.random.default_rng(lg)
    noise = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    psi = [np.exp(-0.5 * ((x - 3 * c) / 8) ** 2) * np.exp(2j * x) + 1e-6 * noise for c in range(ncomp)]
    norm = np.sqrt(float(h["dx"]) * sum((np.abs(p) ** 2).sum() for p in psi))
    psi = [p / norm for p in psi]
    gs = np.array([[10.0, 9.5, 9.0], [9.5, 9.8, 9.1], [9.0, 9.1, 9.7]])[:ncomp, :ncomp]
    kw = dict(Amp=[4.0, 4.0], laser_k=[8.0, 0.0], laser_domh=[16.0, 0.0], beta=[0.3, 0, 0], DeltaL=[0.0, 0.5, 0.2, 0.0])
    V = 0.5 * x * x
    if kind == STEP_BRAGG_AD:
        kw.update(beta=[0.0, 0, 0], DeltaL=[0.0] * 4)
    s = Solver(h, ncomp, PREC_MIXED if mixed else PREC_FP64)
    s.set_bragg_stable(True)
    for c in range(ncomp):
        s.set_psi(c, psi[c])
        s.set_alpha(c, [0.5])
    s.set_gs(gs)
    if kind == STEP_NL:
        s.set_potential(0, V)
    s.set_dt(DT)
    s.block(NK, kind, Laser.make(**kw))
    ref = reference(h, psi, V, gs, kind, kw)
    err = np.sqrt(sum(np.linalg.norm(s.psi(c) - ref[c]) ** 2 for c in range(ncomp)))
    assert err <= (2e-5 if mixed else 1e-9) * np.sqrt(sum(np.linalg.norm(r) ** 2 for r in ref))
    s.close()
