"""1D blocks with the field on chip at every length they take, against a numpy
split step: one and two components, every step kind, block lengths around the
number of pulse amplitudes that travel with the launch (32) and of steps whose
couplings are prepared together (64).

Two exact FP64 transforms differ by a few 2^-53 sqrt(log2 N) of the norm, the
couplings and phases by 2^-53 of arguments up to 30: 70 steps of ~10 roundings
each stay below 1e-12 of the norm.  Complex64: 2^-24 a rounding, random signs:
70 steps below 5e-6."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, STEP_BRAGG_AD, STEP_NL, STEP_NL_IF, STEP_NL_IF_2, Laser, Solver, binfmt

pytestmark = pytest.mark.gpu

DT = 1e-3
KW = dict(Amp=[4.0, 4.0], laser_k=[8.0, 0.0], laser_dk=[0.3, 0.0], laser_domh=[16.0, 0.0], phase=[0.2, 0.0],
          chirp_rate=[0.4, 0.0], chirp=0.3, beta=[0.3, 0, 0], DeltaL=[0.1, 0.5, 0.0, 0.0])


def reference(h, psi, V, gs, kind, F):
    x, k = binfmt.x_coords(h, 0), binfmt.k_coords(h, 0)
    half, full = np.exp(-0.25j * DT * k * k), np.exp(-0.5j * DT * k * k)
    psi = [np.fft.ifft(np.fft.fft(p) * half) for p in psi]
    nk = len(F)
    for j in range(nk):
        rho = [np.abs(p) ** 2 for p in psi]
        ph = [sum(gs[i][m] * rho[m] for m in range(len(psi))) for i in range(len(psi))]
        if kind == STEP_BRAGG_AD:
            t1 = DT * (j + 1)
            W = F[j] * 4.0 * np.cos(8.0 * x - (16.0 + 0.3 * t1 + 0.4 * t1) * t1 + 0.1)
            V1, V2, eta = ph[0] + 0.3 * x, ph[1] - 0.5 + 0.3 * x, np.exp(-0.15j * x)
            m, d = 0.5 * (V1 + V2), 0.5 * (V1 - V2)
            r = np.sqrt(d * d + W * W)
            s, c, e = DT * np.sinc(DT * r / np.pi), np.cos(DT * r), np.exp(-1j * DT * m)
            psi = [e * ((c - 1j * s * d) * psi[0] - 1j * s * W * eta * psi[1]),
                   e * ((c + 1j * s * d) * psi[1] - 1j * s * W * np.conj(eta) * psi[0])]
        else:
            beta = [0.3, -0.7 if kind == STEP_NL_IF_2 else 0.3]
            own = [V[i] if kind == STEP_NL else beta[i] * x - KW["DeltaL"][i] for i in range(len(psi))]
            psi = [p * np.exp(-1j * DT * (q + v)) for p, q, v in zip(psi, ph, own)]
        f = half if j == nk - 1 else full
        psi = [np.fft.ifft(np.fft.fft(p) * f) for p in psi]
    return psi


@pytest.mark.parametrize("n", [128, 256, 512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("case", ["nl1", "nl2", "if1", "if2", "if2s", "bragg"])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nk", [1, 32, 33, 70])
def test_block_matches_numpy(n, case, precision, nk):
    kind = {"nl": STEP_NL, "if": STEP_NL_IF, "br": STEP_BRAGG_AD}[case[:2]] if case != "if2s" else STEP_NL_IF_2
    ncomp = 1 if case.endswith("1") else 2
    L = min(200.0, n * 0.05)
    h = binfmt.make_header(1, [n], [-L / 2], [L / 2])
    x = binfmt.x_coords(h, 0)
    rng = np.random.default_rng(n)
    psi = [np.exp(-0.5 * ((x - 0.02 * L * c) / (L / 16)) ** 2) * np.exp(1.5j * x) * (1.0 - 0.4 * c)
           + 1e-6 * (rng.standard_normal(n) + 1j * rng.standard_normal(n)) for c in range(ncomp)]
    norm = np.sqrt(float(h["dx"]) * sum((np.abs(p) ** 2).sum() for p in psi))
    psi = [p / norm for p in psi]
    gs = np.array([[10.0, 9.5], [9.2, 9.8]])[:ncomp, :ncomp]
    V = [0.5 * x * x, 0.3 * x * x + x]
    F = 0.6 + 0.4 * np.cos(0.1 * np.arange(nk)) if kind == STEP_BRAGG_AD else np.ones(nk)
    s = Solver(h, ncomp, precision)
    s.set_bragg_stable(True)
    for c in range(ncomp):
        s.set_psi(c, psi[c])
        s.set_alpha(c, [0.5])
        if kind == STEP_NL:
            s.set_potential(c, V[c])
    s.set_gs(gs)
    s.set_species2(Laser.make(beta=[-0.7, 0, 0]))
    s.set_dt(DT)
    s.block(nk, kind, Laser.make(**KW), F if kind == STEP_BRAGG_AD else None)
    ref = reference(h, psi, V, gs, kind, F)
    err = np.sqrt(sum(np.linalg.norm(s.psi(c) - ref[c]) ** 2 for c in range(ncomp)))
    assert err <= (1e-12 if precision == PREC_FP64 else 5e-6) * np.sqrt(sum(np.linalg.norm(r) ** 2 for r in ref))
    s.close()
