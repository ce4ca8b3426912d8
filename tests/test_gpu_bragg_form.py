"""Which form of the 2x2 exponential the FP64 Bragg steps take, on every route
a block can go: by default the reference's eigenvalue form, with
set_bragg_stable(True) the eigenvalue-free one.

The two are the same map, so the test looks at what tells them apart: the
eigenvalue form divides by (V11 - E)^2 + Omega^2, which leaves it unitary only
to about 2^-53 |V| / |Omega|, the other is unitary to a few roundings.  The
coupling here is constant, Omega = 2^-10 |V| or so, the kinetic phases are 1
(alpha = 0), and a step multiplies the density of a point, summed over the two
states, by 1 + e.  rms(e) of the eigenvalue form comes from the same formulas
in numpy; a GPU's roundings (fused multiply-adds) scatter alike, so its rms is
held to a factor of 4 of numpy's (1e-13 here).  The eigenvalue-free form and
the four transforms around either (2^-53 sqrt(log2 N) each) stay below 1e-14."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, STEP_BRAGG_AD, STEP_BRAGG_DS_AD, Laser, Solver, binfmt

pytestmark = pytest.mark.gpu

DT, AMP, G = 1e-3, 2.0**-10, np.array([[1.0, 0.8], [0.7, 1.2]])
# one CTA of 2..128 points; on chip, one CTA and a cluster; four-step passes;
# tile passes; small dense grids (components meeting in shared memory, two-
# and three-stage pencils, tiles of 4096); the warp-autonomous pass; three-stage
# pencils of larger grids
SHAPES = [(64,), (512,), (4096,), (1 << 16,), (64, 8), (8, 64), (4, 512), (128, 128), (64, 16, 32), (32, 1024),
          (2, 4096), (4, 4096)]


def fields(shape, seed, n):
    rng = np.random.default_rng(seed)
    return [rng.uniform(0.5, 1.0, shape) * np.exp(2j * np.pi * rng.random(shape)) for _ in range(n)]


def eigen_form(p1, p2):
    r1, r2 = abs(p1) ** 2, abs(p2) ** 2
    V1, V2 = G[0, 0] * r1 + G[0, 1] * r2, G[1, 0] * r1 + G[1, 1] * r2
    root = np.sqrt((V1 - V2) ** 2 + 4 * AMP * AMP)
    out1, out2 = 0, 0
    for E in (0.5 * (V1 + V2 + root), 0.5 * (V1 + V2 - root)):
        g = np.exp(-1j * DT * E) / ((V1 - E) ** 2 + AMP * AMP)
        out1 = out1 + AMP * AMP * g * p1 - AMP * (V1 - E) * g * p2
        out2 = out2 - AMP * (V1 - E) * g * p1 + (V1 - E) ** 2 * g * p2
    return out1, out2


def spread(before, after):
    rho = [sum(abs(p) ** 2 for p in q) for q in (before, after)]
    return float(np.sqrt(np.mean((rho[1] / rho[0] - 1) ** 2)))


def step(shape, psi, kind, stable):
    dim, n = len(shape), len(psi)
    h = binfmt.make_header(dim, list(shape), [-4.0] * dim, [4.0] * dim)
    s = Solver(h, n, PREC_FP64)
    s.set_bragg_stable(stable)
    gs = np.zeros((n, n))
    for i in range(0, n, 2):
        gs[i : i + 2, i : i + 2] = G
    for c in range(n):
        s.set_alpha(c, [0.0] * dim)
        s.set_psi(c, psi[c])
    s.set_gs(gs)
    s.set_species2(Laser.make(Amp=[AMP, 0.0], laser_k=[0.0, 0.0], laser_domh=[0.0, 0.0]))
    s.set_dt(DT)
    s.block(1, kind, Laser.make(Amp=[AMP, 0.0], laser_k=[0.0, 0.0], laser_domh=[0.0, 0.0]))
    out = [s.psi(c) for c in range(n)]
    s.close()
    return out


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["bragg", "bragg_ds"])
def test_default_is_the_eigenvalue_form(shape, kind):
    if kind == "bragg_ds" and shape[-1] > 2048:
        pytest.skip("four components of such pencils do not fit in shared memory")
    psi = fields(shape, 5, 2 if kind == "bragg" else 4)
    number = STEP_BRAGG_AD if kind == "bragg" else STEP_BRAGG_DS_AD
    default, stable = (step(shape, psi, number, q) for q in (False, True))
    for i in range(0, len(psi), 2):
        want = eigen_form(psi[i], psi[i + 1])
        assert np.linalg.norm(np.subtract(default[i : i + 2], want)) <= 1e-11 * np.linalg.norm(want)
        rms = spread(psi[i : i + 2], want)
        assert 3e-14 <= rms <= 1e-11
        assert rms / 4 <= spread(psi[i : i + 2], default[i : i + 2]) <= 4 * rms
        assert spread(psi[i : i + 2], stable[i : i + 2]) <= 1e-14
