"""One-launch reductions at the sizes where their grid changes: one partly
filled block, one full block, a few blocks, more points than one trip of the
full grid.  Against numpy; a sum of n non-negative terms in any order is within
n 2^-53 of exact (pairwise-like trees stay far below), so 1e-12 of the sum of
absolute terms bounds every case here (at most 2^20 terms of ~20 roundings of
the transform behind <p>)."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, Solver, binfmt

pytestmark = pytest.mark.gpu

SHAPES = [(2,), (512,), (1024,), (2048,), (1 << 20,), (2, 4, 2), (64, 32, 128), (1024, 256)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_observables_match_numpy(shape, precision):
    dim = len(shape)
    h = binfmt.make_header(dim, list(shape), [-3.0] * dim, [3.0] * dim)
    rng = np.random.default_rng(5)
    psi = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64).astype(np.complex128)
    s = Solver(h, 1, precision)
    s.set_psi(0, psi)
    rho = np.abs(psi) ** 2
    vol = float(np.prod([h["d" + a] for a in "xyz"[:dim]]))
    total = vol * rho.sum()
    assert abs(s.particle_number(0) - total) <= 1e-12 * total
    assert s.particle_number(0) == s.particle_number(0)
    dk = float(np.prod([h["dk" + a] for a in "xyz"[:dim]]))
    hat = np.abs(np.fft.fftn(psi) * vol / (2 * np.pi) ** (dim / 2)) ** 2
    x, p = s.expval_position(0), s.expval_momentum(0)
    for a in range(dim):
        sh = [-1 if b == a else 1 for b in range(dim)]
        X, K = binfmt.x_coords(h, a).reshape(sh), binfmt.k_coords(h, a).reshape(sh)
        assert abs(x[a] - vol * (X * rho).sum()) <= 1e-12 * vol * (abs(X) * rho).sum()
        assert abs(p[a] - dk * (K * hat).sum()) <= 1e-12 * dk * (abs(K) * hat).sum()
    # two balls: the whole spectrum, and none of it (thr is shared, so one
    # centre far outside); a point inside the first ball stays in bin 0
    thr = 1e3 * float(max(abs(binfmt.k_coords(h, a)).max() for a in range(dim)))
    r = s.rabi_integrals([[0.0] * dim, [1e9 * thr] * dim], thr)
    assert abs(r[0] - dk * hat.sum()) <= 1e-12 * dk * hat.sum() and r[1] == 0.0
    s.close()
