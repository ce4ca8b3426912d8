"""The fused Sobolev iteration (contiguous axis of 32..256 points) at the edges
of that range and beyond, against a plain numpy descent: one and two
components, with and without a potential, 2D and 3D, short other axes.

Both sides do the same FP64 arithmetic up to summation order; a step moves psi
by stepsize * G, so after 20 iterations the states agree to a few roundings of
the transforms (log2 N of 2^-53 each): 1e-12 relative.  The residual is a sum
of squares of a difference that cancels to sqrt(res) of its terms, so it is
held to 1e-9 relative."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, Solver, binfmt

pytestmark = pytest.mark.gpu

STEP, ITERS = 4e-4, 20
SHAPES = [(16, 16), (4, 32), (32, 256), (8, 512), (2, 2, 32), (16, 8, 64), (4, 32, 128)]


def descend(h, psi, V, gs, alpha):
    dim = psi[0].ndim
    vol = float(np.prod([h["d" + a] for a in "xyz"[:dim]]))
    k2 = sum(binfmt.k_coords(h, a).reshape([-1 if b == a else 1 for b in range(dim)]) ** 2 for a in range(dim))
    dot = lambda a, b: float((a.real * b.real + a.imag * b.imag).sum())  # noqa: E731
    psi = [p / np.sqrt(vol * dot(p, p)) for p in psi]
    for _ in range(ITERS):
        grads, res = [], 0.0
        for i, p in enumerate(psi):
            S = 1.0 / (1.0 + alpha[i] * k2)
            f = np.fft.fftn(p)
            W = (V[i] if V[i] is not None else 0.0) + sum(gs[i][j] * np.abs(psi[j]) ** 2 for j in range(len(psi)))
            g = np.fft.ifftn(np.fft.fftn(np.fft.ifftn(f * alpha[i] * k2) + W * p) * S)
            sp = np.fft.ifftn(f * S)
            g = g - dot(p, g) / dot(p, sp) * sp
            grads.append(g)
            res += (vol * dot(g, g)) ** 2
        N = [vol * dot(p, p) for p in psi]
        if any(abs(n - 1) > 1e-5 for n in N):
            psi = [p / np.sqrt(n) for p, n in zip(psi, N)]
        psi = [p - STEP * g for p, g in zip(psi, grads)]
    return psi, np.sqrt(res)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ncomp", [1, 2])
def test_descent_matches_numpy(shape, ncomp):
    dim = len(shape)
    h = binfmt.make_header(dim, list(shape), [-4.0] * dim, [4.0] * dim)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(dim)], indexing="ij")
    rng = np.random.default_rng(11)
    psi = [np.exp(-0.4 * sum(x * x for x in X)) * (1 + 0.1j * (c + 1)) + 0.01 * rng.standard_normal(shape)
           for c in range(ncomp)]
    V = [sum(0.5 * (1 + c) * x * x for x in X) if c == 0 else None for c in range(ncomp)]
    gs = np.array([[10.0, 4.0], [4.0, 6.0]])[:ncomp, :ncomp]
    alpha = [0.5, 0.7][:ncomp]
    s = Solver(h, ncomp, PREC_FP64)
    for c in range(ncomp):
        s.set_psi(c, psi[c])
        if V[c] is not None:
            s.set_potential(c, V[c])
    s.set_gs(gs)
    s.sob_init(alpha, STEP)
    iters, res = s.sob_run(0.0, ITERS)
    ref, ref_res = descend(h, psi, V, gs, alpha)
    assert iters == ITERS
    assert abs(res - ref_res) <= 1e-9 * ref_res
    for c in range(ncomp):
        assert np.linalg.norm(s.psi(c) - ref[c]) <= 1e-12 * np.linalg.norm(ref[c])
    s.close()


def test_descent_follows_changed_parameters():
    """A second descent on the same context with another interaction strength,
    then without the potential, equals a fresh context's (the iterations
    captured by the first hold neither)."""
    shape = (4, 8, 32)
    h = binfmt.make_header(3, list(shape), [-4.0] * 3, [4.0] * 3)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(3)], indexing="ij")
    psi = np.exp(-0.4 * sum(x * x for x in X))
    V = sum(0.5 * x * x for x in X)

    def run(s, g, V):
        s.set_psi(0, psi)
        s.set_gs([g])
        s.set_potential(0, V)
        s.sob_init([0.5], STEP)
        s.sob_run(0.0, ITERS)
        return s.psi(0)

    used = Solver(h, 1, PREC_FP64)
    run(used, 10.0, V)
    for g, pot in ((200.0, V), (200.0, None), (50.0, V)):
        fresh = Solver(h, 1, PREC_FP64)
        np.testing.assert_array_equal(run(used, g, pot), run(fresh, g, pot))
        fresh.close()
    used.close()
