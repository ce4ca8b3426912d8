"""A second descent on a context that was set up once follows a changed
interaction strength, a removed, a new and a changed potential, though its
iterations were captured by the first: each equals, bit for bit, a context
that never ran with other values."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, Solver, binfmt

pytestmark = pytest.mark.gpu

STEP, ITERS = 4e-4, 20


def context(shape, ncomp):
    h = binfmt.make_header(len(shape), list(shape), [-4.0] * len(shape), [4.0] * len(shape))
    s = Solver(h, ncomp, PREC_FP64)
    s.sob_init([0.5] * ncomp, STEP)
    return s, h


def descend(s, psi):
    for c in range(s.ncomp):
        s.set_psi(c, psi)
    s.sob_run(0.0, ITERS)
    return np.stack([s.psi(c) for c in range(s.ncomp)])


# the fused iteration (contiguous axis of 32..256 points) and the general one
@pytest.mark.parametrize("shape", [(4, 8, 32), (8, 8), (64,)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("ncomp", [1, 2])
@pytest.mark.parametrize("change", ["gs", "potential_removed", "potential_new", "potential_values"])
def test_captured_descent_follows(shape, ncomp, change):
    used, h = context(shape, ncomp)
    X = np.meshgrid(*[binfmt.x_coords(h, a) for a in range(len(shape))], indexing="ij")
    r2 = sum(x * x for x in X)
    psi, V = np.exp(-0.4 * r2), 0.5 * r2
    first_V = None if change == "potential_new" else V
    last_V = {"potential_removed": None, "potential_values": 2.0 * V}.get(change, V)
    first_g, last_g = 10.0 * np.ones((ncomp, ncomp)), (200.0 if change == "gs" else 10.0) * np.ones((ncomp, ncomp))
    used.set_gs(first_g)
    used.set_potential(0, first_V)
    first = descend(used, psi)
    if change == "gs":
        used.set_gs(last_g)
    else:
        used.set_potential(0, last_V)
    got = descend(used, psi)
    fresh, _ = context(shape, ncomp)
    fresh.set_gs(last_g)
    fresh.set_potential(0, last_V)
    np.testing.assert_array_equal(got, descend(fresh, psi))
    assert not np.array_equal(got, first)
    used.close()
    fresh.close()
