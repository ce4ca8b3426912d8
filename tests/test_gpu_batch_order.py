"""A batch's uploads, and the copies that the autotuner puts aside and back, are
ordered before the kernels that follow: tuning leaves the fields as they were,
and batches made one after another give the same bits."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, Batch, Laser, binfmt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_tuning_and_uploads_are_ordered(precision):
    sizes = [(1, 1024), (1, 8192), (2, 64), (2, 256), (2, 256)]
    rng = np.random.default_rng(3)
    insts, fields = [], []
    for dim, n in sizes:
        h = binfmt.make_header(dim, [n] * dim, [-16.0] * dim, [16.0] * dim)
        insts.append(dict(header=h, alpha=0.5, gs=[5.0] * 4, pulse=(0.02, 0.01), bragg_stable=True,
                          laser=Laser.make(Amp=[4.0, 4.0], laser_k=[8.0, 0], laser_domh=[2.0, 0])))
        shape = (n,) * dim
        # exact in complex64
        fields.append([(rng.integers(1, 1000, shape) / 1024 + 1j * rng.integers(1, 1000, shape) / 1024) for _ in range(2)])
    first = None
    for _ in range(4):
        b = Batch(insts, precision, 1e-3)
        for i, f in enumerate(fields):
            for c in range(2):
                b.set_psi(i, c, f[c])
        b.run(7)
        ran = [b.psi(i, c) for i in range(len(sizes)) for c in range(2)]
        if first is None:
            first = ran
        for p, q in zip(ran, first):
            np.testing.assert_array_equal(p, q)
        b.tune(3)
        for p, q in zip([b.psi(i, c) for i in range(len(sizes)) for c in range(2)], ran):
            np.testing.assert_array_equal(p, q)
