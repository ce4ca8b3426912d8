"""Several host threads read the fields of one batch at the same time (ctypes
drops the interpreter's lock): each gets its own field.  Complex64 fields are
widened on the device in a buffer that all readers of the batch share."""
import concurrent.futures as cf

import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, Batch, Laser, binfmt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_threads_read_their_own_fields(precision):
    insts, fields = [], []
    for k in range(24):
        dim, n = ((1, 1024), (1, 8192), (2, 64), (2, 256))[k % 4]
        h = binfmt.make_header(dim, [n] * dim, [-16.0] * dim, [16.0] * dim)
        insts.append(dict(header=h, alpha=0.5, gs=[1.0] * 4, laser=Laser.make(Amp=[1.0, 1.0], laser_k=[8.0, 0]),
                          pulse=(1.0, 0.3)))
        # whole numbers below 2^24 in both parts: the same in either precision
        base = np.arange(n**dim, dtype=np.float64).reshape((n,) * dim)
        fields.append([(base + 100000 * k + 1j * (c + 1)).astype(np.complex128) for c in range(2)])
    b = Batch(insts, precision, 1e-3)
    for i, f in enumerate(fields):
        for c in range(2):
            b.set_psi(i, c, f[c])
    jobs = [(i, c) for i in range(len(insts)) for c in range(2)] * 4
    with cf.ThreadPoolExecutor(8) as pool:
        for (i, c), got in zip(jobs, pool.map(lambda q: b.psi(*q), jobs)):
            np.testing.assert_array_equal(got, fields[i][c])
