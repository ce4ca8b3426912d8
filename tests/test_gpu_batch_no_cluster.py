"""A batch's 1D runs where no cluster of CTAs is used (ATUS_CLUSTER1D=0; the
same route serves a device that cannot place one): every length the precision
takes, against the oracle, within the bounds of test_batch.py."""
import numpy as np
import pytest

from atus2_b200 import PREC_FP64, PREC_MIXED, Batch
from test_batch import DT, FP64_TOL, MIXED_TOL, _check, _instances, _oracle_runs, _psi0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_batch_without_clusters_matches_oracle(precision, monkeypatch):
    monkeypatch.setenv("ATUS_CLUSTER1D", "0")
    lengths = [1024, 2048, 4096, 8192] + ([16384] if precision == PREC_MIXED else [])
    insts = _instances(17, [(1, n) for n in lengths] + [(1, lengths[-1])] * 2)
    b = Batch(insts, precision, DT)
    for i, d in enumerate(insts):
        b.set_psi(i, 0, _psi0(d["header"]))
        b.set_psi(i, 1, np.zeros_like(_psi0(d["header"])))
    b.run(25)
    b.tune(3)
    assert "CTAs per instance" not in b.schedule()  # one CTA each
    b.run(1)
    _check(b, insts, _oracle_runs(insts, [25, 1]), FP64_TOL if precision == PREC_FP64 else MIXED_TOL)
