"""Harmonic summing of a warp's few groups, of its whole tile and of the 16-warp form at
the planes where its code changes: hits and powers equal hsum.py's recurrence in float32."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,planes", [(47, 8), (49, 9), (87, 8), (89, 1), (89, 8), (127, 9), (127, 16)])
@pytest.mark.parametrize("quantile", [1e-3, 3e-3, 3e-2])  # below, about and above sixteen groups a tile
def test_hits_equal_recurrence(rows, planes, quantile):
    n = 2333
    fop = np.random.default_rng(rows * planes).exponential(1.0, size=(rows, n)).astype(np.float32)
    hps = O.harmonic_planes(fop, n_planes=planes, dtype=np.float32)
    thr = np.array([np.quantile(h, 1 - quantile) for h in hps], dtype=np.float32)
    _, pwr, plane, row, fbin = O.detections(hps, thr)
    p = make_pipeline(n, log=io.StringIO(), n_templates=rows, n_planes=planes)
    assert p.inject_FOP(fop, FDAS.A), p.last_error
    assert p.perform_harmonic_summing(thr, FDAS.AllAccelerations, FDAS.A), p.last_error
    rec, total, dropped = p.retrieve_candidate_list(FDAS.A)
    assert dropped == 0 and total == pwr.size and total > 0
    got = sorted(zip(rec["harmonic"].tolist(), rec["template_num"].tolist(), rec["bin"].tolist(),
                     rec["power"].tolist()))
    assert got == sorted(zip((plane + 1).tolist(), (row - rows // 2).tolist(), fbin.tolist(), pwr.tolist()))


def test_overflow_of_the_list_with_few_groups():
    """Reservations that cross the list's end keep what fits and count the rest."""
    n, rows, planes, cap = 3000, 85, 8, 1000
    fop = np.random.default_rng(9).exponential(1.0, size=(rows, n)).astype(np.float32)
    hps = O.harmonic_planes(fop, n_planes=planes, dtype=np.float32)
    thr = np.array([np.quantile(h, 1 - 1e-3) for h in hps], dtype=np.float32)
    _, pwr, plane, row, fbin = O.detections(hps, thr)
    assert pwr.size > cap
    p = make_pipeline(n, log=io.StringIO(), n_templates=rows, n_planes=planes, candidate_capacity=cap)
    assert p.inject_FOP(fop, FDAS.A) and p.perform_harmonic_summing(thr, FDAS.AllAccelerations, FDAS.A), p.last_error
    rec, total, dropped = p.retrieve_candidate_list(FDAS.A)
    assert total == pwr.size and dropped == pwr.size - cap and rec.size == cap
    want = set(zip((plane + 1).tolist(), (row - rows // 2).tolist(), fbin.tolist(), pwr.tolist()))
    got = set(zip(rec["harmonic"].tolist(), rec["template_num"].tolist(), rec["bin"].tolist(), rec["power"].tolist()))
    assert len(got) == cap and got <= want
