"""Harmonic summing decides most of a tile from bounds of its sums and sums
only what they leave over: no group, a few groups one cell per lane, or whole
tiles.  On injected FOPs of each density, over banks, planes, halves and ragged
lengths, hits and powers equal hsum.py's recurrence in float32 -- with
infinities and NaN among the cells too."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu

PARTS = {"all": FDAS.AllAccelerations, "pos": FDAS.PositiveAccelerations, "neg": FDAS.NegativeAccelerations}


@pytest.mark.parametrize("rows,planes,part,n,quantile,odd", [
    (85, 8, "all", 3001, 1e-5, False),   # a group here and there
    (85, 8, "all", 3001, 3e-3, False),   # several groups of a warp
    (85, 8, "all", 1024, 0.5, False),    # every warp, every plane
    (85, 16, "all", 4099, 1e-4, False),
    (43, 16, "neg", 2050, 1e-3, False),
    (127, 8, "all", 1500, 1e-3, False),
    (3, 5, "pos", 700, 1e-2, False),
    (1, 1, "all", 255, 1e-2, False),
    (85, 2, "pos", 257, 1e-3, False),
    (85, 9, "all", 2111, 1e-3, True),
])
def test_hits_equal_recurrence(rows, planes, part, n, quantile, odd):
    rng = np.random.default_rng(rows * planes + n)
    fop = rng.exponential(1.0, size=(rows, n)).astype(np.float32)
    if odd:
        for v in (np.inf, np.nan, -np.inf, 0.0, -1.0):
            fop[rng.integers(0, rows, 40), rng.integers(0, n, 40)] = v
    with np.errstate(invalid="ignore"):
        hps = O.harmonic_planes(fop, n_planes=planes, dtype=np.float32)
    thr = np.array([np.quantile(h[np.isfinite(h)], 1 - quantile) for h in hps], dtype=np.float32)
    _, pwr, plane, row, fbin = O.detections(hps, thr, rows=O.part_rows(part, rows))
    p = make_pipeline(n, log=io.StringIO(), n_templates=rows, n_planes=planes)
    assert p.inject_FOP(fop, FDAS.A), p.last_error
    assert p.perform_harmonic_summing(thr, PARTS[part], FDAS.A), p.last_error
    rec, total, dropped = p.retrieve_candidate_list(FDAS.A)
    assert dropped == 0 and total == pwr.size and total > 0
    got = sorted(zip(rec["harmonic"].tolist(), rec["template_num"].tolist(), rec["bin"].tolist(),
                     rec["power"].tolist()))
    want = sorted(zip((plane + 1).tolist(), (row - rows // 2).tolist(), fbin.tolist(), pwr.tolist()))
    assert got == want
