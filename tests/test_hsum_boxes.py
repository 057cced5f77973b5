"""Harmonic summing reads no column past the row of a staged box."""
import io
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_columns_lie_in_their_boxes(tmp_path):
    exe = tmp_path / "hsum_boxes"
    subprocess.run(["g++", "-std=c++17", "-x", "c++", f"-I{ROOT / 'fdas_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "hsum_boxes.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n,quantile", [(43, 4111, 0.3), (85, 4100, 0.5), (127, 1030, 0.2)])
def test_plane_16_of_dense_hits(rows, n, quantile):
    """Whole tiles summed and marked at 16 planes: hits and powers equal hsum.py's
    recurrence in float32."""
    from gpu_util import make_pipeline
    from fdas_gb300.fdas import FDAS
    from oracle import fdas_oracle as O
    fop = np.random.default_rng(rows + n).exponential(1.0, size=(rows, n)).astype(np.float32)
    hps = O.harmonic_planes(fop, n_planes=16, dtype=np.float32)
    # only the last planes' hits, so that plane 16's own marks decide
    thr = np.full(16, 1e30, dtype=np.float32)
    thr[14:] = [np.quantile(h, 1 - quantile) for h in hps[14:]]
    _, pwr, plane, row, fbin = O.detections(hps, thr)
    p = make_pipeline(n, log=io.StringIO(), n_templates=rows, n_planes=16)
    assert p.inject_FOP(fop, FDAS.A), p.last_error
    assert p.perform_harmonic_summing(thr, FDAS.AllAccelerations, FDAS.A), p.last_error
    rec, total, dropped = p.retrieve_candidate_list(FDAS.A)
    assert dropped == 0 and total == pwr.size and total > 0
    got = sorted(zip(rec["harmonic"].tolist(), rec["template_num"].tolist(), rec["bin"].tolist(),
                     rec["power"].tolist()))
    assert got == sorted(zip((plane + 1).tolist(), (row - rows // 2).tolist(), fbin.tolist(), pwr.tolist()))
