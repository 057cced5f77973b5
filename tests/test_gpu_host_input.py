"""Short spectra in pinned host memory are read by the tiling itself: the same tiles
and records as from pageable memory, and the copy it leaves serves the stages after."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300 import synth
from fdas_gb300.fdas import FDAS, PinnedArray
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


def spectrum(n, seed):
    return synth.spectrum(synth.timeseries(2 * n, [dict(r0=0.3 * n, z=8.0, n_harm=3, amp=0.1)], seed=seed))[0]


# one tile, around tile ends (1628 bins a tile), ragged, both sides of the limit of 2^18 bins
@pytest.mark.parametrize("n", [500, 1628, 1629, 4096, 9001, 262144, 262145])
def test_pinned_and_pageable_spectra(n):
    thr = O.chi2_thresholds(1e-4, 8)
    p = make_pipeline(n, log=io.StringIO())
    for ab in (FDAS.A, FDAS.B):
        assert p.upload_templates(template_bank(), ab)
    nc = p.get_candidate_list_sz()
    keep = PinnedArray((n + 2,), np.complex64)
    pinned = keep.array[1:n + 1]  # 8-byte aligned
    loc, pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
    tiles = [np.zeros(p.get_tiles_sz(), np.complex64) for _ in range(2)]
    for seed in (1, 2):
        pageable = spectrum(n, seed).astype(np.complex64)
        pinned[:] = pageable
        keep.array[0] = keep.array[n + 1] = np.nan
        got = []
        for x, t in ((pageable, tiles[0]), (pinned, tiles[1])):
            assert p.launch(x, thr, loc, pwr, FDAS.AllAccelerations, FDAS.A) and p.wait(FDAS.A)
            assert p.retrieve_tiles(t, FDAS.A)
            got.append(p.retrieve_candidate_list(FDAS.A)[0])
        assert np.array_equal(tiles[0], tiles[1]) and np.array_equal(got[0], got[1]) and got[0].size
        # the stages after a launch read the copy, whatever became of the caller's array
        pinned[:] = np.nan
        assert p.perform_harmonic_summing(thr, FDAS.AllAccelerations, FDAS.A)
        assert np.array_equal(p.retrieve_candidate_list(FDAS.A)[0], got[0])
    # with both sets in use the spectrum is copied
    pinned[:] = pageable
    for ab in (FDAS.B, FDAS.A):
        assert p.launch(pinned, thr, loc, pwr, FDAS.AllAccelerations, ab) and p.wait(ab)
        assert np.array_equal(p.retrieve_candidate_list(ab)[0], got[0])
