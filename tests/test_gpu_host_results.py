"""The selection's kernels write the list and the first records into host memory;
retrievals beyond that, of other arrays, and after stage calls read the device's."""
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
    return synth.spectrum(synth.timeseries(2 * n, [], seed=seed))[0]


def handle(n):
    p = make_pipeline(n, log=io.StringIO())
    assert p.upload_templates(template_bank(), FDAS.A)
    return p


def device_list(p, rec, nc):
    """The fixed-size list of the search, one entry per record where the record is in it."""
    loc, pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
    assert p.retrieve_candidates(loc, pwr, FDAS.A)
    by_loc = dict(zip(O.encode_location(rec["harmonic"], rec["template_num"], rec["bin"]).tolist(), rec["power"]))
    keep = loc != O.INVALID_LOCATION
    assert all(by_loc[l] == w for l, w in zip(loc[keep].tolist(), pwr[keep]))
    return loc, pwr


# false alarms of 85 * 8 * n cells: a few, some below and some above 4096 records
@pytest.mark.parametrize("p_false", [1e-6, 5e-4, 3e-3])
def test_records_and_lists(p_false):
    n, thr = 6000, O.chi2_thresholds(p_false, 8)
    p = handle(n)
    nc = p.get_candidate_list_sz()
    a, b = spectrum(n, 1), spectrum(n, 2)
    for x in (a, b, a):
        # arrays of pageable memory, then pinned ones, then stage calls
        loc, pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
        assert p.launch(x, thr, loc, pwr, FDAS.AllAccelerations, FDAS.A) and p.wait(FDAS.A)
        rec, total, dropped = p.retrieve_candidate_list(FDAS.A)
        assert total == rec.size + dropped and dropped == 0
        got = device_list(p, rec, nc)
        assert np.array_equal(got[0], loc) and np.array_equal(got[1], pwr)
        keep = [PinnedArray((nc,), d) for d in (np.uint32, np.float32)]
        assert p.launch(x, thr, keep[0].array, keep[1].array, FDAS.AllAccelerations, FDAS.A) and p.wait(FDAS.A)
        again = device_list(p, rec, nc)
        assert np.array_equal(again[0], loc) and np.array_equal(again[1], pwr)
        assert np.array_equal(keep[0].array, loc) and np.array_equal(keep[1].array, pwr)
        # the list stays that of the last harmonic summing while the next stages run
        other = b if x is a else a
        assert p.perform_input_tiling(other, FDAS.A)
        again = device_list(p, rec, nc)
        assert np.array_equal(again[0], loc) and np.array_equal(again[1], pwr)
        assert p.perform_ft_convolution(FDAS.AllAccelerations, FDAS.A)
        assert np.array_equal(p.retrieve_candidate_list(FDAS.A)[0], rec)
        assert p.perform_input_tiling(x, FDAS.A) and p.perform_ft_convolution(FDAS.AllAccelerations, FDAS.A)
        assert p.perform_harmonic_summing(thr, FDAS.AllAccelerations, FDAS.A)
        assert np.array_equal(p.retrieve_candidate_list(FDAS.A)[0], rec)
        again = device_list(p, rec, nc)
        assert np.array_equal(again[0], loc) and np.array_equal(again[1], pwr)
        if p_false == 3e-3:
            assert rec.size > 4096
        few, total, _ = p.retrieve_candidate_list(FDAS.A, capacity=5)
        assert total == rec.size and np.array_equal(few, rec[:5])
