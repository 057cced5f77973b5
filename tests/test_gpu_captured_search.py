"""A search of a device spectrum captured into a graph: replays search the
spectrum that is there then, and the other set's searches go on as before."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300 import synth
from fdas_gb300.fdas import FDAS
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,planes", [(4096, 8), (20000, 16)])
def test_captured_device_search(n, planes):
    import torch
    thr = O.chi2_thresholds(1e-5, planes)
    p = make_pipeline(n, log=io.StringIO(), n_planes=planes)
    for ab in (FDAS.A, FDAS.B):
        assert p.upload_templates(template_bank(), ab)
    xs = [synth.spectrum(synth.timeseries(2 * n, [dict(r0=0.3 * n, z=8.0 * s, n_harm=3, amp=0.1)], seed=s))[0]
          for s in (1, 2, 3)]
    d = torch.empty(2 * n, dtype=torch.float32, device="cuda")

    def put(i):
        d.copy_(torch.from_numpy(xs[i].view(np.float32)))
        torch.cuda.synchronize()

    def results(ab):
        assert p.synchronize(ab), p.last_error
        nc = p.get_candidate_list_sz()
        loc, pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
        assert p.retrieve_candidates(loc, pwr, ab)
        rec, total, dropped = p.retrieve_candidate_list(ab)
        assert dropped == 0 and rec.size
        return loc, pwr, rec

    want = []
    for i in range(3):  # (both sets in use before the capture)
        put(i)
        for ab in (FDAS.A, FDAS.B):
            assert p.enqueue_search_device(d.data_ptr(), thr, FDAS.AllAccelerations, ab), p.last_error
            assert p.synchronize(ab)
        want.append(results(FDAS.B))
    stream = torch.cuda.ExternalStream(p.stream(FDAS.A))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        assert p.enqueue_search_device(d.data_ptr(), thr, FDAS.AllAccelerations, FDAS.A), p.last_error
    for i in (0, 1, 0):
        put(i)
        for _ in range(2):  # (a replay follows a replay: the control words start from zero each time)
            with torch.cuda.stream(stream):
                g.replay()
        for got, ref in zip(results(FDAS.A), want[i]):
            assert np.array_equal(got, ref)
    # the other set: a spectrum in host memory
    nc = p.get_candidate_list_sz()
    loc, pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
    assert p.launch(xs[2], thr, loc, pwr, FDAS.AllAccelerations, FDAS.B), p.last_error
    assert p.wait(FDAS.B)
    assert np.array_equal(loc, want[2][0]) and np.array_equal(pwr, want[2][1])
    # and a plain search on the captured one
    put(2)
    assert p.enqueue_search_device(d.data_ptr(), thr, FDAS.AllAccelerations, FDAS.A), p.last_error
    for got, ref in zip(results(FDAS.A), want[2]):
        assert np.array_equal(got, ref)
