"""Kernels of one search start on the tail of the one before, and the tiling
zeroes the search's control words for all of them.  Repeated and alternating
searches, stage calls in between, a refused call and a captured call give what
they gave with every kernel on its own."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300 import _lib, synth
from fdas_gb300.fdas import FDAS
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


def spectrum(n, seed):
    return synth.spectrum(synth.timeseries(2 * n, [dict(r0=0.3 * n, z=8.0 * seed, n_harm=3, amp=0.1)], seed=seed))[0]


def handle(n):
    p = make_pipeline(n, log=io.StringIO())
    for ab in (FDAS.A, FDAS.B):
        assert p.upload_templates(template_bank(), ab)
    return p


def stages(p, x, thr, ab):
    assert p.perform_input_tiling(x, ab) and p.perform_ft_convolution(FDAS.AllAccelerations, ab)
    assert p.perform_harmonic_summing(thr, FDAS.AllAccelerations, ab), p.last_error
    return p.retrieve_candidate_list(ab)


def test_chained_searches_equal_stage_calls():
    n, thr = 9001, O.chi2_thresholds(1e-5, 8)
    xs = [spectrum(n, s) for s in (1, 2, 3, 4)]
    want = [stages(handle(n), x, thr, FDAS.A)[0] for x in xs]
    p = handle(n)
    nc = p.get_candidate_list_sz()
    out = [(np.zeros(nc, np.uint32), np.zeros(nc, np.float32)) for _ in range(2)]
    for rep in range(6):  # both sets in flight, every set's words zeroed by its own next search
        for ab in (FDAS.A, FDAS.B):
            assert p.launch(xs[(2 * rep + ab) % 4], thr, *out[ab], FDAS.AllAccelerations, ab)
        for ab in (FDAS.A, FDAS.B):
            assert p.wait(ab)
            rec, total, dropped = p.retrieve_candidate_list(ab)
            ref = want[(2 * rep + ab) % 4]
            assert dropped == 0 and np.array_equal(rec, ref)
        rec = stages(p, xs[rep % 4], thr, FDAS.A)[0]
        assert np.array_equal(rec, want[rep % 4])


def test_refused_search_leaves_the_list():
    import torch
    n, thr = 5000, O.chi2_thresholds(1e-5, 8)
    p = handle(n)
    rec = stages(p, spectrum(n, 2), thr, FDAS.A)[0]
    assert rec.size
    x = torch.from_numpy(spectrum(n, 3).view(np.float32)).cuda()
    st = p._lib.fdas_enqueue_search_device(p._h, x.data_ptr(), None, int(FDAS.AllAccelerations), int(FDAS.A))
    assert st == _lib.ERR_STATE  # no thresholds given or uploaded
    torch.cuda.synchronize()
    again, total, dropped = p.retrieve_candidate_list(FDAS.A)
    assert np.array_equal(again, rec) and dropped == 0


def test_noalloc_in_a_graph():
    import torch
    lib = _lib.load()
    n = 12345
    bank = np.fft.fft(template_bank().astype(np.complex128), 2048, axis=1).astype(np.complex64)
    d_t = torch.from_numpy(bank.view(np.float32)).cuda()
    d_x = torch.from_numpy(spectrum(n, 1).view(np.float32)).cuda()
    plain, graphed = (torch.zeros((85, n), dtype=torch.float32, device="cuda") for _ in range(2))

    def call(out):
        return lib.fdas_ft_convolution_noalloc(d_x.data_ptr(), n, d_t.data_ptr(), int(FDAS.TemplatesFFTNatural), 85, 420,
                                               int(FDAS.AllAccelerations), out.data_ptr(), n, None,
                                               torch.cuda.current_stream().cuda_stream)

    assert call(plain) == _lib.OK
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert call(graphed) == _lib.OK
    d_x.copy_(torch.from_numpy(spectrum(n, 4).view(np.float32)))
    g.replay()
    torch.cuda.synchronize()
    assert call(plain) == _lib.OK
    torch.cuda.synchronize()
    assert torch.equal(plain, graphed)


@pytest.mark.parametrize("pins", [(True, True), (True, False), (False, True), (False, False)])
def test_list_into_pinned_and_pageable_arrays(pins):
    """The selection writes pinned arrays itself, others are copied to: the same list."""
    from fdas_gb300.fdas import PinnedArray
    n, thr = 20000, O.chi2_thresholds(1e-4, 8)
    p = handle(n)
    nc = p.get_candidate_list_sz()
    keep = [PinnedArray((nc,), d) if pin else None for pin, d in zip(pins, (np.uint32, np.float32))]
    loc, pwr = (k.array if k else np.empty(nc, d) for k, d in zip(keep, (np.uint32, np.float32)))
    loc[:], pwr[:] = 7, 7
    for seed in (1, 2):
        assert p.launch(spectrum(n, seed), thr, loc, pwr, FDAS.AllAccelerations, FDAS.A) and p.wait(FDAS.A)
        want_loc, want_pwr = np.zeros(nc, np.uint32), np.zeros(nc, np.float32)
        assert p.retrieve_candidates(want_loc, want_pwr, FDAS.A)
        assert np.array_equal(loc, want_loc) and np.array_equal(pwr, want_pwr)
        ms = p.stage_times(FDAS.A)
        assert (ms >= 0).all() and ms[1] > 0 and ms[2] > 0 and ms[3] > 0 and ms[:5].sum() <= ms[5] + 0.05
