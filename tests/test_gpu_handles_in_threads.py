"""Handles of different sizes used by one thread each at the same time."""
import io
import threading

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


def run_together(jobs, calls):
    """Each job `calls` times in a thread of its own; the number of calls that failed."""
    failed, start = [0] * len(jobs), threading.Barrier(len(jobs))

    def work(i):
        start.wait()
        for _ in range(calls):
            failed[i] += not jobs[i]()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return failed


def test_series_of_different_lengths():
    """The passes of 2^20 points take several times the shared memory of 4096 points'."""
    import torch
    jobs, check = [], []
    for n in (1 << 20, 4096):
        s = torch.from_numpy(np.random.default_rng(n).standard_normal(2 * n).astype(np.float32)).cuda()
        p = make_pipeline(n, log=io.StringIO(), n_templates=3, max_template_len=5, n_planes=1)
        want, got = np.zeros(n, np.complex64), np.zeros(n, np.complex64)
        assert p.series_to_spectrum(s, FDAS.A, spectrum=want)
        jobs.append(lambda p=p, s=s: p.series_to_spectrum(s, FDAS.A))
        check.append((p, s, got, want))
    assert run_together(jobs, 2000) == [0, 0]
    for p, s, got, want in check:
        assert p.series_to_spectrum(s, FDAS.A, spectrum=got) and np.array_equal(got, want)


def test_searches_of_different_planes():
    """Two planes' boxes and histograms take less shared memory than eight planes'."""
    import torch
    n, jobs, check = 4096, [], []
    x = torch.from_numpy(np.random.default_rng(7).standard_normal(2 * n).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    for planes in (8, 2):
        p = make_pipeline(n, log=io.StringIO(), n_planes=planes)
        assert p.upload_templates(template_bank(), FDAS.A)
        thr = O.chi2_thresholds(1e-4, planes)

        def search(p=p, thr=thr):
            return p.enqueue_search_device(x.data_ptr(), thr, FDAS.AllAccelerations, FDAS.A) and p.synchronize(FDAS.A)

        assert search()
        jobs.append(search)
        check.append((p, search, p.retrieve_candidate_list(FDAS.A)[0]))
    assert run_together(jobs, 2000) == [0, 0]
    for p, search, want in check:
        assert search() and np.array_equal(p.retrieve_candidate_list(FDAS.A)[0], want)
