"""fdas_series_to_spectrum waits for its own buffer set's stream only."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS

pytestmark = pytest.mark.gpu


def test_new_length_does_not_wait_for_other_streams():
    import torch
    n, shorter = 65536, 50000
    rng = np.random.default_rng(5)
    samples = torch.from_numpy(rng.standard_normal(2 * n).astype(np.float32)).cuda()
    want = np.zeros(shorter, np.complex64)
    ref = make_pipeline(shorter, log=io.StringIO())  # (also loads the kernels)
    assert ref.series_to_spectrum(samples, FDAS.A, spectrum=want)
    p = make_pipeline(n, log=io.StringIO())
    assert p.series_to_spectrum(samples, FDAS.A)
    assert p.reshape(shorter)
    got = np.zeros(shorter, np.complex64)
    other, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(600_000_000)  # about 0.3 s
        done.record()
    assert p.series_to_spectrum(samples, FDAS.B, spectrum=got)
    assert not done.query()
    torch.cuda.synchronize()
    assert np.array_equal(got, want)
