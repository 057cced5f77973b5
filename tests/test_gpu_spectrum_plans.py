"""Series FFT over the plans its lengths get (one to several passes of composite
radix, ragged last columns, every small radix), from host memory, device memory
and device memory that is not aligned to a pair of samples, and after a reshape;
against FP64 with the tolerance of the spectrum tests."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS
from test_gpu_spectrum import SPEC_TOL

pytestmark = pytest.mark.gpu


def check(x, s, n):
    exact = np.fft.fft(s[:2 * n].astype(np.float64))[:n]
    rms = np.sqrt(np.mean(np.abs(exact) ** 2))
    assert np.abs(x - exact).max() <= SPEC_TOL * rms * max(1.0, np.log2(max(n, 2)) / 11)


@pytest.mark.parametrize("n", [2, 3, 5, 6, 16, 49, 512, 525, 1024, 2187, 16807, 32768, 59049,
                               65536, 117649, 390625, 786432, 1000000])
def test_plans(n):
    import torch
    s = np.random.default_rng(n).standard_normal(2 * n + 1).astype(np.float32)
    p = make_pipeline(n, log=io.StringIO(), n_templates=3)
    out = np.zeros(n, dtype=np.complex64)
    assert p.series_to_spectrum(s, FDAS.A, scale=1.0, spectrum=out), p.last_error
    check(out, s, n)
    d = torch.from_numpy(s).cuda()
    dev = np.zeros(n, dtype=np.complex64)
    assert p.series_to_spectrum(d, FDAS.B, scale=1.0, spectrum=dev), p.last_error
    assert np.array_equal(out, dev)
    assert torch.equal(d.cpu(), torch.from_numpy(s))  # the caller's samples are only read
    odd = torch.empty(2 * n + 2, dtype=torch.float32, device="cuda")[1:]
    odd.copy_(d)
    assert odd.data_ptr() % 8 == 4
    assert p.series_to_spectrum(odd, FDAS.A, scale=1.0, spectrum=dev), p.last_error
    assert np.array_equal(out, dev)


def test_after_reshape():
    n = 9000
    s = np.random.default_rng(3).standard_normal(2 * n).astype(np.float32)
    p = make_pipeline(n, log=io.StringIO(), n_templates=3)
    for m in (9000, 4096, 9000):
        assert p.reshape(m), p.last_error
        out = np.zeros(m, dtype=np.complex64)
        assert p.series_to_spectrum(s, FDAS.A, scale=1.0, spectrum=out), p.last_error
        check(out, s, m)


# every step size (2 to 10, 12, 14 to 16) first, in between and last, ragged last columns,
# and both sides of the two-pass range
@pytest.mark.parametrize("n", [4, 7, 9, 10, 12, 14, 15, 36, 81, 90, 196, 210, 225, 343, 1890, 30870, 50625, 63504, 100000,
                               157464, 262144, 540225, 655360, 656100, 1048576, 1049760])
def test_step_sizes(n):
    s = np.random.default_rng(n).standard_normal(2 * n).astype(np.float32)
    p = make_pipeline(n, log=io.StringIO(), n_templates=3)
    out = np.zeros(n, dtype=np.complex64)
    assert p.series_to_spectrum(s, FDAS.A, scale=1.0, spectrum=out), p.last_error
    check(out, s, n)


@pytest.mark.parametrize("n", [1, 2, 3, 77 * 25 * 4 // 11, 4096, 30870])
def test_spectrum_into_pinned_memory(n):
    """The last kernel writes a pinned array itself, others are copied to: the same spectrum,
    and nothing next to it."""
    from fdas_gb300.fdas import PinnedArray
    s = np.random.default_rng(n).standard_normal(2 * n).astype(np.float32)
    p = make_pipeline(n, log=io.StringIO(), n_templates=3)
    want = np.zeros(n, dtype=np.complex64)
    assert p.series_to_spectrum(s, FDAS.A, scale=1.0, spectrum=want), p.last_error
    keep = PinnedArray((n + 2,), np.complex64)
    keep.array[:] = 7
    assert p.series_to_spectrum(s, FDAS.B, scale=1.0, spectrum=keep.array[1:n + 1]), p.last_error
    assert np.array_equal(keep.array[1:n + 1], want) and keep.array[0] == 7 and keep.array[n + 1] == 7
    raw = PinnedArray((8 * n + 8,), np.uint8)
    shifted = raw.array[4:8 * n + 4].view(np.complex64)  # not aligned for whole stores
    assert shifted.ctypes.data % 8 == 4
    assert p.series_to_spectrum(s, FDAS.A, scale=1.0, spectrum=shifted), p.last_error
    assert np.array_equal(shifted, want)
