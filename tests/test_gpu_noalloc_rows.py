"""The allocation-free FT convolution brings the template rows of its sign half into
the kernels' form beside the tiling: every half and layout, one tile and several,
one to the most rows, equal to the same call on both halves, and rows outside the
half are left alone."""
import numpy as np
import pytest

from fdas_gb300 import _lib
from fdas_gb300.fdas import FDAS
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,t", [(5, 1), (1628, 3), (1629, 85), (9001, 43), (20000, 127)])
def test_halves_and_layouts(n, t):
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(n + t)
    spec = (rng.standard_normal((t, 2048)) + 1j * rng.standard_normal((t, 2048))).astype(np.complex64)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.float32)).cuda()
    x = dev((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64))
    bank = {FDAS.TemplatesFFTNatural: dev(spec), FDAS.TemplatesFFTP4: dev(O.to_p4(spec))}

    def call(layout, part):
        out = torch.full((t, n), -3.0, dtype=torch.float32, device="cuda")
        st = lib.fdas_ft_convolution_noalloc(x.data_ptr(), n, bank[layout].data_ptr(), int(layout), t, 420, int(part),
                                             out.data_ptr(), n, None, torch.cuda.current_stream().cuda_stream)
        assert st == _lib.OK
        torch.cuda.synchronize()
        return out.cpu().numpy()

    every = call(FDAS.TemplatesFFTNatural, FDAS.AllAccelerations)
    # |overlap-save convolution|^2 of the first tile in FP64; the FOP's bound
    # (1e-5 of the row's mean power + 1e-6 of the cell's)
    pad = np.zeros(2048, dtype=np.complex128)
    m = min(n, 1628)
    pad[420:420 + m] = x.cpu().numpy().view(np.complex64)[:m]
    y = np.fft.ifft(np.fft.fft(pad) * spec.astype(np.complex128), axis=1)[:, 420:420 + m]
    want = np.abs(y) ** 2
    assert (np.abs(every[:, :m] - want) <= 1e-5 * want.mean(axis=1, keepdims=True) + 1e-6 * want).all()
    h = t // 2
    for layout in bank:
        assert np.array_equal(call(layout, FDAS.AllAccelerations), every)
        neg, pos = call(layout, FDAS.NegativeAccelerations), call(layout, FDAS.PositiveAccelerations)
        assert np.array_equal(neg[:h + 1], every[:h + 1]) and (neg[h + 1:] == -3.0).all()
        assert np.array_equal(pos[h:], every[h:]) and (pos[:h] == -3.0).all()
