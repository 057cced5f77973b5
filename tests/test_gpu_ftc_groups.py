"""FT convolution at the edges of its work split: eight tiles per group and the
(group, row) steps dealt evenly to the CTAs, so groups are entered and left in
the middle of the bank, last groups are ragged, and tiles end inside the row.
The FOP is compared with the FP64 oracle under the tolerance of the parity
tests."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from test_gpu_parity import fop_within
from fdas_gb300.fdas import FDAS
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu


def noise(n, seed):
    rng = np.random.default_rng(seed)
    return ((rng.standard_normal(n) + 1j * rng.standard_normal(n)) / np.sqrt(2)).astype(np.complex64)


@pytest.mark.parametrize("rows,overlap,tiles,tail,part", [
    (85, 420, 7, 0, FDAS.AllAccelerations),       # less than a group
    (85, 420, 8, 1, FDAS.PositiveAccelerations),  # one group and a tile of one bin
    (85, 420, 24, -5, FDAS.AllAccelerations),     # whole groups, ragged last tile
    (43, 420, 33, 700, FDAS.NegativeAccelerations),
    (85, 600, 9, 0, FDAS.AllAccelerations),       # overlap above 512: no unconditional stores
    (25, 128, 9, 17, FDAS.AllAccelerations),      # overlap below 256: the first outputs are kept
    (1, 420, 17, 0, FDAS.AllAccelerations),       # one row: every step is a new group
    (3, 420, 50, 3, FDAS.AllAccelerations),       # a ring deeper than the rows
])
def test_fop_at_group_edges(rows, overlap, tiles, tail, part):
    first = (85 - rows) // 2
    bank = template_bank()[first:first + rows]
    taps = max(int(np.count_nonzero(r)) for r in bank)
    bank = np.ascontiguousarray(bank[:, :max(taps, 1)])
    n = tiles * (2048 - overlap) + tail
    x = noise(n, 100 + tiles)
    p = make_pipeline(n, log=io.StringIO(), n_templates=rows, max_template_len=bank.shape[1], tile_overlap=overlap)
    assert p.upload_templates(bank, FDAS.A, layout=FDAS.TemplatesTimeDomain), p.last_error
    assert p.perform_input_tiling(x, FDAS.A) and p.perform_ft_convolution(part, FDAS.A), p.last_error
    fop = np.zeros(p.get_fop_sz(), dtype=np.float32)
    assert p.retrieve_FOP(fop, FDAS.A)
    fop = fop.reshape(rows, n)
    half = rows // 2
    done = {FDAS.NegativeAccelerations: np.arange(half + 1), FDAS.PositiveAccelerations: np.arange(half, rows),
            FDAS.AllAccelerations: np.arange(rows)}[part]
    assert fop_within(fop[done], O.fop(x, bank, rows=done)).all()
    assert np.all(np.delete(fop, done, axis=0) == 0)
