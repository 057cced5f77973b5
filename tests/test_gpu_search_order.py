"""Order between the two buffer sets' searches, read from their event times."""
import io

import numpy as np
import pytest

from gpu_util import make_pipeline
from fdas_gb300.fdas import FDAS
from fdas_gb300.templates import template_bank
from oracle import fdas_oracle as O

pytestmark = pytest.mark.gpu

N = 1 << 20  # an FT convolution of about 150 us, several times the time to enqueue a search
FIELDS = ("in_begin", "in_end", "tile_begin", "tile_end", "ftc_begin", "ftc_end", "hsum_begin", "hsum_end",
          "list_begin", "list_end")


def noise(seed):
    rng = np.random.default_rng(seed)
    return ((rng.standard_normal(N) + 1j * rng.standard_normal(N)) * np.sqrt(0.5)).astype(np.complex64)


def handle(log, **kw):
    p = make_pipeline(N, log=log, **kw)
    for ab in (FDAS.A, FDAS.B):
        assert p.upload_templates(template_bank(), ab)
    return p


def events(p, log, ab):
    at = len(log.getvalue())
    p.print_events(ab)
    line = [s for s in log.getvalue()[at:].splitlines() if s.startswith("@@@")][-1]
    return dict(zip(FIELDS, (int(v) for v in line.split(",")[2:])))


@pytest.mark.parametrize("order", [(FDAS.A, FDAS.B), (FDAS.B, FDAS.A)])
def test_device_searches_under_sync_pipeline(order):
    """sync_pipeline: the tiling of one set waits for the other's FT convolution, for
    searches of device spectra as for launches."""
    import torch
    log, thr = io.StringIO(), O.chi2_thresholds(1e-7, 8)
    p = handle(log, sync_pipeline=True)
    x = torch.from_numpy(noise(1).view(np.float32)).cuda()
    torch.cuda.synchronize()
    for rep in range(3):
        for ab in order:
            assert p.enqueue_search_device(x.data_ptr(), thr, FDAS.AllAccelerations, ab), p.last_error
        for ab in order:
            assert p.synchronize(ab)
    first, second = (events(p, log, ab) for ab in order)
    assert second["tile_begin"] >= first["ftc_end"] - 1000  # (ns; the times are floats in ms)


def launched(p, xs, outs, thr, order):
    for x, (loc, pwr), ab in zip(xs, outs, order):
        assert p.launch(x.array, thr, loc.array, pwr.array, FDAS.AllAccelerations, ab), p.last_error
    for ab in order:
        assert p.wait(ab)


def host_arrays(p, count):
    from fdas_gb300.fdas import PinnedArray
    nc = p.get_candidate_list_sz()
    xs = [PinnedArray((N,), np.complex64) for _ in range(count)]
    for i, x in enumerate(xs):
        x.array[:] = noise(i)
    return xs, [(PinnedArray((nc,), np.uint32), PinnedArray((nc,), np.float32)) for _ in range(count)]


def test_stage_times_of_a_search_that_waits():
    """The second of two launches waits for the first: its harmonic summing, which runs
    by itself, takes as long as a lone search's, and its stages fill its total."""
    log, thr = io.StringIO(), O.chi2_thresholds(1e-7, 8)
    p = handle(log)
    xs, outs = host_arrays(p, 2)
    for _ in range(2):
        launched(p, xs, outs, thr, (FDAS.A, FDAS.B))
    lone, both = [], []
    for _ in range(5):
        launched(p, xs[1:], outs[1:], thr, (FDAS.B,))
        lone.append(p.stage_times(FDAS.B))
        launched(p, xs, outs, thr, (FDAS.A, FDAS.B))
        both.append(p.stage_times(FDAS.B))
        assert abs(both[-1][:5].sum() - both[-1][5]) < 0.005
    last, lone, both = both[-1], np.median(lone, axis=0), np.median(both, axis=0)
    print(lone, both)
    assert lone[1] < 0.5 * lone[2] and lone[3] > 0  # (tiling is a tenth of the FT convolution)
    assert both[2] > 0.9 * lone[2]
    assert both[3] < 1.25 * lone[3] + 0.01
    at = events(p, log, FDAS.B)
    assert list(at.values()) == sorted(at.values())
    assert abs(1e-6 * (at["hsum_end"] - at["hsum_begin"]) - last[3]) < 0.001


@pytest.mark.parametrize("order", [(FDAS.A, FDAS.B), (FDAS.B, FDAS.A)])
def test_first_launch_on_the_second_set(order):
    """The FT convolution of a host spectrum waits for the other set's harmonic summing
    from the first launch on the second set on: it ends a whole FT convolution later."""
    log, thr = io.StringIO(), O.chi2_thresholds(1e-7, 8)
    for _ in range(2):  # (the first handle loads the kernels)
        p = handle(log)
        xs, outs = host_arrays(p, 2)
        launched(p, xs[:1], outs[:1], thr, order[:1])
        lone = events(p, log, order[0])
        launched(p, xs, outs, thr, order)
        first, second = (events(p, log, ab) for ab in order)
        p.close()
    assert second["ftc_end"] - first["hsum_end"] >= 0.8 * (lone["ftc_end"] - lone["ftc_begin"])


def queued_times(p, x, thr):
    """Stage times of a search queued behind others on its set, so that the host's
    part of a launch is in none of them; the median of five."""
    times = []
    for _ in range(5):
        for _ in range(3):
            assert p.enqueue_search_device(x.data_ptr(), thr, FDAS.AllAccelerations, FDAS.A), p.last_error
        assert p.synchronize(FDAS.A)
        times.append(p.stage_times(FDAS.A))
    return np.median(times, axis=0)


@pytest.mark.parametrize("quantile", [1e-4, 1e-2])
def test_stages_of_searches_with_many_hits(quantile):
    """Tiling and FT convolution take what they take, however long the selection of
    the hits does."""
    import torch
    p = make_pipeline(N, log=io.StringIO(), candidate_capacity=1 << 24)
    assert p.upload_templates(template_bank(), FDAS.A)
    x = torch.from_numpy(noise(3).view(np.float32)).cuda()
    torch.cuda.synchronize()
    few, many = (queued_times(p, x, O.chi2_thresholds(q, 8)) for q in (1e-7, quantile))
    print(few, many)
    assert many[3] > 1.5 * few[3]
    assert abs(many[1] - few[1]) < 0.008 and abs(many[2] - few[2]) < 0.1 * few[2]


def test_stages_of_the_pipelined_mode():
    """The pair form of the FT convolution, which the pipelined mode takes: tiling is a
    twentieth of it, and the stages fill the search."""
    import torch
    p = handle(io.StringIO(), overlap=True)
    x = torch.from_numpy(noise(1).view(np.float32)).cuda()
    torch.cuda.synchronize()
    ms = queued_times(p, x, O.chi2_thresholds(1e-7, 8))
    print(ms)
    assert 0 < ms[1] < 0.5 * ms[2] and 0.05 < ms[3] < ms[2]
    assert abs(ms[:5].sum() - ms[5]) < 0.005
