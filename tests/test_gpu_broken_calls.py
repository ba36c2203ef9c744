"""Calls of several steps that break off: a step graph that cannot be built
(the first one, or the one the call needs later) or launched.  The failures
are made on the host (SCGPU_FAIL_GRAPH / SCGPU_FAIL_LAUNCH = k: the k-th build
or launch of the object counts as refused).  The bunch must then be in the
state after whole steps, and later calls must give the bits of a context that
never failed."""
import numpy as np
import pytest

from src_b200.bunch import gaussian_bunch, photoinjector_bunch

pytestmark = pytest.mark.gpu

MASS = 0.51099892e6
DT = 1e-12
N = 4001

# (variable, k, whole steps of a call of 9 with a reorder at steps 0 and 4):
# the first graph is the reorder's, the second the plain steps'.  A launch
# that fails after the first of its run is made up for by one step without a graph
FAILURES = [("SCGPU_FAIL_GRAPH", 1, 0), ("SCGPU_FAIL_GRAPH", 2, 1), ("SCGPU_FAIL_LAUNCH", 1, 0),
            ("SCGPU_FAIL_LAUNCH", 2, 1), ("SCGPU_FAIL_LAUNCH", 3, 3), ("SCGPU_FAIL_LAUNCH", 9, 9)]


def _bunch(kind):
    if kind == "bins":
        return photoinjector_bunch(N, nbins=3)
    return (*gaussian_bunch(N, bunch_id=6), None)


def _context(gpu, kind, monkeypatch, failure=None):
    R, P, bins = _bunch(kind)
    if failure:
        monkeypatch.setenv(failure[0], str(failure[1]))
    c = gpu.Context((16, 16, 16), precision=gpu.MIXED if kind == "mixed" else gpu.PLAIN_FP64)
    if failure:
        monkeypatch.delenv(failure[0])
    c.set_reorder_interval(4)
    c.upload(R, P, DT, -1e-9 / N, MASS)
    if bins is not None:
        c.set_energy_bins(bins, 3)
    return c


def _same(c, w):
    for a, b in zip(c.download(), w.download()):
        np.testing.assert_array_equal(a, b)
    s, t = c.tracker_state(), w.tracker_state()
    assert s["step"] == t["step"] and s["path_length"] == t["path_length"] and s["t"] == t["t"]


@pytest.mark.parametrize("kind", ["plain", "mixed", "bins"])
@pytest.mark.parametrize("failure", FAILURES, ids=lambda f: f"{f[0][11:].lower()}{f[1]}")
def test_track_that_breaks_off(gpu, kind, failure, monkeypatch):
    with _context(gpu, kind, monkeypatch, failure) as c, _context(gpu, kind, monkeypatch) as w:
        with pytest.raises(gpu.ScgpuError) as e:
            c.track(9)
        assert e.value.code == -6
        if failure[2]:
            w.track(failure[2])
        _same(c, w)
        np.testing.assert_array_equal(c.beam_parameters()["moments"], w.beam_parameters()["moments"])
        # a call of one step, one with a record, and one that hands positions on
        s, t = np.zeros((2, 1, gpu.NSTATS))
        for x, rec in ((c, s), (w, t)):
            x.track(1)
            x.track(1, rec)
        np.testing.assert_array_equal(s, t)
        _same(c, w)
        c.track(6)
        w.track(6)
        _same(c, w)


# whole steps of a round of 20 after one of 1 (the batch reorders at steps 0
# and 16, the first round after a change of members runs without graphs)
BATCH_FAILURES = [("SCGPU_FAIL_GRAPH", 1, 0), ("SCGPU_FAIL_GRAPH", 2, 15), ("SCGPU_FAIL_LAUNCH", 1, 0),
                  ("SCGPU_FAIL_LAUNCH", 2, 2), ("SCGPU_FAIL_LAUNCH", 16, 15), ("SCGPU_FAIL_LAUNCH", 17, 17)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("failure", BATCH_FAILURES, ids=lambda f: f"{f[0][11:].lower()}{f[1]}")
def test_batch_round_that_breaks_off(gpu, precision, failure, monkeypatch):
    def batch(fail):
        if fail:
            monkeypatch.setenv(fail[0], str(fail[1]))
        b = gpu.Batch(precision=precision)
        if fail:
            monkeypatch.delenv(fail[0])
        for i, (n, m) in enumerate([(N, 16), (700, 20)]):
            R, P = gaussian_bunch(n, bunch_id=i)
            b.add((m, m, m), R, P, DT, -1e-10 / n, MASS)
        b.track(1)
        return b

    def same(b, w):
        for slot in range(2):
            _same(b.member(slot), w.member(slot))

    with batch(failure) as b, batch(None) as w:
        with pytest.raises(gpu.ScgpuError) as e:
            b.track(20)
        assert e.value.code == -6
        b.wait()
        if failure[2]:
            w.track(failure[2])
        same(b, w)
        for x in (b, w):
            x.track(1)
        same(b, w)
        b.launch(6)
        b.wait()
        w.track(6)
        same(b, w)
