"""The step's particle kernels where their work is cut: particle counts around
the warp, chunk and block edges, the exact sums' range switch at |P| = 1024,
weights of exactly 1 in the mixed deposit, and the first half drift handed from
one step of a call to the next (one call of n steps must leave the bits of n
calls of one step)."""
import numpy as np
import pytest

from src_b200.bunch import dc_bunch, gaussian_bunch, photoinjector_bunch

pytestmark = pytest.mark.gpu

MASS = 0.51099892e6
DT = 1e-12
TOL = 1e-12  # the repository's bound against the oracle (norm-wise)


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("n", [2, 31, 33, 64, 65, 255, 257, 1023])
def test_particle_counts_vs_oracle(gpu, n):
    from oracle import oracle as O

    nr = (16, 15, 12)
    R, P = gaussian_bunch(n, bunch_id=7)
    Ro, Po = R.copy(), P.copy()
    with O.exact():
        tr = O.OracleTracker(O.make_params(nr, DT), -1e-12 / n)
        tr.track(Ro, Po, 3)
    with gpu.Context(nr) as c:
        c.upload(R, P, DT, -1e-12 / n, O.electron_mass_ev())
        c.track(3)
        Rg, Pg = c.download()
    assert _rel(Rg, Ro) <= TOL and _rel(Pg, Po) <= TOL


@pytest.mark.parametrize("bg", [1024.0, 3000.0])
def test_large_momenta_vs_oracle(gpu, bg):
    """A bunch across and above |P| = 1024, where the exact momentum sums change accumulators."""
    from oracle import oracle as O

    nr = (16, 16, 16)
    R, P = gaussian_bunch(3000, bg_z=bg, rel_spread=1e-2, bunch_id=3)
    Ro, Po = R.copy(), P.copy()
    with O.exact():
        tr = O.OracleTracker(O.make_params(nr, DT, ref_pz=bg), -1e-13)
        tr.track(Ro, Po, 3)
    with gpu.Context(nr) as c:
        c.upload(R, P, DT, -1e-13, O.electron_mass_ev(), ref_P=(0.0, 0.0, bg))
        c.track(3)
        Rg, Pg = c.download()
        gz = c.mesh()["gammaz"]
        c.upload(R, P, DT, -1e-13, O.electron_mass_ev(), ref_P=(0.0, 0.0, bg))
        c.track(1)
        c.track(2)
        Rs, Ps = c.download()
        assert c.mesh()["gammaz"] == gz
    assert _rel(Rg, Ro) <= TOL and _rel(Pg, Po) <= TOL
    np.testing.assert_array_equal(Rg, Rs)
    np.testing.assert_array_equal(Pg, Ps)


@pytest.mark.parametrize("n", [64, 200])
def test_mixed_deposit_full_weights(gpu, n):
    """n particles on one node (the middle of an odd mesh): every weight of a warp's corner is exactly 1
    (2^26), the sum that does not fit the 32-bit reduction.  The density
    agrees with the plain form's to the mixed form's FP32 storage (2^-24)."""
    R = np.zeros((n + 8, 3))
    R[n:] = 1e-3 * np.array([[(k & 1) * 2 - 1, (k & 2) - 1, (k & 4) / 2 - 1] for k in range(8)])
    P = np.zeros_like(R)
    P[:, 2] = 10.0
    rho = []
    for prec in (gpu.PLAIN_FP64, gpu.MIXED):
        with gpu.Context((15, 15, 15), precision=prec) as c:
            c.compute_self_fields(R, P, -1e-13, DT)
            rho.append(c.field(gpu.FIELD_RHO))
    assert _rel(rho[1], rho[0]) <= 2.0 ** -23


def _state(c):
    R, P = c.download()
    t = c.tracker_state()
    return [R, P, t["path_length"], t["t"], t["q_macro"], t["ref_R"], t["ref_P"], c.field(1)]


@pytest.mark.parametrize("kind", ["plain", "mixed", "tilted", "dc", "dc mixed", "bins"])
@pytest.mark.parametrize("interval", [0, 5, 32])
def test_one_call_equals_single_steps(gpu, kind, interval):
    nr, n, steps = (16, 16, 16), 4001, 21
    prec = gpu.MIXED if "mixed" in kind else gpu.PLAIN_FP64
    R, P = dc_bunch(n, 0.02 * 1.04) if kind.startswith("dc") else gaussian_bunch(n, bunch_id=5)
    bins = None
    if kind == "bins":
        R, P, bins = photoinjector_bunch(n, nbins=3)
    # a reference particle off the axis: its frame update rotates
    ref = (0.01, -0.02, 10.0) if kind == "tilted" else (0.0, 0.0, 10.0)
    got = []
    for calls in ([steps], [1] * steps, [8, 1, 12]):
        with gpu.Context(nr, precision=prec) as c:
            c.set_reorder_interval(interval)
            if kind.startswith("dc"):
                c.set_periodic_z(True)
                c.set_beam_frequency(299792458.0 / 0.02)
            c.upload(R, P, DT, -1e-9 / n, MASS, ref_P=ref)
            if bins is not None:
                c.set_energy_bins(bins, 3)
            for k in calls:
                c.track(k)
            got.append(_state(c))
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)


def test_statistics_between_pushed_steps(gpu):
    """Records are moments of unpushed positions, whichever calls precede them."""
    R, P = gaussian_bunch(3000, bunch_id=2)
    rows = []
    for calls in ([(9, False), (1, True)], [(10, True)]):
        with gpu.Context((16, 16, 16)) as c:
            c.upload(R, P, DT, -1e-9 / 3000, MASS)
            for k, want in calls:
                s = np.zeros((k, gpu.NSTATS))
                c.track(k, s if want else None)
            rows.append(s[-1].copy())
    np.testing.assert_array_equal(rows[0], rows[1])


def test_batch_of_many_bunches_equals_single_steps(gpu):
    """Rounds of several steps against rounds of one, with bunches of one block and of many."""
    got = []
    for calls in ([7, 2], [1] * 9):
        with gpu.Batch(precision=gpu.MIXED) as b:
            slots = []
            for i, (n, m) in enumerate([(40, 16), (33_000, 32), (5000, 24), (1, 16), (260_001, 48)]):
                R, P = gaussian_bunch(n, bunch_id=i)
                slots.append(b.add((m, m, m), R, P, DT, -1e-10 / n, MASS))
            for k in calls:
                b.track(k)
            got.append([a for s in slots for a in b.member(s).download()])
    for a, c in zip(*got):
        np.testing.assert_array_equal(a, c)


@pytest.mark.parametrize("nr", [(16, 16, 16), (20, 12, 9)])
@pytest.mark.parametrize("form", ["plain", "mixed"])
@pytest.mark.parametrize("image", [False, True])
def test_device_solve_in_place(gpu, nr, form, image):
    """A device buffer solved in place, and one that is not aligned to its
    elements (through the context's grids), give the host call's bits."""
    import ctypes as C

    import torch

    prec = gpu.MIXED if form == "mixed" else gpu.PLAIN_FP64
    rho = np.random.default_rng(11).standard_normal(nr[::-1])
    hr = (C.c_double * 3)(1e-3, 1.5e-3, 0.7e-3)
    zs = -3e-3
    L = gpu.lib()
    with gpu.Context(nr, precision=prec) as c:
        want = c.compute_potential_image(rho, hr, zs) if image else c.compute_potential(rho, hr)
        raw = torch.empty(8 * rho.size + 16, dtype=torch.uint8, device="cuda")
        for shift in (0, 8, 4):
            buf = raw[shift:shift + 8 * rho.size]
            buf.copy_(torch.from_numpy(rho.reshape(-1).view(np.uint8)))
            torch.cuda.synchronize()
            p = C.c_void_p(buf.data_ptr())
            rc = (L.scgpu_compute_potential_image_device(c.h, p, hr, zs) if image
                  else L.scgpu_compute_potential_device(c.h, p, hr))
            assert rc == 0
            got = buf.cpu().numpy().view(np.float64).reshape(rho.shape)
            np.testing.assert_array_equal(got, want)
