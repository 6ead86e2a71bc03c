"""The Nystrom form of the Runge-Kutta machines (machines_nystrom.cuh): its
tables against the published DOP853 tableau, its pairs of forces against single
ones, and on the GPU the second-order machines against the first-order one over
the sizes where the warp's rounds and its dense-output queue have edges."""
import os
import re
from fractions import Fraction

import numpy as np
import pytest
import timedep_pots

CSRC = os.path.join(os.path.dirname(__file__), "..", "galpy_b200", "csrc")


def _tableau():
    with open(os.path.join(CSRC, "dop853_tableau.cuh")) as f:
        v = {k: Fraction(x) for k, x in re.findall(r"constexpr double (\w+) = ([-+\d.e]+);",
                                                   f.read())}
    A = [[Fraction(0)] * 16 for _ in range(16)]
    for i in list(range(2, 13)) + [14, 15, 16]:
        for j in range(1, i):
            A[i - 1][j - 1] = v.get(f"a{i}{j}", Fraction(0))
    A[12] = [v.get(f"b{j}", Fraction(0)) for j in range(1, 17)]
    return v, A


def test_dop853_nystrom_table():
    """X = A A, DX = d A, EX = er A, HX = (b - bhh) A, each entry the nearest
    double; entries the order conditions make zero (to the published digits,
    1e-25) are exact zeros."""
    v, A = _tableau()

    def times_A(row):
        return [sum(row[j] * A[j][k] for j in range(16)) for k in range(16)]

    def named(prefix):
        return [v.get(f"{prefix}{j}", Fraction(0)) for j in range(1, 17)]

    hb = list(A[12])
    hb[0] -= v["bhh1"]
    hb[8] -= v["bhh2"]
    hb[11] -= v["bhh3"]
    want = [times_A(A[i])[:14] for i in range(16)]
    want += [times_A(named(f"d{m}"))[:15] for m in (4, 5, 6, 7)]
    want += [times_A(named("er"))[:11], times_A(hb)[:11]]
    with open(os.path.join(CSRC, "dop853_nystrom.cuh")) as f:
        body = f.read().split("static constexpr NyTable kNy")[1]
    rows = [[float(x) for x in m.split(",")] for m in re.findall(r"\{([-\d.e,\s]+)\}", body)]
    assert len(rows) >= len(want)
    for got, w in zip(rows, want):
        assert len(got) == len(w)
        for g, x in zip(got, w):
            if abs(x) < Fraction(1, 10**25):
                assert g == 0.0
            else:
                assert abs(Fraction(g) - x) <= abs(x) * Fraction(1, 2**53)


def _controller(harness, kind, e):
    import ctypes

    dp = ctypes.POINTER(ctypes.c_double)
    e = np.ascontiguousarray(e, dtype=float)
    out = np.empty_like(e)
    harness.lib.harness_controller(kind, len(e), e.ctypes.data_as(dp), out.ctypes.data_as(dp))
    return out


def test_dopr54_step_power(harness):
    """round(log2(0.85 e^(-1/5))) in [-3, 3] (bovy_rk.c:744-752), at and about
    every rounding boundary, for norms that single precision does not hold,
    and for zero, infinity and NaN."""
    edge = (0.85 / 2.0 ** (np.arange(-4, 5) + 0.5)) ** 5
    near = edge[:, None] * (1 + np.outer([1, -1], 10.0 ** np.arange(-15, 0)).ravel())
    e = np.concatenate([edge, near.ravel(), np.logspace(-60, 60, 400),
                        [0.0, 1e-310, 1e300, np.inf]])
    with np.errstate(divide="ignore"):
        x = np.log(0.85 * e ** -0.2) / np.log(2.0)
        want = np.clip(np.sign(x) * np.floor(np.abs(x) + 0.5), -3, 3)
    got = _controller(harness, 0, e)
    with np.errstate(invalid="ignore"):  # (x is infinite at zero)
        tie = np.abs(np.abs(x - np.floor(x)) - 0.5) < 1e-13  # two libraries' logarithms may differ
    assert np.array_equal(got[~tie], want[~tie])
    assert np.isnan(_controller(harness, 0, [np.nan])[0])


def test_dop853_controller_root(harness):
    """e^(-1/8) to rounding on [1e-9, 1e6], constant beyond, where the
    controller's limits hold; NaN is caught before it."""
    e = np.concatenate([np.logspace(-9, 6, 500), [0.0, 1e-300, 1e-9, 1e6, 1e300, np.inf]])
    got = _controller(harness, 1, e)
    want = np.clip(e, 1e-9, 1e6) ** -0.125
    assert np.abs(got / want - 1).max() < 8 * 2.0 ** -53


PAIR_POTS = ["mw14", "hernquist", "loghalo", "logtri", "power", "plummer", "kks", "einasto", "hh",
             "kuzmindisk", "ell_trinfw", *timedep_pots.NAMES, *timedep_pots.WRAPPED]


@pytest.mark.parametrize("name", PAIR_POTS)
@pytest.mark.parametrize("planar", [False, True])
def test_force_pairs(harness, golden, name, planar):
    """Two forces at once against each alone, in both run-time lists and with
    deviations: components evaluated side by side and one after the other,
    continuation records, wrappers with the records they wrap, times of their
    own, and one point given twice (whose second half is copied)."""
    import ctypes

    if name == "hh" and not planar:
        pytest.skip("a planar potential")
    npot = None
    if name in timedep_pots.WRAPPED:
        pt, pa, npot = timedep_pots.wrapped(name, planar=planar)
    elif name in timedep_pots.NAMES:
        pt, pa = timedep_pots.potential(name, planar=planar)
    else:
        key = name + "_planar" if planar and name + "_planar_type" in golden else name
        pt, pa = golden[key + "_type"], golden[key + "_args"]
    pt, pa = np.ascontiguousarray(pt, np.int32), np.ascontiguousarray(pa, float)
    D, n = (2 if planar else 3), 16
    rng = np.random.default_rng(8)
    ptr = lambda a, c=ctypes.c_double: a.ctypes.data_as(ctypes.POINTER(c))  # noqa: E731
    timed = name in timedep_pots.NAMES + timedep_pots.WRAPPED
    full_only = timed or name.startswith("ell")  # (the common list leaves those out)
    for var in (False, True):
        if var and name.startswith("scf"):
            continue  # run on the device only
        for lst in ((0,) if var or full_only else (0, 1)):
            for q_same, t1, t2 in ((False, 0.3, 0.7), (True, 0.4, 0.4), (True, 0.3, 0.7)):
                NA = 2 * D if var else D
                q1 = np.concatenate([rng.uniform(0.3, 1.5, (n, D)), rng.normal(size=(n, NA - D))], 1)
                q2 = q1.copy() if q_same else q1 + rng.uniform(0.1, 0.2, q1.shape)
                a1, a2 = np.zeros_like(q1), np.zeros_like(q1)
                assert harness.lib.harness_force_pairs(
                    int(planar), int(var), lst, n, ptr(q1), ptr(q2), ctypes.c_double(t1),
                    ctypes.c_double(t2), len(pt) if npot is None else npot, ptr(pt, ctypes.c_int),
                    ptr(pa), ptr(a1), ptr(a2)) == 0
                for q, t, a in ((q1, t1, a1), (q2, t2, a2)):
                    z = q[:, 2] if D == 3 else np.zeros(n)
                    acc, tid, _ = harness.forces(q[:, 0], q[:, 1], z, pt, pa, planar=planar, t=t,
                                                 npot=npot)
                    want = acc[:, :D]
                    if var:
                        K = tid[:, [0, 1, 3, 1, 2, 4, 3, 4, 5]].reshape(n, 3, 3)[:, :D, :D]
                        want = np.concatenate([want, np.einsum("nij,nj->ni", K, q[:, D:])], 1)
                    # the same sums up to their order: a few roundings
                    assert np.abs(a - want).max() <= 1e-14 * np.abs(want).max(), (var, lst, t1, t2)


@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("name", ["bar_growing+mw14", "ell_trihern"])
def test_full_list_queued_dense_output(harness, golden, name, planar):
    """The full run-time list's dop853 machine, which is the first-order one:
    rows from its request records against its own dense stages, bit for bit,
    several rows a step and none, forward and backward."""
    from helpers import cyl_to_rect, seeded_ics

    if name in timedep_pots.NAMES:
        pt, pa = timedep_pots.potential(name, planar=planar)
    else:
        key = name + "_planar" if planar else name
        pt, pa = golden[key + "_type"], golden[key + "_args"]
    w = cyl_to_rect(seeded_ics(6, 62, planar=planar))
    for t in (np.linspace(0.0, 8.0, 161), np.linspace(0.0, -6.0, 5)):
        ref = harness.integrate(w, t, pt, pa, "dop853", planar=planar, rtol=1e-10, atol=1e-10)
        got = harness.dop853_queued(w, t, pt, pa, planar=planar, rtol=1e-10, atol=1e-10)
        assert not ref[1].any()
        assert all(np.array_equal(a, b) for a, b in zip(got, ref))


@pytest.mark.gpu
@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 5000])
def test_pair_machine_against_first_order(n, planar):
    """DOP853 in MWPotential2014: the pair machine (compile-time list) against
    the first-order machine of the full run-time list (signature 0), per-orbit
    end times, rows from none to several per step.  Both round differently:
    an orbit either takes the same steps and agrees to its conditioning, or
    one borderline step differs and it moves by its truncation error."""
    import torch

    import galpy_b200 as gb
    from helpers import cyl_to_rect, seeded_ics

    pot = gb.MWPotential2014()
    buf, ncomp = gb.compile_potential(pot, planar=planar)
    comps = torch.from_numpy(buf).cuda()
    w0 = torch.from_numpy(cyl_to_rect(seeded_ics(n, 5, planar=planar)).T.copy()).cuda()
    tend = np.random.default_rng(6).uniform(0.5, 30.0, n)
    t = torch.from_numpy(np.linspace(0.0, 1.0, 67)[None, :] * tend[:, None]).cuda()
    nv = 4 if planar else 6
    got = []
    for sig in (gb.signature(pot, planar=planar), 0):
        out = torch.empty((n, 67, nv), dtype=torch.float64, device="cuda")
        err = torch.empty(n, dtype=torch.int32, device="cuda")
        ns = torch.empty(n, dtype=torch.int64, device="cuda")
        gb.integrate_device(comps, ncomp, w0, t, out, err, "dop853_cuda", planar=planar,
                            nsteps=ns, out_layout="aos_rect", rtol=1e-10, atol=1e-10,
                            signature=sig, comps_host=buf)
        assert not err.any()
        got.append((out.cpu().numpy(), ns.cpu().numpy()))
    (a, na), (b, nb) = got
    d = np.abs(a - b).max(axis=(1, 2))
    assert (na == nb).mean() >= 0.98
    assert np.median(d) < 1e-12 and d.max() < 1e-6, (np.median(d), d.max())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32, 63, 2000])
def test_requests_reuse_the_ring(n):
    """Output times in every step: the warp's 64 request slots are reused many
    times over, and every row is the one of the entry point without a ring
    (its lanes run their own dense stages; a torn request would show at once).
    The same arithmetic either way, so rounding of a few ulp is allowed."""
    import ctypes

    import torch

    import galpy_b200 as gb
    from galpy_b200 import _lib
    from test_zz_no_alloc import _launch, _workload

    pot = gb.MWPotential2014()
    buf, ncomp = gb.compile_potential(pot)
    w, t = _workload(n)
    t = np.linspace(0.0, 1.0, 401)[None, :] * t[:, -1:]
    comps, w0, td = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (buf, w, t))
    got = []
    for entry in ("galpy_cuda_integrate_device", "galpy_cuda_integrate_device_noalloc"):
        out = torch.full((6, 401, n), float("nan"), dtype=torch.float64, device="cuda")
        err = torch.full((n,), -99, dtype=torch.int32, device="cuda")
        ns = torch.empty(n, dtype=torch.int64, device="cuda")
        L = _launch(comps, ncomp, w0, td, out, err, ns, gb.signature(pot), 1)
        L.comps_host = buf.ctypes.data
        assert getattr(_lib.lib(), entry)(ctypes.byref(L)) == 0, _lib.last_error()
        torch.cuda.synchronize()
        assert not err.any()
        got.append((out, ns))
    assert torch.equal(got[0][1], got[1][1])
    assert float((got[0][0] - got[1][0]).abs().max()) < 1e-13
