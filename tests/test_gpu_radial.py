"""MWPotential2014's tabulated radial force (RadialPot, potentials.cuh) on the
GPU: against 40-digit arithmetic over the table's range, at its rows' edges
and outside it, beside the direct form it replaces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# |force error| allowed, in units of 2^-53 |force|: the radial factor (its
# nodes' two to three roundings, averaged over 32 of them, and the table's
# own), the disk's (about five), their sum and the product with the position
# come to ten roundings of half an ulp each at most
BOUND = 10.0


def _exact(P, pa, planar):
    import mpmath as mp

    mp.mp.dps = 40
    d = 3 if planar else 5
    amp, al, rc, am, A, B, an, a = [mp.mpf(float(v)) for v in (*pa[:3], *pa[d:d + 5])]
    out = np.empty(P.shape, dtype=object)
    for i in range(P.shape[1]):
        x, y, z = (mp.mpf(float(v)) for v in P[:, i])
        r2 = x * x + y * y + z * z
        r = mp.sqrt(r2)
        M = 2 * mp.pi * rc ** (3 - al) * mp.gammainc(mp.mpf(3) / 2 - al / 2, 0, r2 / rc ** 2)
        f = -amp * M / r ** 3 + an * (1 / (r2 * (a + r)) - mp.log(1 + r / a) / r ** 3)
        zb = mp.sqrt(z * z + B * B)
        g = -am / mp.sqrt(x * x + y * y + (A + zb) ** 2) ** 3
        out[:, i] = x * (f + g), y * (f + g), z * (f + g * (A + zb) / zb)
    return out


def _points(lo, hi, n, planar, seed):
    rng = np.random.default_rng(seed)
    R = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    ph = rng.uniform(0, 2 * np.pi, n)
    z = np.zeros(n) if planar else 0.1 * R * rng.normal(0, 1, n)
    return np.stack([R * np.cos(ph), R * np.sin(ph), z])


def _errors(P, planar, signature, change=None):
    """Force errors over 2^-53 |force|; change: {argument: value}, the disk's
    and halo's arguments counted from 3."""
    import torch

    import galpy_b200 as gb

    _, pt, pa = gb.parse_pot(gb.MWPotential2014(), planar=planar)
    pa = np.array(pa, float)
    for k, v in (change or {}).items():
        pa[k if k < 3 or planar else k + 2] = v
    buf, n = gb.compile_potential((pt, pa), planar=planar)
    acc = torch.empty((3, P.shape[1]), dtype=torch.float64, device="cuda")
    gb.accel_device(torch.from_numpy(buf).cuda(), n, torch.from_numpy(P).cuda(), acc,
                    planar=planar, signature=signature)
    E = _exact(P, pa, planar)
    a = acc.cpu().numpy()
    k = 2 if planar else 3
    d = np.array([[float(float(a[c, i]) - E[c, i]) for i in range(P.shape[1])] for c in range(k)])
    mag = np.sqrt(sum(np.array([float(v) for v in E[c]]) ** 2 for c in range(k)))
    return np.sqrt((d ** 2).sum(0)) / mag / 2.0 ** -53


@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("lo,hi", [(1e-3, 0.05), (0.05, 0.5), (0.5, 3.0), (3.0, 500.0)])
def test_radial_force_is_closer_than_the_direct_form(lo, hi, planar):
    P = _points(lo, hi, 400, planar, 3)
    rad, direct = _errors(P, planar, 1), _errors(P, planar, 0)
    assert rad.max() <= BOUND, rad.max()
    assert np.sqrt((rad ** 2).mean()) <= np.sqrt((direct ** 2).mean())


# alpha, rc, the halo's scale, and lists with one spherical component: the
# table is built from the launch's own parameters (a row's degree suffices for
# any power law up to r^-3 and for the cutoff at any rc)
@pytest.mark.parametrize("change", [{1: 0.0}, {1: 2.9}, {2: 0.0237}, {2: 2.37}, {0: 0.0}, {6: 0.0},
                                    {7: 0.05}, {7: 50.0}])
@pytest.mark.parametrize("planar", [False, True])
def test_radial_force_with_other_parameters(change, planar):
    P = _points(0.01, 300.0, 400, planar, 9)
    rad, direct = _errors(P, planar, 1, change), _errors(P, planar, 0, change)
    assert rad.max() <= BOUND, rad.max()
    assert np.sqrt((rad ** 2).mean()) <= np.sqrt((direct ** 2).mean())


def test_radial_force_at_row_edges_and_outside():
    """r^2 at, just below and just above rows' edges, in the table's first and
    last rows, and beyond both ends (the direct form answers there)."""
    e = np.array([2.0 ** -30, 2.0 ** -29 * (1 + 63 / 64), 0.25, 0.25 * (1 + 1 / 64), 1.0,
                  1.0 + 63 / 64, 4.0, 2.0 ** 18 * (1 - 1 / 128)])
    r2 = np.concatenate([e * (1 - 2.0 ** -50), e, e * (1 + 2.0 ** -50),
                         [1e-12, 2.0 ** -31, 2.0 ** 18, 1e7]])
    P = np.stack([np.sqrt(r2), 0 * r2, 0 * r2])
    err = _errors(P, False, 1)
    inside = (r2 >= 2.0 ** -30) & (r2 < 2.0 ** 18)
    assert err[inside].max() <= BOUND, err[inside].max()
    # outside, the direct form's own rounding: its halo factor is a difference
    # whose terms exceed it 2 a / r times (4e6 at r = 1e-6), where the halo is
    # 3.1e-5 of the force: each of its four roundings counts up to 124 times
    assert err[~inside].max() <= 4 * 4e6 * 3.1e-5, err[~inside].max()


def test_radial_force_not_finite():
    """A point at infinity or NaN gives no finite force, as the direct form."""
    import torch

    import galpy_b200 as gb

    pot = gb.MWPotential2014()
    buf, n = gb.compile_potential(pot)
    P = np.array([[np.nan, 1.0, np.inf], [1.0, np.nan, 1.0], [0.0, 0.0, 0.0]])
    got = []
    for sig in (1, 0):
        acc = torch.zeros((3, 3), dtype=torch.float64, device="cuda")
        gb.accel_device(torch.from_numpy(buf).cuda(), n, torch.from_numpy(P).cuda(), acc,
                        signature=sig)
        got.append(np.isfinite(acc.cpu().numpy()[:2]).all(axis=0))
    assert np.array_equal(got[0], got[1])


# single precision, in units of 2^-24 |force|: the position's rounding (three:
# the force falls with its square at most), the radii (three), the row and its
# polynomial (four), the disk's hardware root and reciprocal (two ulps each, the
# product of three: fourteen with its own roundings)
BOUND_F32 = 24.0


def _kick_errors(P, planar, signature):
    """The same for the float32 force of one leapfrog step of length one from rest,
    whose velocity change it is."""
    import torch

    import galpy_b200 as gb

    pot = gb.MWPotential2014()
    buf, ncomp = gb.compile_potential(pot, planar=planar)
    _, _, pa = gb.parse_pot(pot, planar=planar)
    k, n = (2 if planar else 3), P.shape[1]
    w = torch.zeros((2 * k, n), dtype=torch.float64, device="cuda")
    w[:k] = torch.from_numpy(P[:k]).cuda()
    out = torch.empty((n, 1, 2 * k), dtype=torch.float64, device="cuda")
    err = torch.empty(n, dtype=torch.int32, device="cuda")
    gb.integrate_device(torch.from_numpy(buf).cuda(), ncomp, w,
                        torch.tensor([0.0, 1.0], dtype=torch.float64, device="cuda"), out, err,
                        "leapfrog_cuda", planar=planar, out_layout="aos_rect", out_row0=1, dt=1.0,
                        precision="f32force", signature=signature, comps_host=buf)
    E = _exact(P, pa, planar)[:k].astype(float)
    a = out.cpu().numpy()[:, 0, k:].T
    return np.sqrt(((a - E) ** 2).sum(0) / (E ** 2).sum(0)) / 2.0 ** -24


@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("lo,hi", [(1e-3, 0.05), (0.05, 3.0), (3.0, 500.0)])
def test_radial_force_in_single_precision(lo, hi, planar):
    P = _points(lo, hi, 400, planar, 5)
    rad, direct = (_kick_errors(P, planar, s) for s in (1, 0))
    assert rad.max() <= BOUND_F32, rad.max()
    assert np.sqrt((rad ** 2).mean()) <= np.sqrt((direct ** 2).mean())


def test_radial_force_in_single_precision_at_row_edges():
    """Rows' edges, the first and last rows, and beyond both ends."""
    e = np.array([2.0 ** -30, 0.25, 0.25 * (1 + 1 / 64), 1.0, 1.0 + 63 / 64,
                  2.0 ** 18 * (1 - 1 / 128)])
    r2 = np.concatenate([e * (1 - 2.0 ** -22), e, e * (1 + 2.0 ** -22), [2.0 ** -31, 2.0 ** 18, 1e7]])
    err = _kick_errors(np.stack([np.sqrt(r2), 0 * r2, 0 * r2]), False, 1)
    assert err.max() <= BOUND_F32, err.max()


def _default_pool_high(reset=False):
    from cuda.bindings import driver, runtime as rt

    _, pool = rt.cudaDeviceGetDefaultMemPool(0)
    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    if reset:
        rt.cudaMemPoolSetAttribute(pool, attr, driver.cuuint64_t(0))
    return int(rt.cudaMemPoolGetAttribute(pool, attr)[1])


@pytest.mark.parametrize("precision", ["fp64", "f32force", "f32force_df"])
@pytest.mark.parametrize("planar", [False, True])
def test_accelerations_are_the_integrators_own(planar, precision):
    """accel_device gives the kicks of a leapfrog step of length one from rest
    (bit for bit in float64; in single precision the two kernels may fuse the
    radii's sums differently, an ulp of each, which the force's second power
    of the radius doubles) and takes no memory from the device's default pool."""
    import torch

    import galpy_b200 as gb

    pot = gb.MWPotential2014()
    buf, ncomp = gb.compile_potential(pot, planar=planar)
    sig = gb.signature(pot, planar=planar)
    P = _points(1e-3, 600.0, 3000, planar, 11)
    if precision == "f32force_df":  # (positions are rounded to the pairs, too)
        P = P.astype(np.float32).astype(float)
    k, n = (2 if planar else 3), P.shape[1]
    comps, pos = torch.from_numpy(buf).cuda(), torch.from_numpy(P).cuda()
    acc = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    before = _default_pool_high(reset=True)
    gb.accel_device(comps, ncomp, pos, acc, planar=planar, signature=sig, precision=precision)
    torch.cuda.synchronize()
    assert _default_pool_high() == before
    w = torch.zeros((2 * k, n), dtype=torch.float64, device="cuda")
    w[:k] = pos[:k]
    out = torch.empty((n, 1, 2 * k), dtype=torch.float64, device="cuda")
    err = torch.empty(n, dtype=torch.int32, device="cuda")
    gb.integrate_device(comps, ncomp, w, torch.tensor([0.0, 1.0], dtype=torch.float64, device="cuda"),
                        out, err, "leapfrog_cuda", planar=planar, out_layout="aos_rect", out_row0=1,
                        dt=1.0, precision=precision, signature=sig, comps_host=buf)
    d, mag = (out[:, 0, k:].T - acc[:k]).abs().max(0).values, acc[:k].norm(dim=0)
    assert float((d / mag).max()) <= (0.0 if precision == "fp64" else 6 * 2.0 ** -24)
