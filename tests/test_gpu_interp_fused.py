"""Orbit interpolation on one shared grid (the fused kernel) against the same
grid given per orbit (the four-pass route), at the edges of the fused kernel's
tiles, query chunks and row lengths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, t, nv, seed):
    rng = np.random.default_rng(seed)
    R, f, ph = rng.uniform(0.5, 2, (n, 1)), rng.uniform(0.2, 2, (n, 1)), rng.uniform(0, 6, (n, 1))
    w = [R * (1 + 0.1 * np.cos(f * t)), 0.1 * np.sin(f * t), 1 + 0.1 * np.cos(f * t)]
    if nv == 6:
        w += [0.05 * np.sin(2 * f * t), 0.05 * np.cos(2 * f * t)]
    w.append(np.mod(ph + f * t + np.pi, 2 * np.pi) - np.pi)
    return np.ascontiguousarray(np.stack(w, -1))


# (orbits, rows, queries): one orbit; the last rows of a tile and of a query
# chunk (128); the shortest spline; one orbit per block (nt = 801); rows of
# one orbit beyond the largest block (nt = 2500), which take the four passes
@pytest.mark.parametrize("n,nt,nq", [(1, 4, 1), (6, 101, 127), (7, 101, 128), (8, 101, 129),
                                     (513, 5, 300), (5, 801, 33), (3, 2500, 40)])
@pytest.mark.parametrize("nv", [4, 6])
@pytest.mark.parametrize("own_queries", [False, True])
def test_shared_grid_against_per_orbit_grid(n, nt, nq, nv, own_queries):
    import torch

    from galpy_b200.orbit_quantities import interpolate_device

    rng = np.random.default_rng(nt)
    t = np.cumsum(rng.uniform(0.02, 0.1, nt))
    rows = torch.from_numpy(_rows(n, t, nv, 1)).cuda()
    lo, hi = t[0] - 0.01, t[-1] + 0.01  # a little outside: the end pieces extrapolate
    tq = rng.uniform(lo, hi, (n, nq) if own_queries else nq)
    td, tqd = torch.from_numpy(t).cuda(), torch.from_numpy(tq).cuda()
    got = [torch.empty((n, nq, nv), dtype=torch.float64, device="cuda") for _ in range(2)]
    interpolate_device(rows, td, tqd, got[0])
    interpolate_device(rows, td.expand(n, nt).contiguous(), tqd, got[1])
    a, b = (g.cpu().numpy() for g in got)
    d = np.abs(a - b)
    d[..., -1] = np.abs(np.mod(a[..., -1] - b[..., -1] + np.pi, 2 * np.pi) - np.pi)
    # both solve the same diagonally dominant system (condition < 10) in
    # double precision: ten roundings of values up to 4
    assert d.max() < 4e-14 / min(1.0, a[..., 0].min()), d.max()


def test_output_over_the_rows():
    """An output that overlaps the rows: all rows are read first."""
    import torch

    from galpy_b200.orbit_quantities import interpolate_device

    n, nt, nq = 300, 41, 30
    t = np.linspace(0.0, 4.0, nt)
    rows = torch.from_numpy(_rows(n, t, 6, 2)).cuda()
    td, tq = torch.from_numpy(t).cuda(), torch.linspace(0.1, 3.9, nq, dtype=torch.float64).cuda()
    ref = torch.empty((n, nq, 6), dtype=torch.float64, device="cuda")
    interpolate_device(rows, td, tq, ref)
    out = rows.view(-1)[: n * nq * 6].view(n, nq, 6)
    interpolate_device(rows, td, tq, out)
    assert float((out - ref).abs().max()) < 1e-13


def test_threads_with_different_grids():
    """Host threads on streams of their own, with grids whose blocks need
    different amounts of shared memory: no call's launch may depend on what
    another asked of the kernel."""
    import threading

    import torch

    from galpy_b200.orbit_quantities import interpolate_device

    failed = []

    def work(nt, calls):
        t = np.linspace(0.0, 0.05 * (nt - 1), nt)
        rows = torch.from_numpy(_rows(1, t, 6, 3)).cuda()
        td, tq = torch.from_numpy(t).cuda(), torch.linspace(0.0, t[-1], 8, dtype=torch.float64).cuda()
        out = torch.empty((1, 8, 6), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        try:
            for _ in range(calls):
                interpolate_device(rows, td, tq, out, stream=stream)
        except Exception as e:  # noqa: BLE001 (the other thread must end too)
            failed.append((nt, str(e)))
        torch.cuda.synchronize()

    threads = [threading.Thread(target=work, args=(nt, 4000)) for nt in (801, 601, 1201, 901)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed, failed
