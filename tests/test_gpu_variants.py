"""Edges of the kernels' variants: sizes around a tile, a word or a chunk, and the calls that a
dispatch sends another way than their neighbours.  Integers are compared bitwise; the bars of
computed values are the ones of the path's own parity tests."""
import ctypes
import math
from fractions import Fraction

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TWO_PI = 2 * np.pi


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def to_dev(a, dev):
    return torch.from_numpy(np.asfortranarray(a)).to(dev)


def relerr(got, want):
    return np.abs(np.asarray(got, dtype=np.float64) - want).max() / max(np.abs(want).max(), 1e-300)


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 255, 257, 4097, 400_003])
def test_traversal_validation_counts_every_entry(gbg, dev, m):
    # the bitmap's word edges and the last, partial word; one entry named twice, one out of range
    rng = np.random.default_rng(m)
    perm = (rng.permutation(m) + 1).astype(np.int32)
    gbg.PointTraversalOrder(torch.from_numpy(perm).to(dev))
    for bad in (0, m + 1, -7):
        broken = perm.copy()
        broken[rng.integers(m)] = bad
        with pytest.raises(gbg.ArgumentError, match="1:%d, but it spans" % m):
            gbg.PointTraversalOrder(torch.from_numpy(broken).to(dev))
    if m > 1:
        twice = perm.copy()
        twice[0] = twice[m - 1]
        with pytest.raises(gbg.ArgumentError, match="names %d of %d" % (m - 1, m)):
            gbg.PointTraversalOrder(torch.from_numpy(twice).to(dev))


def _contribution_sizes(coef, n, pos, q, spacing):
    """Per node the sums over its contributions of |w1 w2 w3 q| and of |q|."""
    width, powers = coef.shape
    ci = pos / spacing
    base = np.floor(ci).astype(np.int64)
    t = ci - base
    w = np.zeros(pos.shape + (width,))
    for p in range(powers - 1, -1, -1):
        w = w * t[..., None] + coef[:, p]
    w = np.abs(w)
    out, reach = np.zeros(tuple(n) + (q.shape[1],)), np.zeros(tuple(n) + (q.shape[1],))
    for k in range(width):
        for j in range(width):
            for i in range(width):
                at = [(base[:, d] - (width // 2 - 1) + s) % n[d] for d, s in enumerate((i, j, k))]
                wt = w[:, 0, i] * w[:, 1, j] * w[:, 2, k]
                for c in range(q.shape[1]):
                    np.add.at(out[..., c], tuple(at), wt * np.abs(q[:, c]))
                    np.add.at(reach[..., c], tuple(at), np.abs(q[:, c]))
    return out, reach


# grids of one brick, of bricks with a last cell of one, and of axes no longer than the stencil; point
# counts below, at and above one staging (508 points of a brick's region); quantities of one size and
# spread over many windows of digits, region by region and point by point
@pytest.mark.parametrize("n,m", [((8, 8, 4), 300), ((8, 8, 4), 509), ((9, 17, 5), 4000), ((25, 9, 13), 20_000),
                                 ((8, 25, 33), 60)])
@pytest.mark.parametrize("width,comps", [(2, 3), (4, 1), (4, 3), (4, 2), (6, 9), (8, 3)])
@pytest.mark.parametrize("spread", [0, 14, 45])
def test_fp64_scatter_per_node(gbg, oracle, dev, n, m, width, comps, spread):
    n = tuple(max(v, width) for v in n)
    rng = np.random.default_rng(1000 * width + m + spread)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    pos = TWO_PI * rng.random((m, 3))
    pos[: m // 4] = pos[0] + 1e-3 * rng.random((m // 4, 3))  # a crowded cell
    q = rng.standard_normal((m, comps)) * 10.0 ** (-spread * rng.random((m, 1)))
    q[rng.random(m) < 0.05] = 0.0
    pos, q = np.asfortranarray(pos), np.asfortranarray(q)
    scheme = gbg.LalescuSpline(width)
    old = np.asfortranarray(rng.standard_normal(n + (comps,)))
    got = _scatter_abi(gbg, grid, dev, old, pos, q, scheme, 0.75, -0.5)
    # the deposit by the oracle, then beta * old (the oracle's own adds onto beta * old would each round there)
    want = oracle.scatter(g, np.zeros(n + (comps,), order="F"), pos, q, scheme.coefficients, alpha=0.75) - 0.5 * old
    size, reach = _contribution_sizes(np.asarray(scheme.coefficients), n, pos, q, TWO_PI / np.array(n))
    # the path's bar for a node (1e-12 of its own contributions), the unit of a node's fixed-point weight
    # (2^(128 - 3 P), P >= 61, a few of them) for each point, and the roundings of beta * old and the sum
    assert np.all(np.abs(got - want) <= 0.75 * (1e-12 * size + 4 * 2.0 ** -55 * reach) + 4e-16 * np.abs(old))
    again = _scatter_abi(gbg, grid, dev, old, pos[::-1], q[::-1], scheme, 0.75, -0.5)
    assert np.array_equal(got, again)  # integers: the points' order is no matter


def _scatter_abi(gbg, grid, dev, old, pos, q, scheme, alpha, beta):
    """gbg_anterpolate for any number of components."""
    from gbgperiodicfields_gb300 import _lib
    f, x, v = (to_dev(np.asfortranarray(a), dev) for a in (old, pos, q))
    st = _lib.load().gbg_anterpolate(grid.c(), _lib.GBG_F64 if f.dtype == torch.float64 else _lib.GBG_F32, q.shape[1],
                                     f.data_ptr(), x.data_ptr(), q.shape[0], v.data_ptr(), None, scheme.c(), alpha, beta,
                                     None, 0, None, torch.cuda.current_stream().cuda_stream)
    _lib.check(st, "scatter")
    torch.cuda.synchronize()
    return f.cpu().numpy()


@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("spread", [0, 20])
def test_fp32_scatter_windows(gbg, oracle, dev, comps, spread):
    n, m = (25, 9, 13), 5000
    rng = np.random.default_rng(comps + spread)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, dtype=torch.float32)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin, dtype=np.float32)
    pos = np.asfortranarray((TWO_PI * rng.random((m, 3))).astype(np.float32))
    q = np.asfortranarray((rng.standard_normal((m, comps)) * 10.0 ** (-spread * rng.random((m, 1)))).astype(np.float32))
    zero = np.zeros(n + (comps,), np.float32, order="F")
    got = _scatter_abi(gbg, grid, dev, zero, pos, q, gbg.CatmullRom, 1.0, 0.0)
    want = oracle.scatter(g, zero.copy(order="F"), pos, q, gbg.CatmullRom.coefficients)
    assert relerr(got, want) <= 2e-5


def test_fp64_scatter_marks_what_a_nan_reaches(gbg, oracle, dev):
    n, m = (20, 16, 12), 3000
    rng = np.random.default_rng(5)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    pos = np.asfortranarray(TWO_PI * rng.random((m, 3)))
    q = np.asfortranarray(rng.standard_normal((m, 3)))
    q[17, 1], q[40, 2] = np.nan, np.inf
    zero = np.zeros(n + (3,), order="F")
    got = _scatter_abi(gbg, grid, dev, zero, pos, q, gbg.CatmullRom, 1.0, 0.0)
    clean = q.copy(order="F")
    clean[17, 1] = clean[40, 2] = 0.0
    want = oracle.scatter(g, zero.copy(order="F"), pos, clean, gbg.CatmullRom.coefficients)
    base = np.floor(pos / (TWO_PI / np.array(n))).astype(int)
    reach = np.zeros(n + (3,), bool)
    for p, c in ((17, 1), (40, 2)):
        reach[np.ix_(*[(base[p, d] - 1 + np.arange(4)) % n[d] for d in range(3)], [c])] = True
    assert np.array_equal(np.isnan(got), reach)
    assert np.abs(got - want)[~reach].max() <= 1e-13 * np.abs(want).max()


# a quarter-warp per point at widths 6 and 8: a few points, a brick's points no multiple of the CTA's
# quarter-warps, bricks with and without a second tile buffer, schemes with fewer powers than nodes
@pytest.mark.parametrize("m", [1, 7, 65, 5000])
@pytest.mark.parametrize("ncomp", [1, 3, 9, 12])
@pytest.mark.parametrize("name", ["L6", "L6m1", "L8", "L8m2", "G8"])
def test_wide_gather_staged_direct_and_batched(gbg, oracle, dev, m, ncomp, name):
    from gbgperiodicfields_gb300 import resident
    scheme = {"L6": gbg.LalescuSpline(6), "L6m1": gbg.LalescuSpline(6, 1), "L8": gbg.LalescuSpline(8),
              "L8m2": gbg.LalescuSpline(8, 2), "G8": gbg.LagrangeSpline(8)}[name]
    n = (19, 16, 21)
    rng = np.random.default_rng(m + 100 * ncomp)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, origin=(0.5, -1.0, 2.0))
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    pos = np.asfortranarray(np.array(grid.origin) + TWO_PI * (rng.random((m, 3)) * 1.2 - 0.1))
    f = np.asfortranarray(rng.standard_normal(n + (ncomp,)))
    want = oracle.gather(g, f, pos, scheme.coefficients)
    field = resident.ResidentField(grid, ncomp, max_stencil_width=8).load(to_dev(f, dev))
    got = {}
    for brick in ((19, 16, 21), (4, 4, 4), (11, 8, 8)):
        # one brick of m points is staged, hundreds of bricks with few points each are read directly
        if (brick[0] + 7) * (brick[1] + 7) * (brick[2] + 7) * (16 if ncomp <= 4 else 48) > 200 * 1024:
            continue
        bins = resident.PointBins(grid, m, brick=brick).build(to_dev(pos, dev))
        got[brick] = resident.interpolate_binned(field, bins, scheme, dtype=torch.float32).cpu().numpy()
        assert relerr(got[brick], want) <= 1e-5
        if scheme.coefficients.shape[1] == scheme.stencil_width:
            out = gbg.empty_colmajor((m, ncomp), torch.float32, dev)
            resident.Batch([dict(field=field, bins=bins, scheme=scheme, out=out)]).run()
            assert np.array_equal(out.cpu().numpy(), got[brick])
    first = next(iter(got.values()))
    assert all(np.array_equal(v, first) for v in got.values())


@pytest.mark.parametrize("ncomp", [1, 4, 5, 12])
@pytest.mark.parametrize("n", [(8, 9, 33), (65, 8, 8), (31, 40, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_import_rows_and_ghosts(gbg, oracle, dev, ncomp, n, dtype):
    # axes no longer than the widest stencil, rows below, at and above a warp's width
    from gbgperiodicfields_gb300 import resident
    rng = np.random.default_rng(ncomp + n[0])
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    f = np.asfortranarray(rng.standard_normal(n + (ncomp,)))
    data = to_dev(f, dev).to(dtype)
    field = resident.ResidentField(grid, ncomp, max_stencil_width=8).load(data)
    assert torch.equal(field.read(torch.float32), data.float())
    pos = np.asfortranarray(np.concatenate([TWO_PI * rng.random((200, 3)), TWO_PI * rng.integers(0, 2, (50, 3))]))
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    scheme = gbg.LalescuSpline(8)
    got = resident.interpolate_binned(field, resident.PointBins(grid, 250).build(to_dev(pos, dev)), scheme)
    assert relerr(got.cpu().numpy(), oracle.gather(g, f, pos, scheme.coefficients)) <= 1e-5


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("origin", [0.0, -0.75, 1e-3])
def test_wrap_around_every_bound(gbg, oracle, dev, T, origin):
    # coordinates a few units either side of every bound that the wrap decides at, and far beyond
    L, o = T(TWO_PI), T(origin)
    grid = gbg.Grid3D((8, 8, 8), (float(L),) * 3, origin=(origin,) * 3,
                      dtype=torch.float64 if T is np.float64 else torch.float32)
    at = [T(0), -T(0), L, -L, L + L, -(L + L), L / T(2), T(3) * L, T(1e6) * L]
    tiny = np.finfo(T).tiny
    xs = [T(v) for v in (np.inf, -np.inf, np.nan, tiny, -tiny, np.finfo(T).max, -np.finfo(T).max, 1e-30, -1e-30)]
    for v in at:
        for k in (-2, -1, 0, 1, 2):
            w = v
            for _ in range(abs(k)):
                w = np.nextafter(w, T(np.inf) if k > 0 else T(-np.inf))
            xs += [w, T(w + o)]
    x = np.asfortranarray(np.stack([np.array(xs, T), np.array(xs[::-1], T), np.array(xs, T)], 1))
    pts = gbg.PointSet(to_dev(x, dev))
    gbg.wrap_(pts, grid)
    want = oracle.displace(x, [], {"domain": grid.domain_size, "origin": grid.origin})
    got = pts.positions.cpu().numpy()
    assert np.array_equal(got.view(np.uint64 if T is np.float64 else np.uint32)[~np.isnan(want)],
                          want.view(np.uint64 if T is np.float64 else np.uint32)[~np.isnan(want)])
    assert np.array_equal(np.isnan(got), np.isnan(want))


# cells at and above the longest run that the placement sorts itself (1024), of one tile of the run sort
# (2048) and of several, alone and together; index widths of one to three passes
@pytest.mark.parametrize("runs", [(1024,), (1025,), (2048, 2049), (1500, 9000, 1025, 70_001)])
@pytest.mark.parametrize("spread", [0, 300, 200_000])
def test_bins_order_with_long_runs(gbg, dev, runs, spread):
    from gbgperiodicfields_gb300 import resident
    n, brick = np.array((20, 18, 16)), np.array((11, 8, 8))
    rng = np.random.default_rng(sum(runs) + spread)
    grid = gbg.Grid3D(tuple(n), tuple(float(v) for v in n))  # cells of edge 1
    pos = [rng.random((spread, 3)) * n]
    for k, c in enumerate(runs):
        pos.append(np.array([3 * k + 1, 17 - 2 * k, k]) + rng.random((c, 3)))
    pos = np.concatenate(pos)
    pos = np.asfortranarray(pos[rng.permutation(len(pos))])
    bins = resident.PointBins(grid, len(pos), brick=tuple(brick)).build(to_dev(pos, dev))
    c = np.floor(pos).astype(np.int64) % n
    nb, br = -(-n // brick), c // brick
    loc = c - br * brick
    key = ((br[:, 2] * nb[1] + br[:, 1]) * nb[0] + br[:, 0]) * brick.prod() + (loc[:, 2] * brick[1] + loc[:, 1]) * brick[0] + loc[:, 0]
    assert np.array_equal(bins.order().cpu().numpy(), np.argsort(key, kind="stable") + 1)
    # the records follow: a linear field is reproduced by the cubic spline inside the box
    x = torch.arange(int(n[0]), dtype=torch.float64, device=dev)[:, None, None].expand(*[int(v) for v in n])
    field = resident.ResidentField(grid, 1, 4).load(gbg.colmajor(x.contiguous()[..., None]))
    got = resident.interpolate_binned(field, bins, gbg.CatmullRom).cpu().numpy()[:, 0]
    inner = (pos[:, 0] >= 2) & (pos[:, 0] < n[0] - 3)
    assert np.abs(got - pos[:, 0])[inner].max(initial=0.0) <= 1e-5 * n[0]


@pytest.mark.parametrize("n", [1, 7, 8, 2047, 2048, 2049, 4096 * 19, 1216 * 2048 + 5, 3 * 1216 * 2048 - 1])
def test_cell_starts_at_every_scan_length(gbg, dev, n):
    # grids of n cells in a row of bricks: the bins' order is the points' order by cell
    from gbgperiodicfields_gb300 import resident
    edge = 1 if n <= 64 else 64
    rows = -(-n // edge)
    ny = next(v for v in range(min(rows, 64), 0, -1) if rows % v == 0)
    grid = gbg.Grid3D((edge, ny, rows // ny), (float(edge), float(ny), float(rows // ny)))
    rng = np.random.default_rng(n)
    m = 5000
    pos = np.asfortranarray(rng.random((m, 3)) * np.array(grid.grid_size))
    bins = resident.PointBins(grid, m, brick=(edge, 1, 1)).build(to_dev(pos, dev))
    c = np.floor(pos).astype(np.int64)
    key = (c[:, 2] * ny + c[:, 1]) * edge + c[:, 0]
    assert np.array_equal(bins.order().cpu().numpy(), np.argsort(key, kind="stable") + 1)


# a group of lanes per point: points no multiple of a CTA's groups, axes shorter than the stencil (which
# wraps more than once), component counts of every chunk, powers fewer than nodes, a bad traversal entry
@pytest.mark.parametrize("n", [(3, 5, 2), (33, 8, 9)])
@pytest.mark.parametrize("m", [1, 3, 65, 4097])
@pytest.mark.parametrize("ncomp", [1, 2, 3, 9])
@pytest.mark.parametrize("name", ["C4", "L6m1", "L6", "G8"])
def test_fp32_gather_rows(gbg, oracle, dev, n, m, ncomp, name):
    from gbgperiodicfields_gb300 import _lib
    scheme = {"C4": gbg.CatmullRom, "L6m1": gbg.LalescuSpline(6, 1), "L6": gbg.LalescuSpline(6),
              "G8": gbg.LagrangeSpline(8)}[name]
    rng = np.random.default_rng(m + ncomp)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, origin=(0.25, -2.0, 1.0), dtype=torch.float32)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin, dtype=np.float32)
    pos = np.asfortranarray((np.array(grid.origin) + TWO_PI * (rng.random((m, 3)) * 3 - 1)).astype(np.float32))
    f = np.asfortranarray(rng.standard_normal(n + (ncomp,)).astype(np.float32))
    fd, pd = to_dev(f, dev), to_dev(pos, dev)
    trav = torch.from_numpy((rng.permutation(m) + 1).astype(np.int32)).to(dev)
    got = []
    for t in (None, trav):
        out = gbg.zeros_colmajor((m, ncomp), torch.float32, dev)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        st = _lib.load().gbg_interpolate(grid.c(), _lib.GBG_F32, ncomp, fd.data_ptr(), pd.data_ptr(), m,
                                         t.data_ptr() if t is not None else None, scheme.c(), out.data_ptr(),
                                         status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        _lib.check(st, "gather")
        assert int(status.item()) == 0
        got.append(out.cpu().numpy())
    assert np.array_equal(got[0], got[1])
    assert relerr(got[0], oracle.gather(g, f, pos, scheme.coefficients)) <= 2e-5
    trav[m // 2] = m + 1
    out, status = gbg.zeros_colmajor((m, ncomp), torch.float32, dev), torch.zeros(1, dtype=torch.int32, device=dev)
    _lib.check(_lib.load().gbg_interpolate(grid.c(), _lib.GBG_F32, ncomp, fd.data_ptr(), pd.data_ptr(), m, trav.data_ptr(),
                                           scheme.c(), out.data_ptr(), status.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), "gather")
    assert int(status.item()) == _lib.GBG_DEV_TRAVERSAL


# every window width: odd and even, powers of two and not, held node tables (to 8) and not; grids no
# longer than the window; the oracle's windowed transform with the same window
@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 13, 16])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("comps", [1, 4])
def test_window_gather_and_spread(gbg, dev, width, dtype, comps):
    from gbgperiodicfields_gb300 import _lib
    T = np.float64 if dtype == torch.float64 else np.float32
    n, m = (9, 16, 12), 700
    rng = np.random.default_rng(width)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, origin=(0.5, 0.0, -1.0), dtype=dtype)
    pos = np.asfortranarray((np.array(grid.origin) + TWO_PI * (rng.random((m, 3)) * 2 - 0.5)).astype(T))
    pos[:20] = np.array(grid.origin, T) + np.array(grid.grid_spacing, T) * rng.integers(0, 9, (20, 3)).astype(T)
    f = np.asfortranarray(rng.standard_normal(n + (comps,)).astype(T))
    q = np.asfortranarray(rng.standard_normal((m, comps)).astype(T))
    beta = float(T(2.3) * T(width))
    # the window's weights in the grid's type, as the reference rounds them, then 64-bit sums
    o, d = np.array(grid.origin, T), np.array(grid.grid_spacing, T)
    ci = (pos - o) / d
    base = np.floor(ci).astype(np.int64)
    t = ci - np.floor(ci)
    half = np.where(t < T(0.5), (width + 1) // 2, width // 2) if width % 2 else np.full(t.shape, width // 2)
    off = np.arange(1, width + 1) - half[..., None]
    z = T(2) * (t[..., None] - off.astype(T)) / T(width)
    w = np.exp(T(beta) * (np.sqrt(np.maximum(T(1) - z * z, T(0))) - T(1))).astype(np.float64)
    at = (base[..., None] + off) % np.array(n)[:, None]
    want, spread = np.zeros((m, comps)), np.zeros(n + (comps,))
    for k in range(width):
        for j in range(width):
            for i in range(width):
                x, y, zz = at[:, 0, i], at[:, 1, j], at[:, 2, k]
                wt = w[:, 0, i] * w[:, 1, j] * w[:, 2, k]
                want += wt[:, None] * f[x, y, zz]
                np.add.at(spread, (x, y, zz), wt[:, None] * q)
    lib, code = _lib.load(), _lib.GBG_F64 if dtype == torch.float64 else _lib.GBG_F32
    import ctypes
    stream, need = torch.cuda.current_stream().cuda_stream, ctypes.c_size_t()
    fd, pd, qd = to_dev(f, dev), to_dev(pos, dev), to_dev(q, dev)
    out, field = gbg.zeros_colmajor((m, comps), dtype, dev), gbg.zeros_colmajor(n + (comps,), dtype, dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    _lib.check(lib.gbg_nufft_interp_workspace_size(grid.c(), code, comps, m, width, ctypes.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device=dev)
    _lib.check(lib.gbg_nufft_interp(grid.c(), code, comps, fd.data_ptr(), pd.data_ptr(), m, None, width, beta, out.data_ptr(),
                                    ws.data_ptr(), ws.numel(), status.data_ptr(), stream))
    _lib.check(lib.gbg_nufft_spread_workspace_size(grid.c(), code, comps, m, width, ctypes.byref(need)))
    ws2 = torch.empty(need.value, dtype=torch.uint8, device=dev)
    _lib.check(lib.gbg_nufft_spread(grid.c(), code, comps, field.data_ptr(), pd.data_ptr(), m, qd.data_ptr(), None, width,
                                    beta, ws2.data_ptr(), ws2.numel(), status.data_ptr(), stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    bar = 1e-12 if dtype == torch.float64 else 1e-5
    assert relerr(out.cpu().numpy(), want) <= bar
    assert relerr(field.cpu().numpy(), spread) <= bar


# rows below, at and above a warp's width; a scatter of nothing with beta = 1 refreshes the ghosts of the
# bricks it reaches and leaves every value
@pytest.mark.parametrize("ncomp", [1, 3, 9, 12])
@pytest.mark.parametrize("n", [(8, 9, 33), (65, 8, 10), (32, 33, 8)])
def test_export_rows_and_refreshed_ghosts(gbg, dev, ncomp, n):
    from gbgperiodicfields_gb300 import resident
    rng = np.random.default_rng(3 * ncomp + n[0])
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    data = to_dev(np.asfortranarray(rng.standard_normal(n + (ncomp,))), dev).to(torch.float32)
    field = resident.ResidentField(grid, ncomp, max_stencil_width=8).load(data)
    pos = to_dev(np.asfortranarray(TWO_PI * rng.random((500, 3))), dev)
    bins, scheme = resident.PointBins(grid, 500).build(pos), gbg.LalescuSpline(8)
    before = resident.interpolate_binned(field, bins, scheme)
    resident.anterpolate_binned(field, bins, scheme, torch.zeros_like(before), beta=1.0)
    assert torch.equal(field.read(torch.float32), data)
    assert torch.equal(field.read(torch.float64), data.double())
    assert torch.equal(resident.interpolate_binned(field, bins, scheme), before)


# a brick's region with as many points as are taken in voted trips, one more, and several stagings
@pytest.mark.parametrize("m", [1023, 1024, 1025, 4000])
@pytest.mark.parametrize("ncomp,name", [(9, "cubic"), (12, "quintic"), (5, "octic")])
def test_wide_scatter_either_side_of_the_vote(gbg, oracle, dev, m, ncomp, name):
    from gbgperiodicfields_gb300 import resident
    rng = np.random.default_rng(m + ncomp)
    grid = gbg.Grid3D((32, 32, 32), (TWO_PI,) * 3)
    scheme = {"cubic": gbg.CatmullRom, "quintic": gbg.LalescuSpline(6), "octic": gbg.LalescuSpline(8)}[name]
    # all of them inside the second brick of every axis, cells 12 to 15
    pos = np.asfortranarray(TWO_PI / 32 * (12 + 3.9 * rng.random((m, 3))))
    q = np.asfortranarray(rng.standard_normal((m, ncomp)))
    field = resident.ResidentField(grid, ncomp, max_stencil_width=8)
    bins = resident.PointBins(grid, m).build(to_dev(pos, dev))
    resident.anterpolate_binned(field, bins, scheme, to_dev(q, dev))
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    want = oracle.scatter(g, np.zeros((32, 32, 32, ncomp), order="F"), pos, q, scheme.coefficients)
    assert relerr(field.read(torch.float64).cpu().numpy(), want) <= 1e-5


def _custom_scheme(gbg, coefficients):
    """gbg_scheme_custom: a caller's own (nodes, powers) coefficient matrix."""
    from gbgperiodicfields_gb300 import _lib, api
    coef = np.asarray(coefficients, dtype=np.float64)
    c = _lib.SchemeC()
    flat = np.ascontiguousarray(coef.T).ravel()
    _lib.check(_lib.load().gbg_scheme_custom(coef.shape[0], coef.shape[1],
                                             flat.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.byref(c)), "custom")
    return api._SplineScheme(c)


# Weights above one in the scatter's digit sums: as many equal points in one stencil as a staging, or a pass
# of a crowded cell, can hold, on both sides of those sizes; sums that no rounding hides
@pytest.mark.parametrize("width", [2, 4])
@pytest.mark.parametrize("weight", [1.25, 1.3, 1.4, 1.5, 1.51, 2.9])
@pytest.mark.parametrize("m", [300, 508, 600, 3000])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_scatter_sums_of_large_weights(gbg, dev, width, weight, m, dtype):
    T = np.float64 if dtype == torch.float64 else np.float32
    n = (8, 9, 10)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, dtype=dtype)
    scheme = _custom_scheme(gbg, np.full((width, 1), weight))
    pos = np.asfortranarray(np.full((m, 3), 2.0, dtype=T))
    w = Fraction(float(T(weight)))
    at = [(int(np.floor(2.0 / (TWO_PI / k))) - (width // 2 - 1) + np.arange(width)) % k for k in n]
    for value in (0.3, -0.1, 0.7, 1.0 - 2.0 ** -40):
        q = np.asfortranarray(np.full((m, 3), value, dtype=T))
        got = _scatter_abi(gbg, grid, dev, np.zeros(n + (3,), T, order="F"), pos, q, scheme, 1.0, 0.0)
        want = np.zeros(n + (3,))
        want[np.ix_(*at, range(3))] = float(w ** 3 * Fraction(float(T(value))) * m)
        # the sum of exact products rounded once; a weight's and the node weight's fixed point are below 2^-55
        assert np.abs(got - want).max() <= (2.0 ** -51 if dtype == torch.float64 else 2.0 ** -23) * np.abs(want).max()


# A region with one large quantity whose other nodes hold small ones only: those below the first window of
# digits (2^-18 in FP64, 2^-23 in FP32 of the region's largest) and crowded ones, in any order of the points
@pytest.mark.parametrize("small", [-20, -60, -90, -110])
@pytest.mark.parametrize("m", [40, 300, 1500, 6000])
@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_scatter_of_small_quantities_beside_a_large_one(gbg, dev, small, m, comps, dtype):
    T = np.float64 if dtype == torch.float64 else np.float32
    n = (16, 16, 8)
    rng = np.random.default_rng(m - small)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, dtype=dtype)
    spacing = TWO_PI / np.array(n)
    pos = np.concatenate([(1 + rng.random((m, 3))), [[6.5, 6.5, 2.5]]]) * spacing
    q = np.concatenate([rng.standard_normal((m, comps)) * 2.0 ** small, np.ones((1, comps))])
    pos, q = np.asfortranarray(pos.astype(T)), np.asfortranarray(q.astype(T))
    zero = np.zeros(n + (comps,), T, order="F")
    got = _scatter_abi(gbg, grid, dev, zero, pos, q, gbg.CatmullRom, 1.0, 0.0)
    for _ in range(4):
        order = rng.permutation(m + 1)
        again = _scatter_abi(gbg, grid, dev, zero, pos[order], q[order], gbg.CatmullRom, 1.0, 0.0)
        assert np.array_equal(got, again)
    want = np.zeros(n + (comps,))
    size, reach = _contribution_sizes(gbg.CatmullRom.coefficients, n, pos.astype(np.float64), q.astype(np.float64), spacing)
    w = np.zeros((m + 1, 3, 4))
    ci = pos.astype(np.float64) / spacing
    base = np.floor(ci).astype(np.int64)
    for p in range(3, -1, -1):
        w = w * (ci - base)[..., None] + gbg.CatmullRom.coefficients[:, p]
    parts = {}
    for k in range(4):
        for j in range(4):
            for i in range(4):
                wt = w[:, 0, i] * w[:, 1, j] * w[:, 2, k]
                for p in range(m + 1):
                    node = tuple((base[p, d] - 1 + s) % n[d] for d, s in enumerate((i, j, k)))
                    parts.setdefault(node, []).append(wt[p] * q[p].astype(np.float64))
    for node, terms in parts.items():
        want[node] = [math.fsum(t[c] for t in terms) for c in range(comps)]
    # the weights' own roundings (a dozen of T's per contribution, the locate's among them), the node weight's
    # fixed point (its unit 2^-59, a few of them) and the quantities' last kept bit, 2^-143 of the largest
    eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    bar = 64 * eps * (size + reach) + 4 * 2.0 ** -59 * reach + 2.0 ** -143 * (m + 1)
    assert np.all(np.abs(got - want) <= bar)


# more components than a full brick's line takes, on grids whose clipped bricks let them in: the integer sums do
# not depend on how many components there are, so the first three are those of a deposit of three
@pytest.mark.parametrize("n,width,comps", [((64, 64, 4), 4, 27), ((33, 4, 9), 4, 45), ((40, 2, 2), 2, 81), ((6, 7, 30), 6, 27),
                                           ((64, 64, 4), 4, 23), ((30, 6, 50), 6, 24)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_scatter_of_many_components_on_thin_grids(gbg, dev, n, width, comps, dtype):
    T = np.float64 if dtype == torch.float64 else np.float32
    rng = np.random.default_rng(comps)
    m = 20_000
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, dtype=dtype)
    scheme = gbg.LalescuSpline(width) if width > 2 else gbg.LagrangeSpline(2)
    pos = np.asfortranarray((TWO_PI * rng.random((m, 3))).astype(T))
    q = np.asfortranarray((0.5 + rng.random((m, comps))).astype(T))
    got = _scatter_abi(gbg, grid, dev, np.zeros(n + (comps,), T, order="F"), pos, q, scheme, 1.0, 0.0)
    for c in range(0, comps, 3):
        some = q[:, c:c + 3]
        few = _scatter_abi(gbg, grid, dev, np.zeros(n + some.shape[1:], T, order="F"), pos, some, scheme, 1.0, 0.0)
        assert np.array_equal(got[..., c:c + 3], few)


# spacings whose reciprocal is no normal number: the same cells and fractions as on the grid scaled by a power
# of two, so the same transfers
@pytest.mark.parametrize("scale", [2.0 ** -1030, 2.0 ** -1010, 2.0 ** -880, 2.0 ** 880, 2.0 ** 1016])
@pytest.mark.parametrize("width", [2, 4, 8])
def test_spacings_without_a_normal_reciprocal(gbg, dev, scale, width):
    n, m = (8, 9, 12), 500
    rng = np.random.default_rng(width)
    # positions and domain of few bits, whole at every scale
    domain = (16.0, 18.0, 12.0)
    pos = np.asfortranarray(rng.integers(-512, 1024, (m, 3)) / 64.0)
    f = np.asfortranarray(rng.standard_normal(n + (3,)))
    q = np.asfortranarray(rng.standard_normal((m, 3)))
    scheme = gbg.LalescuSpline(width) if width > 2 else gbg.LagrangeSpline(2)
    got = {}
    for s in (1.0, scale):
        grid = gbg.Grid3D(n, tuple(s * d for d in domain))
        points = gbg.PointSet(to_dev(np.asfortranarray(pos * s), dev))
        values = gbg.interpolate(gbg.VectorFieldPhysical(to_dev(f, dev), grid), points, scheme).data.cpu().numpy()
        deposit = gbg.anterpolate(grid, points, gbg.VectorPointValues(to_dev(q, dev)), scheme).data.cpu().numpy()
        got[s] = values, deposit
    assert relerr(got[scale][0], got[1.0][0]) <= 1e-13  # another kernel's order of the same sums
    assert np.array_equal(got[scale][1], got[1.0][1])


def _bad_and_good(gbg, dev, m):
    """A gather whose every position is non-finite, and one of a single point."""
    grid = gbg.Grid3D((16, 16, 16), (TWO_PI,) * 3)
    field = gbg.ScalarFieldPhysical(to_dev(np.ones((16, 16, 16)), dev), grid)
    bad = gbg.PointSet(to_dev(np.full((m, 3), np.nan), dev))
    good = gbg.PointSet(to_dev(np.full((1, 3), 1.0), dev))
    out = {p: gbg.ScalarPointValues(gbg.empty_colmajor((p.npoints,), torch.float64, dev)) for p in (bad, good)}
    return [lambda p=p: gbg.interpolate_(out[p], field, p, gbg.CatmullRom) for p in (bad, good)]


def test_status_of_a_call_cut_short_reaches_no_later_call(gbg, dev, monkeypatch):
    from gbgperiodicfields_gb300 import _lib
    bad, good = _bad_and_good(gbg, dev, 3_000_000)
    good()
    check = _lib.check

    def interrupted(st, what):
        monkeypatch.setattr(_lib, "check", check)
        raise KeyboardInterrupt  # as a signal between the launch and the wait

    for _ in range(5):
        monkeypatch.setattr(_lib, "check", interrupted)
        with pytest.raises(KeyboardInterrupt):
            bad()
        good()
        with pytest.raises(gbg.InexactError):
            bad()
        good()


def test_status_of_a_call_inside_another(gbg, dev, monkeypatch):
    from gbgperiodicfields_gb300 import _lib
    bad, good = _bad_and_good(gbg, dev, 100)
    check = _lib.check

    def nested(inner):
        def run(st, what):
            monkeypatch.setattr(_lib, "check", check)
            torch.cuda.synchronize()
            inner()
            return check(st, what)
        return run

    monkeypatch.setattr(_lib, "check", nested(good))
    with pytest.raises(gbg.InexactError):
        bad()
    good()


def test_status_by_thread(gbg, dev):
    import threading
    calls = [_bad_and_good(gbg, dev, 50_000) for _ in range(4)]
    wrong = []

    def work(k):
        bad, good = calls[k]
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(40):
                try:
                    (bad if (i + k) % 2 else good)()
                    reported = False
                except gbg.InexactError:
                    reported = True
                if reported != bool((i + k) % 2):
                    wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("bad", ["positions", "quantities"])
def test_deposit_of_bad_points_only(gbg, dev, bad):
    # every lane of every warp reports
    m = 200_000
    rng = np.random.default_rng(3)
    grid = gbg.Grid3D((32, 32, 32), (TWO_PI,) * 3)
    pos, q = TWO_PI * rng.random((m, 3)), rng.standard_normal((m, 3))
    (pos if bad == "positions" else q)[:] = np.nan
    points, values = gbg.PointSet(to_dev(pos, dev)), gbg.VectorPointValues(to_dev(q, dev))
    for _ in range(2):
        with pytest.raises(gbg.InexactError):
            gbg.anterpolate(grid, points, values, gbg.CatmullRom)


# bricks whose tables take a third, half and all of an SM's memory
@pytest.mark.parametrize("brick", [(11, 8, 8), (16, 8, 8), (20, 10, 10), (32, 8, 8), (16, 16, 8)])
@pytest.mark.parametrize("width,ncomp", [(2, 3), (4, 4), (4, 1)])
@pytest.mark.parametrize("density", [0.05, 1.3])
def test_scatter_of_every_brick_share(gbg, oracle, dev, brick, width, ncomp, density):
    _resident_scatter(gbg, oracle, dev, (40, 33, 24), brick, width, ncomp, density)


def _resident_scatter(gbg, oracle, dev, n, brick, width, ncomp, density):
    """A resident scatter against the oracle, and the batched form's against it bit by bit."""
    from gbgperiodicfields_gb300 import resident
    m = int(density * np.prod(n))
    rng = np.random.default_rng(m + 100 * ncomp + width)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    scheme = gbg.LalescuSpline(width) if width > 2 else gbg.LagrangeSpline(2)
    pos = np.asfortranarray(TWO_PI * rng.random((m, 3)))
    q = np.asfortranarray(rng.standard_normal((m, ncomp)).astype(np.float32))
    want = oracle.scatter(g, np.zeros(n + (ncomp,), order="F"), pos, q.astype(np.float64), scheme.coefficients)
    bins = resident.PointBins(grid, m, brick=brick).build(to_dev(pos, dev))
    dest = resident.ResidentField(grid, ncomp, max_stencil_width=width)
    qd = to_dev(q, dev)
    resident.anterpolate_binned(dest, bins, scheme, qd)
    got = dest.read(torch.float32).cpu().numpy()
    assert relerr(got, want) <= 1e-5
    again = resident.ResidentField(grid, ncomp, max_stencil_width=width)
    resident.Batch([dict(field=dest, bins=bins, scheme=scheme, dest=again, q=qd)]).run()
    assert np.array_equal(again.read(torch.float32).cpu().numpy(), got)


# mean regions below, at and above 7/8 of the smaller staging (710 points at width 4, 1088 at width 2)
@pytest.mark.parametrize("width,density", [(4, 0.30), (4, 0.36), (4, 0.37), (4, 0.5), (4, 0.9), (2, 0.9), (2, 0.97), (2, 0.98), (2, 1.2)])
def test_scatter_either_side_of_the_third_share(gbg, oracle, dev, width, density):
    _resident_scatter(gbg, oracle, dev, (44, 32, 24), (11, 8, 8), width, 3, density)


# regions of few and of many points at the widths whose trips are never voted, and mean regions either side of
# 1024 points at those where they are
@pytest.mark.parametrize("width,density", [(2, 0.1), (2, 1.5), (8, 0.1), (8, 0.4), (4, 0.5), (4, 0.7), (6, 0.3), (6, 0.45)])
@pytest.mark.parametrize("ncomp", [5, 12])
def test_scatter_trips_at_every_width(gbg, oracle, dev, width, density, ncomp):
    _resident_scatter(gbg, oracle, dev, (33, 24, 20), (11, 8, 8), width, ncomp, density)


# runs at and above the longest that one CTA sorts (16384, or a 255th of the points), alone, beside shorter
# ones and nearly as many as there can be, shares of the points that end within a tile
@pytest.mark.parametrize("runs,spread", [((16384,), 0), ((16385,), 0), ((16384, 16385, 1025, 40_000, 1024, 2500), 30_001),
                                         ((200_000,), 1), ((20_000,) * 200, 77), ((16_500,) * 240, 300_000)])
def test_bins_order_with_huge_runs(gbg, dev, runs, spread):
    from gbgperiodicfields_gb300 import resident
    n = np.array((24, 24, 24))
    rng = np.random.default_rng(len(runs) + spread)
    grid = gbg.Grid3D(tuple(n), tuple(float(v) for v in n))  # cells of edge 1
    cells = rng.choice(24 ** 3, len(runs), replace=False)
    pos = [24 * rng.random((spread, 3))]
    for k, c in zip(cells, runs):
        pos.append(np.array([k % 24, (k // 24) % 24, k // 576]) + rng.random((c, 3)))
    pos = np.concatenate(pos)
    pos = np.asfortranarray(pos[rng.permutation(len(pos))])
    bins = resident.PointBins(grid, len(pos), brick=(8, 8, 8))
    c = np.floor(pos).astype(np.int64) % n
    br = c // 8
    loc = c - 8 * br
    key = ((br[:, 2] * 3 + br[:, 1]) * 3 + br[:, 0]) * 512 + (loc[:, 2] * 8 + loc[:, 1]) * 8 + loc[:, 0]
    want = np.argsort(key, kind="stable") + 1
    for _ in range(2):
        bins.build(to_dev(pos, dev))
        assert np.array_equal(bins.order().cpu().numpy(), want)
    # the records follow: a linear field is reproduced by the cubic spline inside the box
    x = torch.arange(24, dtype=torch.float64, device=dev)[:, None, None].expand(24, 24, 24)
    field = resident.ResidentField(grid, 1, 4).load(gbg.colmajor(x.contiguous()[..., None]))
    got = resident.interpolate_binned(field, bins, gbg.CatmullRom).cpu().numpy()[:, 0]
    inner = (pos[:, 0] >= 2) & (pos[:, 0] < 21)
    assert np.abs(got - pos[:, 0])[inner].max(initial=0.0) <= 24e-5


# every remainder of three: a component's sums do not depend on the others beside it, sparse and crowded, with
# quantities of one window and of several
@pytest.mark.parametrize("comps", [1, 2, 3, 4, 5, 7, 8, 10])
@pytest.mark.parametrize("width", [2, 4, 6, 8])
@pytest.mark.parametrize("m,spread", [(2000, 0), (2000, 60), (60_000, 0), (60_000, 30)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_scatter_of_every_component_count(gbg, dev, comps, width, m, spread, dtype):
    T = np.float64 if dtype == torch.float64 else np.float32
    n = (17, 16, 13)
    rng = np.random.default_rng(comps + m)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3, dtype=dtype)
    scheme = gbg.LalescuSpline(width) if width > 2 else gbg.LagrangeSpline(2)
    pos = np.asfortranarray((TWO_PI * rng.random((m, 3))).astype(T))
    q = (rng.standard_normal((m, comps)) * 2.0 ** (-spread * rng.random((m, 1)))).astype(T)
    q[rng.integers(m), rng.integers(comps)] = np.nan
    q = np.asfortranarray(q)
    old = np.asfortranarray(rng.standard_normal(n + (comps,)).astype(T))
    got = _scatter_abi(gbg, grid, dev, old, pos, q, scheme, 1.0, 0.5)
    for c in range(comps):
        alone = _scatter_abi(gbg, grid, dev, old[..., c:c + 1], pos, q[:, c:c + 1], scheme, 1.0, 0.5)
        assert np.array_equal(got[..., c:c + 1], alone, equal_nan=True)


# crowded regions whose points lie in one cell, in one row of cells and in a few: a node's lanes share a row's
# points there, with pieces whose ends cut the rows
@pytest.mark.parametrize("extent", [(1, 1, 1), (6, 1, 1), (2, 2, 1), (5, 5, 4)])
@pytest.mark.parametrize("m", [505, 509, 1777, 40_003])
@pytest.mark.parametrize("width", [2, 4, 8])
def test_scatter_of_crowded_cells(gbg, oracle, dev, extent, m, width):
    n = (16, 11, 9)
    rng = np.random.default_rng(m + width)
    grid = gbg.Grid3D(n, (TWO_PI,) * 3)
    g = oracle.grid_dict(grid.grid_size, grid.domain_size, grid.origin)
    scheme = gbg.LalescuSpline(width) if width > 2 else gbg.LagrangeSpline(2)
    pos = np.asfortranarray((np.array([5.0, 6.0, 3.0]) + rng.random((m, 3)) * extent) * TWO_PI / n)
    q = np.asfortranarray(rng.standard_normal((m, 3)))
    zero = np.zeros(n + (3,), order="F")
    got = _scatter_abi(gbg, grid, dev, zero, pos, q, scheme, 1.0, 0.0)
    want = oracle.scatter(g, zero.copy(order="F"), pos, q, scheme.coefficients)
    size, reach = _contribution_sizes(scheme.coefficients, n, pos, q, TWO_PI / np.array(n))
    assert np.all(np.abs(got - want) <= 1e-12 * size + 4 * 2.0 ** -59 * reach)
    order = rng.permutation(m)
    assert np.array_equal(got, _scatter_abi(gbg, grid, dev, zero, pos[order], q[order], scheme, 1.0, 0.0))
