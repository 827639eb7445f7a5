"""The Lloyd kernel's float row bounds at the edges of their dispatch: crowded
windows (more candidates than a lane's list holds), cells of more rows than the
row list and wider than a 16-pixel chunk, windows above and below one 32-row
word and two, covering bounds beyond the float range, sites in one column or
row, sites at the grid's border.  Moments against the FP64 oracle (1e-5
relative, the engine's contract: FP32 chunks of 16 pixels, two-float sums), and
the lane-per-site and warp-per-site kernels against each other, bit for bit
(they do the same sums in the same order)."""
import numpy as np
import pytest

from workloads import gaussian_density

pytestmark = pytest.mark.gpu


def points(kind, n, rng):
    """Distinct (x, y) of a site set."""
    if kind == "crowd":    # a packed block (windows of hundreds of sites) and a few far ones
        b = np.stack(np.meshgrid(np.arange(24), np.arange(24)), -1).reshape(-1, 2) + n // 2
        return np.concatenate([b, rng.integers(0, n, (30, 2))])
    if kind == "one":      # a single cell: the whole support
        return np.array([[n // 2, n // 3]])
    if kind == "column":   # horizontal slabs, same-column limits on both sides
        return np.stack([np.full(n // 16, n // 2), np.arange(n // 16) * 16 + 3], 1)
    if kind == "row":      # vertical slabs: one row bound per side, tall cells
        return np.stack([np.arange(n // 16) * 16 + 5, np.full(n // 16, n // 2)], 1)
    if kind == "border":   # along the grid's edges
        t = np.arange(0, n, 7)
        return np.concatenate([np.stack([t, 0 * t], 1), np.stack([0 * t + n - 1, t], 1),
                               rng.integers(0, n, (40, 2))])
    return rng.integers(0, n, (int(kind), 2))  # that many at random


@pytest.mark.parametrize("n,kind", [(256, "crowd"), (512, "crowd"), (256, "one"), (1024, "one"),
                                    (512, "column"), (512, "row"), (768, "border"), (512, 12),
                                    (1024, 60), (512, 250), (512, 1200), (512, 6000),
                                    (768, 20000)])
def test_cells_match_fp64_and_each_other(gcvt_lib, oracle, cuda_device, n, kind):
    rng = np.random.default_rng(n)
    q = np.unique(points(kind, n, rng), axis=0)
    sites = gcvt_lib.sites_from_points(n, q[:, 0], q[:, 1])
    rho = gaussian_density(n, 6, 4.0, 0.05, 0.2, 3)
    if kind == "border":
        rho = np.maximum(rho, np.float32(0.25))  # density up to the grid's edge
    mask = np.zeros((n, n), np.uint8)
    _, mom, energy, _ = oracle.lloyd_step(sites, rho, mask, 2.0)
    ctx = gcvt_lib.Context(n)
    ctx.load(sites, rho, mask)
    got = ctx.moments()
    ys, xs = np.nonzero(sites[..., 0] != -32768)
    for k in range(3):
        want, have = mom[k][ys, xs], got[k][ys, xs]
        assert (np.abs(have - want) <= 1e-5 * np.abs(want)).all()
    e = got[3][ys, xs].sum() / (n * n)
    assert abs(e - energy) <= 1e-5 * energy
    runs = []
    for mode in (1, 2):
        ctx.set_tuning(cell_mode=mode)
        ctx.load(sites, rho, mask)
        ctx.iterate(4)
        runs.append((ctx.sites(), ctx.info()))
    assert np.array_equal(runs[0][0], runs[1][0])
    assert runs[0][1] == runs[1][1]
    ctx.close()


@pytest.mark.parametrize("n,m", [(256, 0), (256, 1), (256, 7), (256, 9), (512, 1024), (512, 1025),
                                 (1024, 8185), (1024, 8192), (1024, 8193), (4096, 700),
                                 (4352, 700)])
def test_one_launch_iterations(gcvt_lib, cuda_device, n, m):
    """Few sites' one-launch iterations against the list and the lane-per-site
    kernel, bit for bit: no site, a part of a block, the group counts around the
    two ways of folding them, the site and grid limits of the dispatch."""
    rng = np.random.default_rng(m)
    rho = gaussian_density(n, 6, 4.0, 0.05, 0.2, 3)
    p = rng.choice(np.flatnonzero(rho.ravel() > 0), m, replace=False)
    fixed = np.zeros((n, n), np.uint8)
    fixed.ravel()[p[::5]] = 1
    sites = gcvt_lib.sites_from_points(n, p % n, p // n)
    ctx = gcvt_lib.Context(n)
    runs = []
    for mode in (1, 2):
        ctx.set_tuning(cell_mode=mode)
        ctx.load(sites, rho, fixed)
        ctx.iterate(12)
        runs.append((ctx.sites(), ctx.info()))
    assert np.array_equal(runs[0][0], runs[1][0])
    assert runs[0][1] == runs[1][1]
    ctx.close()


@pytest.mark.parametrize("n,gaussians", [(1024, 2), (1024, 9), (512, 6)])
def test_one_context_with_changing_counts(gcvt_lib, cuda_device, n, gaussians):
    """The form of an iteration and its recorded launches follow the loaded sites: one
    context by its own rule against fresh ones with a site per lane, bit for bit, over the
    one-launch form's size classes and the limits between the forms, up and down."""
    rng = np.random.default_rng(n + gaussians)
    rho = gaussian_density(n, gaussians, 4.0, 0.05, 0.2, 3)
    inside = np.flatnonzero(rho.ravel() > 0)
    fixed = np.zeros((n, n), np.uint8)
    ctx = gcvt_lib.Context(n)
    for m in (700, 9000, 20000, 300, 40000, 8192, 8193, 700, 32768, 32769, 256, 257, 9000, 20):
        p = rng.choice(inside, m, replace=False)
        sites = gcvt_lib.sites_from_points(n, p % n, p // n)
        ctx.load(sites, rho, fixed)
        ctx.iterate(21)
        one = gcvt_lib.Context(n)
        one.set_tuning(cell_mode=1)
        one.load(sites, rho, fixed)
        one.iterate(21)
        assert np.array_equal(ctx.sites(), one.sites()), m
        assert ctx.info() == one.info(), m
        one.close()
    ctx.close()


def crowded(kind, n, rng):
    if kind == "circle":  # cells reach across the empty inside
        t = rng.uniform(0, 2 * np.pi, 700)
        return np.rint(n / 2 + (n * 0.4) * np.stack([np.cos(t), np.sin(t)], 1)).astype(int)
    if kind == "cluster":
        return np.clip(np.rint(n / 3 + rng.normal(0, 9, (800, 2))), 0, n - 1).astype(int)
    if kind == "border":  # every second pixel of the border, two sites inside
        t = np.arange(0, n, 2)
        q = [np.stack([t, 0 * t], 1), np.stack([t, 0 * t + n - 1], 1), np.stack([0 * t, t], 1),
             np.stack([0 * t + n - 1, t], 1)]
        return np.concatenate(q + [np.array([(n // 2, n // 3), (n // 2, n // 3 + 9)])])
    if kind == "line":  # a full column and its neighbours
        t = np.arange(0, n)
        return np.concatenate([np.stack([0 * t + n // 2 + d, t], 1)[d & 1::1 + d % 3] for d in range(5)])
    b = int(kind)  # that many sites around a lone one, so that its window holds them all
    a = np.stack(np.meshgrid(np.arange(12), np.arange(12)), -1).reshape(-1, 2)[:b]
    return np.concatenate([a + n // 2, [(n // 2 + 60, n // 2 + 6)]])


@pytest.mark.parametrize("n,kind", [(512, "circle"), (768, "circle"), (512, "cluster"),
                                    (768, "cluster"), (512, "border"), (512, "line"),
                                    (256, "127"), (256, "128"), (256, "129"), (256, "144")])
def test_crowded_windows_by_warps(gcvt_lib, oracle, cuda_device, n, kind):
    """Windows of more candidates than a warp's list holds (128): a site per warp, with
    and without the list launch, against a site per lane, bit for bit, and the first
    iteration's energy against FP64."""
    rng = np.random.default_rng(n)
    q = np.unique(crowded(kind, n, rng), axis=0)
    sites = gcvt_lib.sites_from_points(n, q[:, 0], q[:, 1])
    rho = gaussian_density(n, 6, 4.0, 0.05, 0.2, 3)
    fixed = np.zeros((n, n), np.uint8)
    fixed[q[::7, 1], q[::7, 0]] = 1
    _, _, energy, _ = oracle.lloyd_step(sites, rho, fixed, 2.0)
    ctx = gcvt_lib.Context(n)
    runs = []
    for mode in (1, 2, 0):
        ctx.set_tuning(cell_mode=mode)
        ctx.load(sites, rho, fixed)
        ctx.iterate(1)
        first = ctx.info()["energy"]
        assert abs(first - energy) <= 1e-5 * energy
        ctx.iterate(3)
        runs.append((ctx.sites(), ctx.info()))
    for r in runs[1:]:
        assert np.array_equal(r[0], runs[0][0]) and r[1] == runs[0][1]
    ctx.close()
