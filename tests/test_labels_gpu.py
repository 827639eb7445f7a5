"""GPU labelling parity: the CUDA labeller against the oracle's literal PBA+
restatement (and the pointwise rule at sizes where the restatement is slow).
Labels are integer work: equality is bit-exact."""
import numpy as np
import pytest

from test_oracle import cases, grid
from workloads import MARKER, config_inputs, disk_sites, gaussian_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_labels_equal_pba_random_and_lattices(gcvt_lib, oracle, cuda_device, seed):
    for n, pts in cases(seed, 24):
        g = grid(n, pts)
        got = gcvt_lib.label_grid(g)
        want = oracle.pba_label(g)
        bad = np.argwhere((got != want).any(-1))
        assert bad.size == 0, (n, len(pts), bad[:3], got[tuple(bad[0])], want[tuple(bad[0])])


def test_labels_equal_pba_1024_dense(gcvt_lib, oracle, cuda_device):
    rng = np.random.default_rng(11)
    for m in (1, 3, 50, 4096, 60000):
        n = 1024
        pick = rng.choice(n * n, size=m, replace=False)
        ys, xs = np.divmod(pick, n)
        g = gcvt_lib.sites_from_points(n, xs, ys)
        assert np.array_equal(gcvt_lib.label_grid(g), oracle.pba_label(g)), m


@pytest.mark.parametrize("n", [2048, 4096])
def test_labels_large_against_pointwise_rule(gcvt_lib, oracle, cuda_device, n):
    rho = gaussian_density(n, 8, 4.0, 0.02, 0.15, seed=n)
    g = disk_sites(n, n * n // 64, seed=n, density=rho)
    assert np.array_equal(gcvt_lib.label_grid(g), oracle.spec_label(g))


def test_labels_non_power_of_two(gcvt_lib, oracle, cuda_device):
    rng = np.random.default_rng(3)
    n = 768
    pick = rng.choice(n * n, size=3000, replace=False)
    ys, xs = np.divmod(pick, n)
    g = gcvt_lib.sites_from_points(n, xs, ys)
    assert np.array_equal(gcvt_lib.label_grid(g), oracle.spec_label(g))


def test_full_row_and_full_column(gcvt_lib, oracle, cuda_device):
    n = 512
    pts = [(x, 77) for x in range(n)] + [(300, y) for y in range(n)]
    g = grid(n, sorted(set(pts)))
    assert np.array_equal(gcvt_lib.label_grid(g), oracle.pba_label(g))


def test_no_sites_gives_marker(gcvt_lib, cuda_device):
    g = np.full((256, 256, 2), MARKER, np.int16)
    out = gcvt_lib.label_grid(g)
    assert (out == MARKER).all()


def test_rejects_bad_grids(gcvt_lib, cuda_device):
    g = np.full((256, 256, 2), MARKER, np.int16)
    g[5, 6] = (7, 5)  # site pixel holding someone else's coordinates
    with pytest.raises(gcvt_lib.GcvtError) as e:
        gcvt_lib.label_grid(g)
    assert e.value.code == 4
    with pytest.raises(gcvt_lib.GcvtError) as e:
        gcvt_lib.label_grid(np.full((200, 200, 2), MARKER, np.int16))
    assert e.value.code == 2


def test_context_label_device_buffers(gcvt_lib, oracle, cuda_device):
    import torch
    sites, rho, mask, _ = config_inputs("plain_1024", seed=2)
    want = oracle.pba_label(sites)
    ctx = gcvt_lib.Context(1024)
    ctx.load(torch.from_numpy(sites).to(cuda_device), torch.from_numpy(rho).to(cuda_device),
             torch.from_numpy(mask).to(cuda_device))
    out = torch.empty((1024, 1024, 2), dtype=torch.int16, device=cuda_device)
    ctx.label(out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    ctx.close()


@pytest.mark.parametrize("n,kind", [(512, "1"), (512, "2"), (768, "3"), (512, "5"), (512, "18"),
                                    (1024, "mirror"), (768, "far"), (2048, "one"), (256, "one"),
                                    (768, "1"), (768, "2"), (768, "5"), (768, "18")])
def test_tile_lists_and_their_overflows(gcvt_lib, oracle, cuda_device, n, kind):
    """The tile labeller's dispatch: a crowded block of one site per 1 to 18 pixels
    beside empty space (window, candidate and block lists at and past their ends,
    tiles far from any site, the row pass behind them and on grids up to 512), mirror pairs across bands seen
    from near and far, lone sites."""
    rng = np.random.default_rng(n)
    if kind == "mirror":  # pairs of one column about band edges and tile rows, far apart
        xs, ys = [], []
        for x in range(40, n, 170):
            for c in (64, 128, 200, 448, 512, 720):
                k = int(rng.integers(1, 40))
                xs += [x, x]
                ys += [c - k, c + k]
        pts = set(zip(xs, ys))
    elif kind == "far":
        pts = {(3, 5), (3, 765), (760, 2), (384, 384), (385, 384), (384, 386)}
    elif kind == "one":
        pts = {(n - 1, n // 3)}
    else:
        b = rng.random((160, 200)) < 1.0 / int(kind)
        ys, xs = np.nonzero(b)
        pts = set(zip((xs + 37).tolist(), (ys + 61).tolist()))
        pts |= {tuple(p) for p in rng.integers(0, n, (9, 2)).tolist()}
    g = grid(n, sorted(pts))
    got, want = gcvt_lib.label_grid(g), oracle.spec_label(g)
    bad = np.argwhere((got != want).any(-1))
    assert bad.size == 0, (len(bad), bad[:3], got[tuple(bad[0])], want[tuple(bad[0])])


@pytest.mark.parametrize("n,kind", [(768, "block380"), (768, "block381"), (1024, "band"),
                                    (2048, "late"), (2304, "late"), (2304, "block380"),
                                    (2304, "block381"), (2304, "band"), (2048, "quarter"),
                                    (2304, "quarter"), (2304, "stripe"), (1024, "uniform13"),
                                    (1024, "uniform12")])
def test_crowded_bands(gcvt_lib, oracle, cuda_device, n, kind):
    """Bands labelled by rows beside bands labelled by tiles: a 64 x 64 block at and past
    the count that sends its band to the rows, a crowded band, tiles whose lists overflow
    in a block below that count, crowded parts of the grid, the count that sends all of
    it there; grids up to and past the size where one such band takes the others along."""
    import torch
    rng = np.random.default_rng(n)
    b = np.zeros((n, n), bool)
    b.ravel()[rng.choice(n * n, n * n // 300, replace=False)] = True
    if kind.startswith("block"):
        q = np.zeros(64 * 64, bool)
        q[rng.choice(64 * 64, int(kind[5:]), replace=False)] = True
        b[128:192, 320:384] = q.reshape(64, 64)
    elif kind == "band":
        b[256:320] = rng.random((64, n)) < 0.3
    elif kind == "late":  # 196 sites of one tile, a lone block far from any other site
        b[300:314, 420:434] = True
        b[n // 2:] = False
        b[n - 70, n - 70] = True
    elif kind == "quarter":
        b[:n // 2, :n // 2] = rng.random((n // 2, n // 2)) < 0.25
    elif kind == "stripe":
        b[:, 700:800] = rng.random((n, 100)) < 0.25
    else:
        b[:] = False
        b.ravel()[rng.choice(n * n, n * n // int(kind[7:]), replace=False)] = True
    ys, xs = np.nonzero(b)
    g = grid(n, list(zip(xs.tolist(), ys.tolist())))
    want = oracle.spec_label(g)
    assert np.array_equal(gcvt_lib.label_grid(g), want)
    d = torch.from_numpy(g).cuda()
    o = torch.empty_like(d)
    if n <= 2048:
        lib = gcvt_lib.load_library()
        assert lib.gcvt_label_grid_static(d.data_ptr(), o.data_ptr(), n, None) == 0
        assert np.array_equal(o.cpu().numpy(), want)


def test_label_into_other_buffers(gcvt_lib, oracle, cuda_device):
    """Kernels write a device buffer of the context's device that holds the labels; any
    other pointer goes through a copy, which refuses what it cannot write.  At odd
    offsets, in pinned host memory passed as device memory, in host memory so passed."""
    import torch
    n = 768
    rng = np.random.default_rng(5)
    p = rng.choice(n * n, 4000, replace=False)
    g = gcvt_lib.sites_from_points(n, p % n, p // n)
    want = oracle.spec_label(g)
    ctx, lib = gcvt_lib.Context(n), gcvt_lib.load_library()
    ctx.load(g, np.ones((n, n), np.float32), np.zeros((n, n), np.uint8))
    raw = torch.zeros(n * n * 2 + 64, dtype=torch.int16, device="cuda")
    for off in (0, 1, 2, 7, 64):
        raw.zero_()
        torch.cuda.synchronize()
        assert lib.gcvt_ctx_label(ctx.h, raw.data_ptr() + 2 * off, 1) == 0
        torch.cuda.synchronize()
        assert np.array_equal(raw.cpu().numpy()[off:off + 2 * n * n].reshape(n, n, 2), want)
        assert not raw[:off].any() and not raw[off + 2 * n * n:].any()
    pinned = torch.zeros((n, n, 2), dtype=torch.int16).pin_memory()
    host = np.zeros((n, n, 2), np.int16)
    for ptr, out in ((pinned.data_ptr(), pinned.numpy()), (host.ctypes.data, host)):
        rc = lib.gcvt_ctx_label(ctx.h, ptr, 1)
        torch.cuda.synchronize()
        assert rc == 3 or (rc == 0 and np.array_equal(out, want))  # GCVT_ERR_CUDA
    assert np.array_equal(ctx.label(), want)  # the context goes on
    ctx.close()


@pytest.mark.parametrize("n,kind", [(768, "circle"), (1024, "circle"), (2304, "circle"),
                                    (1024, "column"), (768, "diagonal"), (2304, "diagonal"),
                                    (2304, "solid"), (1024, "rings"), (768, "late")])
def test_many_candidates(gcvt_lib, oracle, cuda_device, n, kind):
    """Tiles of more candidates than their list holds: the middle of a
    circle of sites (all at one distance, mirror pairs across bands among them), a full
    column or diagonal, concentric circles; and a solid block, whose sites do not fit the
    far blocks' lists either."""
    t = np.arange(6 * n) * (2 * np.pi / (6 * n))
    cs = np.stack([np.cos(t), np.sin(t)], 1)
    q = {"circle": lambda: np.rint(n / 2 + 0.45 * n * cs),
         "rings": lambda: np.concatenate([np.rint(n / 2 + r * n * cs) for r in (0.2, 0.35, 0.48)]),
         "column": lambda: np.stack([np.full(n, n // 2), np.arange(n)], 1),
         "diagonal": lambda: np.stack([np.arange(n), n - 1 - np.arange(n)], 1),
         "solid": lambda: np.stack(np.meshgrid(np.arange(300, 560), np.arange(310, 540)), -1).reshape(-1, 2),
         "late": lambda: np.concatenate([np.stack(np.meshgrid(np.arange(14), np.arange(14)), -1)
                                         .reshape(-1, 2) + (420, 300), [(700, 60)]])}[kind]()
    q = np.unique(q.astype(int), axis=0)
    g = gcvt_lib.sites_from_points(n, q[:, 0], q[:, 1])
    assert np.array_equal(gcvt_lib.label_grid(g), oracle.spec_label(g))
