"""The branches that rows take through the sift kernels by their length and knot density, at the
sizes where they change: against the CPU oracle, bit for bit.

The tile kernels hold a tile's knots in shared memory: rows of up to about 660 knots in their
densest tile (of 2048 samples) go to the sparse form of k_tile_sift, rows of up to about 1780 to
the dense form, denser rows take one envelope after the other there; with few tiles one launch
serves all rows.  k_spline_solve keeps its tables in shared memory up to 256 tiles and solves in
one pass up to 2048 separators.  The end rule is applied by k_tile_knots when the row's first or
last tile holds six knots of the envelope, else by k_spline_solve.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 2048


def _zigzag(n, per_tile, seed):
    """A row with about per_tile extrema in every tile, at random places."""
    rng = np.random.default_rng(seed)
    pos = [0]
    for t0 in range(0, n, TILE):
        m = min(TILE, n - t0)
        k = min(per_tile, m)
        pos += list(t0 + np.sort(rng.choice(m, k, replace=False)))
    pos = np.unique(np.array(pos + [n - 1]))
    val = (1.0 - 2.0 * (np.arange(pos.size) & 1)) * (1.0 + rng.random(pos.size))
    return np.interp(np.arange(n), pos, val)


def _check_envelopes(pkg, orc, cuda, rows, copies=1):
    import torch
    h = torch.tensor(np.tile(rows, (copies, 1)), device=cuda)
    up, lo, _ = pkg.envelopes(h)
    up, lo = up.cpu().numpy(), lo.cpu().numpy()
    for r in range(rows.shape[0]):
        eu = orc.envelope(rows[r], 0, solver=1, chunk=16)
        el = orc.envelope(rows[r], 1, solver=1, chunk=16)
        for k in range(copies):
            i = k * rows.shape[0] + r
            assert np.array_equal(up[i], eu), f"upper envelope of row {i}"
            assert np.array_equal(lo[i], el), f"lower envelope of row {i}"


# knots of a tile: none to all samples, the chunks' edges, both sides of the capacities
DENSITIES = [0, 1, 2, 5, 11, 12, 13, 31, 32, 33, 64, 600, 640, 660, 680, 720, 1500, 1740, 1780,
             1800, 1860, 2000, 2048]


@pytest.mark.parametrize("n", [2 * TILE, 2 * TILE + 1, 3 * TILE - 1, 3 * TILE + 18])
def test_envelopes_of_every_density_one_launch(pkg, orc, cuda, n):
    rows = np.stack([_zigzag(n, k, 31 * k + n) for k in DENSITIES])
    _check_envelopes(pkg, orc, cuda, rows)


@pytest.mark.parametrize("n", [2 * TILE + 3, 3 * TILE])
def test_envelopes_of_mixed_densities_two_launches(pkg, orc, cuda, n):
    # 460 tiles and more: the rows of the two forms in two launches
    rows = np.stack([_zigzag(n, k, 7 * k + n) for k in DENSITIES])
    _check_envelopes(pkg, orc, cuda, rows, copies=12)


@pytest.mark.parametrize("n,per_tile", [
    (34 * TILE + 5, 2048),    # more than 2048 separators: several passes
    (31 * TILE + 1, 2048),    # just fewer
    (256 * TILE, 40),         # the last size whose tables are in shared memory
    (256 * TILE + 1, 40),     # the first whose are not; a tile of one sample
    (300 * TILE + 77, 700),
    (40 * TILE, 1),           # tiles without a knot of one envelope or of both
])
def test_envelopes_of_long_rows(pkg, orc, cuda, n, per_tile):
    _check_envelopes(pkg, orc, cuda, _zigzag(n, per_tile, n)[None, :])


@pytest.mark.parametrize("side", ["first", "last", "both"])
@pytest.mark.parametrize("few", [0, 1, 2, 4, 6, 8, 11])
def test_envelopes_with_sparse_end_tiles(pkg, orc, cuda, side, few):
    n = 4 * TILE + 700
    row = _zigzag(n, 90, few)
    end = _zigzag(n, few, 1000 + few)
    if side in ("first", "both"):
        row[:TILE] = end[:TILE]
    if side in ("last", "both"):
        row[4 * TILE:] = end[4 * TILE:]
    _check_envelopes(pkg, orc, cuda, row[None, :])


def _ensemble(nr, n):
    """Noise rows of every density, so that the forms mix and rows change between them."""
    return np.stack([_zigzag(n, DENSITIES[3:][r % 20], 5 + r) for r in range(nr)])


@pytest.mark.parametrize("nr,n", [(150, 2 * TILE + 1), (230, 2 * TILE - 2), (40, 3 * TILE + 9)])
def test_decomposition_of_mixed_densities(pkg, orc, cuda, wl, monkeypatch, nr, n):
    """The multi-kernel iteration with two launches and with one, and with a row's counts in
    separate words (rows of 2^17 tiles and more) instead of one."""
    import torch
    monkeypatch.setenv("CEEMDAN_SMALL", "0")
    x, noise = wl.eeg_like(n, seed=3), _ensemble(nr, n)

    def run():
        imfs, it = pkg.iceemdan(torch.tensor(x, device=cuda), nr, 4, 12, 0.2,
                                noise=torch.tensor(noise, device=cuda), noise_sift_cap=15,
                                return_iters=True)
        return imfs.cpu().numpy(), list(it)

    got, it = run()
    ref, rit = orc.iceemdan(x, noise, 4, 12, 0.2, solver=1, chunk=16, noise_sift_cap=15,
                            return_iters=True)
    assert it == list(rit)
    assert np.array_equal(got, ref)
    monkeypatch.setenv("CEEMDAN_SPLIT_COUNT", "1")
    split, sit = run()
    assert sit == it
    assert np.array_equal(split, got)


def test_batched_channels_of_mixed_densities(pkg, wl, cuda):
    """Ragged channels in one loop, their rows of both forms at once, against the plain calls."""
    import torch
    lengths = [2 * TILE + 1, 3 * TILE, 9 * TILE - 5]
    ys = [torch.tensor(wl.eeg_like(n, seed=n % 13), device=cuda) for n in lengths]
    kw = dict(noise_sift_cap=25, return_iters=True)
    got, its = pkg.iceemdan_batched(ys, 60, 5, 15, 0.2, seed=11, **kw)
    for c, y in enumerate(ys):
        ref, it = pkg.iceemdan(y, 60, 5, 15, 0.2, seed=11 + c, **kw)
        assert list(its[c]) == list(it)
        assert torch.equal(got[c], ref)


@pytest.mark.parametrize("pair", ["1", "0"])
@pytest.mark.parametrize("n,nr", [
    (5, 3), (33, 75), (4096, 74), (4096, 75),    # two CTAs a realization up to 74 of them
    (5000, 80), (5248, 80), (5312, 80), (5376, 80), (5600, 80),  # both envelopes at once, or not
    (8191, 74), (8191, 75),
])
def test_on_chip_forms_equal_the_multi_kernel_iteration(pkg, wl, cuda, monkeypatch, n, nr, pair):
    import torch
    y = torch.tensor(wl.two_tone_chirp(n, seed=n % 89), device=cuda)
    kw = dict(seed=9, noise_sift_cap=12, return_iters=True)
    monkeypatch.setenv("CEEMDAN_SMALL_PAIR", pair)
    a, ia = pkg.iceemdan(y, nr, 4, 10, 0.2, **kw)
    monkeypatch.setenv("CEEMDAN_SMALL", "0")
    b, ib = pkg.iceemdan(y, nr, 4, 10, 0.2, **kw)
    assert ia == ib
    assert torch.equal(a, b)


@pytest.mark.parametrize("n", [300, 9001, 20011, 45000])
def test_reverse_pass_solves_and_sums(pkg, orc, wl, cuda, n):
    """The transposed solve in shared memory and in global memory, long segments one per warp
    and one per thread."""
    import torch
    nr, nimf = 2, 4
    x, noise = wl.two_tone_chirp(n, seed=2), wl.white_noise(nr, n, 1)
    imfs, tape = pkg.iceemdan_taped(torch.tensor(x, device=cuda), nr, nimf, 8, 0.2,
                                    noise=torch.tensor(noise, device=cuda), noise_sift_cap=10)
    t = orc.Tape(x, noise, nimf, 8, 0.2, solver=1, chunk=16, noise_sift_cap=10)
    w = np.linspace(0.5, 1.5, nimf)[:, None]
    gy = tape.backward(torch.tensor(w, device=cuda) * imfs).cpu().numpy()
    tape.free()
    assert np.array_equal(imfs.cpu().numpy(), t.imfs)
    assert np.array_equal(gy, t.vjp(w * t.imfs))


def test_noise_of_kept_generators(pkg, wl, cuda):
    """A seed's numbers do not depend on the calls before, nor on calls of other threads."""
    import torch
    y = torch.tensor(wl.two_tone_chirp(600, seed=1), device=cuda)

    def call(seed, nr=5):
        return pkg.iceemdan(y, nr, 3, 5, 0.2, seed=seed, noise_sift_cap=5).cpu()

    first = {s: call(s) for s in range(8)}
    assert not torch.equal(first[0], first[1])
    call(3, nr=7)  # another count: an odd position of the generator
    assert torch.equal(call(0), first[0])
    got = {}

    def worker(i):
        with torch.cuda.stream(torch.cuda.Stream(cuda)):
            got[i] = [call(s) for s in (i, (i + 3) % 8)]

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(8):
        assert torch.equal(got[i][0], first[i])
        assert torch.equal(got[i][1], first[(i + 3) % 8])
