"""Rows that end inside a warp's samples of a tile (512 samples a warp, 16 a thread, planes padded
to four): the part of the warp past the row takes the same path as the rest and must count
nowhere.  Against the CPU oracle, bit for bit, with the default thresholds and with thresholds
outside the range in which the sign test decides (every sample then takes the division)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [4, 5, 15, 16, 17, 63, 300, 509, 511, 512, 513, 515, 529, 1023, 1025, 1537, 2047, 2048,
           2049, 2052, 2563, 4097]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("sd,sd2", [(0.05, 0.5), (1e-40, 0.5), (0.05, 1e-40), (1e40, 1e40)])
def test_iterations_of_rows_that_end_inside_a_warp(pkg, orc, wl, cuda, monkeypatch, n, sd, sd2):
    import torch
    monkeypatch.setenv("CEEMDAN_SMALL", "0")
    nr, nimf = 6, 3
    x = wl.two_tone_chirp(n, seed=n % 71)
    noise = wl.white_noise(nr, n, 4)
    noise[1] = np.cumsum(noise[1])                              # few knots
    noise[2] = np.round(2.0 * noise[2])                         # plateaus
    noise[3] = np.cos(2 * np.pi * 1.4 * np.arange(n) / n)       # three knots or fewer
    got, it = pkg.iceemdan(torch.tensor(x, device=cuda), nr, nimf, 6, 0.2,
                           noise=torch.tensor(noise, device=cuda), noise_sift_cap=8, sd=sd,
                           sd2=sd2, return_iters=True)
    want, wit = orc.iceemdan(x, noise, nimf, 6, 0.2, solver=1, chunk=16, noise_sift_cap=8, sd=sd,
                             sd2=sd2, return_iters=True)
    assert list(it) == list(wit)
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("n,nr", [(16, 900), (300, 600), (1100, 500)])
def test_many_short_rows(pkg, orc, wl, cuda, n, nr):
    """More realizations than the on-chip path holds: two launches a class, tiles of one row end."""
    import torch
    x, noise = wl.two_tone_chirp(n, seed=3), wl.white_noise(nr, n, 8)
    got, it = pkg.iceemdan(torch.tensor(x, device=cuda), nr, 3, 6, 0.2,
                           noise=torch.tensor(noise, device=cuda), noise_sift_cap=8,
                           return_iters=True)
    want, wit = orc.iceemdan(x, noise, 3, 6, 0.2, solver=1, chunk=16, noise_sift_cap=8,
                             return_iters=True)
    assert list(it) == list(wit)
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("n", LENGTHS + [6144, 6147])
@pytest.mark.parametrize("shift", [0, 1, 2, 5])
def test_envelopes_into_any_alignment(pkg, orc, cuda, n, shift):
    """Outputs that start `shift` doubles past a 256-byte boundary, rows of every length modulo
    four; nothing around the output is touched."""
    import ctypes
    import torch
    nr = 5
    rng = np.random.default_rng(n)
    rows = rng.standard_normal((nr, n))
    rows[1] = np.cumsum(rows[1])
    rows[2] = np.cos(2 * np.pi * 1.3 * np.arange(n) / n)
    h = torch.tensor(rows, device=cuda)
    bufs = [torch.full((nr * n + 16,), -7.5, dtype=torch.float64, device=cuda) for _ in range(2)]
    p = lambda t, k=0: ctypes.c_void_p(t.data_ptr() + 8 * k)  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert pkg.lib().ceemdan_envelopes_f64(nr, n, p(h), p(bufs[0], shift), p(bufs[1], shift), None,
                                           stream) == 0
    for e, b in enumerate(bufs):
        b = b.cpu().numpy()
        got = b[shift:shift + nr * n].reshape(nr, n)
        for r in range(nr):
            assert np.array_equal(got[r], orc.envelope(rows[r], e, solver=1, chunk=16))
        assert (b[:shift] == -7.5).all() and (b[shift + nr * n:] == -7.5).all()
