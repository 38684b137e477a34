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
