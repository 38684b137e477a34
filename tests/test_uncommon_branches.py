"""Branches that ordinary data hardly reaches: separator systems too long for the shared-memory
workspace, samples that the sign test of sx leaves undecided, rows with infinities, NaN and numbers
whose sums overflow, and the divisions by segment lengths."""
import os
import subprocess

import numpy as np
import pytest

from test_tile_paths import TILE, _check_envelopes, _zigzag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,per_tile", [
    (128 * TILE + 5, 2048),   # about 8,300 separators: the last that fit
    (130 * TILE - 3, 2048),   # more: the workspace in global memory
    (140 * TILE + 5, 2048),
    (600 * TILE + 11, 700),   # and more than 256 tiles
])
def test_envelopes_of_rows_with_thousands_of_separators(pkg, orc, cuda, n, per_tile):
    _check_envelopes(pkg, orc, cuda, _zigzag(n, per_tile, n)[None, :])


# how a call of n samples sifts: the multi-kernel iteration, and the on-chip forms
FORMS = [("0", "1", 5000), ("1", "1", 700), ("1", "1", 5000), ("1", "0", 700), ("1", "0", 5000),
         ("1", "0", 7000)]


def _run(pkg, orc, wl, cuda, monkeypatch, small, pair, x, noise, **kw):
    import torch
    monkeypatch.setenv("CEEMDAN_SMALL", small)
    monkeypatch.setenv("CEEMDAN_SMALL_PAIR", pair)
    nr = noise.shape[0]
    kw.update(noise_sift_cap=9, return_iters=True, return_noise_modes=True)
    got, it, modes = pkg.iceemdan(torch.tensor(x, device=cuda), nr, 4, 7, 0.2,
                                  noise=torch.tensor(noise, device=cuda), **kw)
    want, wit, wmodes = orc.iceemdan(x, noise, 4, 7, 0.2, solver=1, chunk=16, **kw)
    assert list(it) == list(wit)
    assert np.array_equal(modes.cpu().numpy(), wmodes, equal_nan=True)
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("small,pair,n", FORMS)
@pytest.mark.parametrize("kw", [dict(sd=1e-40), dict(sd2=1e-40), dict(sd=1e40, sd2=1e40),
                                dict(sd=1.0, sd2=1.0)])
def test_undecided_samples(pkg, orc, wl, cuda, monkeypatch, small, pair, n, kw):
    """Thresholds outside the sign test's range, and 1, which the end knots' sx is exactly."""
    _run(pkg, orc, wl, cuda, monkeypatch, small, pair, wl.two_tone_chirp(n, seed=2),
         wl.white_noise(5, n, 6), **kw)


def _odd_rows(n, kind):
    rng = np.random.default_rng(5)
    rows = rng.standard_normal((5, n))
    at = rng.choice(n, 6, replace=False)
    if kind == "inf":
        rows[1, at[0]] = np.inf
        rows[2, at[1]] = -np.inf
        rows[3, at[2:4]] = np.inf, -np.inf
        rows[4, 0] = np.inf
    elif kind == "nan":
        rows[1, at[0]] = np.nan
        rows[2, at] = np.nan
        rows[3, 0] = rows[4, n - 1] = np.nan
    elif kind == "huge":  # sums and slopes overflow
        rows[1] *= 4e307
        rows[2, at] = 1.7e308
        rows[3, at] = -1.7e308
        rows[4, -1] = 1e300
    else:  # subnormal, zero, constant
        rows[1] *= 1e-310
        rows[2] = 0.0
        rows[3] = -2.5
        rows[4, n // 3:] = 0.0
    return rows


@pytest.mark.parametrize("small,pair,n", FORMS)
@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "tiny"])
def test_rows_that_are_not_ordinary_numbers(pkg, orc, wl, cuda, monkeypatch, small, pair, n, kind):
    _run(pkg, orc, wl, cuda, monkeypatch, small, pair, wl.two_tone_chirp(n, seed=2),
         _odd_rows(n, kind))


def test_divisions_by_segment_lengths(cuda, tmp_path):
    exe = str(tmp_path / "spline_div_check")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "spline_div_check.cu")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O2", "-std=c++17", "-fmad=false", "-o", exe, src], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["mismatches", "0", "0", "0"]
