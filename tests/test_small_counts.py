"""Knot counts of the on-chip forms on rows with a handful of extrema.

A row's two knot counts decide whether the mean envelope is written (both above 3) and whether a
large sx keeps the row sifting (their sum above 6), and every thread of a CTA takes these
decisions by itself.  Rows of a few slow oscillations pass through the counts around both limits
from one iteration to the next, so a thread that goes by another iteration's count shows in the
IMFs, in the iteration counts or in the knots counted.

The lock-step test can also end differently for the two CTAs of a realization: one sees the
stage's end at its last poll, the other has given up.  Both have to take the same way out.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _slow_rows(nr, n):
    """Rows of one to five extrema of either kind, with a faint faster tone that sifting moves."""
    t = np.linspace(0.0, 1.0, n)
    rows = []
    for r in range(nr):
        f = 0.4 + 2.2 * (r % 23) / 23.0
        rows.append(np.cos(2 * np.pi * (f * t + 0.13 * r)) + 0.3 * t +
                    0.25 * np.cos(2 * np.pi * (2.7 * f * t + 0.31 * r)))
    return np.stack(rows)


@pytest.mark.parametrize("n,nr", [
    (7680, 80), (5600, 75), (8192, 100),   # one envelope after the other
    (2501, 80),                            # both envelopes side by side
    (4096, 20), (8192, 74),                # a cluster of two CTAs
])
@pytest.mark.parametrize("slow", [True, False])
def test_few_knots_equal_the_multi_kernel_iteration(pkg, wl, cuda, monkeypatch, n, nr, slow):
    import torch
    y = torch.tensor(wl.two_tone_chirp(n, seed=n % 83), device=cuda)
    kw = dict(seed=21, noise_sift_cap=40, return_iters=True)
    if slow:
        kw["noise"] = torch.tensor(_slow_rows(nr, n), device=cuda)
    nimf = 5 if slow else 12

    def run():
        prof = {}
        imfs, it = pkg.iceemdan(y, nr, nimf, 25, 0.2, profile=prof, **kw)
        return imfs, list(it), prof["counters"]["knots"], prof["ms"]["sift_small"]

    a, ia, ka, on_chip = run()
    assert on_chip > 0
    monkeypatch.setenv("CEEMDAN_SMALL", "0")
    b, ib, kb, off_chip = run()
    assert off_chip == 0
    assert ia == ib
    assert ka == kb
    assert torch.equal(a, b)


def _tone_rows(nr, n):
    """Rows whose envelopes are symmetric: their first iteration is their last."""
    t = np.arange(n) / n
    return np.stack([np.cos(2 * np.pi * (40 + r % 7) * t) for r in range(nr)])


@pytest.mark.parametrize("n,nr", [(2048, 8), (4096, 60), (2501, 80), (7680, 80)])
@pytest.mark.parametrize("ending", [True, False])
def test_one_cta_of_a_realization_gives_up(pkg, wl, cuda, n, nr, ending):
    """With a negative spin limit the first CTA of every realization gives up in iteration 1; the
    second one of a pair meanwhile sees the stage end there (tones) or go on (white noise)."""
    import torch
    y = torch.tensor(wl.two_tone_chirp(n, seed=7), device=cuda)
    rows = _tone_rows(nr, n) if ending else wl.white_noise(nr, n, 3)
    kw = dict(noise=torch.tensor(rows, device=cuda), noise_sift_cap=30)
    a, it = pkg.iceemdan(y, nr, 4, 10, 0.2, return_iters=True, **kw)
    assert (it[0] == 1) == ending
    for _ in range(3):
        with pytest.raises(pkg.CeemdanError) as ei:
            pkg.iceemdan(y, nr, 4, 10, 0.2, spin_limit=-200000, **kw)
        assert ei.value.status == 5
    # the context is usable and the next call gives the usual result
    assert torch.equal(a, pkg.iceemdan(y, nr, 4, 10, 0.2, **kw))
