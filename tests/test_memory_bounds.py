"""The device memory that the library plans with is what its arrays take: as many channels to a
wave and realizations to a block as fit, and no more."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,nr", [([61440, 50001, 40000, 30007], 30),
                                        ([4096] * 20, 25), ([700, 300, 5000, 2049] * 6, 10)])
def test_waves_hold_what_fits(pkg, wl, cuda, lengths, nr):
    import torch
    ys = [torch.tensor(wl.eeg_like(n, seed=n % 17), device=cuda) for n in lengths]

    def run(budget, ys=ys):
        prof = {}
        outs = pkg.iceemdan_batched(ys, nr, 5, 6, 0.2, noise_sift_cap=6, wave_bytes=budget,
                                    profile=prof)
        return outs, prof["counters"]["waves"], prof["counters"]["peak_bytes"]

    outs, waves, need = run(1 << 40)
    assert waves == 1
    # all of it in one wave, with a few percent for the rounding of every channel's arrays
    slack = 64 * 1024 * len(lengths)
    same, waves, peak = run(need + need // 20 + slack)
    assert waves == 1 and peak == need
    # and never more than the budget, or than the longest channel by itself
    alone = run(1, [max(ys, key=len)])[2]
    for part in (2, 3):
        budget = need // part + slack
        again, waves, peak = run(budget)
        assert waves > 1 and peak <= max(budget, alone)
        for a, b in zip(outs, again):
            assert torch.equal(a, b)
    for a, b in zip(outs, same):
        assert torch.equal(a, b)


def test_checkpointed_blocks_use_the_free_memory(pkg, wl, cuda):
    """With 4 GB left the reverse pass takes blocks that use more than half of what it may."""
    import torch
    n, nr, nimf, left = 61440, 440, 4, 4 << 30
    y = torch.tensor(wl.eeg_like(n, seed=3), device=cuda)
    g = torch.randn((nimf, n), dtype=torch.float64, device=cuda,
                    generator=torch.Generator(device=cuda).manual_seed(2))
    _, tape = pkg.iceemdan_taped(y, nr, nimf, 4, 0.2, noise_sift_cap=4, checkpoint=True)
    try:
        want = tape.backward(g)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        st = pkg.memory_stats()
        free = torch.cuda.mem_get_info()[0] + st["reserved"] - st["used"]
        # what the pool keeps is free for the call too, so the ballast is the rest
        size = min(free - left, torch.cuda.mem_get_info()[0] - (256 << 20))
        ballast = torch.empty(size, dtype=torch.uint8, device=cuda)
        st = pkg.memory_stats(reset_peak=True)
        free = torch.cuda.mem_get_info()[0] + st["reserved"] - st["used"]
        got = tape.backward(g)
        torch.cuda.synchronize()
        took = pkg.memory_stats()["peak"] - st["used"]
        del ballast
    finally:
        tape.free()
        torch.cuda.empty_cache()
    assert torch.equal(got, want)
    assert 0.4 * free < took < 0.8 * free
