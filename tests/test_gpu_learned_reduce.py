"""The sum of the weight gradients' per-CTA partials over small and large batches: the loss is a mean over the
crops, so a batch's gradients are the mean of its crops' own (each checked against the oracle elsewhere)."""
import numpy as np
import pytest

from sqwheel import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crops", [1, 2, 5, 32])
def test_batch_gradients_are_the_mean_of_the_crops(gpu_ok, crops):
    import torch
    gen = torch.Generator("cuda:0").manual_seed(crops)
    lo = torch.randint(-2**31, 2**31, (80, 160), generator=gen, device="cuda:0", dtype=torch.int64).to(torch.int32)
    hi = torch.randint(-2**31, 2**31, (160, 320), generator=gen, device="cuda:0", dtype=torch.int64).to(torch.int32)
    u = learned.Upscaler(0, seed=4)
    try:
        items = [(lo, hi, k % 33, (k * 5) % 17) for k in range(crops)]
        g, loss = u.gradients(items)
        again, _ = u.gradients(items)
        assert np.array_equal(g, again)
        single = [u.gradients([i]) for i in items]
        want = np.mean([s[0].astype(np.float64) for s in single], axis=0)
        # f32 sums of crops * 16 partials: a few ulps of the sum of magnitudes, here bounded by the crops' norms
        scale = np.mean([np.linalg.norm(s[0]) for s in single])
        assert np.linalg.norm(g - want) <= 1e-5 * scale
        assert loss == pytest.approx(np.mean([s[1] for s in single]), rel=1e-5)
    finally:
        u.close()
