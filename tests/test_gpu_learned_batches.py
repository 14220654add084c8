"""The training kernels at batches that give a CTA of the convolutions two, three, four and up to seven rows (an epilogue
group takes every second of them) and CTAs whose rows cross from one crop into the next: loss and gradients of every
layer against the oracle, with the tolerance of the three-crop test (bf16 activations and gradients, f32 sums)."""
import numpy as np
import pytest

import upscaler_oracle as uo
from sqwheel import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crops", [1, 10, 15, 31])
def test_gradients_of_batches(gpu_ok, crops):
    import torch
    rng = np.random.default_rng(crops)

    def frame(h, w):
        a = np.repeat(np.repeat(rng.integers(0, 236, (h // 8, w // 8, 4)), 8, 0), 8, 1) + rng.integers(0, 20, (h, w, 4))
        return (a[..., 0] | (a[..., 1] << 8) | (a[..., 2] << 16) | (a[..., 3] << 24)).astype(np.uint32)

    lo, hi = frame(72, 136), frame(144, 272)
    dev = [torch.from_numpy(f.view(np.int32)).to("cuda:0") for f in (lo, hi)]
    spots = [(k % 9, (3 * k) % 9) for k in range(crops)]
    u = learned.Upscaler(0, seed=6)
    try:
        g, loss = u.gradients([(*dev, x, y) for x, y in spots])
        want, want_loss = uo.gradients(u.params(), [(lo, hi, x, y) for x, y in spots])
    finally:
        u.close()
    assert loss == pytest.approx(want_loss, rel=1e-4)
    off = 0
    for ci, co in uo.LAYERS:
        for n in (co * 9 * ci, co):
            assert np.linalg.norm(g[off:off + n] - want[off:off + n]) < 1e-3 * np.linalg.norm(want[off:off + n])
            off += n
