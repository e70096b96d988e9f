"""Particle preparation in the half spectrum against its steps in float64 numpy: odd and even sides, every flag
combination, images with an offset and a gradient, and shapes that take turns beyond the kept plans."""
import numpy as np
import pytest
import torch

from gisapr_gb300 import ingest

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def stepwise(img, flags, freq, apix):
    v = img.astype(np.float64)
    h, w = v.shape
    if flags & ingest.SPECTRUM:
        ptr, pix, cnt = ingest.radial_bins(h, w)
        F = np.fft.fft2(v).ravel()
        for b in range(1, len(cnt)):
            at = pix[ptr[b]:ptr[b + 1]]
            F[at] *= 1.0 / (np.abs(F[at]).sum() / cnt[b])
        v = np.fft.ifft2(F.reshape(h, w)).real
    if flags & ingest.NORMALIZE:
        y, x = np.mgrid[:h, :w]
        A = np.stack([x.ravel(), y.ravel(), np.ones(h * w)], 1)
        v = v - (A @ np.linalg.lstsq(A, v.ravel(), rcond=None)[0]).reshape(h, w)
        v = (v - v.mean()) / v.std()
    if flags & ingest.HIGHPASS:
        v = np.fft.ifft2(np.fft.fft2(v) * ingest.highpass_mask(h, w, freq, apix)).real
    return v


@pytest.mark.parametrize("size", [32, 45, 64, 91])
@pytest.mark.parametrize("flags", [1, 3, 4, 5, 6, 7])
def test_flags_against_the_steps(size, flags):
    rng = np.random.default_rng(size * 8 + flags)
    images = rng.standard_normal((3, size, size)).astype(np.float32) + np.float32(5.0)
    images += np.linspace(-2, 2, size, dtype=np.float32)[None, :, None]
    out = ingest.preprocess_stack(images, device=DEV, flags=flags, highpass_freq=20.0, angpix=1.5).cpu().numpy()
    for got, img in zip(out, images):
        want = stepwise(img, flags, 20.0, 1.5)
        # FP64 throughout, rounded once to float32: 2^-24 of the largest value, twice that for the rounding of the
        # comparison's own route
        assert np.abs(got - want).max() <= 2.0 ** -23 * np.abs(want).max()


def test_more_shapes_than_kept_plans_and_two_streams():
    rng = np.random.default_rng(3)
    stacks = [torch.from_numpy(rng.standard_normal((n, s, s)).astype(np.float32)).to(DEV)
              for n, s in [(2, 32), (3, 32), (2, 40), (2, 48), (5, 64), (2, 33)]]
    first = [ingest.preprocess_stack(s, None, 0, True, True, 20.0, 1.5) for s in stacks]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    again = []
    for s in stacks * 2:
        with torch.cuda.stream(side if len(again) % 2 else torch.cuda.current_stream()):
            again.append(ingest.preprocess_stack(s, None, 0, True, True, 20.0, 1.5))
    torch.cuda.synchronize()
    for a, b in zip(first * 2, again):
        assert torch.equal(a, b)
    # one bad image leaves the others alone
    bad = stacks[1].clone()
    bad[1, 3, 3] = float("nan")
    got = ingest.preprocess_stack(bad, None, 0, True, True, 20.0, 1.5)
    assert torch.isnan(got[1]).all() and torch.equal(got[0], first[1][0]) and torch.equal(got[2], first[1][2])
