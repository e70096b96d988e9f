"""gisapr_ingest_stack with the caller's own tables, against its steps in float64 numpy on the full spectrum (the real
part of every inverse transform): bins that are not radial, that list a part of the pixels or list them in another
order, and masks that are not their own mirror image, on sides that are odd, even and unequal and too large for the
amplitudes to be kept in shared memory; the radial tables again at those sizes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300 import _native as nat  # noqa: E402
from gisapr_gb300 import ingest  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


def _bins(kind, h, w, rng):
    if kind == "radial":
        return ingest.radial_bins(h, w)
    if kind == "rows":
        of = np.repeat(np.arange(h) // 3, w)
    elif kind == "random":
        of = rng.integers(0, 17, h * w)
    else:
        ptr, pix, cnt = ingest.radial_bins(h, w)
        if kind == "shuffled":  # the radial bins, each listed in another order
            return ptr, np.concatenate([rng.permutation(pix[ptr[b]:ptr[b + 1]]) for b in range(len(cnt))]), cnt
        of = np.empty(h * w, np.int64)  # "part": the radial bins without some of their pixels
        for b in range(len(cnt)):
            of[pix[ptr[b]:ptr[b + 1]]] = b
        of[rng.random(h * w) < 0.3] = -1
    n_bins = int(of.max()) + 1
    pix = np.concatenate([np.nonzero(of == b)[0] for b in range(n_bins)])
    count = np.bincount(of[of >= 0], minlength=n_bins)
    return np.concatenate([[0], np.cumsum(count)]), pix, count.astype(np.float64)


def _steps(img, flags, bins, mask):
    v = img.astype(np.float64)
    h, w = v.shape
    if flags & 1:
        ptr, pix, cnt = bins
        F = np.fft.fft2(v).ravel()
        d = np.ones(h * w)
        for b in range(1, len(cnt)):
            at = pix[ptr[b]:ptr[b + 1]]
            if cnt[b] > 0:
                d[at] = 1.0 / (np.abs(F[at]).sum() / cnt[b])
        v = np.fft.ifft2((F * d).reshape(h, w)).real
    if flags & 2:
        y, x = np.mgrid[:h, :w]
        A = np.stack([x.ravel(), y.ravel(), np.ones(h * w)], 1)
        v = v - (A @ np.linalg.lstsq(A, v.ravel(), rcond=None)[0]).reshape(h, w)
        v = (v - v.mean()) / v.std()
    if flags & 4:
        v = np.fft.ifft2(np.fft.fft2(v) * mask).real
    return v


def _run(images, flags, bins, mask):
    n, h, w = images.shape
    dev = torch.device(DEV)
    ptr, pix, cnt = (torch.from_numpy(np.ascontiguousarray(v)).to(dev) for v in
                     (bins[0].astype(np.int32), bins[1].astype(np.int32), bins[2]))
    m, src = torch.from_numpy(np.ascontiguousarray(mask)).to(dev), torch.from_numpy(images).to(dev)
    out = torch.empty((n, h, w), device=dev)
    work = torch.empty(n * h * w * 2, dtype=torch.float64, device=dev)
    nat.call("gisapr_ingest_stack", nat.Context.for_device(dev).handle, nat.stream_of(dev), nat.ptr(src), n, h, w, None, h,
             w, flags, nat.ptr(ptr), nat.ptr(pix), nat.ptr(cnt), len(cnt), nat.ptr(m), nat.ptr(work), nat.ptr(out))
    return out.cpu().numpy()


@pytest.mark.parametrize("h, w", [(32, 32), (45, 45), (33, 64), (64, 33), (230, 230), (261, 240)])
@pytest.mark.parametrize("kind", ["radial", "shuffled", "rows", "random", "part"])
def test_any_tables(h, w, kind):
    rng = np.random.default_rng(h * w + len(kind))
    images = rng.standard_normal((2, h, w)).astype(np.float32) + np.float32(2.0)
    images += np.linspace(-1, 1, w, dtype=np.float32)
    bins = _bins(kind, h, w, rng)
    for flags in (1, 3, 4, 5, 7):
        mask = rng.uniform(0, 1, (h, w)) if kind != "radial" else ingest.highpass_mask(h, w, 20.0, 1.5)
        for got, img in zip(_run(images, flags, bins, mask), images):
            want = _steps(img, flags, bins, mask)
            # FP64 throughout, rounded once to float32: 2^-24 of the largest value, twice that for the rounding of the
            # comparison's own route
            assert np.abs(got - want).max() <= 2.0 ** -23 * np.abs(want).max(), flags
