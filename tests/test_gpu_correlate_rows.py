"""The plain correlation with the particle's spectrum in registers, against the
correlation map in float64, and its launch shapes against one another.

raw(y, x) is a sum of n (n/2 + 1) products. A first maximum taken in float32 is
the value of some map position within the rounding of that sum of the largest:
16-point and n/16-point transforms over rows, then a sum over n/2 + 1 columns,
each rounding by 2^-24 of terms whose 2-norm is the map's: 40 * 2^-24 times the
norm of the products bounds it with room."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300 import _native as nat  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


def _call(bank, stack, counts, idx, crop, subset=None, cluster=0, sizes=None):
    cand, _, n = bank.shape[:3]
    parts, psi = stack.shape[:2]
    ptr = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    nnz = int(sum(counts))
    score = torch.full((cand, nnz, psi), -7.0, device=DEV)
    y = torch.full((cand, nnz, psi), -7, dtype=torch.int32, device=DEV)
    x = y.clone()
    sub = None if subset is None else torch.tensor(subset, dtype=torch.uint8, device=DEV)
    ctx = nat.Context.for_device(DEV).handle
    nat.call("gisapr_set_tuning", ctx, nat.TUNE_CORR_CLUSTER, n, cluster)
    try:
        nat.call("gisapr_correlate_batch_subset", ctx, nat.stream_of(torch.device(DEV)), nat.ptr(bank),
                 bank.stride(0) // 2 if cand > 1 else 0, cand, nat.ptr(stack), nat.ptr(ptr), nat.ptr(idx), parts, nnz,
                 psi, n, crop, nat.ptr(sub) if sub is not None else None, nat.ptr(score), nat.ptr(y), nat.ptr(x))
    finally:
        nat.call("gisapr_set_tuning", ctx, nat.TUNE_CORR_CLUSTER, n, 0)
    return score.cpu(), y.cpu(), x.cpu()


# every size and window of the form; one to many directions (more than a group),
# psi angles beyond one CTA's, candidates with a subset, few and many particles
@pytest.mark.parametrize("n, crop, parts, psi, cand", [
    (64, 10, 3, 3, 2), (64, 16, 700, 1, 1), (96, 12, 5, 4, 1), (96, 8, 300, 2, 1), (128, 12, 1, 3, 1),
    (128, 12, 330, 3, 2), (128, 14, 4, 5, 3), (192, 12, 3, 2, 1), (192, 16, 2, 3, 1), (256, 14, 2, 3, 2),
    (256, 8, 90, 1, 1)])
def test_maps_and_shapes(n, crop, parts, psi, cand):
    H, dirs = n // 2 + 1, 9
    gen = torch.Generator().manual_seed(n + crop)
    bank = torch.randn(cand, dirs, n, H, 2, generator=gen).to(DEV)
    stack = torch.randn(parts, psi, n, H, 2, generator=gen).to(DEV)
    counts = [(0, 1, 5, 8, 9, 17, 3)[(p + 4) % 7] for p in range(parts)]
    idx = torch.randint(0, dirs, (sum(counts),), generator=gen, dtype=torch.int32).to(DEV)
    subset = None
    if cand > 1:
        subset = np.ones((cand, parts), np.uint8)
        subset[0, ::3] = 0
        subset[-1, 1::2] = 0
    score, ys, xs = _call(bank, stack, counts, idx, crop, subset)
    off = torch.arange(crop, dtype=torch.float64, device=DEV) - crop // 2
    ey = torch.exp(2j * np.pi * off[:, None] * torch.arange(n, device=DEV) / n)
    w = torch.full((H,), 2.0, dtype=torch.float64, device=DEV)
    w[0] = w[-1] = 1.0
    ex = w[:, None] * torch.exp(2j * np.pi * torch.arange(H, device=DEV)[:, None] * off / n)
    start = np.concatenate([[0], np.cumsum(counts)])
    for p in sorted({0, 1, 2, parts // 2, parts - 1} & set(range(parts))):
        for c in range(cand):
            for e in range(start[p], start[p + 1]):
                if subset is not None and not subset[c, p]:
                    assert (score[c, e] == -7.0).all() and (ys[c, e] == -7).all()
                    continue
                t = torch.view_as_complex(bank[c, int(idx[e])]).to(torch.complex128)
                for a in range(psi):
                    q = t * torch.view_as_complex(stack[p, a]).to(torch.complex128)
                    raw = (ey @ q @ ex).real.cpu()
                    tol = 40 * 2.0 ** -24 * float((q.abs().square() @ w.to(torch.float64).square()).sum().sqrt())
                    got = float(score[c, e, a]) / 1024.0
                    yi, xi = int(ys[c, e, a]), int(xs[c, e, a])
                    assert abs(got - float(raw[yi, xi])) <= tol
                    assert float(raw[yi, xi]) >= float(raw.max()) - 2 * tol
    # the maps do not depend on the particles of the call, nor, beyond the order of the tiles' sums, on the cluster
    one = [k for k in range(parts) if counts[k]][0]
    s1, y1, x1 = _call(bank, stack[one:one + 1].contiguous(), counts[one:one + 1],
                       idx[start[one]:start[one + 1]].contiguous(), crop)
    live = slice(None) if subset is None else torch.tensor(subset[:, one].astype(bool))
    rows = slice(int(start[one]), int(start[one + 1]))
    scale = score[live][:, rows].abs().max()
    assert (s1[live] - score[live][:, rows]).abs().max() <= 1e-5 * scale
    for k in (2, 3, 8):
        try:
            sk, _, _ = _call(bank, stack, counts, idx, crop, subset, cluster=k)
        except ValueError:  # refused for the shared memory it would take
            continue
        assert (sk - score).abs().max() <= 1e-5 * score.abs().max()
