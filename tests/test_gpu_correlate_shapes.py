"""The plain correlation's register form over its launch shapes: every number of CTAs per particle is taken (none is
refused for shared memory that only the general kernel needs) and gives the same maps up to the order of the tiles'
sums, more psi angles than a CTA holds, and the windows whose rows do not divide among a column's lanes. A tuned number
that the general kernel cannot take gives way to its default.

raw(y, x) is a sum of n (n/2 + 1) products: 40 * 2^-24 times the norm of the products bounds its float32 rounding with
room (16-point and n/16-point transforms over rows, then a sum over columns)."""
import math

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


def _call(bank, stack, ptr, idx, n, crop, cluster):
    parts, psi = stack.shape[:2]
    s = torch.empty(idx.numel(), psi, device=DEV)
    y = torch.empty(idx.numel(), psi, dtype=torch.int32, device=DEV)
    x = torch.empty_like(y)
    ctx = nat.Context.for_device(DEV).handle
    nat.call("gisapr_set_tuning", ctx, nat.TUNE_CORR_CLUSTER, n, cluster)
    try:
        nat.call("gisapr_correlate", ctx, nat.stream_of(torch.device(DEV)), nat.ptr(bank), nat.ptr(stack), nat.ptr(ptr),
                 nat.ptr(idx), parts, psi, n, crop, nat.ptr(s), nat.ptr(y), nat.ptr(x))
    finally:
        nat.call("gisapr_set_tuning", ctx, nat.TUNE_CORR_CLUSTER, n, 0)
    return s, y, x


@pytest.mark.parametrize("n, crop, psi", [(64, 10, 3), (96, 14, 7), (128, 10, 3), (128, 12, 40), (192, 8, 3), (256, 10, 3),
                                          (256, 12, 2), (256, 16, 11), (128, 6, 1), (256, 4, 3), (48, 12, 3)])
def test_every_cluster_size(n, crop, psi):
    H, dirs, parts = n // 2 + 1, 5, 3
    g = torch.Generator(device=DEV).manual_seed(n + crop + psi)
    bank = torch.randn(dirs, n, H, 2, generator=g, device=DEV)
    stack = torch.randn(parts, psi, n, H, 2, generator=g, device=DEV)
    ptr = torch.tensor([0, 11, 11, 14], dtype=torch.int32, device=DEV)  # more than a group, none, few
    idx = torch.randint(0, dirs, (14,), generator=g, device=DEV, dtype=torch.int32)
    off = torch.arange(crop, dtype=torch.float64, device=DEV) - crop // 2
    ey = torch.exp(2j * math.pi * off[:, None] * torch.arange(n, device=DEV) / n)
    w = torch.full((H,), 2.0, dtype=torch.float64, device=DEV)
    w[0] = w[-1] = 1.0
    ex = w[:, None] * torch.exp(2j * math.pi * torch.arange(H, device=DEV)[:, None] * off / n)
    T, P = (torch.view_as_complex(v).to(torch.complex128) for v in (bank, stack))
    part = torch.tensor([0] * 11 + [2] * 3, device=DEV)
    q = T[idx.long()][:, None] * P[part]
    raw = (ey @ q @ ex).real.reshape(14, psi, -1)
    tol = 40 * 2.0 ** -24 * (q.abs().square() @ w.square()).sum(-1).sqrt()
    for cluster in range(9):
        s, y, x = _call(bank, stack, ptr, idx, n, crop, cluster)
        got = s.double() / 1024
        at = raw.gather(2, (y * crop + x).long()[..., None])[..., 0]
        assert bool(((got - at).abs() <= tol).all()), cluster
        assert bool((at >= raw.amax(-1) - 2 * tol).all()), cluster
