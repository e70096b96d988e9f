"""The register form of the plain correlation is no less exact than the general kernel, which takes the same templates when
they do not start on 16 bytes: error against float64 of the maxima of one particle that holds one of its templates (a
peak, where all terms have one sign) and of one that holds none, over 9,600 maps each. The roundings of two maps are as
good as independent, so a ratio of two such errors varies by about 1%; three times that is the margin."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300 import _native as nat  # noqa: E402

DEV = "cuda:0"
DIRS, PSI, SEEDS = 40, 3, 80


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


def _spectra(n, peak, g):
    shape = (n, n // 2 + 1, 2)
    rand = lambda k: torch.view_as_complex(torch.randn(k, *shape, generator=g, device=DEV, dtype=torch.float64))
    unit = lambda v: v / v.abs().square().sum((-2, -1), keepdim=True).sqrt()
    T, P = unit(rand(1) + rand(DIRS)), unit(rand(PSI))
    if peak:
        P = unit(P + 0.05 * T[:1].conj())
    return T.to(torch.complex64), P.to(torch.complex64)


@pytest.mark.parametrize("n, crop", [(64, 10), (96, 12), (128, 12), (192, 12), (256, 14)])
@pytest.mark.parametrize("peak", [True, False])
def test_error_against_64_bits(n, crop, peak):
    H = n // 2 + 1
    g = torch.Generator(device=DEV).manual_seed(n + peak)
    off = torch.arange(crop, dtype=torch.float64, device=DEV) - crop // 2
    ey = torch.exp(2j * math.pi * off[:, None] * torch.arange(n, device=DEV) / n)
    w = torch.full((H,), 2.0, dtype=torch.float64, device=DEV)
    w[0] = w[-1] = 1.0
    ex = w[:, None] * torch.exp(2j * math.pi * torch.arange(H, device=DEV)[:, None] * off / n)
    ptr = torch.tensor([0, DIRS], dtype=torch.int32, device=DEV)
    idx = torch.arange(DIRS, dtype=torch.int32, device=DEV)
    ctx = nat.Context.for_device(DEV).handle
    error = [0.0, 0.0]
    for _ in range(SEEDS):
        T, P = _spectra(n, peak, g)
        raw = (ey @ (T[:, None].to(torch.complex128) * P.to(torch.complex128)) @ ex).real.reshape(DIRS, PSI, -1)
        for kernel, shift in enumerate((0, 1)):  # one complex value off: 8 bytes off 16
            bank = torch.empty(DIRS * n * H + 1, dtype=torch.complex64, device=DEV)[shift:shift + DIRS * n * H].view(DIRS, n, H)
            bank.copy_(T)
            s = torch.empty(DIRS, PSI, device=DEV)
            y = torch.empty(DIRS, PSI, dtype=torch.int32, device=DEV)
            x = torch.empty_like(y)
            nat.call("gisapr_correlate", ctx, nat.stream_of(torch.device(DEV)), nat.ptr(bank), nat.ptr(P), nat.ptr(ptr),
                     nat.ptr(idx), 1, PSI, n, crop, nat.ptr(s), nat.ptr(y), nat.ptr(x))
            at = raw.gather(2, (y * crop + x).long()[..., None])[..., 0]
            error[kernel] += float((s.double() / 1024 - at).square().sum())
    print(f"error ratio at {n}/{crop} peak {peak}: {math.sqrt(error[0] / error[1]):.3f}")
    assert error[0] <= 1.03 ** 2 * error[1]
