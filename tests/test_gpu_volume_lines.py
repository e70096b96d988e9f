"""The volume transform of power-of-two boxes against the cuFFT path where a
misplaced line, output parity or sign of w^j shows: densities of a few single
voxels at the ends and the middle of the axes, where every spectrum value has
the same size.

Tolerance: three float32 transforms of 2N points and their twiddles are good to
about 3 log2(2N) 2^-24 < 2e-6 of a value, the interpolation and the whitening of
a flat spectrum keep that within a small factor; a misplaced value is off by its
whole size. 1e-4 in relative RMS lies far from both."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.search import IntegratedProjector, PackedFourierLayout  # noqa: E402
from gisapr_gb300.tables import model_angles_from_lists  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


@pytest.mark.parametrize("n", [32, 64, 128, 256])
def test_single_voxels_equal_the_whole_transform(n):
    angles = model_angles_from_lists([0.0, 35.0, 120.0, 300.0], [0.0, 90.0, 47.0, 133.0])
    fsc = torch.ones((n, n // 2 + 1))
    proj = IntegratedProjector(DEV, n, n, PackedFourierLayout(n, 8, DEV), None, fsc)
    for z, y, x in ((n // 2, n // 2, n // 2), (0, n // 2, n - 1), (n - 1, 1, 0), (n // 2 - 1, n - 1, n // 2 + 1)):
        vol = torch.zeros((n,) * 3, device=DEV)
        vol[z, y, x] = 1.0
        vol[n // 2, n // 2, n // 2] += 0.5
        out = []
        for blocked in (True, False):
            proj.blocked_fft = blocked
            out.append(proj.build_templates(vol, angles).cpu().numpy().astype(np.complex128))
        got, want = out
        rms = np.sqrt((np.abs(got - want) ** 2).sum(axis=(1, 2)) / (np.abs(want) ** 2).sum(axis=(1, 2)))
        assert (rms < 1e-4).all(), (n, (z, y, x), rms)
