"""Particle spectra of the shared-memory plane kernel against the oracle: every box it takes, crops, psi counts,
job counts around the number of CTAs (an image is shared by its psi jobs and handed on between buffers), with and
without a mask, and a NaN particle that must stay alone."""
import numpy as np
import pytest
import torch

from gisapr_gb300.search import PackedFourierLayout, ParticleFourierPreparer, PsiGridBank
from gisapr_gb300.tables import generate_soft_mask
from oracle import gisapr_oracle as O

from .helpers import rrms

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# float32 transforms of length N and float32 sampling weights: a few times 2^-24 sqrt(log2 N^2) times the
# bilinear sum's own rounding, an order below this
RRMS = 5e-6


@pytest.mark.parametrize("box,nb,n,psi,masked", [
    (32, 32, 7, 3, True), (32, 16, 1, 1, False), (64, 64, 300, 5, True), (64, 48, 3, 2, False),
    (96, 96, 110, 3, True), (96, 32, 2, 1, True), (128, 128, 1, 1, False), (128, 112, 51, 3, True),
    (128, 128, 120, 4, True), (192, 192, 52, 3, True), (192, 176, 1, 2, False)])
def test_spectra_against_the_oracle(box, nb, n, psi, masked):
    rng = np.random.default_rng(box + nb + n)
    images = rng.standard_normal((n, box, box)).astype(np.float32)
    images[n // 2] *= 1e3
    angles = [[float(a) for a in rng.choice(np.arange(1, 48) * 7.5, psi, replace=False)] for _ in range(n)]
    ctf = rng.uniform(-1, 1, (n, nb, nb // 2 + 1)).astype(np.float32)
    mask = generate_soft_mask((box, box), round(0.43 * box), 3) if masked else None
    bank = PsiGridBank(box, DEV, sorted({a for row in angles for a in row}))
    prep = ParticleFourierPreparer(box, nb, DEV, PackedFourierLayout(nb, 8, DEV),
                                   None if mask is None else torch.from_numpy(mask).to(DEV), bank)
    index = torch.stack([bank.indices_for_angles(row) for row in angles])
    got = prep.prepare_batch(torch.from_numpy(images).to(DEV), index, torch.from_numpy(ctf).to(DEV)).cpu().numpy()
    for i in sorted({0, n // 2, n - 1}):
        ref = O.prepare_particle(images[i], angles[i], ctf[i], mask, nb)
        assert rrms(got[i], ref) < RRMS
    assert np.isfinite(got.view(np.float32)).all()


@pytest.mark.parametrize("box", [64, 128, 192])
def test_a_nan_particle_stays_alone(box):
    rng = np.random.default_rng(box)
    images = torch.from_numpy(rng.standard_normal((4, box, box)).astype(np.float32)).to(DEV)
    bank = PsiGridBank(box, DEV, [15.0, 30.0])
    prep = ParticleFourierPreparer(box, box, DEV, PackedFourierLayout(box, 8, DEV), None, bank)
    index = torch.tensor([[0, 1]] * 4, dtype=torch.int32, device=DEV)
    ctf = torch.ones((4, box, box // 2 + 1), device=DEV)
    clean = prep.prepare_batch(images, index, ctf).clone()
    images[1, box // 2, box // 2] = float("nan")
    got = prep.prepare_batch(images, index, ctf)
    assert torch.isnan(torch.view_as_real(got[1])).all()
    assert torch.equal(torch.view_as_real(got[[0, 2, 3]]), torch.view_as_real(clean[[0, 2, 3]]))
