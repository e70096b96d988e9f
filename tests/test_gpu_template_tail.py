"""Templates of the pair-plane tail against the oracle: every box it takes, Fourier crops down to 16, no mask, one
direction and more directions than CTAs, and slots written out of order."""
import numpy as np
import pytest
import torch

from gisapr_gb300 import synthetic as syn
from gisapr_gb300.search import IntegratedProjector, PackedFourierLayout
from gisapr_gb300.tables import expand_radial_values, centered_to_packed_np, generate_soft_mask, model_angles_from_lists
from oracle import gisapr_oracle as O

from .helpers import TEMPLATE_RRMS, rrms

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("box,nb,n_dirs,masked", [
    (32, 32, 1, True), (32, 16, 1000, False), (64, 48, 7, False), (64, 64, 2, True), (128, 128, 1, False),
    (128, 16, 5, True), (128, 112, 330, True)])
def test_templates_against_the_oracle(box, nb, n_dirs, masked):
    rng = np.random.default_rng(box + nb)
    volume = syn.blob_density(box, 3)
    rot = rng.uniform(-180, 180, n_dirs)
    tilt = np.rad2deg(np.arccos(rng.uniform(-1, 1, n_dirs)))
    rot[0], tilt[0] = 90.0, 0.0  # a slice along the grid's own axes
    angles = model_angles_from_lists(rot.tolist(), tilt.tolist())
    fsc = centered_to_packed_np(expand_radial_values(rng.uniform(0.2, 1.0, box).astype(np.float32), nb))
    mask = generate_soft_mask((box, box), round(0.43 * box), 4) if masked else None
    projector = IntegratedProjector(DEV, box, nb, PackedFourierLayout(nb, 8, DEV),
                                    None if mask is None else torch.from_numpy(mask).to(DEV),
                                    torch.from_numpy(np.ascontiguousarray(fsc)).to(DEV))
    vol = torch.from_numpy(volume).to(DEV)
    bank = projector.build_templates(vol, angles)
    assert bool(torch.isfinite(torch.view_as_real(bank)).all())
    some = sorted({0, n_dirs // 2, n_dirs - 1})
    ref = O.build_templates(volume, np.asarray(angles.rotation_matrices_t)[some], nb, mask, fsc)
    got = bank.cpu().numpy()
    for k, i in enumerate(some):
        assert rrms(got[i], ref[k]) < TEMPLATE_RRMS
    # the same directions into other slots, backwards
    dirs = torch.tensor(some[::-1], dtype=torch.int32, device=DEV)
    slots = torch.tensor(list(range(len(some)))[::-1], dtype=torch.int32, device=DEV)
    out = torch.empty((len(some), nb, nb // 2 + 1), dtype=torch.complex64, device=DEV)
    projector.project(angles, dirs, out, slots)
    assert torch.equal(torch.view_as_real(out), torch.view_as_real(bank[some]))
