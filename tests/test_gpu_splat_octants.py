"""The binned splat against the deposit that walks every atom in input order: the same float32 sums, so the same
bits. Odd boxes, atoms on and past the faces, a brick with more atoms than its list holds, empty input bricks in
place, and a density that already holds values."""
import numpy as np
import pytest
import torch

from gisapr_gb300 import _native as nat
from gisapr_gb300.pdb2mrc import MovedChainDensity, density_from_coords, density_parameters

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def walked(xyz, z, box, apix, volume):
    w, rp, kn = density_parameters(apix, 2 * apix)
    out = volume.clone()
    x, zz = torch.from_numpy(xyz).to(DEV), torch.from_numpy(z).to(DEV)
    nat.call("gisapr_deposit_noalloc", nat.stream_of(DEV), nat.ptr(x), nat.ptr(zz), len(xyz), nat.ptr(out), box, w,
             apix, rp, kn)
    return out


@pytest.mark.parametrize("box,apix,n,spread", [(32, 3.0, 1, 0.0), (33, 1.3, 40, 0.6), (47, 1.0, 700, 0.5),
                                               (64, 1.5, 3000, 0.02), (90, 1.1, 2000, 0.3), (128, 1.1, 3000, 0.15),
                                               (256, 1.5, 500, 0.1)])
def test_bits_of_the_walked_deposit(box, apix, n, spread):
    rng = np.random.default_rng(box + n)
    xyz = (rng.standard_normal((n, 3)) * spread * box * apix).astype(np.float32)
    xyz[::7] = np.round(xyz[::7] / apix) * np.float32(apix)  # voxel centres: ties of the bounds
    if n > 3:
        xyz[1] = (box // 2 - 0.25) * apix
        xyz[2] = -(box // 2) * apix - 0.1
    z = rng.choice([0, 1, 6, 7, 8, 16], n).astype(np.float32)
    volume = torch.from_numpy(rng.standard_normal((box,) * 3).astype(np.float32)).to(DEV)
    got = density_from_coords(xyz, z, box, apix, 2 * apix, device=DEV, _initial_volume=volume)
    assert torch.equal(got, walked(xyz, z, box, apix, volume))


@pytest.mark.parametrize("box", [31, 64, 96])
def test_moved_chain_is_the_fixed_density_plus_the_moved_atoms(box):
    """The identity pose of 8.3 coordinates moves nothing, so the density is the deposit of the chain's own atoms."""
    rng = np.random.default_rng(box)
    lines, xyz = [], np.round(rng.standard_normal((400, 3)) * box * 0.2, 3)
    for i, p in enumerate(xyz):
        lines.append("ATOM  %5d  CA  ALA %s%4d    %8.3f%8.3f%8.3f  1.00  0.00           C\n"
                     % (i + 1, "A" if i < 150 else "B", i % 999, *p))
    model = MovedChainDensity("".join(lines), "A", box, 1.2, 2.4, DEV, from_text=True)
    got = model.generate(np.zeros(6))
    # the pose's float32 difference and FP64 sum return the written coordinates
    z = np.full(150, 6.0, np.float32)
    assert torch.equal(got, walked(xyz[:150].astype(np.float32), z, box, 1.2, model.fixed))
