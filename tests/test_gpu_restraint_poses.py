"""The poses of one call, reduced as their densities are computed, against each
pose's own splat (gisapr_deposit) counted on the host. A pose's density is the
same sum in the same order either way, so count and squared distance are equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.pdb2mrc import density_from_coords  # noqa: E402
from gisapr_gb300.restraint import GeometryRestraint, rotate_coords_rotvec  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


def _pdb(path, rng, moving, fixed, spread):
    lines = []
    for i in range(moving + fixed):
        c = rng.normal(size=3) * spread + (0.6 * spread if i < moving else -0.4 * spread)
        lines.append("ATOM  %5d  %-3s ALA %s%4d    %8.3f%8.3f%8.3f  1.00  0.00          %2s"
                     % (i % 99999 + 1, "CA", "A" if i < moving else "B", i % 9999 + 1, *c, rng.choice(list("CNOS"))))
    path.write_text("\n".join(lines) + "\nEND\n")
    return str(path)


# odd and even boxes, one atom, crowded bricks (more than 1,024 atoms in one),
# more poses than one launch takes, poses partly and wholly outside the box,
# and a threshold below zero, where unreached voxels of the bounds count too
@pytest.mark.parametrize("box, apix, moving, spread, poses, threshold",
                         [(33, 1.5, 1, 4.0, 5, 1.0), (48, 1.5, 400, 9.0, 70, 0.0), (64, 1.0, 2500, 4.0, 3, 2.0),
                          (127, 2.0, 900, 30.0, 33, 1.0), (40, 1.5, 60, 8.0, 4, -1.0)])
def test_poses_equal_single_splats(tmp_path, box, apix, moving, spread, poses, threshold):
    rng = np.random.default_rng(box)
    r = GeometryRestraint(_pdb(tmp_path / "m.pdb", rng, moving, 800, spread), "A", device=DEV, boxsize=box, apix=apix,
                          threshold=threshold)
    half = 0.5 * box * apix
    p = np.concatenate([rng.uniform(-180, 180, (poses, 3)), rng.uniform(-half, half, (poses, 3))], axis=1)
    p[-1, 3:] = 40 * half  # wholly outside
    mask = r.mainbody_mask.cpu().numpy().astype(bool)
    dist = r.mainbody_distance.cpu().numpy()
    want = []
    for pose in p:
        moved = rotate_coords_rotvec(r.chain_coords, *pose)
        chain = density_from_coords(moved, r.chain_numbers, box, apix, r.res, device=DEV).cpu().numpy() > threshold
        if threshold < 0.0:
            b = r._bounds(moved)
            inside = np.zeros_like(chain)
            inside[b[0]:b[3], b[1]:b[4], b[2]:b[5]] = True
            chain &= inside
        overlap = int(np.count_nonzero(chain & mask))
        want.append((overlap, 0.0) if overlap else (0, float(dist[chain].min()) * apix) if chain.any()
                    else (0, r._empty_distance()))
    assert r.evaluate_many(p) == want
    assert [r.evaluate(q) for q in p[:2]] == want[:2]
    with pytest.raises(ValueError):
        r.evaluate_many(np.zeros((0, 6)))
