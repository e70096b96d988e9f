"""A restraint holds no density volume unless its threshold asks for one."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.restraint import GeometryRestraint  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


@pytest.mark.parametrize("threshold, volumes", [(1.0, 0), (-1.0, 1)])
def test_memory_held(tmp_path, threshold, volumes):
    """Mask (one byte) and squared distances (four) a voxel, and the volume (four) where it is needed; atoms and
    allocation blocks take less than half a volume."""
    path = tmp_path / "m.pdb"
    path.write_text("".join("ATOM  %5d  CA  ALA %s%4d    %8.3f%8.3f%8.3f  1.00  0.00           C\n"
                            % (i + 1, "AB"[i % 2], i + 1, 3.0 * (i % 7), 2.0 * i - 20.0, 6.0 * (i % 2)) for i in range(20)) + "END\n")
    n = 128
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    r = GeometryRestraint(str(path), "A", device=DEV, boxsize=n, apix=1.5, threshold=threshold)
    first = r.evaluate_many([[0, 0, 0, 0, 0, 0], [10, 0, 0, 5, 0, 0]])
    held = (torch.cuda.memory_allocated() - before) / n ** 3
    assert 5 + 4 * volumes <= held < 7 + 4 * volumes
    assert r.evaluate_many([[0, 0, 0, 0, 0, 0], [10, 0, 0, 5, 0, 0]]) == first
