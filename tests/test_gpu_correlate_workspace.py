"""The per-particle correlation call uploads nothing and waits for nothing once its workspace holds the number of
templates: a stream capture, which refuses both, records it, and the replay follows new inputs. Template counts
that grow and shrink keep their own offsets."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.search import (CorrelationWorkspace, PackedFourierLayout,  # noqa: E402
                                 correlate_templates_and_particle)

DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import __graft_entry__ as g
    g.build()


def _inputs(n, n_a, n_b, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    make = lambda k: torch.view_as_complex(torch.randn(k, n, n // 2 + 1, 2, generator=g, device=DEV))
    return make(n_a), make(n_b)


@pytest.mark.parametrize("n, crop, n_a, n_b", [(32, 6, 1, 1), (64, 10, 17, 2), (128, 12, 6, 3)])
def test_a_warm_call_is_captured_and_follows_its_inputs(n, crop, n_a, n_b):
    layout, work = PackedFourierLayout(n, crop, DEV), CorrelationWorkspace(DEV)
    T, P = _inputs(n, n_a, n_b, 1)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        correlate_templates_and_particle(T, P, layout, work)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = correlate_templates_and_particle(T, P, layout, work)
    for seed in (2, 3):
        t, p = _inputs(n, n_a, n_b, seed)
        T.copy_(t)
        P.copy_(p)
        graph.replay()
        got = [v.clone() for v in out]
        for a, b in zip(got, correlate_templates_and_particle(t, p, layout, CorrelationWorkspace(DEV))):
            assert torch.equal(a, b)


def test_template_counts_that_grow_and_shrink():
    layout, work = PackedFourierLayout(64, 8, DEV), CorrelationWorkspace(DEV)
    T, P = _inputs(64, 40, 3, 7)
    want = [v.clone() for v in correlate_templates_and_particle(T, P, layout, CorrelationWorkspace(DEV))]
    for n_a in (1, 16, 17, 5, 40, 39, 1):
        got = correlate_templates_and_particle(T[:n_a], P, layout, work)
        for a, b in zip(got, want):
            assert torch.equal(a, b[:n_a])
