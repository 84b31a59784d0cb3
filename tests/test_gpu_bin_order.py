"""dem_broad_phase_noalloc behind and ahead of other work on its stream: calls
that share the scratch back to back, positions written just before, and the
same call captured into a graph.  Whole numbers, equal to numpy's stable sort."""
import numpy as np
import pytest

from test_zz_no_alloc import _lib, _numpy_broad_phase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("captured", [False, True])
def test_calls_back_to_back(captured):
    torch = pytest.importorskip("torch")
    L, dev = _lib(), torch.device("cuda", 0)
    jobs = []
    for q, n in enumerate([700001, 33, 400003, 5000]):
        gw, gh = [(509, 509), (7, 3), (16, 32), (300, 200)][q]
        rng = np.random.default_rng(n)
        pr = np.zeros((n, 4), np.float32)
        pr[:, 0] = rng.uniform(-0.05, 1.05, n) * gw
        pr[:, 1] = rng.uniform(-0.05, 1.05, n) * gh
        pr[:, 2] = rng.random(n) > 0.01
        out = [torch.full((k,), -7, dtype=torch.int32, device=dev) for k in (n, n, gw * gh + 2)]
        jobs.append((pr, torch.from_numpy(pr).to(dev), torch.zeros((n, 4), device=dev), (0.0, 0.0, 1.0, gw, gh), out))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def calls():
        for pr, src, d_pr, g, out in jobs:
            d_pr.copy_(src)
            assert L.dem_broad_phase_noalloc(d_pr.data_ptr(), pr.shape[0], *g, *[o.data_ptr() for o in out],
                                             stream.cuda_stream) == 0, L.dem_noalloc_last_error()

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            calls()
        graph.replay()
    else:
        with torch.cuda.stream(stream):
            calls()
            later = [o.clone() for j in jobs for o in j[4]]
    torch.cuda.synchronize()
    if not captured:
        for o, c in zip([o for j in jobs for o in j[4]], later):
            assert torch.equal(o, c)
    for pr, _, _, g, out in jobs:
        for got, want in zip(out, _numpy_broad_phase(pr, *g)):
            assert np.array_equal(got.cpu().numpy(), want)
