"""Losses of a trainer whose call was captured into a CUDA graph: the captured
call leaves nothing behind that an eager one then takes for computed."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(n, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    r = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731
    return r(n, 3) * 2 - 1, r(n, 3), r(n) * 0.1


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_eager_after_capture(precision):
    from mplicits_gb300.model import SIREN
    from mplicits_gb300.train import ResidualTrainer
    torch.manual_seed(0)
    m = SIREN(3, 1, [128, 128, 128], w0=30).cuda()
    tr = ResidualTrainer(m, precision=precision)
    want, _ = ResidualTrainer(m, precision=precision).loss_and_grads(*_batch(300, 1))
    tr.loss_and_grads(*_batch(500, 2))  # buffers and packed weights
    batch = _batch(300, 1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        captured, _ = tr.loss_and_grads(*batch)
    got, _ = tr.loss_and_grads(*batch)  # the graph has not run yet
    # sums of 300 terms in another atomic order: 300 x 2^-24
    tol = 2e-5 * want.abs().max()
    assert (got - want).abs().max() <= tol
    graph.replay()
    torch.cuda.synchronize()
    assert (captured - want).abs().max() <= tol


def test_replay_after_other_batch_sizes():
    from mplicits_gb300.model import SIREN
    from mplicits_gb300.train import ResidualTrainer
    torch.manual_seed(0)
    m = SIREN(3, 1, [128, 128, 128], w0=30).cuda()
    tr = ResidualTrainer(m)
    tr.loss_and_grads(*_batch(500, 2))
    batch = _batch(300, 1)
    want = tr.loss_and_grads(*batch)[0].clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        captured, _ = tr.loss_and_grads(*batch)
    for n in (400, 200, 100):
        tr.loss_and_grads(*_batch(n, 3))
        torch.full((3,), 1e30, device="cuda")  # takes up what was given back
    graph.replay()
    torch.cuda.synchronize()
    assert (captured - want).abs().max() <= 2e-5 * want.abs().max()
