"""The calls around the kernels: packed weights follow every way a parameter
can change, gradients that a call returned are the caller's, and autograd asks
for parameter gradients only where they are wanted."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _siren(hidden=(64, 64, 64), seed=0):
    from mplicits_gb300.model import SIREN
    torch.manual_seed(seed)
    return SIREN(3, 1, list(hidden), w0=30).cuda()


def _fresh(m):
    """The same level, built and packed anew."""
    from mplicits_gb300.model import SIREN
    n = SIREN(3, 1, [l.out_features for l in m.linears()[:-1]], w0=m.w0, delay_init=True).cuda()
    n.load_state_dict(m.state_dict())
    return n


def test_packed_weights_follow_the_parameters():
    m, x = _siren(), torch.rand(257, 3, device="cuda")
    lin = m.net[1][0]
    with torch.no_grad():
        a = m(x)["model_out"]
        lin.weight.mul_(1.01)                                     # in place
        b = m(x)["model_out"]
        lin.weight = torch.nn.Parameter(lin.weight * 0.9)         # another Parameter
        c = m(x)["model_out"]
        lin.bias.data = lin.bias.data + 0.1                       # another storage
        d = m(x)["model_out"]
        m.net[2][0] = torch.nn.Linear(64, 64, device="cuda")      # another module
        e = m(x)["model_out"]
        for got in (a, b, c, d):
            assert not torch.equal(got, e)
        assert torch.equal(e, _fresh(m)(x)["model_out"])
        torch.nn.utils.parametrizations.weight_norm(m.net[1][0])  # a computed weight
        m.net[1][0].parametrizations.weight.original0.mul_(1.5)
        f = m(x)["model_out"]
    assert not torch.equal(e, f)


def test_inputs_of_every_kind():
    m = _siren()
    x = torch.rand(6, 5, 3, device="cuda")
    with torch.no_grad():
        want = m(x.reshape(-1, 3))["model_out"].reshape(6, 5, 1)
        assert torch.equal(m(x)["model_out"], want)
        assert torch.equal(m(x.double())["model_out"], want)
        assert torch.equal(m(x.transpose(0, 1))["model_out"], want.transpose(0, 1))
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            y = m(x)["model_out"]
        torch.cuda.current_stream().wait_stream(s)
        assert torch.equal(y, want)
    out = m(x)
    assert out["model_in"].requires_grad and out["model_in"] is not x
    assert torch.equal(out["model_out"].detach(), want)


@pytest.mark.parametrize("hidden,precision", [((64, 64, 64), "fp32"), ((40, 50, 60), "fp32"),
                                              ((256, 256, 256), "fp32"),
                                              ((256, 256, 256), "bf16"),
                                              ((128, 200, 140), "bf16")])
def test_returned_gradients_stay(hidden, precision):
    from mplicits_gb300.train import ResidualTrainer
    m = _siren(hidden)
    tr = ResidualTrainer(m, precision=precision)
    g = torch.Generator("cuda").manual_seed(0)
    batch = lambda n: (torch.rand(n, 3, device="cuda", generator=g),  # noqa: E731
                       torch.rand(n, 3, device="cuda", generator=g),
                       torch.rand(n, device="cuda", generator=g))
    b = batch(300)
    _, first = tr.loss_and_grads(*b)
    kept = [t.clone() for t in first]
    assert [t.shape for t in first] == [p.shape for p in m.parameters()]
    tr.loss_and_grads(*batch(500))
    tr.step(*batch(700))
    for a, k in zip(first, kept):
        assert torch.equal(a, k)


def test_parameter_gradients_only_where_wanted(monkeypatch):
    from mplicits_gb300 import train
    m, x = _siren(), torch.rand(300, 3, device="cuda")
    calls = []
    real = train.param_grads
    monkeypatch.setattr(train, "param_grads",
                        lambda *a, **k: calls.append(1) or real(*a, **k))
    out = m(x)
    G = torch.autograd.grad(out["model_out"].sum(), out["model_in"], create_graph=True)[0]
    assert not calls
    (out["model_out"].sum() + G.square().sum()).backward()
    assert len(calls) == 2
    both = [p.grad.clone() for p in m.parameters()]
    # the same two terms one at a time
    parts = []
    for i in range(2):
        m.zero_grad()
        out = m(x)
        G = torch.autograd.grad(out["model_out"].sum(), out["model_in"], create_graph=True)[0]
        (out["model_out"].sum() if i == 0 else G.square().sum()).backward()
        parts.append([p.grad.clone() if p.grad is not None else 0 for p in m.parameters()])
    for b, p, q in zip(both, *parts):
        # atomic sums in another order: 2^-24 of the largest entry a few times over
        assert (b - (p + q)).abs().max() <= 1e-5 * b.abs().max()
    # frozen parameters: no gradient node, d(model_in) still there
    m.requires_grad_(False)
    calls.clear()
    out = m(x)
    out["model_out"].sum().backward()
    assert out["model_in"].grad is not None and not calls
