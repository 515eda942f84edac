"""A caller's CUDA graphs and the resident time loops: a captured call takes
the same loops as a direct one and leaves the same things in the workspace, so
graph replays and direct calls of one plan can be mixed."""
import pytest

import cases
from helpers import product

pytestmark = pytest.mark.gpu

KINDS = [("tiny_dxr", {}), ("tiny_dxr", {"adjoint": "exact"}), ("tiny_dtscale", {"adjoint": "exact"}),
         ("tiny_s8", {"energy_balancing": True}), ("tiny_chpr", {})]


def _graph(call):
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    return g


@pytest.mark.parametrize("name,extra", KINDS, ids=lambda v: str(v))
def test_replays_and_direct_calls_mix(name, extra):
    import torch
    case = cases.by_name(name)
    W = product(case, **extra)
    plan = W.plan
    assert plan.resident
    models = [[torch.from_numpy(case[m][k]).cuda() for k in ("vp", "vs", "rho")] for m in ("model_est", "model_obs")]
    damp, traces = W._damping(), None
    buf = [t.clone() for t in models[0]]  # the model the graphs read
    nrs = int(W.ns) * int(W.nr)
    gen = torch.Generator(device="cuda").manual_seed(3)
    res = [torch.randn((plan.nt_ext, nrs), device="cuda", generator=gen) for _ in range(5)]
    grad = torch.empty((3, plan.nz, plan.nx), device="cuda")

    def model(q):
        for b, m in zip(buf, models[q]):
            b.copy_(m)
        plan.set_model(*buf, *damp)

    want, wave = [], []
    for q in (0, 1):
        model(q)
        n = plan.launches()
        traces = plan.forward(W._wavelet, traces)
        plan.gradient(res, 1, grad=grad)
        direct = plan.launches() - n
        want.append(grad.clone())
        wave.append(traces.clone())
    assert not torch.equal(want[0], want[1])

    model(0)
    n = plan.launches()
    whole = _graph(lambda: (plan.set_model(*buf, *damp), plan.forward(W._wavelet, traces)))
    backward = _graph(lambda: plan.gradient(res, 1, grad=grad))
    captured = plan.launches() - n
    for q in (0, 1):
        # a direct forward pass, then the captured gradient
        model(q)
        plan.forward(W._wavelet, traces)
        backward.replay()
        assert torch.equal(grad, want[q]), ("captured gradient", q)
        # a captured forward pass (of the other model before it), then the direct gradient
        model(1 - q)
        plan.forward(W._wavelet, traces)
        for b, m in zip(buf, models[q]):
            b.copy_(m)
        whole.replay()
        assert torch.equal(traces, wave[q])
        plan.gradient(res, 1, grad=grad)
        assert torch.equal(grad, want[q]), ("captured forward pass", q)
        # and both captured
        whole.replay()
        backward.replay()
        assert torch.equal(grad, want[q]), ("both captured", q)
    plan.check_device()
    assert captured <= direct + 8  # the same loops, and the model's kernels
