"""What a resident loop that gave up a wait leaves behind, and who is told.  The
error word is set on purpose (a bounded wait of 20 ms that nothing ends)."""
import pytest

import cases
from helpers import product

pytestmark = pytest.mark.gpu


def _setup(name="tiny_dxr", **extra):
    import torch
    case = cases.by_name(name)
    W = product(case, **extra)
    model = {k: torch.from_numpy(v).cuda() for k, v in case["model_est"].items()}
    obs = {k: v.clone() for k, v in W.forward_modeling({k: torch.from_numpy(v).cuda() for k, v in
                                                        case["model_obs"].items()}).items()}
    assert W.plan.resident
    return W, model, obs


@pytest.mark.parametrize("kind", ["forward", "misfit", "gradient"])
def test_a_later_call_on_tensors_raises_and_the_next_one_works(kind):
    import torch
    from pyfwi_b200._native import NativeError
    W, model, obs = _setup()

    def call():
        if kind == "forward":
            return W.forward_modeling(model)
        if kind == "misfit":
            return W.misfit_gradient(model, obs)[1]
        return W.gradient({k: v - obs[k] for k, v in W.forward_modeling(model).items()})
    clean = {k: v.clone() for k, v in call().items()}
    torch.cuda.synchronize()
    W.plan.barrier_selftest(20_000_000)
    bad = call()
    assert any(bool(torch.isnan(v).any()) for v in bad.values())
    torch.cuda.synchronize()
    with pytest.raises(NativeError, match="device error word 3"):
        call()
        torch.cuda.synchronize()
        call()  # the first was looked at before the wait ran out
    for _ in range(2):
        again = call()
        torch.cuda.synchronize()
    for k in clean:
        assert torch.equal(again[k], clean[k]), k
    W.plan.check_device()


def _same(a, b):
    """Finite values alike."""
    import torch
    return bool(((a == b) | ~(torch.isfinite(a) | torch.isfinite(b))).all())


BLOWN = [("tiny_dxr", {}, 6.0), ("tiny_dtscale", {}, 8.0), ("tiny_both", {}, 5.0), ("c1", {}, 4.0), ("tiny_s8", {"energy_balancing": True}, 6.0),
         ("tiny_s8", {"energy_balancing": False}, 9.0), ("tiny_chpr", {}, 6.0), ("tiny_dxr", {"adjoint": "exact"}, 6.0),
         ("c1", {"adjoint": "exact"}, 4.0)]


@pytest.mark.parametrize("name,extra,factor", BLOWN, ids=lambda v: str(v))
def test_overflows_spread_as_in_the_step_kernels(name, extra, factor):
    """A model too fast for its time step overflows: the same samples are finite,
    with the same bits (infinity or NaN is not told apart: where the damping is
    zero the resident loops do not multiply by it), and the next model is modelled
    as if nothing had been."""
    import torch
    W, model, obs = _setup(name, **extra)
    S = product(cases.by_name(name), persist=False, **extra)
    S.forward_modeling(model)
    fast = {k: v * (factor if k != "rho" else 1.0) for k, v in model.items()}
    out = []
    for P in (W, S):
        d = {k: v.clone() for k, v in P.forward_modeling(fast).items()}
        raw = P._traces.clone()
        g = P.gradient({k: v - obs[k] for k, v in d.items()})
        out.append([raw] + list(d.values()) + list(g.values()))
    assert any(not bool(torch.isfinite(t).all()) for t in out[1])
    assert all(_same(a, b) for a, b in zip(*out))
    again = W.misfit_gradient(model, obs)[1]
    for k, v in S.misfit_gradient(model, obs)[1].items():
        assert torch.equal(again[k], v), k
    assert W.plan.frame_check() == 0  # what overflowed into a frame is overwritten


@pytest.mark.parametrize("name,extra", [("tiny_dxr", {}), ("c1", {}), ("tiny_s8", {"energy_balancing": True}), ("tiny_chpr", {}),
                                        ("tiny_dxr", {"adjoint": "exact"})], ids=lambda v: str(v))
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3e38])
def test_residuals_that_are_not_numbers(name, extra, value):
    import torch
    W, model, obs = _setup(name, **extra)
    S = product(cases.by_name(name), persist=False, **extra)
    out = []
    for P in (W, S):
        d = {k: v.clone() for k, v in P.forward_modeling(model).items()}
        res = {k: (v - obs[k]).clone() for k, v in d.items()}
        first = res[next(iter(res))].view(-1)
        first[first.numel() // 2 + 1] = value
        g = P.gradient(res)
        out.append(list(g.values()))
    assert all(_same(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("adjoint", ["reference", "exact"])
def test_receivers_outside_the_grid_add_nothing(adjoint):
    """Only the C interface takes them; such plans keep the step kernels."""
    import torch
    from pyfwi_b200 import _native as N
    from pyfwi_b200.engine import Plan
    W, model, _ = _setup(adjoint=adjoint)
    geom, grads = W._geometry(), []
    geom.lines[0].col0 -= geom.npml + 3  # the first three columns lie left of the grid
    for persist in (2, 0):
        o = N.Options()
        o.persist, o.store_diffs = persist, 1
        o.adjoint = N.ADJOINT_EXACT if adjoint == "exact" else N.ADJOINT_REFERENCE
        plan = Plan(geom, W.srcx, W.srcz, o, W.device)
        plan.set_model(*(model[k] for k in ("vp", "vs", "rho")), *W._damping())
        traces = plan.forward(W._wavelet)
        grads.append(plan.gradient([t.contiguous() + 1.0 for t in traces], 1))
        assert plan.frame_check() == 0, persist
    assert torch.equal(*grads)


def test_a_replayed_batch_reports_a_loop_that_gave_up():
    """The graph of a batch whose plan was built with resident loops."""
    import torch
    from pyfwi_b200._native import NativeError
    from pyfwi_b200.batch import SurveyBatch
    W, model, obs = _setup()
    batch = SurveyBatch([W], graph=True)
    clean = {k: v.clone() for k, v in batch.misfit_gradient([model], [obs])[0][1].items()}
    torch.cuda.synchronize()
    W.plan.barrier_selftest(20_000_000)
    batch.misfit_gradient([model], [obs])
    torch.cuda.synchronize()
    with pytest.raises(NativeError, match="device error word 3"):
        for _ in range(3):
            batch.misfit_gradient([model], [obs])
            torch.cuda.synchronize()
    again = batch.misfit_gradient([model], [obs])[0][1]
    assert all(torch.equal(again[k], clean[k]) for k in clean)
