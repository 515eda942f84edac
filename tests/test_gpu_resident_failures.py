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
