"""Plans whose two passes run differently, because the step kernels are faster
in one of them: the step kernels' bits all the same."""
import pytest

from test_gpu_resident import _run, _survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,chpr,extra", [((300, 500, 64, 9, 8), 100, {"energy_balancing": True}),
                                             ((300, 500, 64, 9, 8), 100, {"energy_balancing": True, "segment": 4}),
                                             ((480, 520, 16, 41), 10, {}), ((200, 400, 64, 30), 20, {"shot_batch": 40})],
                         ids=lambda v: str(v))
def test_one_pass_on_chip(size, chpr, extra):
    case = dict(_survey(*size), chpr=chpr)
    Wr, r = _run(case, **extra)
    Ws, s = _run(case, persist=False, **extra)
    assert Wr.plan.resident and not Ws.plan.resident
    for k in s:  # (cells that nothing reached in so few steps have no energy to balance with: 0 / 0)
        assert bool(((r[k] == s[k]) | ((r[k] != r[k]) & (s[k] != s[k]))).all()) and bool((s[k] == s[k]).any()), k
    assert Wr.plan.frame_check() == 0
    launches = []
    for W in (Wr, Ws):
        n = W.plan.launches()
        W.forward_modeling({k: v for k, v in case["model_est"].items()})
        launches.append(W.plan.launches() - n)
    nt = int(Wr.nt)
    assert (launches[0] >= nt) == (chpr == 100) and launches[1] >= nt  # the forward pass: step kernels where states are stored
