"""Plans with resident loops used from several threads, each on a stream of its
own: the loops of one plan neither disturb nor wait for another's."""
import threading

import pytest

from helpers import product
from test_gpu_resident import _survey

pytestmark = pytest.mark.gpu


def test_plans_of_other_sizes_on_other_threads():
    """The same kernels with other shared-memory sizes (few and many receivers)."""
    import torch
    cases = []
    for receivers in (120, 9, 40):
        c = _survey(100, 120, 2, 60)
        c["rec_loc"] = c["rec_loc"][:receivers]
        cases.append(c)
    failed, start = [], threading.Barrier(len(cases))

    def evaluate(case):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                W = product(case)
                model = {k: torch.from_numpy(v).cuda() for k, v in case["model_est"].items()}
                d = {k: 0.5 * v for k, v in W.forward_modeling(model).items()}
                first = {k: v.clone() for k, v in W.misfit_gradient(model, d)[1].items()}
                assert W.plan.resident
                start.wait(60)
                for _ in range(40):
                    g = W.misfit_gradient(model, d)[1]
                    assert all(torch.equal(first[k], g[k]) for k in g)
                W.plan.check_device()
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))
            start.abort()
    threads = [threading.Thread(target=evaluate, args=(c,)) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
