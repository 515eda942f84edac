"""The exact adjoint gives the same bits by every route: the resident loop, the
step kernels, a batch of surveys -- with sources at tile borders, wells whose
vz traces record vx, sub-stepped time, recompute segments and shot groups."""
import pytest

import cases
from helpers import product
from test_gpu_resident import _run, _survey

pytestmark = pytest.mark.gpu

SURVEYS = [("tiny_dxr", {}), ("tiny_dtscale", {}), ("tiny_crosswell", {}), ("tiny_water", {}), ("tiny_s8", {"energy_balancing": False}),
           ("tiny_both", {"segment": 40, "shot_batch": 1}), ("c1", {}), ((37, 61, 1, 90), {}), ((101, 203, 17, 100), {"segment": 30}),
           ((150, 301, 9, 70, 8), {}), ((33, 900, 2, 60), {}), ((300, 260, 3, 60), {})]


@pytest.mark.parametrize("what,extra", SURVEYS, ids=lambda v: str(v))
def test_resident_loop_and_step_kernels(what, extra):
    case = cases.by_name(what) if isinstance(what, str) else _survey(*what)
    Wr, r = _run(case, adjoint="exact", **extra)
    Ws, s = _run(case, adjoint="exact", persist=False, **extra)
    assert Wr.plan.resident and not Ws.plan.resident
    for k in s:
        assert bool((r[k] == s[k]).all()) and bool((s[k] == s[k]).all()), k


@pytest.mark.parametrize("graph", [False, True])
def test_a_batch_and_single_surveys(graph):
    import torch
    from pyfwi_b200.batch import SurveyBatch
    names = ["tiny_dxr", "tiny_dtscale", "c1"]
    props = [product(cases.by_name(n), adjoint="exact") for n in names]
    models = [{k: torch.from_numpy(v).cuda() for k, v in cases.by_name(n)["model_est"].items()} for n in names]
    obs = [{k: v.clone() for k, v in W.forward_modeling({k: torch.from_numpy(v).cuda() for k, v in
                                                        cases.by_name(n)["model_obs"].items()}).items()}
           for W, n in zip(props, names)]
    alone = [{k: v.clone() for k, v in W.misfit_gradient(m, o)[1].items()} for W, m, o in zip(props, models, obs)]
    props[1] = product(cases.by_name(names[1]), adjoint="exact")  # its plan is built in the batch, the others' were before
    batch = SurveyBatch(props, graph=graph)
    for _ in range(2):
        for q, (_, g) in enumerate(batch.misfit_gradient(models, obs)):
            for k in g:
                assert torch.equal(g[k], alone[q][k]), (names[q], k)
