"""Per-kernel timing of plans with resident loops: a launch counts the cells of
all its steps under the kind of step it runs."""
import pytest

import cases
from helpers import product
from test_gpu_resident import _survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["tiny_chpr", "reverse", "tiny_dxr"])
def test_kinds_and_cells_as_with_step_kernels(what):
    import torch
    case = dict(_survey(100, 121, 3, 150), chpr=5) if what == "reverse" else cases.by_name(what)
    model = {k: torch.from_numpy(v).cuda() for k, v in case["model_est"].items()}
    cells = []
    for extra in ({}, {"persist": False, "graph": False}):
        W = product(case, **extra)
        d = {k: v.clone() for k, v in W.forward_modeling(model).items()}
        W.plan.profile()
        W.misfit_gradient(model, {k: 0.5 * v for k, v in d.items()})
        torch.cuda.synchronize()
        cells.append([W.plan.profile_read(kind)[2] for kind in (0, 1, 2)])
        assert W.plan.resident == (not extra)
    assert cells[0] == cells[1]
