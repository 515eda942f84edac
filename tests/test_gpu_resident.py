"""The resident time loops (the default where a grid fits on chip) against
the step kernels: the same seismograms, misfits and gradients bit for bit,
whatever the tiling -- both stencils, blocks of 1 to 3 rows, one shot per
launch to all of them, grids whose rows and columns leave remainders,
recompute segments, shot groups, sub-stepped time, wells beside a surface
line, more source samples than travel with one launch -- and the bounded
wait's failure path."""
import numpy as np
import pytest

import cases
from helpers import product

pytestmark = pytest.mark.gpu


def _survey(nz, nx, ns, nt, order=4, **inpa):
    """A surface survey over a layered model with scatter."""
    c = dict(cases.c2())
    c["inpa"] = dict(c["inpa"], sdo=order, **inpa)
    c["inpa"]["t"] = (nt - 0.5) * c["inpa"]["dt"]
    rng = np.random.default_rng(1)

    def model(s):
        vp = (2000 + 1000 * np.linspace(0, 1, nz)[:, None] + s * rng.standard_normal((nz, nx))).astype(np.float32)
        return {"vp": vp, "vs": (vp / 1.8).astype(np.float32), "rho": (310 * vp ** 0.25).astype(np.float32)}

    c["model_obs"], c["model_est"] = model(30.0), model(5.0)
    dh = c["inpa"]["dh"]
    c["src_loc"] = np.stack([np.linspace(5, nx - 6, ns).astype(np.int32) * dh, np.full(ns, 2 * dh)], 1).astype(np.float32)
    c["rec_loc"] = np.stack([np.arange(nx) * dh, np.full(nx, 2 * dh)], 1).astype(np.float32)
    return c


def _run(case, **extra):
    import torch
    W = product(case, **extra)
    est, obs = ({k: torch.from_numpy(v).cuda() for k, v in case[m].items()} for m in ("model_est", "model_obs"))
    d_obs = {k: v.clone() for k, v in W.forward_modeling(obs).items()}
    d = {k: v.clone() for k, v in W.forward_modeling(est).items()}
    grad = W.gradient({k: d[k] - d_obs[k] for k in d}, parameterization=case["param"])
    rms, fused = W.misfit_gradient(est, d_obs, parameterization=case["param"])
    W.plan.check_device()
    out = {"rms": rms}
    for n, t in (("d", d), ("g", grad), ("m", fused)):
        out.update({n + "_" + k: v for k, v in t.items()})
    return W, out


NAMED = [("tiny_dxr", {}), ("tiny_dtscale", {}), ("tiny_both", {}), ("tiny_water", {}), ("c1", {}),
         ("c1", {"segment": 50, "shot_batch": 3}), ("tiny_s8", {"energy_balancing": False, "segment": 11})]
SIZED = [((37, 61, 1, 90), {}), ((300, 500, 3, 40), {}), ((150, 301, 2, 70, 8), {}), ((201, 403, 7, 150), {"segment": 40}),
         ((500, 1000, 2, 60), {}), ((130, 170, 5, 90, 8), {}), ((33, 45, 2, 1300), {"fdom": 2.0}),
         ((23, 1400, 2, 40), {}), ((900, 40, 2, 40), {})]


@pytest.mark.parametrize("what,extra", NAMED + SIZED, ids=lambda v: str(v))
def test_resident_loops_give_the_step_kernels_bits(what, extra):
    case = cases.by_name(what) if isinstance(what, str) else _survey(*what)
    Wr, r = _run(case, **extra)
    Ws, s = _run(case, persist=False, **extra)
    assert Wr.plan.resident and not Ws.plan.resident
    for k in s:
        assert bool((r[k] == s[k]).all()) and bool((s[k] == s[k]).all()), k
    assert Wr.plan.frame_check() == 0  # nothing written outside the grid's planes
    assert Wr.plan.launches() * 4 < Ws.plan.launches()


def _reverse(percent, *size):
    return dict(_survey(*size), chpr=percent)


@pytest.mark.parametrize("what,extra", [("tiny_s8", {}), ("tiny_s8", {"segment": 11}), ("c1", {"energy_balancing": True}),
                                        ("tiny_chpr", {}), ("tiny_crosswell", {}), ((10, 190, 291, 5, 200), {}),
                                        ((5, 100, 121, 3, 150), {"shot_batch": 2}), ((60, 61, 70, 2, 90), {}),
                                        ((20, 75, 90, 2, 120, 8), {}), ((10, 33, 45, 2, 2100), {}), ((4, 300, 500, 2, 75), {})], ids=lambda v: str(v))
def test_sets_formed_from_states(what, extra):
    """Energy terms (states stored) and reconstructed states: the difference
    sets are formed a chunk of steps at a time.  The step kernels' bits."""
    case = cases.by_name(what) if isinstance(what, str) else _reverse(*what)
    Wr, r = _run(case, **extra)
    Ws, s = _run(case, persist=False, **extra)
    assert Wr.plan.resident and not Ws.plan.resident
    for k in s:
        assert bool((r[k] == s[k]).all()), k
    assert Wr.plan.frame_check() == 0


@pytest.mark.parametrize("what,extra", [("tiny_dxr", {}), ("tiny_dtscale", {}), ("tiny_both", {"segment": 40, "shot_batch": 1}),
                                        ("c1", {}), ((37, 61, 1, 90), {}), ((101, 203, 4, 100), {"segment": 30}),
                                        ((150, 301, 2, 70, 8), {}), ((33, 900, 2, 60), {})], ids=lambda v: str(v))
def test_exact_adjoint_on_chip(what, extra):
    """The exact adjoint's resident loop against its step kernels: the traces'
    bits; the gradient sums the same terms with roundings of their own (the
    source's part of a stress difference is added to the stress, not to the
    difference), so it agrees to float32 rounding."""
    case = cases.by_name(what) if isinstance(what, str) else _survey(*what)
    Wr, r = _run(case, adjoint="exact", **extra)
    Ws, s = _run(case, adjoint="exact", persist=False, **extra)
    assert Wr.plan.resident and not Ws.plan.resident
    for k in s:
        if k.startswith("d_") or k == "rms":
            assert bool((r[k] == s[k]).all()), k
        else:
            assert float((r[k] - s[k]).norm()) <= 1e-6 * float(s[k].norm()), k
    assert Wr.plan.frame_check() == 0


def test_steps_kernels_where_they_are_asked_for():
    case = cases.by_name("tiny_dxr")
    for asked in ({"tile": 1}, {"adj_tile": 1}, {"graph": True}, {"persist": False}, {"store": "states"}, {"overlap": True, "segment": 20}):
        assert not product(case, **asked).plan.resident, asked
    with pytest.raises(ValueError, match="persist"):
        product(case, persist=2).plan


def test_a_loop_that_gave_up_raises_and_leaves_nan():
    import torch
    from pyfwi_b200._native import NativeError
    case = cases.by_name("tiny_dxr")
    W = product(case)
    assert W.plan.resident
    clean = W.forward_modeling(case["model_est"])
    W.plan.barrier_selftest(20_000_000)  # sets the error word, as a wait that ran out does
    with pytest.raises(NativeError, match="device error word 3"):
        W.forward_modeling(case["model_est"])
    W.plan.barrier_selftest(20_000_000)
    d = W.forward_modeling({k: torch.from_numpy(v).cuda() for k, v in case["model_est"].items()})
    assert d and all(bool(torch.isnan(v).any()) for v in d.values())
    with pytest.raises(NativeError, match="device error word 3"):
        W.plan.check_device()
    again = W.forward_modeling(case["model_est"])
    for k in clean:
        assert np.array_equal(again[k], clean[k]), k
