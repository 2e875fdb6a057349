"""Ensembles that run as two concurrent halves from fewer members on (finer
grids, FP64), with halves of whole tiles: the one-group run's results, bit for
bit, and its gradients up to the order of the atomic sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,B,precision", [(42, 11, "fp64"), (42, 33, "fp64"), (63, 17, "fast"), (63, 7, "fp64"),
                                           (106, 10, "fast"), (106, 4, "fp64")])
def test_split_equals_one_group(cuda, monkeypatch, M, B, precision):
    from my_swampe_gb300 import model

    assert B * model._SPLIT_WEIGHT[precision][M] >= model._SPLIT_MIN_B
    rng = np.random.default_rng(M)
    p = {k: torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True)
         for k, v in dict(taurad=10.0 ** rng.uniform(4.5, 5.5, B), DPhieq=rng.uniform(1e5, 4e6, B)).items()}
    res = []
    for least in (64, 10**9):
        monkeypatch.setattr(model, "_SPLIT_MIN_B", least)
        last = model.run_model_scan_final(M=M, dt=840.0 / M, tmax=6, Phibar=4.0e6, omega=3.2e-5, a=8.2e7, taudrag=5e4,
                                          precision=precision, **p)["last_state"]
        res.append((last, torch.autograd.grad((last.Phi_curr.double() ** 2).mean(), list(p.values()))))
    (a, ga), (b, gb) = res
    for name in ("eta_curr", "delta_curr", "Phi_curr", "U_curr", "V_curr", "Phi_prev", "etam_curr", "Am_curr"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    for x, y in zip(ga, gb):
        torch.testing.assert_close(x, y, rtol=1e-12 if precision == "fp64" else 1e-5, atol=0)


@pytest.mark.parametrize("M,B,precision", [(42, 29, "fast"), (42, 10, "fp64"), (106, 5, "fast")])
@pytest.mark.parametrize("scheme", [dict(semi_implicit=True), dict(expflag=True), dict(raw_filter=True),
                                    dict(semi_implicit=True, raw_filter=True)])
def test_split_schemes_equal_one_group(cuda, monkeypatch, M, B, precision, scheme):
    """Every field of the final State, the lagged remainders and the filtered
    prev carries of the opt-in schemes among them."""
    from my_swampe_gb300 import model

    rng = np.random.default_rng(B)
    p = {k: torch.tensor(v, dtype=torch.float64, device="cuda")
         for k, v in dict(taurad=10.0 ** rng.uniform(4.5, 5.5, B), DPhieq=rng.uniform(1e5, 4e6, B),
                          alpha=rng.uniform(0.01, 0.05, B)).items()}
    kind = "fast other schemes" if precision == "fast" and set(scheme) != {"raw_filter"} else precision
    weight = dict(model._SPLIT_WEIGHT, fast={M: 64})  # raw_filter's threshold in the fast precision is Euler's
    assert B * weight[kind][M] >= model._SPLIT_MIN_B
    monkeypatch.setattr(model, "_SPLIT_WEIGHT", weight)
    res = []
    for least in (64, 10**9):
        monkeypatch.setattr(model, "_SPLIT_MIN_B", least)
        res.append(model.run_model_scan_final(M=M, dt=840.0 / M, tmax=7, Phibar=4.0e6, omega=3.2e-5, a=8.2e7,
                                              taudrag=5e4, precision=precision, **p, **scheme)["last_state"])
    for name in res[0]._fields:
        assert torch.equal(getattr(res[0], name), getattr(res[1], name)), name
