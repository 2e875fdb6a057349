"""The forms of the parameters that build_static and set_params take, and what
a Static record shares: nothing with the next one."""
import dataclasses
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BASE = dict(dt=600.0, a=8.2e7, omega=3.2e-5, g=9.8, Phibar=3.0e5, taurad=36000.0, taudrag=21600.0, DPhieq=1.0e6,
            K6=1.24e33, K6Phi=None)


def _build(**kw):
    from my_swampe_gb300.model import build_static

    return build_static(M=42, test=None, **dict(BASE, **kw))


def test_one_value_beside_an_ensemble(cuda):
    """A (1,) parameter broadcasts against (B,) ones, and keeps its shape."""
    v = torch.tensor([3.0e4, 5.0e4, 9.0e4], dtype=torch.float64, device="cuda")
    one = torch.tensor([2.0e6], dtype=torch.float64, device="cuda")
    got, want = _build(taurad=v, DPhieq=one), _build(taurad=v, DPhieq=one.expand(3))
    assert got.DPhieq.shape == (1,) and got.taurad.shape == (3,)
    for f in dataclasses.fields(got):
        x, y = getattr(got, f.name), getattr(want, f.name)
        if torch.is_tensor(y):
            assert torch.all((x - y).abs() <= 40 * 2.3e-16 * y.abs()), f.name


def test_under_vmap(cuda):
    v = torch.tensor([1.0e6, 2.0e6], dtype=torch.float64, device="cuda")
    Phieq, sigma = torch.func.vmap(lambda DP, K: (lambda s: (s.Phieq, s.sigma_exp))(_build(DPhieq=DP, K6=K)))(v, v * 1e27)
    for b in range(2):
        s = _build(DPhieq=v[b], K6=v[b] * 1e27)
        torch.testing.assert_close(Phieq[b], s.Phieq, rtol=1e-14, atol=0)
        torch.testing.assert_close(sigma[b], s.sigma_exp, rtol=1e-14, atol=0)


def test_given_tensors_are_carried_as_they_are(cuda):
    """A tensor parameter is the record's own: also one that requires grad, given under no_grad."""
    p = torch.tensor([3.0e4, 5.0e4], dtype=torch.float64, device="cuda", requires_grad=True)
    q = torch.tensor(2.0e4, dtype=torch.float64, device="cuda")
    with torch.no_grad():
        s = _build(taurad=p, taudrag=q)
    assert s.taurad.requires_grad and s.taurad is p and s.taudrag.shape == (2,) and torch.equal(s.taudrag[1], q)


def test_non_finite_parameters_stay_visible(cuda):
    nan = float("nan")
    for kw in (dict(a=nan), dict(K6=nan), dict(dt=nan), dict(a=math.inf)):
        got = _build(**kw)
        want = _build(**kw, g=torch.tensor(9.8, dtype=torch.float64, device="cuda", requires_grad=True))
        for name in ("tstepcoeffmn", "sigma", "sigmaPhi", "sigma_exp", "sigmaPhi_exp", "tstepcoeff", "tstepcoeff2"):
            x, y = getattr(got, name), getattr(want, name).detach()
            assert torch.equal(torch.isnan(x), torch.isnan(y)), (kw, name)


def test_records_share_nothing_that_was_their_own(cuda):
    names = ("lambdas", "Pmnw", "Hmnw", "marray", "mJarray", "narray")
    first = _build()
    want = {k: getattr(first, k).clone() for k in names}
    Phieq = _build(DPhieq=torch.tensor(1.0e6, dtype=torch.float64, device="cuda", requires_grad=True)).Phieq.detach()
    for k in names:
        torch.as_strided(getattr(first, k), (1,), (1,)).fill_(1.0e3)  # through an expanded view too
    first.lambdas.fill_(0.25)
    again = _build()
    for k in names:
        assert torch.equal(getattr(again, k), want[k]), k
    after = _build(DPhieq=torch.tensor(1.0e6, dtype=torch.float64, device="cuda", requires_grad=True)).Phieq.detach()
    assert torch.equal(Phieq, after)


def test_set_params_refuses_another_length(cuda):
    from my_swampe_gb300.engine import PARAM_NAMES, Engine

    eng = Engine([(42, 3)], "fp64")
    kw = {k: 1.0 for k in PARAM_NAMES}
    for bad in (torch.tensor([1.0]), torch.tensor([1.0, 2.0])):
        with pytest.raises(RuntimeError):
            eng.set_params(0, **dict(kw, taurad=bad))
    eng.set_params(0, **dict(kw, taurad=torch.tensor([1.0, 2.0, 3.0])))
    assert eng.groups[0]["params"][4].tolist() == [1.0, 2.0, 3.0]


def test_constants_formed_on_another_stream(cuda):
    from my_swampe_gb300.engine import Engine
    from my_swampe_gb300.model import build_static

    want = _build()
    eng, side = Engine([(42, 1)], "fp64"), torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)
        eng.geometry(0)
    got = build_static(M=42, test=None, engine=eng, **BASE)
    for k in ("mus", "Pmn", "lambdas", "Hmnw", "narray"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k
    torch.cuda.synchronize()
