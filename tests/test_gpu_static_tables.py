"""build_static's one-launch tables (csrc/static_tables.cu) against its tensor
expressions (which parameters that carry derivatives take), scalars and
ensembles, every truncation, forced and not."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu

BASE = dict(dt=600.0, a=8.2e7, omega=3.2e-5, g=9.8, Phibar=3.0e5, taurad=36000.0, taudrag=21600.0, DPhieq=1.0e6,
            K6=1.24e33, K6Phi=None)


@pytest.mark.parametrize("M", [42, 63, 106])
@pytest.mark.parametrize("test", [None, 2])
@pytest.mark.parametrize("vector", [(), ("taurad", "DPhieq"), ("dt", "a", "omega", "Phibar", "K6", "K6Phi")])
def test_tables_match_the_tensor_expressions(cuda, M, test, vector):
    from my_swampe_gb300.model import build_static

    kw = dict(BASE)
    for k in vector:
        v = kw[k] if kw[k] is not None else 2.0e33
        kw[k] = torch.tensor([v, 1.5 * v, 0.7 * v], dtype=torch.float64, device="cuda")
    got = build_static(M=M, test=test, **kw)
    tracked = dict(kw, g=torch.tensor(kw["g"], dtype=torch.float64, device="cuda", requires_grad=True))
    want = build_static(M=M, test=test, **tracked)
    for f in dataclasses.fields(got):
        x, y = getattr(got, f.name), getattr(want, f.name)
        if torch.is_tensor(y):
            y = y.detach()
            assert x.shape == y.shape and x.dtype == y.dtype, f.name
            # a dozen roundings; the sigmas' n^6 factor and powers of a add a few
            assert torch.all((x - y).abs() <= 40 * 2.3e-16 * y.abs()), f.name
        else:
            assert x == y, f.name
