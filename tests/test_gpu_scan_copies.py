"""simulate_scan_last's reverse mode runs a small ensemble's parameter tangents
as copies of its members in one run: the same bits as one run per parameter,
from two-level and stepped states, single members and ensembles."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,dtype", [(0, torch.float64), (0, torch.float32), (5, torch.float32)])
@pytest.mark.parametrize("semi", [False, True])
@pytest.mark.parametrize("stepped", [False, True])
def test_copies_equal_single_runs(cuda, monkeypatch, B, dtype, semi, stepped):
    from my_swampe_gb300 import model

    gen = torch.Generator(device="cuda").manual_seed(4)
    shape = (B, 64, 128) if B else (64, 128)
    Phi = 1e3 * torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    z = torch.zeros(shape, dtype=torch.float64, device="cuda")
    flags = model.RunFlags(diagnostics=False, semi_implicit=semi)
    base = model.build_static(M=42, dt=300.0, a=8.2e7, omega=3.2e-5, g=9.8, Phibar=3.0e5, taurad=36000.0,
                              taudrag=21600.0, DPhieq=1.0e6, K6=1.24e33, K6Phi=None, test=None)
    eta = (2 * 3.2e-5 * base.mus)[:, None].expand(shape)
    f = [x.to(dtype).contiguous() for x in (eta, z, Phi, z, z)]
    state = model._init_state_from_fields(static=base, flags=flags, test=None, eta0=f[0], delta0=f[1], Phi0=f[2],
                                          U0=f[3], V0=f[4])
    kw = dict(flags=flags, test=None, Uic=f[3], Vic=f[4])
    if stepped:
        state = model.simulate_scan_last(static=base, state0=state, t_seq=range(2, 6), **kw)
    t0 = 6 if stepped else 2

    def grads(members):
        monkeypatch.setattr(model, "_TANGENT_MEMBERS", members)
        p = {k: torch.full((B,) if B else (), getattr(base, k).item(), dtype=torch.float64, device="cuda",
                           requires_grad=True) for k in ("taurad", "taudrag", "DPhieq")}
        last = model.simulate_scan_last(static=dataclasses.replace(base, **p), state0=state, t_seq=range(t0, t0 + 5), **kw)
        return torch.autograd.grad((last.Phi_curr.double() ** 2).mean() + last.U_curr.double().mean(), list(p.values()))

    for x, y in zip(grads(24), grads(1)):
        assert torch.equal(x, y) and bool((x != 0).all())
