"""State fields given once for a whole ensemble (a scalar dead flag, Fourier
fields with a member axis of one), forward and backward."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(B):
    from my_swampe_gb300 import model

    gen = torch.Generator(device="cuda").manual_seed(4)
    Phi = (1e3 * torch.randn((1, 64, 128), dtype=torch.float64, device="cuda", generator=gen)).expand(B, 64, 128)
    z = torch.zeros((B, 64, 128), dtype=torch.float64, device="cuda")
    flags = model.RunFlags(diagnostics=False)
    static = model.build_static(M=42, dt=300.0, a=8.2e7, omega=3.2e-5, g=9.8, Phibar=3.0e5, taurad=36000.0,
                                taudrag=21600.0, DPhieq=1.0e6, K6=1.24e33, K6Phi=None, test=None)
    eta = (2 * 3.2e-5 * static.mus)[:, None].expand(B, 64, 128)
    state = model._init_state_from_fields(static=static, flags=flags, test=None, eta0=eta, delta0=z, Phi0=Phi, U0=z, V0=z)
    return model, static, flags, state, z


def _run(model, static, flags, state, z, B, grad):
    p = {k: torch.linspace(0.8, 1.2, B, dtype=torch.float64, device="cuda") * getattr(static, k) for k in ("taurad", "taudrag")}
    p = {k: v.requires_grad_(grad) for k, v in p.items()}
    last = model.simulate_scan_last(static=dataclasses.replace(static, **p), flags=flags, state0=state,
                                    t_seq=range(2, 6), test=None, Uic=z, Vic=z)
    return torch.autograd.grad(last.Phi_curr.mean(), list(p.values())) if grad else [last.Phi_curr]


@pytest.mark.parametrize("B", [1, 4])
@pytest.mark.parametrize("grad", [False, True])
def test_scalar_dead_flag(cuda, B, grad):
    model, static, flags, state, z = _case(B)
    scalar = state._replace(dead=torch.zeros((), dtype=torch.bool, device="cuda"))
    for x, y in zip(_run(model, static, flags, scalar, z, B, grad), _run(model, static, flags, state, z, B, grad)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("grad", [False, True])
def test_fourier_fields_of_one_member(cuda, grad):
    B = 4
    model, static, flags, state, z = _case(B)
    one = state._replace(**{k: getattr(state, k)[:1] for k in ("Am_curr", "Phim_prev", "PhiFm_curr")})
    for x, y in zip(_run(model, static, flags, one, z, B, grad), _run(model, static, flags, state, z, B, grad)):
        assert torch.equal(x, y)
