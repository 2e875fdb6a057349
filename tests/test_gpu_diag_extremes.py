"""The least speed of a step's diagnostics up to the largest whose square is
finite (the comparison is one of squares)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [1.0e-150, 3.0, 1.0e140, 1.0e151, 1.0e153])
def test_least_speed(cuda, speed):
    from my_swampe_gb300.model import run_model_scan

    z = torch.zeros((64, 128), dtype=torch.float64, device="cuda")
    U = torch.full_like(z, speed)
    U[:, ::2] *= 1.25
    outs = run_model_scan(M=42, dt=30.0, tmax=4, Phibar=3.0e5, omega=3.2e-5, a=8.2e7, eta0_init=z, delta0_init=z,
                          Phi0_init=z, U0_init=U, V0_init=z, precision="fp64")["outs"]
    # the squares may be subnormal: their root is then off by the spacing at the bottom of the range
    assert float(outs["spin_min"][0]) == pytest.approx(speed, rel=1e-12)
