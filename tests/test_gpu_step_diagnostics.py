"""The per-step diagnostics (least speed, extremes of Phi), compared as integers
and kept by integer atomics: against the history rows, alike for one member and
for the same member in an ensemble (other rows per CTA), untouched by a member
of NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [42, 63, 106])
@pytest.mark.parametrize("precision", ["fp64", "fast"])
@pytest.mark.parametrize("scale", [1.0, -1.0])
def test_diagnostics_follow_the_fields(cuda, M, precision, scale):
    from my_swampe_gb300 import run_model_scan
    from my_swampe_gb300.model import _SUPPORTED_M

    J, I, _ = _SUPPORTED_M[M]
    rng = np.random.default_rng(M)
    lat = np.linspace(-1.4, 1.4, J)[:, None]
    lam = np.linspace(-np.pi, np.pi, I, endpoint=False)[None, :]
    phi = scale * np.stack([3e4 * (k + 1.5 + np.cos(lam + k) * np.cos(lat)) for k in range(9)])  # one sign per run
    ics = dict(eta0_init=6.4e-5 * np.sin(lat) + 0 * phi, delta0_init=0 * phi, Phi0_init=phi,
               U0_init=20 * np.cos(lat) + rng.standard_normal(phi.shape), V0_init=0 * phi)

    def run(members, nan=None):
        f = {k: torch.tensor(v[members], device="cuda") for k, v in ics.items()}
        if nan is not None:
            f["Phi0_init"][nan, 3, 5] = float("nan")
        out = run_model_scan(M=M, dt=840.0 / M, tmax=7, Phibar=4e6, omega=3.2e-5, a=8.2e7, taudrag=5e4, DPhieq=1e5,
                             precision=precision, **f)["outs"]
        return {k: v.cpu() for k, v in out.items()}

    full = run(list(range(9)))
    s2 = full["U"].double() ** 2 + full["V"].double() ** 2
    want = torch.sqrt(s2.amin((-1, -2)))[:, :-1]  # the state after step t is row t + 1's
    torch.testing.assert_close(full["spin_min"][:, 1:], want, rtol=1e-15, atol=0)
    assert torch.isfinite(full["phi_min"]).all() and (full["phi_min"] < full["phi_max"]).all()
    assert (torch.sign(full["phi_min"]) == scale).all()
    for b in (0, 8):
        one = run([b])
        for k in ("spin_min", "phi_min", "phi_max"):
            assert torch.equal(one[k][0], full[k][b]), k
        torch.testing.assert_close(one["rms"][0], full["rms"][b], rtol=1e-12, atol=0)
    mixed = run(list(range(9)), nan=4)
    for k in ("spin_min", "phi_min", "phi_max", "dead"):
        assert torch.equal(mixed[k][[0, 8]], full[k][[0, 8]]), k
