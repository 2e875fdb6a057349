"""The cluster kernels of the emission stage (csrc/emission.cu) at the sizes
where their work split has edges: fewer latitudes than warps of a cluster, row
lengths that are no multiple of a warp, more longitudes than one block of the
phase curve, phase counts around a warp, one pixel."""
import numpy as np
import pytest
import torch

from oracle import emission_oracle as eo

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("JI,phases,B", [((1, 1), 1, 1), ((5, 7), 3, 2), ((64, 128), 257, 3), ((3, 513), 33, 1),
                                         ((70, 1100), 40, 2), ((160, 320), 64, 1)])
def test_simple_phase_curve_sizes(cuda, JI, phases, B):
    from my_swampe_gb300.emission import simple_phase_curve

    rng = np.random.default_rng(JI[0] * 1000 + JI[1])
    phi = rng.standard_normal((B,) + JI) + 0.5
    ph = np.linspace(-7.0, 7.0, phases)
    got = simple_phase_curve(torch.tensor(phi, device="cuda"), ph).cpu().numpy()
    mu = np.polynomial.legendre.leggauss(JI[0])[0]
    aw = np.sqrt(1.0 - mu**2)
    for b in range(B):
        want = eo.simple_phase_curve(phi[b], ph)
        # each cosine carries a few rounding errors (of its argument, up to 10, and of
        # the products): 32 eps of the sum of |terms|, over the mean |flux|
        flux = np.array([np.sum(phi[b] * np.maximum(np.cos(np.linspace(-np.pi, np.pi, JI[1], endpoint=False)[None, :] - p), 0)
                                * aw[:, None]) for p in ph])
        norm = np.mean(np.abs(flux)) or 1.0
        bound = 32 * EPS * np.sum(np.abs(phi[b]) * aw[:, None]) / norm * 2
        assert np.max(np.abs(got[b] - want)) <= bound, (b, np.max(np.abs(got[b] - want)), bound)


@pytest.mark.parametrize("mode,scale", [("geopotential", 3780.0), ("geopotential", 0.5), ("linear", 600.0),
                                        ("linear", 0.25)])
@pytest.mark.parametrize("JI", [(1, 1), (3, 5), (65, 33), (130, 70)])
def test_planck_map_sizes(cuda, JI, mode, scale):
    """The Planck intensity from Phi directly (with the division by the scale
    folded into its argument where the scale is at least 1), against T and the
    library exponential.  Arguments from 0.003 to past the clip at 80."""
    from my_swampe_gb300.emission import EmissionConfig, _map, temperature_to_intensity

    rng = np.random.default_rng(JI[1])
    T = 10.0 ** rng.uniform(1.4, 6.0, (2,) + JI)
    Phibar, T_ref = 100.0, 50.0
    phi = (T * scale - Phibar) if mode == "geopotential" else (T - T_ref) * scale
    kw = dict(emission_temp_mode=mode, R_d=scale, T_ref=T_ref, phi_to_T_scale=scale, emission_model="planck")
    got = _map(torch.tensor(phi, device="cuda"), Phibar, EmissionConfig(**kw), 0, 1)[0].cpu().numpy()
    Tx = eo.phi_to_temperature(phi, Phibar, temp_mode=mode, R_d=scale, T_ref=T_ref, phi_to_T_scale=scale)
    want = eo.planck_intensity_relative(Tx, 4.5e-6)
    # x carries 4 roundings, each x e^x / (e^x - 1) <= 81 times in the intensity; the rest is a few ulp
    assert np.max(np.abs(got / want - 1.0)) <= (4 * 81 + 8) * EPS
    again = temperature_to_intensity(torch.tensor(Tx, device="cuda"), EmissionConfig(**kw)).cpu().numpy()
    assert np.max(np.abs(again / want - 1.0)) <= (4 * 81 + 8) * EPS
