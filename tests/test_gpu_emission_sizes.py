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


@pytest.mark.parametrize("npix,ncoef,B", [(1, 1, 1), (63, 5, 2), (65, 16, 16), (510, 17, 17), (8192, 121, 3),
                                          (513, 129, 33), (70001, 3, 2)])
@pytest.mark.parametrize("kind", ["noise", "constant", "range"])
def test_projection_sizes(cuda, npix, ncoef, B, kind):
    """The sliced projection against extended precision: tiles of 16 members and
    128 coefficients and eighths of the pixels with remainders, more pixels than
    one conversion of the integer sums; constant rows (all digits alike, the
    largest integer sums) and rows that span 40 powers of ten."""
    from my_swampe_gb300.emission import _project

    rng = np.random.default_rng(npix + ncoef)
    P = rng.standard_normal((ncoef, npix))
    r = rng.standard_normal((B, npix)) + 1.0
    if kind == "constant":
        P[:], r[:] = -(1.0 - 2.0**-53) / 3.0, 0.1
    if kind == "range":
        P *= 10.0 ** rng.uniform(-40, 0, P.shape)
        r *= 10.0 ** rng.uniform(0, 5, r.shape)
    P[0] = np.abs(P[0]) + 1e-3
    r = np.abs(r)
    ok = torch.ones(B, dtype=torch.int32, device="cuda")
    y = _project(torch.tensor(r, device="cuda").reshape(B, 1, npix), ok, torch.tensor(P, device="cuda")).cpu().numpy()
    want = (r.astype(np.longdouble) @ P.T.astype(np.longdouble))
    # each operand is truncated to 2^-53 of its row's maximum, a product's dropped
    # digits are below 2^-59, the eight partial sums and y0's quotient round once each
    unit = 2.0**-51 * npix * np.max(np.abs(r), axis=1, keepdims=True) * np.max(np.abs(P), axis=1)
    err = unit + 9 * EPS * np.abs(r) @ np.abs(P).T
    bound = (err + np.abs(want / want[:, :1]) * err[:, :1]) / np.abs(want[:, :1]) + 2 * EPS * np.abs(want / want[:, :1])
    assert np.all(np.abs(y - want / want[:, :1]) <= bound)


def test_projection_of_non_finite_members(cuda):
    """An infinity or a NaN anywhere in a member gives NaN for it and leaves the others of its tile alone."""
    from my_swampe_gb300.emission import _project

    rng = np.random.default_rng(5)
    P, r = np.abs(rng.standard_normal((20, 300))), np.abs(rng.standard_normal((5, 300)))
    ok = torch.ones(5, dtype=torch.int32, device="cuda")
    clean = _project(torch.tensor(r, device="cuda").reshape(5, 1, 300), ok, torch.tensor(P, device="cuda"))
    r[1, 7], r[3, 299] = np.inf, np.nan
    y = _project(torch.tensor(r, device="cuda").reshape(5, 1, 300), ok, torch.tensor(P, device="cuda"))
    assert torch.isnan(y[[1, 3]]).all() and torch.equal(y[[0, 2, 4]], clean[[0, 2, 4]])
