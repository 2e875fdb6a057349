"""Accuracy of the emission kernels output by output: the projection onto bases
of local support, whose coefficients see only a faint part of the map, against
the FP64 bound of each sum; the digits that the sliced projection keeps; the
Planck intensity relative to its own size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0**-53


def _check(r, P, y):
    """y (B, ncoef) against sum_p P r / (the first coefficient's), each output within
    its own bound: a lane's chain of FMAs is npix / 32 long, or slices drop at most
    npix 2^-59 of the sum of magnitudes, 24 conversions and additions, the quotient."""
    npix = r.shape[1]
    want = r.astype(np.longdouble) @ P.T.astype(np.longdouble)
    gone = np.abs(want[:, 0]) <= 1e-30  # the guard of y0: all NaN
    assert np.all(np.isnan(y[gone]))
    r, want, y = r[~gone], want[~gone], y[~gone]
    err = (npix / 32 + 24) * U * (np.abs(r) @ np.abs(P).T)
    q = want / want[:, :1]
    bound = (err + np.abs(q) * err[:, :1]) / np.abs(want[:, :1]) + 2 * U * np.abs(q)
    assert np.all(np.abs(y - q) <= bound)


def _project(r, P):
    from my_swampe_gb300.emission import _project as project

    ok = torch.ones(r.shape[0], dtype=torch.int32, device="cuda")
    return project(torch.tensor(r, device="cuda").reshape(r.shape[0], 1, -1), ok, torch.tensor(P, device="cuda")).cpu().numpy()


@pytest.mark.parametrize("wavelength", [1.6e-6, 2.2e-6, 3.6e-6, 4.5e-6])
@pytest.mark.parametrize("basis", ["sectors", "night", "patches"])
def test_local_basis_on_a_day_night_map(cuda, wavelength, basis):
    """A planet of 344 K by day and 79 K by night: the first coefficient is the
    antistellar part's, 10^-8 and less of the map's maximum."""
    from my_swampe_gb300.emission import EmissionConfig, _map, build_projector

    J, I, B = 64, 128, 3
    mu, w = np.polynomial.legendre.leggauss(J)
    lam = np.linspace(-np.pi, np.pi, I, endpoint=False)
    day = np.maximum(np.cos(lam), 0.0)[None, :] * np.sqrt(1.0 - mu * mu)[:, None]
    rng = np.random.default_rng(1)
    phi = 1.0e6 * day + 50.0 * rng.standard_normal((B, J, I))
    sector = np.floor(((lam - np.pi + np.pi / 8) % (2 * np.pi)) / (np.pi / 4)).astype(int)
    if basis == "sectors":
        cols = [np.broadcast_to(sector == k, (J, I)) for k in range(8)]
    elif basis == "night":
        cols = [np.broadcast_to(np.cos(lam) < -0.1, (J, I)), np.ones((J, I))]
    else:
        at = [(32, 0), (3, 1), (60, 100), (32, 64)]
        cols = [(np.abs(np.arange(J)[:, None] - j) < 2) & (np.abs(np.arange(I)[None, :] - i) < 2) for j, i in at]
    design = np.stack([np.asarray(c, dtype=np.float64).reshape(-1) for c in cols], 1)
    cfg = EmissionConfig(emission_model="planck", planck_wavelength_m=wavelength, planck_x_clip=700.0)
    wt = torch.tensor(w, device="cuda")
    rhs, ok, _ = _map(torch.tensor(phi, device="cuda"), 3.0e5, cfg, 0, 2, wt)
    P = build_projector(torch.tensor(design, device="cuda"), wt, ridge=0.0).cpu().numpy()
    r = rhs.cpu().numpy().reshape(B, -1)
    assert bool(ok.all())
    _check(r, P, _project(r, P))


@pytest.mark.parametrize("npix", [2, 64, 200, 1000, 8192, 20000])
def test_rows_that_meet_where_both_are_faint(cuda, npix):
    """The largest element of a map where a projector row is faint and the reverse:
    down to and beyond the digits of a common scale, and the ends of FP64's range."""
    rng = np.random.default_rng(npix)
    half = npix // 2
    for lo in (1e-3, 1e-9, 1e-15, 1e-20, 1e-30):
        r = rng.uniform(0.5, 1.0, (18, npix))
        P = rng.uniform(0.5, 1.0, (5, npix))
        r[:, :half] *= lo
        P[:, half:] *= lo
        P[3] = rng.standard_normal(npix)
        P[4, :half] = 0.0
        _check(r, P, _project(r, P))
    for scale in (1e-250, 1e-290, 1e250, 1e290):
        r = rng.uniform(0.5, 1.0, (2, npix)) * scale
        P = rng.uniform(0.5, 1.0, (3, npix)) / scale
        _check(r, P, _project(r, P))


def test_outputs_do_not_depend_on_the_tile_of_members(cuda):
    rng = np.random.default_rng(3)
    r = rng.uniform(0.5, 1.0, (19, 4000)) * 10.0 ** rng.uniform(-25, 0, (19, 4000))
    P = rng.uniform(0.5, 1.0, (70, 4000)) * 10.0 ** rng.uniform(-25, 0, (70, 4000))
    P[::3] *= rng.uniform(size=(24, 4000)) < 0.01  # few pixels each
    y = _project(r, P)
    for b in (0, 7, 15, 16, 18):
        assert np.array_equal(_project(r[b:b + 1], P)[0], y[b])


@pytest.mark.parametrize("B,ncoef", [(144, 121), (145, 129), (160, 121)])
def test_outputs_do_not_depend_on_the_tile_of_coefficients(cuda, B, ncoef):
    """Members of launches on both sides of the rule for coefficients per CTA, alone."""
    rng = np.random.default_rng(B)
    r, P = rng.uniform(0.5, 1.0, (B, 700)), rng.standard_normal((ncoef, 700))
    P[0] = np.abs(P[0])
    y = _project(r, P)
    for b in (0, 31, B - 1):
        assert np.array_equal(_project(r[b:b + 1], P)[0], y[b])
    assert np.array_equal(_project(r, P[:40]), y[:, :40])


@pytest.mark.parametrize("npix", [64, 128, 512])
def test_every_digit_counts(cuda, npix):
    """Pairs of pixels whose products cancel to 2^-30: the rounding of the result is
    then far below what a digit less would lose.  Operands below 1: each product is off
    by the dropped digit products (7 of 2^14 at 2^-76, and smaller ones) and the operands'
    own 2^-62, below 2^-59 in all."""
    rng = np.random.default_rng(npix)
    r = rng.uniform(0.5, 1.0, (32, npix))
    P = rng.uniform(-1.0, 1.0, (60, npix))
    d = 2.0**-30 * rng.uniform(-1.0, 1.0, (32, npix // 2))
    r[:, 1::2] = r[:, 0::2] + d
    r = np.minimum(r, 1.0 - 2.0**-53)
    P[:, 1::2] = -P[:, 0::2]
    P[0] = 0.0
    P[0, 0] = 1.0  # y0 = r[0], exactly
    y = _project(r, P)
    rl, Pl = r.astype(np.longdouble), P.astype(np.longdouble)
    pair = (rl[:, None, 0::2] - rl[:, None, 1::2]) * Pl[None, :, 0::2]
    pair[:, 0] = 0.0
    want = pair.sum(axis=2) / rl[:, :1]
    bound = (npix * 2.0**-59 + 24 * U * np.abs(pair).sum(axis=2)) / r[:, :1]
    assert np.all(np.abs(y - want)[:, 1:] <= bound[:, 1:].astype(np.float64))


@pytest.mark.parametrize("x_clip", [80.0, 700.0, 1000.0, 0.5, -1.0, -800.0])
def test_planck_intensity_relative_accuracy(cuda, x_clip):
    """1 / (expm1(x) + tiny) at x = h c / (lambda kB T) from 10^-6 to past 709, where
    expm1 overflows.  x carries two roundings, each kappa = x e^x / (e^x - 1) times in
    the intensity; its expm1, sum and reciprocal four ulp."""
    from my_swampe_gb300.emission import EmissionConfig, temperature_to_intensity

    ld = np.longdouble
    hck = ld("6.62607015e-34") * ld("299792458.0") / ld("1.380649e-23")
    x = np.concatenate([10.0 ** np.linspace(-6, np.log10(709.0), 4096), np.linspace(0.002, 0.03, 4096),
                        np.linspace(695.0, 1100.0, 4096)])
    T = (hck / (ld(4.5e-6) * x)).astype(np.float64)
    cfg = EmissionConfig(emission_model="planck", planck_x_clip=x_clip, Tmin_K=1e-3)
    got = temperature_to_intensity(torch.tensor(T.reshape(96, 128), device="cuda"), cfg).cpu().numpy().reshape(-1)
    xe = np.minimum(np.maximum(hck / (ld(4.5e-6) * T.astype(ld)), 0), ld(x_clip))
    with np.errstate(over="ignore"):
        want = 1 / (np.expm1(xe) + ld(1e-30))
        kappa = np.abs(xe / (1 - np.exp(-xe)))
    # beyond 709.7 expm1 overflows in FP64 and the intensity, below 10^-307, is lost
    small = xe > 709.0
    assert np.all(np.abs(got / want - 1)[~small] <= ((kappa + 4) * 2 * U)[~small])
    assert np.all(np.abs(got - want)[small] <= 2e-308)
