"""The FP64 kernels on integer slices (csrc/slices.cuh, spectral_f64.cu): their
sums are exact and scaled per row, so no result may depend on how members are
tiled.  Members of an ensemble are compared bit for bit with the same members
run alone, at ensemble sizes around the tile rules and with remainders."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(M, B, sel=None, nan=None, total=None):
    """FP64 engine of B members; with sel, member sel of the ensemble of `total` members alone."""
    from my_swampe_gb300 import workloads
    from my_swampe_gb300.engine import Engine

    big = Engine([(M, total or B)], "fp64")
    wl = workloads.forced_ensemble(big, seed=7, dt=840.0 / M)
    ics, par = wl["ics"].clone(), wl["params"]
    if nan is not None:
        ics[2, nan, 3, 5] = float("nan")
    if sel is None:
        workloads.apply_params(big, 0, par)
        return big, ics
    one = Engine([(M, 1)], "fp64")
    workloads.apply_params(one, 0, {k: v[sel:sel + 1] if torch.is_tensor(v) else v for k, v in par.items()})
    return one, ics[:, sel:sel + 1].contiguous()


def _run(eng, ics, scheme, adjoint):
    from my_swampe_gb300.adjoint import Integration
    from my_swampe_gb300.engine import RunFlagsC

    flags = RunFlagsC(scheme=scheme)
    if not adjoint:
        eng.init_state([ics], flags)
        eng.forward(flags, 2, 3)
        return [eng.groups[0]["fourier"].clone()]
    integ = Integration(eng, flags, 2, 3)
    out = integ.run_forward([ics])[0]
    dic, grad = integ.run_backward([torch.sin(out)])
    return [out, dic[0], grad[0].clone()]


@pytest.mark.parametrize("M,B", [(42, 3), (42, 9), (42, 17), (42, 33), (63, 2), (63, 11), (106, 2)])
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("adjoint", [False, True])
def test_members_do_not_depend_on_the_tile(cuda, M, B, scheme, adjoint):
    eng, ics = _engine(M, B)
    got = _run(eng, ics, scheme, adjoint)
    for b in (0, B - 1):
        one, ic = _engine(M, B, sel=b)
        want = _run(one, ic, scheme, adjoint)
        for k, (x, y) in enumerate(zip(got, want)):
            if k == 2:  # gradients: sums over latitudes and m by atomics, in no fixed order
                assert torch.allclose(x[:, b], y[:, 0], rtol=1e-12, atol=1e-12 * float(x.abs().max()))
            else:
                dim = 2 if not adjoint else 1
                assert torch.equal(x.select(dim, b), y.select(dim, 0)), (b, k)


def test_non_finite_member_stays_alone(cuda):
    eng, ics = _engine(42, 5, nan=3)
    got = _run(eng, ics, 0, False)[0]
    clean, ics = _engine(42, 5)
    want = _run(clean, ics, 0, False)[0]
    assert torch.isnan(torch.view_as_real(got[5, :, 3])).all()  # Phi at every m and latitude
    keep = [0, 1, 2, 4]
    assert torch.equal(got[:, :, keep], want[:, :, keep])
