"""A member whose fields hold a NaN or an infinity is NaN in every Fourier
coefficient after FP64 steps, also where a wavenumber's basis underflows to zero
(M = 106, the highest m): zero times a NaN is a NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [42, 63, 106])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("scheme", [0, 2])
def test_whole_member(cuda, M, bad, scheme):
    from my_swampe_gb300 import _lib, workloads
    from my_swampe_gb300.engine import Engine, RunFlagsC

    eng, flags = Engine([(M, 2)], "fp64"), RunFlagsC(scheme=scheme)
    wl = workloads.forced_ensemble(eng, seed=7, dt=840.0 / M)
    workloads.apply_params(eng, 0, wl["params"])
    ics = wl["ics"].clone()
    ics[2, 1, 3, 5] = bad
    eng.init_state([ics], flags)
    eng.forward(flags, 2, 3)
    four = torch.view_as_real(eng.groups[0]["fourier"])
    for k in (_lib.F_ETA, _lib.F_DELTA, _lib.F_PHI):
        assert torch.isnan(four[k, :, 1]).all() and torch.isfinite(four[k, :, 0]).all()
