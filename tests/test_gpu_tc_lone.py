"""The tensor-core Legendre kernels' one-CTA-per-SM form (few members, M = 42):
states and initial-field gradients of the same members in an ensemble that runs
the two-CTA form, bit for bit.  16 and 24 members are the last counts of the
forward and the adjoint form; 7 and 17 leave a tile ragged."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("raw", [False, True])
def test_few_members_equal_those_of_a_larger_ensemble(cuda, raw):
    from my_swampe_gb300 import workloads
    from my_swampe_gb300.adjoint import Integration
    from my_swampe_gb300.engine import Engine, RunFlagsC

    wl = workloads.forced_ensemble(Engine([(42, 41)], "fast"), seed=5, dt=20.0)

    def run(B):
        eng = Engine([(42, B)], "fast")
        workloads.apply_params(eng, 0, {k: v[:B] if torch.is_tensor(v) else v for k, v in wl["params"].items()})
        ics, flags = [wl["ics"][:, :B].contiguous()], RunFlagsC(raw_filter=raw)
        if raw:
            eng.init_state(ics, flags)
            eng.forward(flags, 2, 8)
            return eng.groups[0]["fourier"].clone(), None
        integ = Integration(eng, flags, 2, 8)
        out = integ.run_forward(ics)[0]
        four = eng.groups[0]["fourier"].clone()
        return four, integ.run_backward([torch.sin(out)])[0][0].clone()

    four, dic = run(41)
    assert torch.isfinite(torch.view_as_real(four)).all()
    for B in (1, 7, 16, 17, 24):
        f, d = run(B)
        assert torch.equal(torch.view_as_real(f), torch.view_as_real(four[:, :, :B])), B
        if not raw:
            assert torch.equal(d, dic[:, :B]), B
