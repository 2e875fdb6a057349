"""Device memory of a plan's packed matrices: none without steps, one set for the
groups of a truncation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _used(groups, **kw):
    """Bytes that an engine holds beyond its own tensors."""
    from my_swampe_gb300.engine import Engine

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, held = torch.cuda.mem_get_info()[0], torch.cuda.memory_reserved()
    eng = Engine(groups, "fp64", **kw)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0] - (torch.cuda.memory_reserved() - held)
    return eng, used


def test_packed_matrices(cuda):
    _used([(106, 1)])  # modules and context
    geo, none = _used([(106, 1)], steps=False)
    one, single = _used([(106, 1)])
    two, double = _used([(106, 1), (106, 2)], concurrent=True)
    # the sliced bases are 137 MB; geometry and coefficients of a group about 30 MB
    assert none < 60e6 and single - none > 100e6 and double - single < 60e6
    assert torch.equal(geo.geometry()["Pmn"], one.geometry()["Pmn"])
    ics = torch.rand((2, 1, 160, 320), dtype=torch.float64, device="cuda")
    assert torch.equal(geo.diagnose_winds([ics])[0], one.diagnose_winds([ics])[0])


def test_a_plan_without_steps_refuses_them(cuda):
    from my_swampe_gb300.engine import Engine, RunFlagsC

    with pytest.raises(ValueError):
        Engine([(42, 1)], "fast", steps=False)
    eng = Engine([(42, 1)], "fp64", steps=False)
    flags = RunFlagsC()
    for call in (lambda: eng.init_state([torch.zeros((5, 1, 64, 128), device="cuda")], flags),
                 lambda: eng.forward(flags, 2, 1), lambda: eng.output_physical(flags)):
        with pytest.raises(RuntimeError):
            call()
    torch.cuda.synchronize()


def test_groups_that_share_them(cuda):
    """A plan of equal and unequal truncations: each group's results are its own engine's."""
    from my_swampe_gb300.engine import Engine, RunFlagsC
    from my_swampe_gb300 import workloads

    spec = [(42, 2), (63, 1), (42, 3)]
    eng, flags, ics = Engine(spec, "fp64"), RunFlagsC(), []
    for g in range(3):
        wl = workloads.forced_ensemble(eng, g=g, seed=g)
        workloads.apply_params(eng, g, wl["params"])
        ics.append(wl["ics"])
    eng.init_state(ics, flags)
    eng.forward(flags, 2, 3)
    for g, (M, B) in enumerate(spec):
        one = Engine([(M, B)], "fp64")
        workloads.apply_params(one, 0, workloads.forced_ensemble(one, seed=g)["params"])
        one.init_state([ics[g]], flags)
        one.forward(flags, 2, 3)
        assert torch.equal(one.groups[0]["fourier"], eng.groups[g]["fourier"])
        del one
    del eng
    torch.cuda.synchronize()
