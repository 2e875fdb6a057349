"""FP32 kernels whose work split follows the number of members (rows per CTA of
k_grid, register tiles and units of k_spectral): a member's results are the
same bits whatever the split."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(M, B, members):
    """Fast engine of the given members of a seeded ensemble of B."""
    from my_swampe_gb300 import workloads
    from my_swampe_gb300.engine import Engine

    wl = workloads.forced_ensemble(Engine([(M, B)], "fast"), seed=3, dt=840.0 / M)
    eng = Engine([(M, len(members))], "fast")
    workloads.apply_params(eng, 0, {k: v[members] if torch.is_tensor(v) else v for k, v in wl["params"].items()})
    return eng, wl["ics"][:, members].contiguous()


@pytest.mark.parametrize("M,B", [(42, 7), (42, 40), (63, 5), (63, 11), (106, 3), (106, 5)])
def test_grid_rows_follow_the_members(cuda, M, B):
    from my_swampe_gb300.adjoint import Integration
    from my_swampe_gb300.engine import RunFlagsC

    def run(members):
        eng, ics = _engine(M, B, members)
        integ = Integration(eng, RunFlagsC(), 2, 3)
        out = integ.run_forward([ics])[0]
        dic, grad = integ.run_backward([torch.sin(out)])
        return out, dic[0], grad[0].clone()

    got = run(list(range(B)))
    for b in (0, B - 1):
        want = run([b])
        assert torch.equal(got[0][:, b], want[0][:, 0]) and torch.equal(got[1][:, b], want[1][:, 0])
        # gradients: partial sums per CTA in FP32, then FP64 atomics
        assert torch.allclose(got[2][:, b], want[2][:, 0], rtol=1e-5, atol=1e-6 * float(got[2].abs().max()))


@pytest.mark.parametrize("M,B", [(42, 9), (63, 3), (106, 3)])
@pytest.mark.parametrize("scheme", [1, 2, "tangent"])
def test_simt_legendre_tiles(cuda, M, B, scheme):
    from my_swampe_gb300 import _lib
    from my_swampe_gb300.adjoint import Integration
    from my_swampe_gb300.engine import RunFlagsC

    res = []
    for tile in (1, 2, 4, 8):
        eng, ics = _engine(M, B, list(range(B)))
        if eng.lib.swp_plan_set_tile(eng._plan, 0, tile) != _lib.SWP_OK:
            continue  # does not fit in shared memory
        if scheme == "tangent":
            rows = torch.ones((_lib.NTANGENT, B), dtype=torch.float64, device="cuda")
            integ = Integration(eng, RunFlagsC(), 2, 3)
            res.append(integ.run_tangent([ics], [torch.ones_like(ics)], [rows])[0])
        else:
            integ = Integration(eng, RunFlagsC(scheme=scheme), 2, 3)
            out = integ.run_forward([ics])[0]
            res.append(torch.stack([out, integ.run_backward([torch.sin(out)])[0][0]]))
    assert len(res) >= 3
    for r in res[1:]:
        assert torch.equal(r, res[0])
