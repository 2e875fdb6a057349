"""The FP64 longitude transform on integer slices (csrc/grid_f64.cu) at the
longitude I/2, the alternating sum of a row's coefficients, in exact arithmetic:
it takes part of every digit, as the other longitudes do."""
from fractions import Fraction

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [42, 63, 106])
def test_alternating_longitude(cuda, M):
    from my_swampe_gb300 import _lib
    from my_swampe_gb300.engine import Engine, RunFlagsC

    eng = Engine([(M, 1)], "fp64")
    gd = eng.groups[0]
    J, I = gd["J"], gd["I"]
    rng = np.random.default_rng(M)
    # rows of three kinds: flat, steep, and with a sum that cancels to its last digits
    Y = rng.uniform(-1.0, 1.0, (M + 1, J)) + 1j * rng.uniform(-1.0, 1.0, (M + 1, J))
    Y[:, 1::3] *= 10.0 ** (-0.3 * np.arange(M + 1))[:, None]
    w = np.where(np.arange(M + 1) == 0, 1, 2) * (-1) ** np.arange(M + 1)
    for j in range(2, J, 3):
        rest = sum(Fraction(float(Y[m, j].real)) * int(w[m]) for m in range(1, M + 1))
        Y[1:, j] *= 0.5 / max(1.0, abs(float(rest)))
        Y[0, j] = -float(sum(Fraction(float(Y[m, j].real)) * int(w[m]) for m in range(1, M + 1)))
    four = gd["fourier"]
    four.zero_()
    four[_lib.F_PHI, :, 0] = torch.tensor(Y, device="cuda")
    gd["member"].zero_()
    got = eng.output_physical(RunFlagsC())[0][2, 0, :, I // 2].cpu().numpy()
    for j in range(J):
        want = sum(Fraction(float(Y[m, j].real)) * int(w[m]) for m in range(M + 1))
        top = max(max(abs(Y[:, j].real)), max(abs(Y[:, j].imag)))
        # every coefficient within half of 2^-62 of twice the row's maximum (its scale is a
        # power of two), with weights 1 and 2; the result rounded once
        bound = (2 * M + 1) * 2.0**-62 * top + 2.0**-53 * abs(float(want))
        assert abs(float(Fraction(float(got[j])) - want)) <= bound, (j, float(want), float(got[j]))
