"""The z/y plane kernels with one, two and four blocks per box row (chosen by the number of rows and
their size): the long-range field against the z-pass + cuFFT planes on the same lattice, at sizes on
both sides of every line of the rule.  Both transforms are FP32: each is within about 3e-7 of the
field's largest component (1.3e-7 rms measured for cuFFT), so 2e-6 bounds their difference."""
import numpy as np
import pytest

import asd_b200 as A
import asd_lattice as LT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(110, 4, 4), (110, 64, 9), (110, 64, 17), (106, 33, 33),      # more than 320 rows
                               (64, 16, 32), (64, 17, 33), (60, 65, 49), (50, 128, 65),       # 149 to 320
                               (9, 16, 31), (9, 17, 33), (10, 100, 100)])                    # fewer than the SMs
def test_rows_shared_by_clusters(gpu, L):
    s = LT.sc_ferromagnet(L, pbc=(0, 0, 0), dipole=True, J=1e-30)
    S0 = LT.random_spins(s.nspins, 3)
    f = []
    for flag in (0, A.FLAG_CUFFT_PLANES):
        with A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED | flag), s) as h:
            assert ("plane kernels" in h.tuning()) == (flag == 0), h.tuning()
            h.set_spins(S0)
            h.step(2)
            f.append(h.get_field())
    assert np.abs(f[0] - f[1]).max() <= 2e-6 * np.abs(f[1]).max()
