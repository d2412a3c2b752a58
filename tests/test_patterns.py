"""The stage kernels' row patterns (each row a 2-byte number into the distinct sequences of
(column - row, tensor)): bit-identical to the SELL gather of the same entries at ragged sizes,
with boundary rows of every length, uneven replicas, full tensors and DIA input; a matrix whose
rows do not repeat keeps its words."""
import numpy as np
import pytest

import asd_b200 as A
import asd_lattice as LT

pytestmark = pytest.mark.gpu

CASES = {
    "sc_periodic_one_past_a_block": lambda: [LT.sc_ferromagnet((257, 3, 3), T=100.0)],
    "sc_open_ragged": lambda: [LT.sc_ferromagnet((9, 7, 11), pbc=(0, 0, 0), T=100.0)],
    "sc_mixed_boundaries": lambda: [LT.sc_ferromagnet((5, 33, 8), pbc=(1, 0, 1))],
    "uneven_replicas": lambda: [LT.sc_ferromagnet(e, T=50.0 * r, stream=r) for r, e in enumerate((5, 16, 7, 11))],
    "bct2_full_csr": lambda: [LT.bct2_antiferromagnet((7, 6, 9), T=300.0)],
    "bct2_full_dia": lambda: [LT.bct2_antiferromagnet((6, 7, 5), layout="dia", T=300.0)],
    "film_dia": lambda: [LT.film_dia(17, 14, 3, dipole=False)],
}


def run(systems, prec, integ, shape=None):
    flags = A.FLAG_COMPENSATED if prec == A.FP32 else 0
    n = sum(s.nspins for s in systems)
    with A.Handle(A.RunParams(precision=prec, flags=flags, integrator=integ, seed=4), systems) as h:
        if shape:
            h.set_launch_shape(*shape)
        h.set_spins(LT.random_spins(n, 5))
        h.step(40)
        return h.get_spins(), h.tuning()


@pytest.mark.parametrize("prec", [A.FP32, A.FP64_FUSED])
@pytest.mark.parametrize("integ", [A.HEUN, A.RK5])
@pytest.mark.parametrize("case", CASES)
def test_patterns_bit_identical_to_sell(gpu, case, integ, prec):
    s = CASES[case]()
    got, tune = run(s, prec, integ)
    assert "staging=pattern" in tune, tune
    for shape in ((256, 1), (64, 0)):
        want, tune = run(s, prec, integ, shape)
        assert "pattern" not in tune, tune
        assert np.array_equal(got, want), shape


def test_rows_that_do_not_repeat_keep_their_words(gpu):
    n = 600
    rng = np.random.default_rng(1)
    adj = np.concatenate([rng.choice(n, 5, replace=False) for _ in range(n)]).astype(np.uint32)
    val = np.tile(np.diag([5.0, 5.0, 5.0]).reshape(9), (5 * n, 1))
    s = A.SpinSystem(nspins=n, materials=[A.MaterialSpec()], exch=A.EXCH_CSR, csr_val=val, adjncy=adj,
                     xadj=np.arange(0, 5 * n + 1, 5, dtype=np.uint32))
    got, tune = run([s], A.FP32, A.HEUN)
    assert "staging=words" in tune, tune
    assert np.array_equal(got, run([s], A.FP32, A.HEUN, (64, 0))[0])
