"""The stage kernels' row patterns (each row a 2-byte number into the distinct sequences of
(column - row, tensor)): bit-identical to the SELL gather of the same entries at ragged sizes,
with boundary rows of every length, uneven replicas, full tensors and DIA input; a matrix whose
rows do not repeat keeps its words.  Single steps run the stage kernels, which whole chunks of these
small lattices in FP32 do not (tests/test_resident_steps.py); the kernels that only larger lattices
take are run at the sizes where each begins."""
import re

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


def run(systems, prec, integ, shape=None, steps=40, single=False):
    flags = A.FLAG_COMPENSATED if prec == A.FP32 else 0
    n = sum(s.nspins for s in systems)
    with A.Handle(A.RunParams(precision=prec, flags=flags, integrator=integ, seed=4), systems) as h:
        if shape:
            h.set_launch_shape(*shape)
        h.set_spins(LT.random_spins(n, 5))
        for k in [1] * steps if single else [steps]:
            h.step(k)
        return h.get_spins(), h.tuning()


@pytest.mark.parametrize("prec", [A.FP32, A.FP64_FUSED])
@pytest.mark.parametrize("integ", [A.HEUN, A.RK5])
@pytest.mark.parametrize("case", CASES)
def test_patterns_bit_identical_to_sell(gpu, case, integ, prec):
    s = CASES[case]()
    got, tune = run(s, prec, integ)
    assert "staging=pattern" in tune, tune
    assert np.array_equal(got, run(s, prec, integ, single=True)[0])
    for shape in ((256, 1), (64, 0)):
        want, tune = run(s, prec, integ, shape)
        assert "pattern" not in tune, tune
        assert np.array_equal(got, want), shape


# FP32, one wave of 4 blocks of 256 per SM being 151,552 rows: the last size of the early-loading
# kernels and the first past it, diagonal tensors of 6 neighbours (48 registers past one wave) and of
# 18 (64 up to two waves, then 48), and full tensors (64)
@pytest.mark.parametrize("integ", [A.HEUN, A.RK4])
@pytest.mark.parametrize("make", [lambda: LT.sc_ferromagnet((148, 32, 32), T=100.0),
                                  lambda: LT.sc_ferromagnet((148, 32, 33), T=100.0),
                                  lambda: LT.film_dia(148, 74, 14, dipole=False),
                                  lambda: LT.film_dia(148, 74, 28, dipole=False),
                                  lambda: LT.bct2_antiferromagnet((37, 64, 33), T=100.0)],
                         ids=["one_wave", "diag6", "diag18_two_waves", "diag18", "full"])
def test_large_lattice_kernels_bit_identical_to_sell(gpu, make, integ):
    s = make()
    got, tune = run([s], A.FP32, integ, steps=6)
    assert "staging=pattern" in tune and "several" not in tune, tune
    assert np.array_equal(got, run([s], A.FP32, integ, (256, 1), steps=6)[0])


def alloy(L, vecs, seed, nsp=2):
    """Full pair tensors that go with the two sites' species: 2 to the power of (neighbours + 1) patterns."""
    n = L[0] * L[1] * L[2]
    J = np.array([1.0, 0.03, -0.03, -0.03, 1.0, 0.03, 0.03, -0.03, 1.0]) * 1e-21
    xadj, adj, val = LT.build_csr(L, (1, 1, 1), [LT.MU_SC], [0] * len(vecs), [0] * len(vecs), vecs, [J] * len(vecs))
    sp = np.random.default_rng(seed).integers(0, nsp, n)
    rows = np.repeat(np.arange(n), np.diff(xadj))
    val = np.ascontiguousarray(val.reshape(-1, 9) * (1.0 - 0.4 * sp[rows] - 0.3 * sp[adj])[:, None])
    return A.SpinSystem(nspins=n, materials=[A.MaterialSpec(mu=LT.MU_SC, lam=0.1)], full=True, temperature=100.0,
                        exch=A.EXCH_CSR, xadj=xadj, adjncy=adj, csr_val=val)


def test_alloy_takes_the_faster_of_patterns_and_words(gpu):
    """Many patterns: FP32 times both and keeps the faster; the results are the same.  FP64, and an alloy
    that runs several steps per launch, go by patterns untimed."""
    s = alloy((48, 48, 36), LT.SC_NNN, 3)
    got, tune = run([s], A.FP32, A.HEUN)
    m = re.search(r"staging=(\w+) \(timed: pattern ([\d.]+), words ([\d.]+)", tune)
    assert m, tune
    assert (m[1] == "words") == (float(m[3]) < float(m[2])) or m[2] == m[3], tune
    want = run([s], A.FP32, A.HEUN, (64, 0))[0]
    assert np.array_equal(got, want)
    with A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED), s) as h:    # timing leaves no trace
        assert h.t == 0 and not h.get_det_field().any()
        assert np.array_equal(h.get_spins(), np.tile([0.0, 0.0, 1.0], (s.nspins, 1)))
        f = h.get_field()
    s.nr, s.mesh = LT.dipole_nr((48, 48, 36))
    s.lr, s.mesh_xyz = A.LR_DIPOLE, LT.sc_mesh_xyz((48, 48, 36))
    with A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED), s) as h:    # nor in the dipole field
        assert "timed:" in h.tuning(), h.tuning()
        assert np.array_equal(h.get_field(), f)
    s.lr = A.LR_NONE
    assert "staging=pattern" in run([s], A.FP64_FUSED, A.HEUN)[1]
    assert "staging=pattern (default)" in run([alloy((25, 25, 25), LT.SC_NN, 3)], A.FP32, A.HEUN)[1]


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
