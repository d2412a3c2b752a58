"""Small lattices run several steps in one cooperative launch, a grid barrier between the stages:
bit-identical to one launch per stage (ASD_FLAG_SERIAL_LAUNCH), at the sizes where its block size
changes and at the largest lattice that takes it, through whole chunks, remainders and single
steps, with each integrator, several replicas, a site-field pulse, the det field and rows of fewer
neighbours than the gather loads at a time.  Which of the two forms ran is read from the tuning line
and from the launch count of a whole chunk."""
import numpy as np
import pytest

import asd_b200 as A
import asd_lattice as LT

pytestmark = pytest.mark.gpu
SM = 148


def run(systems, flags, integ=A.HEUN, chunks=(32, 5, 1, 34), pulse=False):
    n = sum(s.nspins for s in systems)
    with A.Handle(A.RunParams(precision=A.FP32, flags=flags, integrator=integ, seed=6, applied=(0.1, 0.0, 0.2)), systems) as h:
        h.set_spins(LT.random_spins(n, 2))
        if pulse:
            h.set_site_field_pulse(0.1, 2e-15, 1e-15)
        for k in chunks:
            h.step(k)
            h.set_applied((0.05 * k, 0.0, -0.1))
        h.sync()
        out = h.get_spins(), h.get_det_field()
        several = "several per launch" in h.tuning()
        # a whole chunk of 32 steps: the launch, the field and step scalars and the counter; or every stage
        assert (h.time_steps(32)[1] < 10) == several
        return *out, several


def same(systems, base=A.FLAG_COMPENSATED, several=True, **kw):
    a = run(systems, base, **kw)
    b = run(systems, base | A.FLAG_SERIAL_LAUNCH, **kw)
    assert a[2] == several and not b[2]
    assert np.array_equal(a[0], b[0]), np.abs(a[0] - b[0]).max()
    assert np.array_equal(a[1], b[1])


# spins: one block; blocks of 64, 128 and 256; the largest that is resident and the first that is not
@pytest.mark.parametrize("L", [(7, 6, 5), (SM, 8, 8), (SM, 8, 9), (SM, 16, 8), (SM, 16, 9), (SM, 32, 16), (SM, 27, 19)])
def test_block_sizes(gpu, L):
    same([LT.sc_ferromagnet(L, T=100.0)], several=np.prod(L) <= 75776)


# full tensors: 37 x 16 x 16 cells of two are the most that are resident
@pytest.mark.parametrize("L", [(37, 16, 16), (43, 13, 17)])
def test_full_tensors_at_the_limit(gpu, L):
    same([LT.bct2_antiferromagnet(L, T=100.0)], several=2 * np.prod(L) <= 18944)


# 2, 4, 3 (padded to 4) and 5 (to 6) entries per row; 18 rows are too few for their six patterns, which
# may hold no more than a quarter of the entries
@pytest.mark.parametrize("L, pbc, several", [((700, 1, 1), (0, 0, 0), True), ((33, 21, 1), (0, 0, 0), True),
                                             ((9, 1, 2), (1, 0, 0), False), ((90, 1, 2), (1, 0, 0), True),
                                             ((12, 11, 2), (1, 1, 0), True)])
def test_few_neighbours(gpu, L, pbc, several):
    same([LT.sc_ferromagnet(L, pbc=pbc, T=100.0)], several=several)


@pytest.mark.parametrize("integ", [A.HEUN, A.RK4, A.RK5])
@pytest.mark.parametrize("base", [A.FLAG_COMPENSATED, 0])
def test_integrators_full_tensors(gpu, integ, base):
    same([LT.bct2_antiferromagnet((9, 7, 11), T=200.0)], base=base, integ=integ)


def test_replicas_film_and_pulse(gpu):
    same([LT.sc_ferromagnet(e, T=60.0 * r, stream=r) for r, e in enumerate((8, 13, 9))])
    same([LT.film_dia(33, 21, 3, dipole=False)], integ=A.RK4, pulse=True)


@pytest.mark.parametrize("s", [LT.sc_ferromagnet((7, 6, 5)), LT.sc_ferromagnet((16, 16, 8), pbc=(0, 0, 0)),
                               LT.bct2_antiferromagnet((6, 7, 6))], ids=["sc7x6x5", "sc_open_dia", "bct2"])
def test_autotuner_keeps_several_steps(gpu, s):
    """One stage's launch time does not decide against the several-steps launch (launch noise did, on
    two of three handles of the smallest lattice)."""
    for _ in range(4):
        with A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED | A.FLAG_AUTOTUNE), s) as h:
            assert "staging=pattern; " in h.tuning() and "several per launch" in h.tuning(), h.tuning()


def test_two_handles_at_once(gpu):
    """Two handles' streams hold such launches at the same time: each gets its own results."""
    s = LT.sc_ferromagnet((40, 40, 40), T=50.0)
    want = [run([s], A.FLAG_COMPENSATED | A.FLAG_SERIAL_LAUNCH, chunks=(320,))[0]] * 2
    hs = [A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED, seed=6, applied=(0.1, 0.0, 0.2)), s) for _ in range(2)]
    for h in hs:
        h.set_spins(LT.random_spins(s.nspins, 2))
    for _ in range(10):
        for h in hs:
            h.step(32)
    for h, w in zip(hs, want):
        h.sync()
        assert np.array_equal(h.get_spins(), w)
        assert "several per launch" in h.tuning()
        h.close()
