"""Small lattices run several steps in one cooperative launch, a grid barrier between the stages:
bit-identical to one launch per stage (ASD_FLAG_SERIAL_LAUNCH), at the sizes where its block size
changes and at the largest lattice that takes it, through whole chunks, remainders and single
steps, with each integrator, several replicas, a site-field pulse and the det field."""
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
        return h.get_spins(), h.get_det_field()


def same(systems, base=A.FLAG_COMPENSATED, **kw):
    a = run(systems, base, **kw)
    b = run(systems, base | A.FLAG_SERIAL_LAUNCH, **kw)
    assert np.array_equal(a[0], b[0]), np.abs(a[0] - b[0]).max()
    assert np.array_equal(a[1], b[1])


# spins: one block; blocks of 64, 128 and 256; the largest that is resident and the first that is not
@pytest.mark.parametrize("L", [(7, 6, 5), (SM, 8, 8), (SM, 8, 9), (SM, 16, 8), (SM, 16, 9), (SM, 32, 16), (SM, 27, 19)])
def test_block_sizes(gpu, L):
    same([LT.sc_ferromagnet(L, T=100.0)])


@pytest.mark.parametrize("integ", [A.HEUN, A.RK4, A.RK5])
@pytest.mark.parametrize("base", [A.FLAG_COMPENSATED, 0])
def test_integrators_full_tensors(gpu, integ, base):
    same([LT.bct2_antiferromagnet((9, 7, 11), T=200.0)], base=base, integ=integ)


def test_replicas_film_and_pulse(gpu):
    same([LT.sc_ferromagnet(e, T=60.0 * r, stream=r) for r, e in enumerate((8, 13, 9))])
    same([LT.film_dia(33, 21, 3, dipole=False)], integ=A.RK4, pulse=True)


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
        h.close()
