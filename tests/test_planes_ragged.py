"""Long-range field on meshes whose axes are not powers of two: the library moves N_r to the
shortest mesh of the plane kernels' lengths (powers of two and 3 x powers of two) that holds twice
the box.  Against the FP64 direct-sum oracle on the caller's mesh; each
new length is reached at an edge of its range.  Tolerances as in the power-of-two tests: FP32
1e-5, fused FP64 with the FP32 transform 1e-8."""
import numpy as np
import pytest

import asd_b200 as A
import asd_lattice as LT
from helpers import maxdiff
from oracle import oracle as O

pytestmark = pytest.mark.gpu
PLANES = "long-range: plane kernels"


FP32 = (A.FP32, A.FLAG_COMPENSATED, 1e-5)
FUSED64 = (A.FP64_FUSED, 0, 1e-8)


def check(s, steps, forms=(FP32, FUSED64), path=PLANES):
    S0 = LT.random_spins(s.nspins, 0)
    o = O.Oracle(s)
    o.set_spins(S0)
    o.step(steps)
    for prec, flags, tol in forms:
        with A.Handle(A.RunParams(precision=prec, flags=flags), s) as h:
            assert path in h.tuning(), h.tuning()
            h.set_spins(S0)
            h.step(steps)
            g = h.get_spins()
        assert maxdiff(g, o.spins()) <= tol, (prec, maxdiff(g, o.spins()))


# x, y, z lengths the box leads to in the comments
@pytest.mark.parametrize("L", [(9, 11, 1),       # 24, 32, 8 (caller's mesh z: 2)
                               (12, 20, 3),      # 24, 48, 8
                               (20, 3, 23),      # 48, 8, 48
                               (2, 37, 33),      # 4, 96, 96
                               (40, 5, 17),      # 96, 16, 48
                               (67, 3, 5),       # 192, 8, 16
                               (1, 66, 70),      # 4, 192, 192: one row, clusters of 4
                               (100, 33, 1),     # 256, 96, 8: 300 rows of one block
                               (87, 9, 3)])      # 192, 32, 8
def test_ragged_dipole_matches_oracle(gpu, L):
    check(LT.sc_ferromagnet(L, pbc=(0, 0, 0), dipole=True), 10)


@pytest.mark.parametrize("L, path", [(125, "cuFFT"), (97, PLANES), (96, PLANES), (128, "cuFFT")])
def test_chain(gpu, L, path):
    """A chain along x stays on cuFFT where its mesh length has small factors and would go to 256."""
    check(LT.sc_ferromagnet((L, 1, 1), pbc=(0, 0, 0), dipole=True), 20, path=path)


def test_ragged_box_away_from_origin(gpu):
    s = LT.sc_ferromagnet((5, 6, 3), pbc=(0, 0, 0), dipole=True)
    s.nr, s.mesh = LT.dipole_nr((9, 7, 5))
    s.mesh_xyz = (LT.sc_mesh_xyz((5, 6, 3)) + np.array((11, 3, 6), dtype=np.uint32)).astype(np.uint32)
    check(s, 20)


def test_ragged_general_interaction_matrix(gpu):
    """Neither symmetric nor even: 9 complex N_k components on the new mesh."""
    s = LT.sc_ferromagnet((5, 9, 7), pbc=(0, 0, 0), dipole=True)
    rng = np.random.default_rng(7)
    s.nr = s.nr + rng.uniform(-0.05, 0.05, s.nr.shape) * np.abs(s.nr).max()
    check(s, 20)


def test_ragged_fft_exchange_mode(gpu):
    """The whole field from N_k (FP32 form, as for the power-of-two meshes: the fused FP64 form's
    1e-8 is the dipole's, a thousandth of the field)."""
    check(LT.sc_fft((6, 5, 7)), 40, (FP32,))


@pytest.mark.parametrize("L", [(24, 24, 24), (32, 32, 32), (90, 75, 41), (128, 128, 32)])
def test_transforms_have_no_common_factor(gpu, L):
    """The field of random spins from the plane kernels, projected on the FP64 one: the constants'
    roundings leave a common factor within 2e-8 of one (per axis, there and back, below 0.8e-8, and
    1.8e-8 at 24 points; the projection's own noise is below 1e-9).  Nearest rounding of every constant leaves -1.2e-7 on
    the powers of two, and sin(2 pi / 3) rounded up in both directions 5e-8 to 9e-8 on the others, the
    same at every step."""
    s = LT.sc_fft(L)
    S0 = LT.random_spins(s.nspins, 5)
    f = []
    for prec in (A.FP32, A.FP64_PLAIN):
        with A.Handle(A.RunParams(precision=prec), s) as h:
            assert (PLANES in h.tuning()) == (prec == A.FP32)
            h.set_spins(S0)
            f.append(h.get_field().ravel())
    gain = np.dot(f[0], f[1]) / np.dot(f[1], f[1]) - 1.0
    assert abs(gain) <= 2e-8, gain


def test_box_wider_than_the_plane_kernels(gpu):
    """An axis of more than 128 points has no plane-kernel length: cuFFT runs the caller's mesh."""
    s = LT.sc_ferromagnet((131, 2, 3), pbc=(0, 0, 0), dipole=True)
    S0 = LT.random_spins(s.nspins, 0)
    o = O.Oracle(s)
    o.set_spins(S0)
    o.step(10)
    with A.Handle(A.RunParams(precision=A.FP32, flags=A.FLAG_COMPENSATED), s) as h:
        assert "cuFFT" in h.tuning(), h.tuning()
        h.set_spins(S0)
        h.step(10)
        assert maxdiff(h.get_spins(), o.spins()) <= 1e-5
