"""FP64 plain form of a typed matrix (values from the tensor table, entries by row pattern or word, one
launch per stage) against its general form (ASD_FLAG_STREAMED_EXCHANGE: the caller's values,
field and stage launches apart): bit-identical, also with replicas at T = 0 and above, the Cdzz quirk, explicit
zero entries and rows that do not repeat."""
import numpy as np
import pytest

import asd_b200 as A
import asd_lattice as LT

pytestmark = pytest.mark.gpu


def random_graph():
    n, rng = 700, np.random.default_rng(3)
    lens = rng.integers(0, 7, n)
    adj = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.uint32)
    tens = rng.standard_normal((5, 9)) * 20.0
    tens[0] = 0.0                                     # an explicit zero entry
    s = A.SpinSystem(nspins=n, materials=[A.MaterialSpec()], full=True, exch=A.EXCH_CSR, adjncy=adj,
                     csr_val=tens[rng.integers(0, 5, len(adj))], temperature=50.0,
                     xadj=np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32))
    return [s]


CASES = {
    "sc_open": lambda: [LT.sc_ferromagnet((9, 7, 5), pbc=(0, 0, 0), T=100.0)],
    "replicas": lambda: [LT.sc_ferromagnet(e, T=80.0 * r, stream=r) for r, e in enumerate((6, 9, 5))],
    "bct2_csr": lambda: [LT.bct2_antiferromagnet((5, 7, 6), T=300.0)],
    "bct2_dia": lambda: [LT.bct2_antiferromagnet((6, 5, 7), layout="dia", T=300.0)],
    "film_dia_pulse": lambda: [LT.film_dia(13, 10, 3, dipole=False)],
    "dipole": lambda: [LT.sc_ferromagnet((6, 5, 4), pbc=(0, 0, 0), dipole=True)],
    "random_graph": random_graph,
}


@pytest.mark.parametrize("integ", [A.HEUN, A.RK4, A.RK5])
@pytest.mark.parametrize("case", CASES)
def test_typed_bit_identical_to_general(gpu, case, integ):
    systems = CASES[case]()
    n = sum(s.nspins for s in systems)
    out = []
    for flags in (0, A.FLAG_STREAMED_EXCHANGE, A.FLAG_GPU_DZZ_FROM_DYY, A.FLAG_GPU_DZZ_FROM_DYY | A.FLAG_STREAMED_EXCHANGE):
        with A.Handle(A.RunParams(precision=A.FP64_PLAIN, integrator=integ, flags=flags, seed=8), systems) as h:
            h.set_spins(LT.random_spins(n, 1))
            if "pulse" in case:
                h.set_site_field_pulse(0.2, 2e-15, 1e-15)
            h.step(25)
            out.append((h.get_spins(), h.get_field()))
    for a, b in ((0, 1), (2, 3)):
        assert np.array_equal(out[a][0], out[b][0])
        assert np.array_equal(out[a][1], out[b][1])
