"""The device enumeration at the edges of its chunks (a thread each, 4 states at least) against the oracle, bit for bit:
no or all spins up, one state, totals that are no multiple of a chunk, and a sector past 64 states a chunk's start; and
that a sector's tables are complete when the call returns, for a stream that waits for no other."""
import numpy as np
import pytest

from oracle import oracle as O
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("spec", [lat.chain_sector(4, 0, 0), lat.chain_sector(4, 4, 0), lat.chain_sector(5, 1, 2),
                                  lat.chain_sector(13, 6, 0), lat.chain_sector(20, 10, 7), lat.chain_sector(24, 11, 5),
                                  lat.chain_a1_flip_sector(24), lat.square_k0_sector(6, 4, 11)],
                         ids=lambda s: f"{s.label} up={s.n_up}")
def test_enumeration_equals_the_oracle(spec):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    r1, w1 = D.Sector(spec).reps()
    r2, w2 = O.Sector(spec).reps()
    assert np.array_equal(r1, r2)
    assert np.array_equal(w1.view(np.uint64), w2.view(np.uint64))


@pytest.mark.parametrize("lookup", [0, 1, 2, 4])   # chosen, rank table, buckets, wide hash slots
@pytest.mark.parametrize("n,mom", [(20, 7), (24, 5), (25, 0)])
def test_sector_is_complete_on_return(n, mom, lookup):
    """Created, or made from representatives, and applied at once on a non-blocking stream: the oracle's y bit for bit."""
    from qed_spin_b200 import device as D
    spec = lat.chain_sector(n, 6, mom)
    host = ops.row_program(ops.from_products(n, ops.xxz_products(lat.chain_bonds(n), 1.0, 0.7)))
    So = O.Sector(spec)
    reps, inv = So.reps()
    x = np.random.default_rng(3).normal(size=(So.dim, 2)).view(np.complex128)[:, 0].copy()
    want = So.gather(O.Program(host), x).view(np.uint64)
    P, xd, st = D.Program(host), torch.from_numpy(x).cuda(), torch.cuda.Stream()
    yd = torch.empty_like(xd)
    torch.cuda.synchronize()
    for i in range(6):
        S = D.Sector(spec, lookup=lookup) if i % 2 else D.Sector(spec, lookup=lookup, reps=reps, inv_norms=inv)
        D.matvec(S, S, P, [xd], [yd], stream=st)
        st.synchronize()
        assert np.array_equal(yd.cpu().numpy().view(np.uint64), want)
        S.close()


def test_empty_sector_from_representatives():
    from qed_spin_b200 import device as D
    spec = lat.chain_sector(12, 6, 0)
    S = D.Sector(spec, reps=np.zeros(0, np.uint64), inv_norms=np.zeros(0))
    assert S.dim == 0
    idx, _ = S.index_and_projection(np.array([0b111111], np.uint64))
    assert idx[0] == -1
