"""Square tori against the oracle bit for bit: representatives, projections and y = H x through every walk, the block walk and
the CSR build, at real and complex characters, few spins up (many tied rows) and more. 6x6 takes its candidates from
pairs of rows; 5x5 (32-bit states), and 6x6 with its elements in another order, a subgroup or a reflection, do not."""
import numpy as np
import pytest

from oracle import oracle as O
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _torus(L, up, kx, ky, order=None):
    perms = lat.square_translations(L, L)
    g = np.arange(L * L)
    chars = np.exp(-2j * np.pi * (kx * (g % L) + ky * (g // L)) / L)
    if kx == ky == 0:
        chars = np.ones(L * L, np.complex128)
    if order is not None:
        perms, chars = perms[order], chars[order]
    return lat.SectorSpec(L * L, up, perms, chars, None, f"{L}x{L} up={up} k=({kx},{ky})")


SHUFFLED = np.concatenate([[0], 1 + np.random.default_rng(1).permutation(35)])
EVEN_ROWS = np.array([g for g in range(36) if (g // 6) % 2 == 0])


def _reflected(up):
    """6x6 translations and their products with the reflection of the rows, trivial characters."""
    t = lat.square_translations(6, 6)
    flip = np.array([(5 - i % 6) + 6 * (i // 6) for i in range(36)])
    perms = np.concatenate([t, t[:, flip]])
    return lat.SectorSpec(36, up, perms, np.ones(72, np.complex128), None, f"6x6 up={up} with reflection")


SPECS = [_torus(5, 2, 0, 0), _torus(5, 7, 0, 0), _torus(5, 6, 1, 2), _torus(6, 4, 0, 0), _torus(6, 5, 3, 1),
         _torus(6, 3, 2, 0), _torus(6, 5, 3, 1, SHUFFLED), _torus(6, 4, 0, 0, EVEN_ROWS), _reflected(4)]
IDS = ["5x5-2", "5x5-7", "5x5-6 k=(1,2)", "6x6-4", "6x6-5 k=(3,1)", "6x6-3 k=(2,0)", "6x6-5 shuffled", "6x6-4 subgroup",
       "6x6-4 reflected"]


def _bits(y):
    return np.ascontiguousarray(y).view(np.uint64)


@pytest.mark.parametrize("spec", SPECS, ids=IDS)
def test_torus_equals_the_oracle(spec):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    L = int(round(spec.n_sites ** 0.5))
    nn, nnn = lat.square_j1j2_bonds(L, L)
    prog = ops.row_program(ops.from_products(spec.n_sites, ops.heisenberg_products(nn) + ops.heisenberg_products(nnn, 0.5)))
    S, So = D.Sector(spec), O.Sector(spec)
    r1, w1 = S.reps()
    r2, w2 = So.reps()
    assert np.array_equal(r1, r2) and np.array_equal(w1.view(np.uint64), w2.view(np.uint64))
    g = np.random.default_rng(2)
    x = g.normal(size=(3, S.dim)) + 1j * g.normal(size=(3, S.dim))
    P, Po = D.Program(prog), O.Program(prog)
    want = [So.gather(Po, v) for v in x]
    xd = [torch.from_numpy(v).cuda() for v in x]
    xb = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    try:
        for shape in range(6):   # a thread a row, a warp's rows compacted, teams of 8, 16, 32 and 4 lanes
            D.tune_force("walk", shape)
            D.tune_force("walk_team", shape % 4)
            for n in (1, 2) if shape < 2 else (1,):
                yd = [torch.empty_like(v) for v in xd[:n]]
                D.matvec(S, S, P, xd[:n], yd)
                for y, z in zip(yd, want):
                    assert np.array_equal(_bits(y.cpu().numpy()), _bits(z)), (shape, n)
            yb = torch.empty_like(xb)
            D.matvec_block(S, S, P, xb, yb, 3)
            for y, z in zip(yb.cpu().numpy().T, want):
                assert np.array_equal(_bits(y), _bits(z)), shape
    finally:
        D.tune_force("walk", -1)
        D.tune_force("walk_team", -1)
    for a, b in zip(D.Csr(S, S, P).download(), So.csr(Po)):
        assert np.array_equal(a, np.asarray(b, a.dtype))
    states = np.array([int(sum(1 << int(b) for b in g.choice(spec.n_sites, spec.n_up, replace=False))) for _ in range(300)],
                      np.uint64)
    idx, proj = S.index_and_projection(states)
    for s, i, p in zip(states, idx, proj):
        j, q = So.index_and_projection(int(s))
        assert i == j and (j < 0 or (p.real == q.real and p.imag == q.imag))


def test_the_pair_table_is_made_for_translations_in_their_order():
    """The table's 16 KB are in the sector's bytes, and gone when the elements come in another order."""
    from qed_spin_b200 import device as D
    for up, kx, ky in ((5, 3, 1), (4, 0, 0)):
        with_table = D.Sector(_torus(6, up, kx, ky)).info()["device_bytes"]
        without = D.Sector(_torus(6, up, kx, ky, SHUFFLED)).info()["device_bytes"]
        assert with_table - without == 4 << 12


def test_large_torus_csr_equals_the_oracle():
    """A sector the one-walk build takes: its slab walk reads the row pairs too."""
    from qed_spin_b200 import device as D
    spec = _torus(6, 7, 2, 1)
    nn, nnn = lat.square_j1j2_bonds(6, 6)
    prog = ops.row_program(ops.from_products(36, ops.heisenberg_products(nn) + ops.heisenberg_products(nnn, 0.5)))
    S, So = D.Sector(spec), O.Sector(spec)
    assert S.dim >= 65536
    for a, b in zip(D.Csr(S, S, D.Program(prog)).download(), So.csr(O.Program(prog))):
        assert np.array_equal(a, np.asarray(b, a.dtype))
