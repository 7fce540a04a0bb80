"""The candidates of the key order, from the lists (two blocks, or three at real characters) or collected as masks (other
key orders; groups of up to 64, up to 128 and more elements), against the oracle bit for bit: y = H x through every walk,
one vector and two, and projections, at real and complex characters. The larger groups are a chain's translations listed
three or six times, up to 150 elements whose characters add up as any group's do."""
import numpy as np
import pytest

from oracle import oracle as O
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _tiled(spec, times):
    return lat.SectorSpec(spec.n_sites, spec.n_up, np.concatenate([spec.perms] * times),
                          np.concatenate([spec.chars] * times), None, f"{spec.label} x{times}")


def _dihedral(n, up):
    perms = lat.chain_dihedral(n)
    return lat.SectorSpec(n, up, perms, np.ones(len(perms), np.complex128), None, f"D{n} up={up}")


@pytest.mark.parametrize("spec", [lat.chain_sector(24, 8, 5), lat.chain_sector(27, 7, 3), _dihedral(36, 5),
                                  lat.chain_a1_flip_sector(24), _tiled(lat.chain_sector(24, 8, 5), 6),
                                  _tiled(lat.chain_sector(24, 6, 0), 6), _tiled(lat.chain_sector(25, 5, 1), 6),
                                  _tiled(lat.chain_sector(25, 6, 0), 6), _tiled(lat.chain_sector(25, 6, 2), 3),
                                  _tiled(lat.chain_sector(27, 5, 4), 3), lat.chain_sector(25, 7, 0),
                                  lat.chain_sector(27, 6, 0), lat.square_k0_sector(8, 4, 5)],
                         ids=lambda s: f"{s.label} G={s.group_size}")
def test_candidates_equal_the_oracle(spec):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    n = spec.n_sites
    prog = ops.row_program(ops.from_products(n, ops.xxz_products(lat.chain_bonds(n), 1.0, 0.7) +
                                             ops.xxz_products(lat.chain_bonds(n, 2), 0.4, 0.3)))
    S, So = D.Sector(spec), O.Sector(spec)
    assert S.info()["slc_L"] > 0 and np.array_equal(S.reps()[0], So.reps()[0])
    g = np.random.default_rng(4)
    x = g.normal(size=(2, S.dim)) + 1j * g.normal(size=(2, S.dim))
    want = [So.gather(O.Program(prog), v).view(np.uint64) for v in x]
    xd, P = [torch.from_numpy(v).cuda() for v in x], D.Program(prog)
    try:
        for shape in range(6):   # a thread a row, a warp's rows compacted, teams of 8, 16, 32 and 4 lanes
            D.tune_force("walk", shape)
            for n_vec in (1, 2) if shape < 2 else (1,):
                yd = [torch.empty_like(v) for v in xd[:n_vec]]
                D.matvec(S, S, P, xd[:n_vec], yd)
                for y, z in zip(yd, want):
                    assert np.array_equal(y.cpu().numpy().view(np.uint64), z), (shape, n_vec)
    finally:
        D.tune_force("walk", -1)
    states = np.array([int(sum(1 << int(b) for b in g.choice(n, spec.n_up, replace=False))) for _ in range(200)], np.uint64)
    idx, proj = S.index_and_projection(states)
    for s, i, p in zip(states, idx, proj):
        j, q = So.index_and_projection(int(s))
        assert i == j and (j < 0 or (p.real == q.real and p.imag == q.imag))
