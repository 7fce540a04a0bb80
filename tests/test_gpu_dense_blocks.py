"""The dense tail's one-pass reduction against numpy's dense solve of the oracle's matrix, 1e-11 of the scale: one and two
states, sizes around a warp, around the largest block of 256 threads (64 states), 1,001 states, exactly the largest block
the device takes (1,024) and one that the host takes (1,035), a diagonal operator (zero columns: no reflections),
64-bit states, an attached CSR, and blocks of several programs."""
import numpy as np
import pytest

from oracle import oracle as O
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _no_symmetry(n, up):
    return lat.SectorSpec(n, up, np.arange(n, dtype=np.int32)[None, :], np.ones(1, np.complex128))


def _levels(spec, prog):
    S = O.Sector(spec)
    rp, col, val = S.csr(O.Program(prog))
    A = np.zeros((S.dim, S.dim), np.complex128)
    rows = np.repeat(np.arange(S.dim), np.diff(np.asarray(rp).astype(np.int64)))
    A[rows, np.asarray(col)] = val
    return np.linalg.eigvalsh(A)


def _chiral(n):
    return ops.row_program(ops.from_products(n, ops.heisenberg_products(lat.chain_bonds(n)) + ops.chiral_products(
        [(i, (i + 1) % n, (i + 2) % n) for i in range(n)], 0.3)))


def _pairs(m):
    """m disjoint pairs of sites with one spin up in each: 2^m states of 2m sites, closed under flips within a pair."""
    n = 2 * m
    prods = []
    for i in range(m):
        prods += ops.xxz_products([(2 * i, 2 * i + 1)], 0.4 + 0.1 * i, 0.0)
        prods += ops.xxz_products([(2 * i, (2 * i + 2) % n)], 0.0, 0.7 + 0.03 * i)
    reps = np.sort(np.array([sum(1 << (2 * i + ((s >> i) & 1)) for i in range(m)) for s in range(1 << m)], np.uint64))
    A = np.zeros((len(reps), len(reps)))
    index = {int(r): i for i, r in enumerate(reps)}
    for r, i in index.items():
        up = [((r >> (2 * q)) & 1) - 0.5 for q in range(m)]
        A[i, i] = sum((0.7 + 0.03 * q) * up[q] * up[(q + 1) % m] for q in range(m))
        for q in range(m):
            A[index[r ^ (3 << (2 * q))], i] += 0.5 * (0.4 + 0.1 * q)
    return _no_symmetry(n, m), ops.row_program(ops.from_products(n, prods)), reps, A


CASES = [("one", lat.chain_sector(6, 0, 0), _chiral(6)), ("two", lat.chain_sector(6, 2, 1), _chiral(6)),
         ("k=5", lat.chain_sector(11, 5, 5), _chiral(11)), ("36", _no_symmetry(9, 2), _chiral(9)),
         ("1001", _no_symmetry(14, 4), _chiral(14)), ("35 sites", _no_symmetry(35, 1), _chiral(35)),
         *((str(n), _no_symmetry(n, 1), _chiral(n)) for n in (31, 32, 33, 63, 64)),
         ("66", _no_symmetry(12, 2), _chiral(12)), ("1035", _no_symmetry(46, 2), _chiral(46)),
         ("ising", lat.chain_sector(12, 6, 0),
          ops.row_program(ops.from_products(12, ops.xxz_products(lat.chain_bonds(12), 0.0, 1.0))))]


@pytest.mark.parametrize("name", [c[0] for c in CASES])
@pytest.mark.parametrize("csr", [False, True])
def test_dense_levels(name, csr):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    _, spec, prog = next(c for c in CASES if c[0] == name)
    S, P = D.Sector(spec), D.Program(prog)
    if csr:
        A = D.Csr(S, S, P)
        A.attach(P)
    got, ref = D.dense_levels(S, P), _levels(spec, prog)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-11 * max(1.0, np.abs(ref).max()))


def test_dense_blocks_of_several_sizes_and_state_widths():
    from qed_spin_b200 import device as D
    picks = [c for c in CASES if c[0] in ("two", "k=5", "36")]
    for _, spec, prog in picks:
        secs = [D.Sector(spec), D.Sector(lat.chain_sector(spec.n_sites, 1, 0)), D.Sector(spec)]
        out = D.dense_levels_blocks(secs, D.Program(prog))
        assert np.array_equal(out[0], out[2])
        np.testing.assert_array_equal(out[0], D.dense_levels(secs[0], D.Program(prog)))


@pytest.mark.parametrize("m", [6, 10])   # 64 and 1,024 states
def test_dense_levels_of_exactly_the_limits(m):
    from qed_spin_b200 import device as D
    spec, prog, reps, A = _pairs(m)
    S = D.Sector(spec, reps=reps, inv_norms=np.ones(len(reps)))
    ref = np.linalg.eigvalsh(A)
    np.testing.assert_allclose(D.dense_levels(S, D.Program(prog)), ref, rtol=0, atol=1e-11 * np.abs(ref).max())
