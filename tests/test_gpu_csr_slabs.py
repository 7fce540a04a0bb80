"""The one-walk CSR build of large sectors (from 65,536 rows) against the oracle's merged rows, bit for bit: real and complex
characters, rows with repeated columns (a dihedral group with spin flip), an operator between two sectors, no symmetry,
64-bit states; what it hands to the general path: more than 256 values, a budget that holds the merged entries
only; and that the matrix is complete when the call returns, for a stream that waits for no other."""
import numpy as np
import pytest

from oracle import oracle as O
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _no_symmetry(n, up):
    return lat.SectorSpec(n, up, np.arange(n, dtype=np.int32)[None, :], np.ones(1, np.complex128))


def _chain(n, chiral=0.0):
    prods = ops.xxz_products(lat.chain_bonds(n), 1.0, 0.7)
    if chiral:
        prods = prods + ops.chiral_products([(i, (i + 1) % n, (i + 2) % n) for i in range(n)], chiral)
    return ops.from_products(n, prods)


def _random_bonds(n):
    g = np.random.default_rng(5)
    return ops.from_products(n, sum((ops.xxz_products([b], *g.uniform(0.5, 1.5, 2)) for b in lat.chain_bonds(n)), []))


CASES = {
    "k=0": (lat.chain_sector(24, 12, 0), None, lambda: ops.row_program(_chain(24))),
    "k=5 chiral": (lat.chain_sector(24, 11, 5), None, lambda: ops.row_program(_chain(24, 0.2))),
    "dihedral, flip": (lat.chain_a1_flip_sector(26), None, lambda: ops.row_program(_chain(26))),
    "40 sites": (lat.chain_sector(40, 6, 0), None, lambda: ops.row_program(_chain(40))),
    "no symmetry": (_no_symmetry(20, 8), None, lambda: ops.row_program(_chain(20))),
    "past 256 values": (_no_symmetry(20, 8), None, lambda: ops.row_program(_random_bonds(20))),
    "two handles": (lat.chain_sector(24, 11, 5), lat.chain_sector(24, 11, 5), lambda: ops.row_program(_chain(24, 0.2))),
    "k=2 to k=5": (lat.chain_sector(24, 12, 5), lat.chain_sector(24, 12, 2), None),
}


@pytest.mark.parametrize("name", list(CASES))
def test_csr_equals_the_oracle(name):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    row, col, prog = CASES[name]
    if prog is None:
        prog = ops.cross_row_program(ops.from_products(24, ops.sz_q_products(24, 2 * np.pi * 3 / 24)), row, col)
    else:
        prog = prog()
    S = D.Sector(row)
    C = S if col is None else D.Sector(col)
    So = O.Sector(row)
    Co = None if col is None else O.Sector(col)
    assert S.dim >= 65536
    A = D.Csr(S, C, D.Program(prog))
    rp, c, v = A.download()
    rp2, c2, v2 = So.csr(O.Program(prog), Co) if Co is not None else So.csr(O.Program(prog))
    assert np.array_equal(rp, np.asarray(rp2, np.uint64))
    assert np.array_equal(c, c2)
    assert np.array_equal(v.view(np.uint64), np.ascontiguousarray(v2).view(np.uint64))
    assert (A.info()["n_dict"] > 256 or A.info()["n_dict"] == -1) == (name in ("past 256 values", "k=2 to k=5"))


def test_budget_of_the_merged_entries():
    from qed_spin_b200 import device as D
    from qed_spin_b200._lib import ResourceLimit
    spec, _, prog = CASES["dihedral, flip"]
    S, P = D.Sector(spec), D.Program(prog())
    A = D.Csr(S, S, P)
    info = A.info()
    need = (S.dim + 1) * 8 + info["nnz"] * 5 + info["n_dict"] * 16
    B = D.Csr(S, S, P, max_bytes=need)
    for a, b in zip(A.download(), B.download()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    with pytest.raises(ResourceLimit):
        D.Csr(S, S, P, max_bytes=need - 1)


def _projected(n):
    """Flips of a bond that act only with the next site up: half the entries a row emits are exact zeros, dropped."""
    prods = ops.xxz_products(lat.chain_bonds(n), 0.0, 0.7)
    for i in range(n):
        for a, b in ((i, (i + 1) % n), ((i + 1) % n, i)):
            prods += [("+-", [a, b], 0.25), ("+-z", [a, b, (i + 2) % n], 0.5)]
    return ops.row_program(ops.from_products(n, prods))


@pytest.mark.parametrize("name", ["projected", "no room for slices"])
def test_matrix_is_complete_on_return(name):
    """Applied at once on a non-blocking stream, bit for bit against the same entries uploaded. "projected" ends with the
    trim of a third of its entries' room, gigabytes-long copies on a large sector; without slices no kernel follows it."""
    from qed_spin_b200 import device as D
    n = 24
    S = D.Sector(lat.chain_sector(n, 12, 3))
    P = D.Program(_projected(n) if name == "projected" else ops.row_program(_chain(n)))
    A = D.Csr(S, S, P)
    info = A.info()
    U = D.Csr.upload(S, S, *A.download())
    # the slab build wants room for the entries before the merge; one byte less than the sliced copy's room leaves it out
    reps = S.reps()[0]
    flips = sum(int((((reps >> np.uint64(i)) ^ (reps >> np.uint64((i + 1) % n))) & np.uint64(1)).sum()) for i in range(n))
    unmerged = (S.dim + 1) * 8 + ((flips + S.dim + 3) & ~3) * 5 + 256 * 16
    budget = max(unmerged, (S.dim + 1) * 8 + info["nnz"] * 9 - 1)
    sliced = info["bytes"] > (S.dim + 1) * 8 + info["nnz"] * 8
    assert sliced
    if name == "projected":
        assert flips > 1.5 * info["nnz"]
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    x = torch.randn(S.dim, dtype=torch.complex128, device="cuda", generator=g)
    want = torch.empty_like(x)
    U.matvec(x, want)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    for limit in (budget, 0):
        for _ in range(4):
            y = torch.zeros_like(x)
            torch.cuda.synchronize()
            B = D.Csr(S, S, P, max_bytes=limit)
            B.matvec(x, y, stream=st)
            st.synchronize()
            assert torch.equal(torch.view_as_real(y).view(torch.int64), torch.view_as_real(want).view(torch.int64))
            if limit and name != "projected":
                assert B.info()["bytes"] < info["bytes"]
            B.close()
