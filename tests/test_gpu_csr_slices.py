"""The sliced one-vector CSR apply of large sectors against the CSR's own kernels on the same entries (an uploaded CSR has no
sliced copy): FP64 storage bit for bit, FP32 storage within the rounding of its output (1.2e-7). Row counts that are no
multiple of a slice or a block, rows of 1 to 75 entries, complex values, a matrix between two sectors, and row counts on
both sides of each form's last wave; and the same copy whichever way the matrix was built."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from qed_spin_b200 import lattice as lat
from qed_spin_b200 import operators as ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _chain(n, jz=0.7, chiral=0.0):
    prods = ops.xxz_products(lat.chain_bonds(n), 1.0, jz)
    if chiral:
        prods = prods + ops.chiral_products([(i, (i + 1) % n, (i + 2) % n) for i in range(n)], chiral)
    return ops.row_program(ops.from_products(n, prods))


def _square(Lx=6, Ly=4):
    nn, nnn = lat.square_j1j2_bonds(Lx, Ly)
    return ops.row_program(ops.from_products(Lx * Ly, ops.heisenberg_products(nn) + ops.heisenberg_products(nnn, 0.5)))


@pytest.mark.parametrize("name,spec,prog,two", [
    ("chiral", lat.chain_sector(24, 11, 5), lambda: _chain(24, chiral=0.2), False),
    ("no diagonal", lat.chain_sector(25, 9, 0), lambda: _chain(25, jz=0.0), False),
    ("square", lat.square_k0_sector(6, 4, 12), _square, False),
    ("two handles", lat.chain_sector(24, 12, 3), lambda: _chain(24), True),
    ("six blocks an SM", lat.chain_sector(26, 10, 1), lambda: _chain(26), False),          # 204 k rows on 148 SMs
    ("a short second wave", lat.square_k0_sector(6, 6, 7), lambda: _square(6, 6), False),   # 232 k rows of 47 entries
    ("a second wave", lat.chain_sector(28, 9, 3), lambda: _chain(28, chiral=0.2), False)], ids=lambda v: v if isinstance(v, str) else "")
def test_sliced_apply(name, spec, prog, two):
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from qed_spin_b200 import device as D
    S = D.Sector(spec)
    C = D.Sector(spec) if two else S
    assert S.dim >= 65536
    A = D.Csr(S, C, D.Program(prog()))
    B = D.Csr.upload(S, C, *A.download())
    assert A.info()["bytes"] >= B.info()["bytes"] + 4 * A.info()["nnz"] - 64
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.randn(S.dim, dtype=torch.complex128, device="cuda", generator=g)
    y, z = torch.empty_like(x), torch.empty_like(x)
    A.matvec(x, y)
    B.matvec(x, z)
    assert torch.equal(torch.view_as_real(y).view(torch.int64), torch.view_as_real(z).view(torch.int64))
    x, y, z = x.to(torch.complex64), y.to(torch.complex64), z.to(torch.complex64)
    A.matvec(x, y, dtype="c64")
    B.matvec(x, z, dtype="c64")
    assert float((y - z).abs().max()) <= 1.2e-7 * float(z.abs().max())


def test_slices_of_a_matrix_built_the_general_way():
    """A budget with room for the merged entries and their slices, not for the entries before the merge (most of them exact
    zeros: flips that act only with the next two sites up), sends the build the general way. The same apply follows."""
    from qed_spin_b200 import device as D
    n = 24
    prods = []
    for i in range(n):
        j, k, m = (i + 1) % n, (i + 2) % n, (i + 3) % n
        for a, b in ((i, j), (j, i)):   # S+ S- (1/2 + Sz)(1/2 + Sz)
            prods += [("+-", [a, b], 0.25), ("+-z", [a, b, k], 0.5), ("+-z", [a, b, m], 0.5), ("+-zz", [a, b, k, m], 1.0)]
    S = D.Sector(lat.chain_sector(n, 12, 5))
    P = D.Program(ops.row_program(ops.from_products(n, prods)))
    A = D.Csr(S, S, P)
    info = A.info()
    reps = S.reps()[0]
    flips = sum(int((((reps >> np.uint64(i)) ^ (reps >> np.uint64((i + 1) % n))) & np.uint64(1)).sum()) for i in range(n))
    unmerged = (S.dim + 1) * 8 + ((flips + 3) & ~3) * 5 + 256 * 16
    budget = (S.dim + 1) * 8 + (info["nnz"] + 4) * 9 + 256 * 16
    assert budget < unmerged and info["n_dict"] <= 256
    B = D.Csr(S, S, P, max_bytes=budget)
    assert B.info()["bytes"] >= (S.dim + 1) * 8 + info["nnz"] * 9
    for a, b in zip(A.download(), B.download()):
        assert np.array_equal(a, b)
    x = torch.randn(S.dim, dtype=torch.complex64, device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    A.matvec(x, y, dtype="c64")
    B.matvec(x, z, dtype="c64")
    assert torch.equal(torch.view_as_real(y).view(torch.int32), torch.view_as_real(z).view(torch.int32))


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_first_apply_of_a_process_under_capture(dtype):
    """A process whose first sliced apply is captured in a graph: the replay equals the apply."""
    code = f"""
import sys
import torch
from qed_spin_b200 import device as D, lattice as lat, operators as ops
S = D.Sector(lat.chain_sector(24, 11, 5))
A = D.Csr(S, S, D.Program(ops.row_program(ops.from_products(24, ops.heisenberg_products(lat.chain_bonds(24))))))
x = torch.randn(S.dim, dtype=torch.{'complex64' if dtype == 'c64' else 'complex128'}, device="cuda")
y, z = torch.zeros_like(x), torch.empty_like(x)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    A.matvec(x, y, dtype="{dtype}", stream=torch.cuda.current_stream())
g.replay()
A.matvec(x, z, dtype="{dtype}", stream=torch.cuda.current_stream())
torch.cuda.synchronize()
sys.exit(0 if torch.equal(y, z) and float(y.abs().max()) > 0 else 1)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
