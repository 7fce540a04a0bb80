"""Shared test set-up: the `gpu` marker, the golden fixtures, and the checkers under oracle/."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (runs the sm_100a library)")


@pytest.fixture(scope="session")
def fixtures():
    return dict(np.load(os.path.join(GOLDEN, "fixtures.npz")))


@pytest.fixture(scope="session")
def golden():
    with open(os.path.join(GOLDEN, "golden.json")) as fh:
        return json.load(fh)


def need_reference(lib="libqed_ref.so"):
    """Goes on when oracle/_ref/`lib` is there: the reference's own code, compiled from its sources (oracle/Makefile, run by
    __graft_entry__.build()). Skips where neither it nor the sources are, as nothing can be compared there; sources without
    the library fail."""
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", lib)):
        return
    r = subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle"), "print-ref"], capture_output=True, text=True)
    if r.returncode == 0 and os.path.isdir(os.path.join(r.stdout.strip(), "include", "ed")):
        pytest.fail(f"oracle/_ref/{lib} is not built (oracle/Makefile, run by __graft_entry__.build())")
    pytest.skip(f"oracle/_ref/{lib} is not here, nor are the reference's sources")


def host_program(fx, name):
    """The reference's compiled row program of a fixture case, as a host Program."""
    from qed_spin_b200.operators import Program
    g = lambda k: fx[f"{name}/prog/{k}"]
    return Program(g("group_flip"), g("group_setbits"), g("group_vbegin"), g("vsub_val"), g("vsub_tbegin"),
                   g("term_sign"), g("term_coeff").view(np.complex128))
