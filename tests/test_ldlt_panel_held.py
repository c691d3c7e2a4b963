"""The LDL^T panel's two ways through its own columns, on the CPU emulation: the next columns held up
to date while the own rows fit the room for them, and each column formed when it is looked at beyond
it. Built with room for 40 rows, fronts below, at and above it (several panels, so that one front
takes both ways) come out the oracle's bit for bit."""
import subprocess

import numpy as np
import pytest

from native import emulation as E
from test_ldlt_panel_emulated import bits, dense_csr, indefinite, oracle_ldlt


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    lib = tmp_path_factory.mktemp("emulation") / "libheld.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-ffp-contract=off", "-Wall", "-Wextra",
                    "-DFC_LDLT_HELD_ROWS=40", f"-I{E.HEADER.parent.parent}", "-o", str(lib), str(E.SRC)], check=True)
    return lib


@pytest.mark.parametrize("n", [3, 39, 40, 41, 64, 104, 105, 150])
@pytest.mark.parametrize("zero_every", [2, 1000])
def test_both_ways_are_the_oracles(library, monkeypatch, n, zero_every):
    monkeypatch.setattr(E, "LIB", library)
    monkeypatch.setattr(E, "_lib", None)
    a = indefinite(n, seed=n, zero_every=zero_every)
    _, f = oracle_ldlt(dense_csr(a))
    rc, F, piv, order, _ = E.factor_front(np.tril(a), n, np.max(np.abs(a), axis=0), threads=7)
    opiv, oorder = f.pivots()
    assert rc == -1 and np.array_equal(piv, opiv) and np.array_equal(order, oorder)
    assert np.array_equal(bits(E.packed(F, n)), bits(f.values()))
