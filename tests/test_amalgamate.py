"""The merged supernodes that the device factors by (fieldcraft_b200/csrc/host/amalgamate.cpp), on the
CPU: a new order of the columns with descendants before ancestors, every row of the reference's
structure in the merged one, each child's rows among its parent's (what the assembly's relative maps
need), explicit zeros within the share the rule allows, and a batch's systems merged each as alone.
merge = 0 gives the reference's supernodes as they are."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import Symbolic, UpperColumns, _lib, problems


def amalgamated(sym, merge=1):
    lib = _lib.load()
    fn = lib.fc_test_amalgamate
    sizes = np.zeros(2, np.int64)
    none = [C.c_void_p(None)] * 5
    fn(sym.handle, merge, C.c_void_p(sizes.ctypes.data), *none)
    ns, rows = int(sizes[0]), int(sizes[1])
    out = dict(place=np.zeros(sym.n, np.int32), first=np.zeros(ns + 1, np.int64), rptr=np.zeros(ns + 1, np.int64),
               rows=np.zeros(rows, np.int32), sparent=np.zeros(ns, np.int64))
    fn(sym.handle, merge, C.c_void_p(sizes.ctypes.data), *(C.c_void_p(a.ctypes.data) for a in out.values()))
    return out


def dense(n):
    a = np.full((n, n), 0.1) + n * np.eye(n)
    return H.rows_to_csr([[(j, a[i, j]) for j in range(n)] for i in range(n)])


def diagonal(n):
    return H.rows_to_csr([[(i, 2.0)] for i in range(n)])


CASES = {
    "empty": lambda: diagonal(0),
    "one": lambda: diagonal(1),
    "forest of ones": lambda: diagonal(40),
    "dense": lambda: dense(150),
    "grid": lambda: H.shifted_grid([9, 8, 7], -0.5)[0],
    "saddle pattern": lambda: H.saddle(8, 3),
    "cantilever": lambda: problems.cantilever().csr,
    "block": lambda: problems.lognormal_block(9, nrhs=1).csr,
    "plate": lambda: problems.plate(20, 14, 2).csr,
}


@pytest.mark.parametrize("name", list(CASES))
def test_the_merged_structure_holds_the_references(name):
    up = UpperColumns.from_symmetric(CASES[name]())
    sym = Symbolic(up, 2**62)
    a, g = sym.arrays(), amalgamated(sym)
    n, ns, place = up.n, a["ns"], g["place"].astype(np.int64)
    assert np.array_equal(np.sort(place), np.arange(n))
    width, height = np.diff(g["first"]), np.diff(g["rptr"])
    assert g["first"][-1] == n and np.all(width >= 1) and np.all(height >= width)
    group = np.repeat(np.arange(width.size), width)  # of each new column
    rows = [g["rows"][g["rptr"][k]:g["rptr"][k + 1]].astype(np.int64) for k in range(width.size)]
    for k, r in enumerate(rows):
        assert np.array_equal(r[:width[k]], np.arange(g["first"][k], g["first"][k + 1]))
        assert np.all(np.diff(r) > 0)
        q = g["sparent"][k]
        if height[k] > width[k]:
            assert q > k and group[r[width[k]]] == q and np.all(np.isin(r[width[k]:], rows[q]))
        else:
            assert q < 0
    held = 0
    for s in range(ns):
        own = place[a["first"][s]:a["first"][s + 1]]
        assert np.array_equal(own, np.arange(own[0], own[0] + own.size)) and np.all(group[own] == group[own[0]])
        ref = place[a["rows"][a["rptr"][s]:a["rptr"][s + 1]]]
        assert np.all(np.isin(ref, rows[group[own[0]]]))
        assert np.all(ref[own.size:] > own[-1])  # a row stays below its column
        held += own.size * ref.size - own.size * (own.size - 1) // 2
    stored = int(np.sum(width * height - width * (width - 1) // 2))
    assert held == a["entries"] and stored >= held
    # the rule's shares of what a supernode stores, by its width, or its fixed number of zeros
    share = np.where(width <= 16, 0.8, np.where(width <= 48, 0.1, 0.05))
    allowed = np.maximum(share * (width * height - width * (width - 1) // 2), 4000)
    assert stored - held <= np.sum(allowed)


@pytest.mark.parametrize("name", ["grid", "cantilever", "plate"])
def test_unmerged_is_the_reference(name):
    up = UpperColumns.from_symmetric(CASES[name]())
    sym = Symbolic(up, 2**62)
    a, g = sym.arrays(), amalgamated(sym, 0)
    assert np.array_equal(g["place"], np.arange(up.n)) and np.array_equal(g["first"], a["first"])
    assert np.array_equal(g["rptr"], a["rptr"]) and np.array_equal(g["rows"], a["rows"])


def test_a_batch_merges_each_system_as_alone():
    parts = [UpperColumns.from_symmetric(CASES[k]()) for k in ("cantilever", "grid", "dense")]
    whole = amalgamated(Symbolic.batch(parts, 2**62)[0])
    alone = [amalgamated(Symbolic(p, 2**62)) for p in parts]
    offset = np.cumsum([0] + [p.n for p in parts])
    assert np.array_equal(whole["place"], np.concatenate([g["place"] + o for g, o in zip(alone, offset)]))
    assert np.array_equal(np.diff(whole["first"]), np.concatenate([np.diff(g["first"]) for g in alone]))


def test_merging_shortens_the_tree():
    """The 24^3 block: at most a third of the supernodes and half of the levels are left."""
    up = problems.lognormal_block(24, nrhs=1).upper()
    sym = Symbolic(up, 2**62)

    def levels(g):
        lev = np.zeros(g["sparent"].size, int)
        for k, q in enumerate(g["sparent"]):
            if q >= 0:
                lev[q] = max(lev[q], lev[k] + 1)
        return lev.max() + 1

    before, after = amalgamated(sym, 0), amalgamated(sym)
    assert 3 * after["sparent"].size <= before["sparent"].size and 2 * levels(after) <= levels(before)
