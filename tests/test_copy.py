"""Copies into an empty relation, and the recursion that follows them.

A copy that keeps every column of distinct rows claims nothing and leaves the seen set to the SCC
that needs it; every other one (repeated data columns, a dropped or doubled column, two rules, a
relation that holds rows already) removes repetitions.  Both against the oracle, on the evaluators that need no seen set
and on the hash set, twice per program."""
import os

import numpy as np
import pytest

import oracle as O
import parallel_ra_b200 as P

pytestmark = pytest.mark.gpu

FULL, DELTA = P.programs.FULL, P.programs.DELTA


def build(p, case, n, seed):
    rng = np.random.default_rng(seed)
    arity = 3 if case == "dropped" else 2
    rows = np.zeros((n, arity + 1), dtype=np.uint64)
    rows[:, :arity] = rng.integers(0, max(2, n), size=(n, arity))
    if case == "repeated" and n > 3:
        rows[n // 2:, :2] = rows[: n - n // 2, :2]
    else:
        rows = np.unique(rows, axis=0)
    rows[:, arity] = np.arange(len(rows)) + 7
    G = p.relation(1, arity, 256, "G", FULL)
    E = p.relation(1, 2, 258, "E", FULL)
    T = p.relation(1, 2, 257, "T", FULL)
    p.load_rows(G, rows)
    edges = np.zeros((n, 3), dtype=np.uint64)
    edges[:, :2] = rng.integers(0, max(2, n), size=(n, 2))
    edges[:, 2] = np.arange(n)
    p.load_rows(E, edges)
    p.load_rows(T, rows[: n // 3 + 1, [1, 0, 2]] if case == "stored" else np.empty((0, 3), dtype=np.uint64))
    copy = p.scc(False, 2)
    p.add_relation(copy, G, False)
    p.add_relation(copy, T, True)
    if case == "filtered":
        p.copy(copy, T, G, FULL, [1, 0], P.programs.COPY_FILTER, P.programs.PRED_NE)
    else:
        p.copy(copy, T, G, FULL, {"doubled": [1, 1], "dropped": [2, 0], "kept": [0, 1]}.get(case, [1, 0]))
    if case == "two rules":
        p.copy(copy, T, G, FULL, [0, 1])
    join = p.scc(True, 1)
    p.add_relation(join, E, False)
    p.add_relation(join, T, True)
    p.join(join, T, T, DELTA, E, FULL, [3, 1])
    p.depend(copy, join)
    return {"G": G, "E": E, "T": T}


@pytest.mark.parametrize("case", ["swapped", "kept", "filtered", "repeated", "doubled", "dropped", "two rules", "stored"])
@pytest.mark.parametrize("n", [1, 40, 3000])
@pytest.mark.parametrize("ids,dense", [(P.engine.IDS_EMISSION, None), (P.engine.IDS_EMISSION, 0.0),
                                       (P.engine.IDS_REFERENCE, None)])
def test_copy_then_recursion(case, n, ids, dense):
    o = O.OracleProgram()
    ro = build(o, case, n, n)
    o.execute(1)
    p = P.Program(0, id_order=ids)
    if dense is not None:
        p.set_tuning(dense_max_bytes=dense)
    rp = build(p, case, n, n)
    for _ in range(2):
        p.execute(1)
        assert p.history() == o.history()
        for name in rp:
            a, b = p.dump_full(rp[name]), o.dump_full(ro[name])
            if ids == P.engine.IDS_EMISSION:
                a, b = a[:, :-1], b[:, :-1]
            assert np.array_equal(a, b), name
    p.close()


def write_dump(path, name, rows):
    P.datagen.write_relation(os.path.join(path, name + "_delta"), rows)
    with open(os.path.join(path, "scc_metadata"), "w") as f:
        f.write("99\n")


@pytest.mark.parametrize("version", [FULL, DELTA])
@pytest.mark.parametrize("n", [2, 40, 9000])
def test_copy_of_restart_rows_that_repeat(tmp_path, n, version):
    """A dump's delta rows may share data columns (under other ids), among themselves and with the
    loaded ones: a copy of them keeps one of each."""
    rng = np.random.default_rng(n)
    rows = np.zeros((n, 3), dtype=np.uint64)
    rows[:, :2] = np.unique(rng.integers(0, n, size=(4 * n, 2)), axis=0)[:n]
    rows[:, 2] = np.arange(n) + 7
    again = rows.copy()
    again[:, 2] += n
    delta = np.concatenate([rows, again]) if version == DELTA else again
    write_dump(str(tmp_path), "R", delta)
    p = P.Program(0)
    R, X, Y = (p.relation(1, 2, 256 + k, name, FULL) for k, name in enumerate("RXY"))
    p.load_rows(R, rows)
    for r in (X, Y):
        p.load_rows(r, np.empty((0, 3), dtype=np.uint64))
    first = p.scc(False, 1)
    p.add_relation(first, R, True)
    p.add_relation(first, Y if version == FULL else X, True)
    p.copy(first, Y if version == FULL else X, R, version, [0, 1])
    if version == FULL:   # R's rows of both kinds are in its full version by then
        second = p.scc(False, 2)
        p.add_relation(second, X, True)
        p.copy(second, X, R, FULL, [0, 1])
        p.depend(first, second)
    p.set_restart(str(tmp_path))
    for _ in range(2):
        p.execute(1)
        assert np.array_equal(p.dump_full(X)[:, :2], rows[:, :2])
    p.close()


@pytest.mark.parametrize("dense", [None, 0.0])
def test_copy_of_a_relation_that_two_restarted_sccs_list(tmp_path, dense):
    """Every SCC that lists a relation takes its delta from the dump, so the rows stand in it twice
    after two of them: a third SCC's copy holds each once, the closure that the oracle derives."""
    edges = P.datagen.with_row_ids(P.datagen.erdos_renyi(300, 360, 8))
    write_dump(str(tmp_path), "T", edges[:, [1, 0, 2]])
    p = P.Program(0)
    if dense is not None:
        p.set_tuning(dense_max_bytes=dense)
    T, G = p.relation(1, 2, 257, "T", FULL), p.relation(1, 2, 256, "G", FULL)
    X, Y = p.relation(1, 2, 258, "X", FULL), p.relation(1, 2, 259, "Y", FULL)
    p.load_rows(G, edges)
    for r in (T, X, Y):
        p.load_rows(r, np.empty((0, 3), dtype=np.uint64))
    join, other, copy = p.scc(True, 1), p.scc(False, 2), p.scc(False, 3)
    for r in (G, T):
        p.add_relation(join, r, r == T)
    p.join(join, T, T, DELTA, G, FULL, [3, 1])
    p.add_relation(other, T, False)
    p.add_relation(other, Y, True)
    p.copy(other, Y, G, FULL, [0, 1])
    p.add_relation(copy, X, True)
    p.copy(copy, X, T, FULL, [0, 1])
    p.depend(join, other)
    p.depend(other, copy)
    p.set_restart(str(tmp_path))
    p.execute(1)
    o = O.OracleProgram()
    ro = P.programs.build_tc(o, edges)
    o.execute(1)
    assert np.array_equal(p.dump_full(X)[:, :2], o.dump_full(ro["T"])[:, :2])
    p.close()
