"""Loading: small relations (one block sorts them and drops repetitions) and larger ones, at the
edges between the two, and small and larger join indexes, against numpy and the oracle."""
import time

import numpy as np
import pytest

import oracle as O
import parallel_ra_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1024, 1025, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("kind", ["distinct", "shared_data", "repeated"])
def test_loaded_rows_are_sorted_and_distinct(n, kind):
    rng = np.random.default_rng(n)
    rows = np.empty((n, 4), dtype=np.uint64)
    rows[:, 0] = rng.permutation(n) if kind == "distinct" else rng.integers(0, max(1, n // 3), size=n)
    rows[:, 1] = rows[:, 0] * 7 % 11
    rows[:, 2] = 3
    rows[:, 3] = rng.integers(0, 2**63, size=n, dtype=np.uint64) if kind != "repeated" else rows[:, 0] % 5
    p = P.Program(0)
    r = p.relation(1, 3, 9, "R")
    for _ in range(2):   # the second run restores what the first one loaded
        p.load_rows(r, rows)
        p.execute(1)
        assert np.array_equal(p.dump_full(r), np.unique(rows, axis=0))
        p.execute(1)
        assert np.array_equal(p.dump_full(r), np.unique(rows, axis=0))


@pytest.mark.parametrize("n", [4095, 4096])
@pytest.mark.parametrize("kind", ["distinct", "shared_data", "repeated"])
def test_rows_at_the_line_between_the_loads(n, kind):
    test_loaded_rows_are_sorted_and_distinct(n, kind)


def test_a_row_more_is_not_the_faster_load():
    """The one-block load ends where the sort over the grid takes over with a gain."""
    best = {}
    for n in (4096, 4097, 8192, 8193):
        rows = np.random.default_rng(n).integers(0, 1 << 20, size=(n, 3), dtype=np.uint64)
        p = P.Program(0)
        r = p.relation(1, 2, 9, "R")
        times = []
        for _ in range(40):
            t = time.perf_counter()
            p.load_rows(r, rows)
            p.execute(1)
            times.append(time.perf_counter() - t)
        best[n] = min(times)
        p.close()
    assert best[4096] < 1.2 * best[4097] and best[8192] < 1.2 * best[8193], best


# join indexes: rows up to / above 4,096, key ranges up to / above 2^16, a row of more than 4,096
@pytest.mark.parametrize("rows_n,values,hub", [(4096, 3000, 0), (4097, 3000, 0), (4096, 65_535, 0), (3000, 70_000, 0),
                                               (4000, 20, 0), (5000, 6000, 4500)])
@pytest.mark.parametrize("ids", [P.engine.IDS_EMISSION, P.engine.IDS_REFERENCE])
def test_joins_over_small_and_large_indexes(rows_n, values, hub, ids):
    rng = np.random.default_rng(rows_n + values)
    g = rng.integers(0, values, size=(rows_n, 2)).astype(np.uint64)
    g[:hub, 0] = 1
    g[:hub, 1] = np.arange(hub)
    g[-1] = values - 1
    f = np.stack([np.arange(40), rng.integers(0, values, size=40)], axis=1).astype(np.uint64)
    f[:3, 1] = (0, 1, values - 1)
    got = []
    for p in (P.Program(0, id_order=ids), O.OracleProgram()):
        G, F, J = p.relation(1, 2, 300, "G"), p.relation(1, 2, 301, "F"), p.relation(1, 2, 302, "J")
        p.load_rows(G, P.datagen.with_row_ids(np.unique(g, axis=0)))
        p.load_rows(F, P.datagen.with_row_ids(f[:, ::-1].copy()))
        p.load_rows(J, np.empty((0, 3), dtype=np.uint64))
        s = p.scc(False, 1)
        for r in (G, F):
            p.add_relation(s, r, False)
        p.add_relation(s, J, True)
        p.join(s, J, F, 1, G, 1, [1, 3])
        p.execute(1)
        got.append((p.history(), p.dump_full(J)[:, :-1]))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
