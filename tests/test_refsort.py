"""Reference id order: each new delta sorted by digits or by buckets of its top digit.

The rows of T's first delta (a copy of G reversed) are given their top-digit bucket sizes, at the
edges of the ways to sort a bucket (512 rows, 2,048 rows) and of the digits (two digits: no
buckets); the order shows in the ids of the tuples joined from it, which must be the oracle's."""
import numpy as np
import pytest

import oracle as O
import parallel_ra_b200 as P

pytestmark = pytest.mark.gpu


def edges(values, sizes, seed):
    """Rows (x, y), x over all values and y over the s-th range of 1/256 of the values."""
    rng = np.random.default_rng(seed)
    bits = int(values - 1).bit_length()
    width = max(1, (1 << bits) >> 8)
    out = [np.array([[0, values - 1]])]   # fixes the bits of a column
    for s, size in enumerate(sizes):
        lo = min(s * 37 % 256 * width, values - width - 1)   # ranges apart from one another
        pick = rng.choice(values * width, size=size, replace=False)
        out.append(np.stack([pick // width, lo + pick % width], axis=1))
    return np.unique(np.concatenate(out), axis=0).astype(np.uint64)


@pytest.mark.parametrize("values,sizes", [
    (200, [150, 90]), (4096, [1]), (4096, [1, 2, 31, 32, 33, 255, 256, 257]), (4096, [511, 512, 513]),
    (4096, [2046, 3]), (4096, [2048]), (4096, [2049, 700]), (4096, [2100, 1, 30]), (100_000, [600, 2000, 17]),
    (100_000, [40] * 7), (100_000, [3000, 3000]), (1 << 20, [513, 2048, 5])])
def test_ids_over_bucket_sizes(values, sizes):
    rows = P.datagen.with_row_ids(edges(values, sizes, values + len(sizes)))
    o = O.OracleProgram()
    ro = P.programs.PROGRAMS["tc"](o, rows)
    o.execute(1)
    p = P.Program(0, id_order=P.engine.IDS_REFERENCE)
    rp = P.programs.PROGRAMS["tc"](p, rows)
    for _ in range(2):   # the second run replays the first one's graph
        p.execute(1)
        assert p.history() == o.history()
        for name in rp:
            assert np.array_equal(p.dump_full(rp[name]), o.dump_full(ro[name])), name
    p.close()


def test_top_digits_of_many_rows_in_the_run():
    """Deltas whose largest bucket has 1,500 rows, 7,500 rows and 1,500 rows in turn."""
    n = 1500
    chain = np.array([[n, n + 1], [n + 3, n + 4]] + [[n + 1, i] for i in range(5)] + [[i, n + 3] for i in range(5)])
    fan = np.stack([np.arange(n), np.full(n, n)], axis=1)   # every value to one value, then to five, then to one
    rows = P.datagen.with_row_ids(np.concatenate([fan, chain]).astype(np.uint64))
    o = O.OracleProgram()
    ro = P.programs.PROGRAMS["tc"](o, rows)
    o.execute(1)
    p = P.Program(0, id_order=P.engine.IDS_REFERENCE)
    rp = P.programs.PROGRAMS["tc"](p, rows)
    p.execute(1)
    assert p.history() == o.history()
    for name in rp:
        assert np.array_equal(p.dump_full(rp[name]), o.dump_full(ro[name])), name
    p.close()
