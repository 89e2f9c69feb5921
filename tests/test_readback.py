"""Rows read back to host memory: small ones by one copy, larger ones (12 MB up) chunk by chunk
through a pinned ring and several threads; every size gives the loaded rows in trie order."""
import threading

import numpy as np
import pytest

import parallel_ra_b200 as P

pytestmark = pytest.mark.gpu

CHUNK = 2 << 20


def rows_of(nbytes, width, top, seed):
    n = -(-nbytes // (8 * width))
    rng = np.random.default_rng(seed)
    rows = np.empty((n, width), dtype=np.uint64)
    rows[:, 0] = rng.permutation(n).astype(np.uint64)
    rows[:, 1:] = rng.integers(0, top, size=(n, width - 1), dtype=np.uint64)
    return rows


@pytest.mark.parametrize("width,top", [(3, 1000), (3, 2**62)])   # packed and wide tuples
def test_sizes_around_the_ring(width, top):
    p = P.Program(0)
    r = p.relation(1, width - 1, 7, "R")
    for k, nbytes in enumerate((24, 6 * CHUNK - 48, 6 * CHUNK, 6 * CHUNK + 24, 7 * CHUNK - 24, 13 * CHUNK + 24,
                                20 * CHUNK, 3 << 20)):
        rows = rows_of(nbytes, width, top, k)
        p.load_rows(r, rows)
        p.execute(1)
        assert np.array_equal(p.dump_full(r), rows[np.argsort(rows[:, 0])]), nbytes
    p.release()
    p.execute(1)
    assert np.array_equal(p.dump_full(r), rows[np.argsort(rows[:, 0])])


def test_two_programs_read_at_once():
    # one read has the ring, the other one goes without
    out, progs = {}, []
    for k in range(2):
        p = P.Program(0)
        r = p.relation(1, 2, 7, "R")
        rows = rows_of(15 * CHUNK, 3, 1000, k)
        p.load_rows(r, rows)
        p.execute(1)
        progs.append((p, r, rows))

    def read(k):
        p, r, _ = progs[k]
        out[k] = [p.dump_full(r) for _ in range(4)]

    ts = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, (p, r, rows) in enumerate(progs):
        want = rows[np.argsort(rows[:, 0])]
        assert all(np.array_equal(g, want) for g in out[k])
        p.close()
