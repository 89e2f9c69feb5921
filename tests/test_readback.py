"""Rows read back to host memory: by one copy, into large fresh memory (12 MB up) while several
threads make its pages, or through a ring; every size gives the loaded rows in trie order."""
import ctypes as C
import mmap
import threading
import time

import numpy as np
import pytest
import torch

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
    # both while threads make their pages
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


def loaded(nbytes):
    p = P.Program(0)
    r = p.relation(1, 2, 7, "R")
    rows = rows_of(nbytes, 3, 1000, 5)
    p.load_rows(r, rows)
    p.execute(1)
    return p, r, rows[np.argsort(rows[:, 0])]


def read_into(p, r, address, n):
    got = C.c_uint64()
    t = time.perf_counter()
    assert p._L.ra_relation_dump_full(p.handle, r, C.cast(address, C.POINTER(C.c_uint64)), n, C.byref(got)) == 0
    assert got.value == n
    return time.perf_counter() - t


def mapped(nbytes, how):
    """Fresh memory of nbytes, its address off the start of a page (and an object that keeps it)."""
    m = mmap.mmap(-1, nbytes + 8192)
    if how == "some touched":
        m[:nbytes // 3] = b"\1" * (nbytes // 3)
    if how == "all touched":
        m[:] = b"\1" * len(m)
    return C.addressof(C.c_char.from_buffer(m)) + 40, m


@pytest.mark.parametrize("how", ["fresh", "some touched", "all touched", "page-locked"])
@pytest.mark.parametrize("nbytes", [6 * CHUNK, 11 * CHUNK + 24, 40 << 20])
def test_memory_of_every_kind(how, nbytes):
    p, r, want = loaded(nbytes)
    if how == "page-locked":
        keep = torch.zeros(want.size, dtype=torch.int64, pin_memory=True)
        at = keep.data_ptr()
    else:
        at, keep = mapped(want.nbytes, how)
    for _ in range(2):
        read_into(p, r, at, len(want))
        got = np.ctypeslib.as_array(C.cast(at, C.POINTER(C.c_uint64)), want.shape)
        assert np.array_equal(got, want)
    p.close()


def test_page_locked_rows_are_read_by_one_copy():
    """45 MB into page-locked rows take the time of the copy (half as much again for the rest of the call)."""
    p, r, want = loaded(45 << 20)
    host = torch.empty(want.size, dtype=torch.int64, pin_memory=True)
    dev = torch.zeros(want.size, dtype=torch.int64, device="cuda")
    copies = []
    for _ in range(10):
        torch.cuda.synchronize()
        t = time.perf_counter()
        host.copy_(dev)
        torch.cuda.synchronize()
        copies.append(time.perf_counter() - t)
    reads = [read_into(p, r, host.data_ptr(), len(want)) for _ in range(10)]
    assert min(reads) < 1.5 * min(copies)
    p.close()


def test_a_program_s_first_read_costs_no_set_up():
    """Programs that are made for one read: the first read takes about as long as the next (the
    first of a process aside), whatever was read or closed before."""
    first, again = [], []
    at, keep = mapped(15 << 20, "all touched")
    for _ in range(4):
        p, r, want = loaded(14 << 20)
        first.append(read_into(p, r, at, len(want)))
        again += [read_into(p, r, at, len(want)) for _ in range(3)]
        p.close()
    assert min(first) < 2 * min(again) + 1e-3


def test_a_process_that_goes_on_reading():
    """From the fourth read of 24 MB or more on through a ring, made with the reads and given back with
    the last program: whole, odd and partial chunks, several programs, then all closed and again."""
    for _ in range(2):
        progs = [loaded(n) for n in (12 * CHUNK, 12 * CHUNK + 24, 13 * CHUNK - 24, 20 * CHUNK + 24)]
        for k in range(3):
            for p, r, want in progs:
                assert np.array_equal(p.dump_full(r), want), k
        at, keep = mapped(progs[3][2].nbytes, "some touched")
        for p, r, want in progs:
            read_into(p, r, at, len(want))
            assert np.array_equal(np.ctypeslib.as_array(C.cast(at, C.POINTER(C.c_uint64)), want.shape), want)
        for p, r, want in progs:
            p.close()


def test_a_program_s_first_large_read_costs_no_ring():
    """Programs made for one read of 30 MB, one after the other: no read pays for a ring."""
    at, keep = mapped(31 << 20, "all touched")
    first, plain = [], []
    for k in range(8):
        p, r, want = loaded(30 << 20)
        first.append(read_into(p, r, at, len(want)))
        plain += [read_into(p, r, at, len(want)) for _ in range(2)]   # the second and third read: none yet
        p.close()
    assert np.median(first) < 1.5 * np.median(plain) + 1e-3
