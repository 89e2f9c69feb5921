"""Bitmap relations: joins that claim a row's matches word by word, and the select that
takes the new tuples from the claimed bits.  Same generation over graphs with short,
long (more matches than a thread walks alone) and shared rows, alone and in waves,
against the oracle and plain runs."""
import numpy as np
import pytest

import oracle as O
import parallel_ra_b200 as P

pytestmark = pytest.mark.gpu


def rows_of(edges):
    e = np.unique(np.array(edges, dtype=np.uint64), axis=0)
    return P.datagen.with_row_ids(e)


def layered(degrees, parents, seed):
    """Layers of nodes; a node has `degrees`-many children, drawn from the next layer, so
    children are shared (a pair is derived many times) when parents is large."""
    rng = np.random.default_rng(seed)
    layers, first = [], 0
    for width in (4, 9, 70, 300):
        layers.append(np.arange(first, first + width))
        first += width
    edges = []
    for up, down in zip(layers, layers[1:]):
        for i, p in enumerate(up):
            d = min(degrees[i % len(degrees)], down.size)
            edges += [(p, c) for c in rng.choice(down, size=d, replace=False)]
        for _ in range(parents):
            edges.append((rng.choice(up), rng.choice(down)))
    return rows_of(edges)


@pytest.mark.parametrize("degrees,parents", [((1, 2, 3), 0), ((15, 16, 17), 0), ((1, 33, 64), 10), ((5, 70), 200)])
def test_same_generation_matches_oracle(degrees, parents):
    rows = layered(degrees, parents, len(degrees) + parents)
    g = P.Program(0)
    grels = P.programs.build_sg(g, rows)
    g.execute(1)
    assert g.stats().bitmap_relations == 2
    o = O.OracleProgram()
    orels = P.programs.build_sg(o, rows)
    o.execute(1)
    assert g.history() == o.history()
    for name in grels:
        assert np.array_equal(g.dump_full(grels[name])[:, :-1], o.dump_full(orels[name])[:, :-1]), name


# 1, 2 and 4 rows per warp of the select: more rows, fewer words per row
@pytest.mark.parametrize("count,n", [(3, 1500), (40, 400), (100, 400)])
def test_waves_match_plain_runs(count, n):
    insts = [P.datagen.with_row_ids(P.datagen.random_tree(n + i % 7, i)) for i in range(count)]
    wave = P.batch.Runner("sg").run_wave(insts)
    plain = P.batch.Runner("sg")
    for i in range(0, count, max(1, count // 8)):
        assert wave[i].key() == plain.run_plain(insts[i]).key(), i
