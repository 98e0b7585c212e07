"""Searches of one warp per query and construction with visited tables of all sizes, from 64 entries that forget nearly every id
to one that is sized by the engine: what is expanded and found must not depend on it.  Lists around the sizes where the
ranking changes, rows of one and two chunks, data full of exact ties, against the oracle.  (Batches of up to ten nodes per SM,
as in the first test, are built by one CTA per node, larger ones by one warp.)"""
import numpy as np
import pytest

import oracle
from conftest import assert_same_bits, engine_options, oracle_graph_of
from cuhnsw_b200 import CuHNSW

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [0, 64, 1024])
@pytest.mark.parametrize("d,max_m0,dist_type,values", [(5, 8, "l2", 2), (40, 33, "dot", 3), (64, 64, "l2", 1000),
                                                       (100, 24, "dot", 2), (200, 40, "l2", 3), (700, 16, "dot", 1000)])
def test_the_table_changes_no_answer(d, max_m0, dist_type, values, table):
  rng = np.random.default_rng(d + table)
  n = 2500
  base = rng.integers(-values, values + 1, (n, d)).astype(np.float32)
  opt = dict(dist_type=dist_type, max_m=max(max_m0 // 2, 4), max_m0=max_m0, ef_construction=max(48, max_m0), seed=3,
             batch_max=512, search_team=0, visited_table_size=table)
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  levels, rows0, rows_u = eng.obj.get_graph()
  built = oracle.build_graph(base, levels, opt["max_m"], max_m0, dist_type, opt["ef_construction"], 0.25, False,
                             bmax=512, ramp_div=4)
  assert (rows0 == built.rows0).all() and (rows_u[:built.rowsU.shape[0]] == built.rowsU).all()
  g = oracle_graph_of(eng, base, opt)
  q = (base[rng.integers(0, n, 60)] + rng.integers(-1, 2, (60, d))).astype(np.float32)
  # (2600: more keys than the index reaches)
  for ef, topk in ((1, 1), (2, 2), (31, 31), (32, 32), (33, 33), (100, 10), (300, 100), (1000, 1), (2600, 2600)):
    want = oracle.search(g, q, topk, ef, counters=True)
    eng.obj.enable_stats(True)
    got = eng.search_knn(q, topk, ef)
    stats = eng.obj.get_stats()
    eng.obj.enable_stats(False)
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all(), ef
    assert_same_bits(got[1], want[1])
    assert stats["expansions"] == int(want[3][:, 1].sum()), ef


def _check(eng, g, q, sizes, label):
  """Searches of the first nq queries with every (nq, ef, topk) against the oracle, expansions included."""
  for nq, ef, topk in sizes:
    want = oracle.search(g, q[:nq], topk, ef, counters=True)
    eng.obj.enable_stats(True)
    got = eng.search_knn(q[:nq], topk, ef)
    stats = eng.obj.get_stats()
    eng.obj.enable_stats(False)
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all(), (label, nq, ef)
    assert_same_bits(got[1], want[1])
    assert stats["expansions"] == int(want[3][:, 1].sum()), (label, nq, ef)


# 64 entries: 16 buckets of four tags or 32 of two.  524 289 to 1 048 576 rows: 16 bits tell the ids of a bucket apart in
# buckets of four (tags of 32 bits), 15 in buckets of two; above both need 32.
@pytest.mark.parametrize("n,d,row", [(600_000, 8, "f32"), (1_100_000, 8, "f32"), (600_000, 70, "f32"), (1_100_000, 70, "f16"),
                                     (600_000, 130, "f16"), (1_100_000, 130, "f32")])
def test_tags_of_16_and_of_32_bits(n, d, row):
  """Tables of 64 entries over so many rows that a tag does not fit into 15 bits, in every search kernel: one warp, one CTA on
  a list and one CTA on a frontier per query."""
  rng = np.random.default_rng(n + d)
  base = rng.integers(-3, 4, (n, d), dtype=np.int8).astype(np.float32)
  opt = dict(dist_type="l2", max_m=8, max_m0=16, ef_construction=24, seed=3, row_dtype=row)
  q = (base[rng.integers(0, n, 500)] + rng.integers(-1, 2, (500, d))).astype(np.float32)
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  graph = eng.obj.get_graph()
  g = oracle_graph_of(eng, base, opt)
  # the same graph behind handles of each kind: construction does not depend on the table
  for team in (0, 1):
    one = CuHNSW(engine_options(opt, search_team=team, visited_table_size=64))
    one.set_data(base)
    one.build()
    for a, b in zip(one.obj.get_graph(), graph):
      assert (a == b).all()
    _check(one, g, q, ((40, 20, 10), (40, 120, 120), (33, 300, 10), (500, 120, 10)), (n, d, row, team))
