"""Searches and construction of one warp per query or node with visited tables of all sizes, from 64 entries that forget nearly
every id to one that is sized by the engine: what is expanded and found must not depend on it.  Lists around the sizes where
the ranking changes, rows of one and two chunks, data full of exact ties, against the oracle."""
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
