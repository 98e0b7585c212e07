"""One CTA per query (walk.cuh): several nodes are prepared at a time, but list, visited nodes and results must be those
of the literal walk.  Every shape of the kernel around the sizes where the choice, the list or a row's lanes change, on
data full of exact ties, against the oracle."""
import numpy as np
import pytest

import oracle
from conftest import assert_same_bits, engine_options, oracle_graph_of
from cuhnsw_b200 import CuHNSW

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,max_m0,dist_type,values", [(7, 8, "l2", 3), (32, 33, "dot", 40), (33, 64, "l2", 2),
                                                       (64, 24, "dot", 1000), (96, 32, "l2", 4), (128, 40, "dot", 3),
                                                       (129, 16, "l2", 3), (512, 64, "dot", 1000), (513, 24, "l2", 4),
                                                       (1030, 8, "dot", 2)])
def test_walk_equals_the_oracle(d, max_m0, dist_type, values):
  rng = np.random.default_rng(d)
  n = 2500
  base = rng.integers(-values, values + 1, (n, d)).astype(np.float32)
  opt = dict(dist_type=dist_type, max_m=max(max_m0 // 2, 4), max_m0=max_m0, ef_construction=max(48, max_m0), seed=11,
             batch_max=512, search_team=1)
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  g = oracle_graph_of(eng, base, opt)
  q = (base[rng.integers(0, n, 700)] + rng.integers(-1, 2, (700, d))).astype(np.float32)
  # one key; lists of 32 and 33; short and long walks; more keys than the index reaches
  for nq, ef in ((1, 1), (9, 1), (8, 32), (40, 33), (700, 100), (8, 101), (9, 101), (600, 300), (40, 2600)):
    topk = min(ef, 10)
    want = oracle.search(g, q[:nq], topk, ef, counters=True)
    eng.obj.enable_stats(True)
    got = eng.search_knn(q[:nq], topk, ef)
    stats = eng.obj.get_stats()
    eng.obj.enable_stats(False)
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all(), (nq, ef)
    assert_same_bits(got[1], want[1])
    assert stats["expansions"] == int(want[3][:, 1].sum()) and stats["sweeps"] == int(want[3][:, 2].sum())


@pytest.mark.parametrize("d,ef,nq", [(20, 40, 2072), (50, 200, 3996), (50, 200, 5328), (140, 40, 1480),
                                     (600, 120, 592), (600, 120, 2072)])
def test_batches_on_both_sides_of_a_change_of_kernel(d, ef, nq):
  """Batches around sizes at which kernel, shape or order of service change, against one warp per query."""
  _same_as_one_warp_per_query(d, ef, nq)


@pytest.mark.parametrize("row_dtype,d,max_m0,ef,per_sm", [
  ("f32", 20, 16, 10, 6), ("f32", 20, 16, 40, 8), ("f32", 20, 24, 100, 12), ("f32", 20, 32, 1000, 11),
  ("f32", 50, 16, 100, 21), ("f32", 50, 24, 1500, 10), ("f32", 50, 25, 300, 30), ("f32", 50, 32, 1000, 11),
  ("f32", 50, 16, 4000, 36), ("f32", 100, 16, 15, 4), ("f32", 100, 16, 30, 14), ("f32", 100, 16, 50, 14),
  ("f32", 100, 16, 800, 17), ("f32", 100, 16, 2000, 24), ("f16", 100, 16, 30, 6), ("f16", 100, 16, 60, 14),
  ("bf16", 100, 16, 2000, 14), ("f32", 140, 16, 300, 10), ("f32", 140, 16, 301, 7), ("f32", 140, 16, 2000, 10),
  ("f32", 600, 16, 100, 2), ("f16", 600, 16, 200, 14), ("f32", 600, 16, 201, 10), ("f32", 600, 16, 1200, 14)])
def test_batches_at_the_lines_of_the_choice(row_dtype, d, max_m0, ef, per_sm):
  """The largest batch of one kernel (queries per SM) and one query more, against one warp per query."""
  import torch
  _same_as_one_warp_per_query(d, ef, per_sm * torch.cuda.get_device_properties(0).multi_processor_count, row_dtype,
                               max_m0)


def _same_as_one_warp_per_query(d, ef, nq, row_dtype="f32", max_m0=16):
  rng = np.random.default_rng(nq)
  base = rng.standard_normal((4000, d)).astype(np.float32)
  q = rng.standard_normal((nq + 1, d)).astype(np.float32)
  opt = dict(dist_type="l2", max_m=8, max_m0=max_m0, ef_construction=32, seed=4, batch_max=1024, row_dtype=row_dtype)
  engines = []
  for team in (-1, 0):
    engines.append(CuHNSW(engine_options(dict(opt, search_team=team))))
    engines[-1].set_data(base)
    engines[-1].build()
  for count in (nq, nq + 1):
    got, want = (e.search_knn(q[:count], 10, ef) for e in engines)
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all()
    assert_same_bits(got[1], want[1])
