"""One CTA per query on a frontier (frontier.cuh, frontier_walk.cuh), for few queries: every shape of the kernel at the batch sizes
where the choice changes, rows of one and two chunks of links, visited tables so small that most ids are forgotten and have
to be looked up, lists that run out of slots, results ranked in registers and sorted in place, data full of exact ties."""
import numpy as np
import pytest

import oracle
from conftest import assert_same_bits, engine_options, oracle_graph_of
from cuhnsw_b200 import CuHNSW

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,max_m0,dist_type,values,table", [
  (9, 64, "l2", 2, 64), (50, 24, "dot", 1000, 0), (64, 33, "l2", 3, 512), (96, 48, "dot", 2, 0), (128, 16, "l2", 1000, 64),
  (200, 64, "dot", 3, 0), (600, 24, "l2", 2, 64), (1000, 40, "dot", 1000, 0)])
def test_frontier_equals_the_oracle(d, max_m0, dist_type, values, table):
  import torch
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  rng = np.random.default_rng(d + table)
  n = 2500
  base = rng.integers(-values, values + 1, (n, d)).astype(np.float32)
  opt = dict(dist_type=dist_type, max_m=max(max_m0 // 2, 4), max_m0=max_m0, ef_construction=max(48, max_m0), seed=5,
             batch_max=512, search_team=1, visited_table_size=table)
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  g = oracle_graph_of(eng, base, opt)
  q = (base[rng.integers(0, n, 3 * sms + 1)] + rng.integers(-1, 2, (3 * sms + 1, d))).astype(np.float32)
  # the last one: more keys than the index reaches
  for nq, ef, topk in ((1, 1, 1), (3, 31, 2), (sms, 32, 32), (sms + 1, 33, 33), (2 * sms, 100, 10), (2 * sms + 1, 101, 100),
                       (sms, 300, 33), (3 * sms, 300, 1), (3 * sms + 1, 60, 60), (3 * sms + 1, 200, 10), (3 * sms, 250, 40),
                       (20, 2600, 2600)):
    want = oracle.search(g, q[:nq], topk, ef, counters=True)
    eng.obj.enable_stats(True)
    got = eng.search_knn(q[:nq], topk, ef)
    stats = eng.obj.get_stats()
    eng.obj.enable_stats(False)
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all(), (nq, ef)
    assert_same_bits(got[1], want[1])
    assert stats["expansions"] == int(want[3][:, 1].sum()) and stats["sweeps"] == int(want[3][:, 2].sum()), (nq, ef)


def _index(base, opt):
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  return eng, oracle_graph_of(eng, base, opt)


def _equal(got, want, label):
  assert (got[0] == want[0]).all() and (got[2] == want[2]).all(), label
  assert_same_bits(got[1], want[1])


@pytest.mark.parametrize("d,row", [(40, "f32"), (70, "f32"), (70, "f16"), (140, "f32")])
def test_list_and_frontier_around_the_lines(d, row):
  """The smallest lists that are walked on a frontier, and tables whose size the shared memory decides: a number of buckets
  that is no power of two (three CTAs per SM at ef 6000, six or five at ef 2000)."""
  import torch
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  rng = np.random.default_rng(d)
  n = 9000
  base = rng.integers(-9, 10, (n, d)).astype(np.float32)
  opt = dict(dist_type="l2", max_m=16, max_m0=64, ef_construction=64, seed=6, search_team=1, row_dtype=row)
  eng, g = _index(base, opt)
  q = (base[rng.integers(0, n, 7 * sms)] + rng.integers(-1, 2, (7 * sms, d))).astype(np.float32)
  few = 24
  for nq, ef, topk in ((sms, 47, 10), (sms, 48, 10), (sms + 1, 55, 10), (sms + 1, 56, 10), (sms + 1, 79, 10),
                       (sms + 1, 80, 10), (sms, 100, 10), (sms, 101, 10), (sms + 1, 6000, 100), (2 * sms + 1, 6000, 100),
                       (7 * sms, 2000, 10), (7 * sms, 199, 10), (7 * sms, 200, 10), (7 * sms, 249, 10), (7 * sms, 250, 10)):
    got = eng.search_knn(q[:nq], topk, ef)
    at = np.r_[:few, nq - few:nq]
    _equal([part[at] for part in got], oracle.search(g, q[at], topk, ef), (nq, ef))


@pytest.mark.parametrize("d", [30, 200])
def test_searches_in_turn_on_several_streams(d):
  """Which kernel a small search gets depends on what the searches on other streams were; what it finds does not."""
  import torch
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  rng = np.random.default_rng(d)
  n, k = 6000, 10
  base = rng.standard_normal((n, d)).astype(np.float32)
  eng = CuHNSW(engine_options(dict(dist_type="l2", max_m=12, max_m0=24, ef_construction=64, seed=2)))
  eng.set_data(base)
  eng.build()
  eng.obj.set_stream(torch.cuda.current_stream().cuda_stream)

  def search(q, ef):
    out = (torch.empty((len(q), k), dtype=torch.int32, device="cuda"), torch.empty((len(q), k), device="cuda"),
           torch.empty((len(q),), dtype=torch.int32, device="cuda"))
    eng.obj.search_knn_device(q.data_ptr(), len(q), k, ef, *(t.data_ptr() for t in out))
    return out

  q = torch.from_numpy(rng.standard_normal((6 * sms, d)).astype(np.float32)).cuda()
  sizes = [1, 37, sms // 2, sms, sms + 1, 2 * sms, 3 * sms, 6 * sms]
  alone = {(nq, ef): search(q[:nq], ef) for nq in sizes for ef in (40, 90, 300)}
  torch.cuda.synchronize()
  streams = [torch.cuda.Stream() for _ in range(10)]  # more than the engine keeps sets of scratch for
  for ef in (40, 90, 300):
    for count in (2, 4, 10):
      for nq in sizes:
        got = []
        for i in range(2 * count):
          eng.obj.set_stream(streams[i % count].cuda_stream)
          got.append(search(q[:nq], ef))
        torch.cuda.synchronize()
        for out in got:
          assert all(torch.equal(a, b) for a, b in zip(out, alone[nq, ef])), (ef, count, nq)


@pytest.mark.parametrize("d,topk", [(20, 33), (20, 64), (20, 65), (60, 257), (60, 600), (200, 33), (200, 300)])
def test_many_results_of_few_queries(d, topk):
  """More than 32 results, ranked by all warps of a CTA: as many as are expanded, fewer, and more than the index holds; alone,
  and several queries per CTA in turn."""
  import torch
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  rng = np.random.default_rng(topk)
  for n in (500, 3000):
    base = rng.integers(-3, 4, (n, d)).astype(np.float32)
    opt = dict(dist_type="l2", max_m=12, max_m0=24, ef_construction=64, seed=4, search_team=1)
    eng, g = _index(base, opt)
    q = base[rng.integers(0, n, 2 * sms + 3)]
    for nq, ef in ((1, topk), (3, max(topk, 150)), (sms, max(topk, 150)), (2 * sms + 3, max(topk, 180))):
      at = np.arange(min(nq, 40))
      _equal([part[at] for part in eng.search_knn(q[:nq], topk, ef)], oracle.search(g, q[at], topk, ef), (n, nq, ef))
