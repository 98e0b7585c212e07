"""Transfers between ordinary host arrays and the device go through page-locked buffers of 8 MB, in pieces: sizes
around the edges of a piece and of the in-place path (256 KB), against the device-buffer search and the numpy reader of
index files."""
import concurrent.futures
import os
import resource
import time

import numpy as np
import pytest

from conftest import assert_same_bits, engine_options
from cuhnsw_b200 import CuHNSW
from oracle import index_file

pytestmark = pytest.mark.gpu

PIECE = 8 << 20


def _index(n, d, **opt):
  rng = np.random.default_rng(n + d)
  base = rng.integers(-8, 9, (n, d)).astype(np.float32)
  opt = dict(dict(dist_type="l2", max_m=4, max_m0=8, ef_construction=8, seed=5, batch_max=4096), **opt)
  eng = CuHNSW(engine_options(opt))
  eng.set_data(base)
  eng.build()
  return eng, base, rng


@pytest.mark.parametrize("d,topk", [(7, 1), (20, 100)])
def test_host_searches_around_the_edges_of_the_staging_sizes(d, topk):
  import torch
  eng, _, rng = _index(3000, d)
  per_query = 4 * (d + 2 * topk + 1)
  in_place, piece = (256 << 10) // per_query, (PIECE - 1024) // per_query
  q = rng.standard_normal((5 * piece + 13, d)).astype(np.float32)
  dq = torch.from_numpy(q).cuda()
  ids = torch.empty((len(q), topk), dtype=torch.int32, device="cuda")
  dist = torch.empty((len(q), topk), dtype=torch.float32, device="cuda")
  found = torch.empty((len(q),), dtype=torch.int32, device="cuda")
  eng.obj.search_knn_device(dq.data_ptr(), len(q), topk, 100, ids.data_ptr(), dist.data_ptr(), found.data_ptr())
  eng.obj.synchronize()
  want = ids.cpu().numpy(), dist.cpu().numpy(), found.cpu().numpy()
  for nq in (1, in_place, in_place + 1, piece, piece + 1, 2 * piece + 1, len(q)):
    got = eng.search_knn(q[:nq], topk, 100)
    assert (got[0] == want[0][:nq]).all() and (got[2] == want[2][:nq]).all(), nq
    assert_same_bits(got[1], want[1][:nq])


@pytest.mark.parametrize("queries", [300, 60_000])
def test_a_blocking_host_search_comes_behind_the_work_on_the_handles_stream(queries):
  """In place and in pieces, on a stream of the caller's and on the legacy default stream."""
  import torch
  eng, _, rng = _index(3000, 20)
  q = rng.standard_normal((queries, 20)).astype(np.float32)
  want = eng.search_knn(q, 10, 40)
  a = torch.randn((4096, 4096), device="cuda")
  for stream in (torch.cuda.Stream(), torch.cuda.default_stream()):
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
      for _ in range(100):  # some tens of ms
        a = a @ a * 1e-2
      before = torch.cuda.Event()
      before.record(stream)
    eng.obj.set_stream(stream.cuda_stream)
    got = eng.search_knn(q, 10, 40)
    assert before.query()
    assert eng.obj.current_stream() == stream.cuda_stream
    assert (got[0] == want[0]).all() and (got[2] == want[2]).all()
    assert_same_bits(got[1], want[1])
  eng.obj.set_stream(0)


@pytest.mark.parametrize("n,d,row_dtype,max_m0", [(40_000, 104, "f32", 8), (33_001, 77, "f32", 64),
                                                  (50_001, 50, "f16", 33), (300, 9, "bf16", 8)])
def test_rows_graph_and_files_of_several_pieces(n, d, row_dtype, max_m0, tmp_path):
  """Rows with and without padding, 16-bit rows, adjacency tables and files of more than three pieces; a file saved
  over a longer one is cut to its length; small integers are exact in every row type."""
  eng, base, _ = _index(n, d, row_dtype=row_dtype, max_m0=max_m0)
  path = str(tmp_path / "x.index")
  with open(path, "wb") as out:
    out.write(b"\xff" * (n * (4 * d + 4 * max_m0 + 12) + (1 << 20)))
  eng.save_index(path)
  levels, rows0, rows_u = eng.obj.get_graph()
  g = index_file.load(path, "l2")
  assert (g.vec == base).all() and (g.levels == levels).all() and (g.rows0 == rows0).all()
  assert (g.rowsU == rows_u[:g.rowsU.shape[0]]).all() and (g.labels == np.arange(n)).all()
  labels = np.arange(n, dtype=np.int64) * (1 << 33) + 7
  index_file.save(path, g, g.header["mult"], g.header["ef_construction"], labels=labels)
  other = CuHNSW(engine_options(dict(dist_type="l2", row_dtype=row_dtype)))
  other.load_index(path)
  again = str(tmp_path / "y.index")
  other.save_index(again)
  assert open(path, "rb").read() == open(again, "rb").read()
  assert (other.obj.get_graph()[1] == rows0).all()


def test_an_interrupted_save_over_an_index_leaves_nothing_that_loads(tmp_path):
  """The write fails half way through a file of the same shape; a second name keeps what was written so far."""
  eng, _, _ = _index(30_000, 50)
  path, kept = str(tmp_path / "x.index"), str(tmp_path / "kept.index")
  eng.save_index(path)
  os.link(path, kept)
  whole = open(path, "rb").read()
  soft, hard = resource.getrlimit(resource.RLIMIT_FSIZE)
  resource.setrlimit(resource.RLIMIT_FSIZE, (len(whole) // 2, hard))
  try:
    with pytest.raises(RuntimeError, match="short write"):
      eng.save_index(path)
  finally:
    resource.setrlimit(resource.RLIMIT_FSIZE, (soft, hard))
  assert not os.path.exists(path) and os.path.getsize(kept) == len(whole)
  with pytest.raises(RuntimeError, match="index file"):
    CuHNSW(engine_options(dict(dist_type="l2"))).load_index(kept)
  eng.save_index(kept)
  assert open(kept, "rb").read() == whole


def test_an_index_saved_into_a_pipe_is_the_file_byte_for_byte(tmp_path):
  eng, _, _ = _index(30_000, 50)
  path, pipe = str(tmp_path / "x.index"), str(tmp_path / "pipe")
  eng.save_index(path)
  os.mkfifo(pipe)
  with concurrent.futures.ThreadPoolExecutor(1) as pool:
    got = pool.submit(lambda: open(pipe, "rb").read())
    eng.save_index(pipe)
    assert got.result() == open(path, "rb").read()


def test_calls_of_other_threads_do_not_wait_for_a_file_that_is_slow_to_write(tmp_path):
  """Three saves into pipes that nobody reads yet hold all page-locked buffers; everything else takes another way."""
  slow = [_index(150_000, 50)[0] for _ in range(3)]  # 37 MB, five pieces
  eng, base, rng = _index(60_000, 50)
  q = rng.standard_normal((40_000, 50)).astype(np.float32)
  path = str(tmp_path / "x.index")
  eng.save_index(path)
  want = eng.search_knn(q, 10, 40), eng.obj.get_graph()
  pipes = [str(tmp_path / f"pipe{i}") for i in range(3)]
  for p in pipes:
    os.mkfifo(p)
  with concurrent.futures.ThreadPoolExecutor(7) as pool:
    saves = [pool.submit(e.save_index, p) for e, p in zip(slow, pipes)]
    readers = [open(p, "rb") for p in pipes]  # returns when the save has opened its end

    def everything():
      time.sleep(1)
      eng.set_data(base)
      eng.build()
      few, many = eng.search_knn(q[:100], 10, 40), eng.search_knn(q, 10, 40)
      assert (few[0] == want[0][0][:100]).all() and (many[0] == want[0][0]).all()
      assert all((a == b).all() for a, b in zip(eng.obj.get_graph(), want[1]))
      eng.save_index(path + "2")
      eng.load_index(path + "2")

    try:
      pool.submit(everything).result(timeout=30)
      assert not any(s.done() for s in saves)
    finally:
      read = [pool.submit(r.read) for r in readers]
      for r, s in zip(read, saves):
        s.result()
        assert len(r.result()) > 4 * PIECE
  assert open(path, "rb").read() == open(path + "2", "rb").read()


def test_what_trails_an_index_in_its_file_is_not_read(tmp_path):
  """Link lists of several pieces of 4 MB, and a file with a hole of 6 GB behind them; cut within the lists it is
  refused."""
  rng = np.random.default_rng(3)
  n = 70_000
  eng = CuHNSW(engine_options(dict(dist_type="l2", max_m=32, max_m0=32, ef_construction=8, batch_max=4096)))
  eng.set_data(rng.integers(-8, 9, (n, 3)).astype(np.float32))
  eng.obj.set_random_levels((np.arange(n) % 2).astype(np.int32))
  eng.obj.build_graph()
  path = str(tmp_path / "x.index")
  eng.save_index(path)
  size, want = os.path.getsize(path), eng.obj.get_graph()
  assert size - 96 - n * (4 * 32 + 4 * 3 + 12) > (4 << 20)
  os.truncate(path, size + (6 << 30))
  other = CuHNSW(engine_options(dict(dist_type="l2")))
  before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
  other.load_index(path)
  assert resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before < (1 << 20)  # kB
  for a, b in zip(other.obj.get_graph(), want):
    assert (a == b).all()
  for cut in (1, (4 << 20) + 5):
    os.truncate(path, size - cut)
    with pytest.raises(RuntimeError, match="truncated"):
      other.load_index(path)


def test_a_smaller_corpus_hands_device_memory_back():
  import torch
  eng = CuHNSW(engine_options(dict(dist_type="l2")))
  rows = np.zeros((500_000, 104), np.float32)
  eng.set_data(rows)
  torch.cuda.synchronize()
  held = 500_000  # rows there is room for
  for n, room in ((500_000, 500_000), (300_000, 300_000), (280_000, 300_000), (240_000, 240_000)):
    before = torch.cuda.mem_get_info()[0]
    eng.set_data(rows[:n])
    torch.cuda.synchronize()
    given = torch.cuda.mem_get_info()[0] - before
    assert abs(given - (held - room) * 416) <= (4 << 20), (n, given)
    held = room


def test_what_a_build_keeps_goes_back_when_the_device_is_out_of_memory():
  """The scratch of the second build stays for a third; rows that fit the device only without it must still fit."""
  import torch
  eng, base, _ = _index(400_000, 8, max_m=12, max_m0=24)
  eng.build()
  graph = eng.obj.get_graph()
  torch.cuda.synchronize()
  fill = torch.empty(torch.cuda.mem_get_info()[0] - (24 << 20), dtype=torch.uint8, device="cuda")
  try:
    eng.set_data(np.tile(base, 4))  # 51 MB, 13 of them in the place of the former rows
  finally:
    del fill
    torch.cuda.empty_cache()
  eng.set_data(base)
  eng.build()
  for a, b in zip(eng.obj.get_graph(), graph):
    assert (a == b).all()


@pytest.mark.parametrize("rows,d", [(1, 3), (40_000, 50), (42_000, 50), (70_001, 33)])
def test_set_data_copies_and_normalises_like_one_thread(rows, d):
  """Below and above the size from which several threads share the work; a second corpus over the first."""
  rng = np.random.default_rng(rows)
  eng = CuHNSW(engine_options(dict(dist_type="dot", nrz=True)))
  for _ in range(2):
    x = rng.standard_normal((rows, d))
    eng.set_data(x)
    want = np.array(x, dtype=np.float32)
    want /= np.linalg.norm(want, axis=1, keepdims=True)
    assert_same_bits(eng.data, want)
  kept = eng.data
  before = kept.copy()
  eng.set_data(-x)
  assert_same_bits(kept, before)  # an array the caller holds is not written over
