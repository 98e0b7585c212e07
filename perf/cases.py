"""The work a program has this engine do, as timed cases: searches from one query to a hundred thousand, batches in
flight, searches on device buffers, construction, and the index file in both directions.

A case is a dict of plain values:

  kind    "search"  ``CuHNSW.search_knn`` on numpy arrays
          "stream"  ``CuHNSW.search_knn_batches``: ``batches`` arrays of ``nq`` queries each
          "device"  ``search_knn_device``: queries and results are CUDA tensors, nothing is copied
          "build"   ``set_data`` + ``build`` of a corpus that is in host memory
          "save"    ``save_index``
          "load"    ``load_index``
  data    "angular"  Gaussian mixture, rows L2-normalised by the engine (``nrz``), dot product
          "integer"  whole numbers 0..255 (image descriptors), squared L2
          "uniform"  tight clusters around uniform centres (long descriptors), squared L2
  n, d    rows and dimensions;  m, efc  ``max_m`` (``max_m0`` is twice that) and ``ef_construction``
  row     storage type of the rows;  save_remains, coef  options of the neighbour selection
  nq, k, ef  queries, results per query, ``ef_search``
"""
import math
import os
import tempfile

import numpy as np
import torch

from cuhnsw_b200 import CuHNSW


def _case(name, kind, data, n, d, m, efc, nq=0, k=0, ef=0, batches=1, row="f32", save_remains=False, coef=0.25):
  return dict(name=name, kind=kind, data=data, n=n, d=d, m=m, efc=efc, nq=nq, k=k, ef=ef, batches=batches, row=row,
              save_remains=save_remains, coef=coef)


def listed():
  return [
    # one user, one question: a single vector against a small corpus (the toy configuration of the benchmark)
    _case("one query", "search", "angular", 100_000, 50, 12, 110, nq=1, k=10, ef=300),
    # a web request or a re-ranking step: a few dozen queries at once, rows in half precision, ragged count
    _case("37 queries, f16 rows", "search", "angular", 300_000, 96, 16, 100, nq=37, k=10, ef=128, row="f16"),
    # a model on the same GPU looks up neighbours of its own embeddings: CUDA tensors in and out
    _case("1000 queries on the device", "device", "integer", 500_000, 128, 16, 200, nq=1000, k=10, ef=128),
    # the benchmark's headline: one 10 000-query batch from host memory at the ef that reaches recall@10 0.95
    _case("10000 queries", "search", "angular", 1_183_514, 50, 12, 110, nq=10_000, k=10, ef=200),
    # the same with 512-byte rows, whole-number data (exact ties) and its configuration's largest ef
    _case("10000 queries, 128-d", "search", "integer", 1_000_000, 128, 16, 200, nq=10_000, k=10, ef=256),
    # GIST-like rows: 3840 bytes each, few queries
    _case("1000 queries, 960-d", "search", "uniform", 150_000, 960, 16, 200, nq=1000, k=10, ef=300),
    # a serving loop: batch after batch, several in flight
    _case("batches in flight", "stream", "angular", 1_183_514, 50, 12, 110, nq=5_000, k=10, ef=100, batches=8),
    # offline join: every row of a table against the index, a hundred neighbours each (the walk-through's protocol)
    _case("100000 queries, top 100", "search", "angular", 1_000_000, 96, 16, 100, nq=100_000, k=100, ef=128, row="bf16"),
    # a small corpus indexed from scratch, as a program does at start-up
    _case("small build", "build", "angular", 100_000, 50, 12, 110, coef=0.0),
    # a full corpus indexed from scratch
    _case("large build", "build", "integer", 1_000_000, 128, 16, 200),
    # the index file, out and in
    _case("save", "save", "angular", 250_000, 96, 16, 100),
    _case("load", "load", "angular", 250_000, 96, 16, 100),
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["search"] * 5 + ["device"] * 2 + ["stream", "build", "build", "save", "load"])
  data = rng.choice(["angular", "angular", "integer", "uniform"])
  d = {"angular": _log_int(rng, 16, 128), "integer": _log_int(rng, 32, 128), "uniform": _log_int(rng, 129, 1024)}[data]
  files = kind in ("save", "load")
  n = _log_int(rng, 20_000, min(1_200_000, (26_000_000 if files else 128_000_000) // d))
  m = rng.choice([8, 12, 16, 24])
  efc = rng.choice([64, 100, 110, 150, 200])
  row = rng.choice(["f32", "f32", "f16", "bf16"])
  case = _case("", kind, data, n, d, m, efc, row=row, save_remains=rng.random() < 0.25,
               coef=rng.choice([0.0, 0.25, 0.25]))
  if kind in ("search", "device", "stream"):
    case["ef"] = _log_int(rng, 40, 400)
    case["k"] = min(case["ef"], rng.choice([1, 5, 10, 10, 20, 50, 100]))
    # no drawn search walks more than the largest listed one
    most = min(100_000, 12_800_000 // case["ef"]) if d <= 128 else min(2_000, 400_000 // case["ef"])
    if kind == "stream":
      case["batches"] = rng.randint(3, 10)
      most = min(10_000, most // case["batches"])
    case["nq"] = _log_int(rng, 200 if kind == "stream" and most > 400 else 1, most)
  del case["name"]
  return case


def _options(case):
  return dict(dist_type="dot" if case["data"] == "angular" else "l2", nrz=case["data"] == "angular", max_m=case["m"],
              max_m0=2 * case["m"], ef_construction=case["efc"], level_mult=1.0 / math.log(2 * case["m"]), seed=777,
              row_dtype=case["row"], save_remains=case["save_remains"], heuristic_coef=case["coef"],
              c_log_level=1, py_log_level=1)


class _Source:
  """Rows and queries of one seed: draws from one mixture, as host arrays."""

  def __init__(self, case, seed):
    self.case = case
    self.gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, d = case["data"], case["d"]
    count = {"angular": max(50, case["n"] // 1000), "integer": 256, "uniform": 500}[kind]
    if kind == "angular":
      self.centres = torch.randn((count, d), generator=self.gen, device="cuda")
    elif kind == "integer":
      self.centres = torch.randint(0, 96, (count, d), generator=self.gen, device="cuda").float()
    else:
      self.centres = torch.rand((count, d), generator=self.gen, device="cuda")

  def rows(self, count):
    kind, d = self.case["data"], self.case["d"]
    out = np.empty((count, d), np.float32)
    step = max(1, (32 << 20) // d)
    for lo in range(0, count, step):
      hi = min(count, lo + step)
      c = self.centres[torch.randint(0, len(self.centres), (hi - lo,), generator=self.gen, device="cuda")]
      x = torch.randn((hi - lo, d), generator=self.gen, device="cuda")
      if kind == "angular":
        x = c + 0.3 * x
      elif kind == "integer":
        x = (c + 40.0 * x.abs()).round().clamp(0, 255)
      else:
        x = c + 0.05 * x
      torch.from_numpy(out[lo:hi]).copy_(x)
    return out

  def queries(self, count):
    q = self.rows(count)
    return q / np.linalg.norm(q, axis=1, keepdims=True) if self.case["data"] == "angular" else q


class _State:
  pass


def prepare(case, seed):
  s = _State()
  s.case = case
  source = _Source(case, seed)
  rows = source.rows(case["n"])
  s.index = CuHNSW(_options(case))
  kind = case["kind"]
  if kind == "build":
    s.rows = rows
    return s
  s.index.set_data(rows)
  s.index.build()
  if kind in ("save", "load"):
    s.folder = tempfile.TemporaryDirectory()
    s.path = os.path.join(s.folder.name, "corpus.index")
    if kind == "load":
      s.index.save_index(s.path)
      s.index = CuHNSW(_options(case))
  elif kind == "stream":
    s.queries = [source.queries(case["nq"]) for _ in range(case["batches"])]
  else:
    s.queries = source.queries(case["nq"])
    if kind == "search" and case["nq"] == 1:
      s.queries = s.queries[0]
  if kind == "device":
    s.queries = torch.from_numpy(s.queries).cuda()
    s.ids = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
    s.distances = torch.empty((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
    s.found = torch.empty((case["nq"],), dtype=torch.int32, device="cuda")
    s.index.obj.set_stream(torch.cuda.current_stream().cuda_stream)
  return s


def run(s):
  case, kind = s.case, s.case["kind"]
  if kind == "search":
    return s.index.search_knn(s.queries, case["k"], case["ef"])
  if kind == "stream":
    return [part for batch in s.index.search_knn_batches(s.queries, case["k"], case["ef"]) for part in batch]
  if kind == "device":
    s.index.obj.search_knn_device(s.queries.data_ptr(), case["nq"], case["k"], case["ef"], s.ids.data_ptr(),
                                  s.distances.data_ptr(), s.found.data_ptr())
    return s.ids, s.distances, s.found
  if kind == "build":
    s.index.set_data(s.rows)
    s.index.build()
    return s.index.obj.get_graph()  # levels, layer-0 rows, upper rows
  if kind == "save":
    s.index.save_index(s.path)
    return np.memmap(s.path, dtype=np.uint8, mode="r")
  s.index.load_index(s.path)
  return s.index.obj.get_graph()


def work(case):
  """Bytes and operations of one pass.  A walk of width ef expands about ef nodes (one adjacency row each) and meets
  about 5.3 new rows per expansion; an inserted node evaluates about 9.2 rows and touches about 1.3 adjacency rows
  per unit of ef_construction (counted on the benchmark's configurations by the CPU restatement)."""
  n, d, links = case["n"], case["d"], 4 * (2 * case["m"] + 1)
  row = d * (4 if case["row"] == "f32" else 2)
  kind = case["kind"]
  if kind == "build":
    rows = 9.2 * case["efc"] * n
    return dict(bytes=rows * row + 1.3 * case["efc"] * n * 2 * links + 4 * n * d, flops=2 * d * rows)
  if kind in ("save", "load"):
    return dict(bytes=n * (4 * d + links + 8) + n * (row + links), flops=0)
  nq = case["nq"] * case["batches"]
  rows = min(n, 5.3 * case["ef"])
  return dict(bytes=nq * (rows * row + min(n, case["ef"]) * links + 4 * d + 8 * case["k"]), flops=nq * 2 * d * rows)


def tolerance(case):
  """Ids, counts, links and file bytes are whole numbers, and the order of the fp32 sums of a distance is part of
  the engine's contract, so distances are the same bits too."""
  return "exact"
