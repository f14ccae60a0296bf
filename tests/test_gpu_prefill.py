"""The tensor-core (tcgen05) matmul for many rows against the oracle's fp32 NumPy matmul over the same dequantised
weights: max relative error 1e-2 for bf16 results, 1e-4 for fp32 results (relative error as in docs/workload.md:141)."""
import ctypes
import numpy as np
import pytest
from oracle import bfp_oracle as o
from helpers import acts, bf16, check_matmul, upload, weights

pytestmark = pytest.mark.gpu


def deq(w, fmt):
  """The oracle's dequantised weights for any N: columns padded with zeros to whole tiles, as the tensor stores them."""
  pad = -w.shape[1] % 32
  return o.dequant(np.pad(w, ((0, 0), (0, pad))), fmt)[:, :w.shape[1]]


def many_rows(rt, tx, tw, tw2, add, epilogue, alpha, dtype):
  """The kernel for many rows (bt_gemm_bfp, x laid out by rows for it), whatever Tensor's rule would take."""
  from baretile_b200.tensor import EPILOGUE, FMT_CODE, Tensor
  m, k = tx.rows, tx.tc * 32
  rows, out = rt.dram_alloc(2 * m * k), Tensor(rt, m, tw.cols, dtype=dtype or "bf16")
  rt.launch("bt_untilize", (2, tx.addr, rows, 1, m, k), name="rows")
  rt.launch("bt_gemm_bfp", (FMT_CODE[tw.dtype], EPILOGUE[epilogue], m, k, tw.cols, rows, tw.addr, tw2.addr if tw2 is not None else 0, add.addr if add is not None else 0,
                            add.rows if add is not None else 0, 1.0 if alpha is None else alpha, out.addr, FMT_CODE[out.dtype], rt.work), name="many rows")
  rt.dram_free(rows)
  return out.numpy()


def run(rt, x, w, fmt, epilogue="none", w2=None, dtype=None, add=None, alpha=None):
  """The matmul as an expression, which takes the kernel that the rule expects to be the faster one, and by the kernel for many rows beside it:
  both within the bounds, and both exact where the one is."""
  tx, tw, tadd = upload(rt, x), upload(rt, w).cast(fmt).columns(), upload(rt, add) if add is not None else None
  tw2 = upload(rt, w2).cast(fmt).columns() if w2 is not None else None
  y, ref = tx.matmul(tw, dtype=dtype), x.astype(np.float32) @ deq(w, fmt)
  if alpha is not None: y, ref = y * alpha, ref * np.float32(alpha)
  if add is not None: y, ref = y + tadd, ref + add
  if epilogue == "relu": y, ref = y.relu(), np.maximum(ref, 0)
  elif epilogue == "silu": y, ref = y.silu(), o.silu(ref)
  elif epilogue == "glu": y, ref = y.silu() * tx.matmul(tw2, dtype=dtype), o.silu(ref) * (x.astype(np.float32) @ deq(w2, fmt))
  rt.log = []
  got = y.realize()
  rt.wait()
  names, rt.log = [n for *_, n in rt.log], None
  assert sum(n.startswith("prefill") for n in names) == 1, names    # a tensor-core kernel ran, once, not the decode loop
  out, many, tol = got.numpy(), many_rows(rt, tx, tw, tw2, tadd, epilogue, alpha, dtype), 1e-2 if dtype != "fp32" else 1e-4
  for result in (out, many):
    # every element of a linear or ReLU result within 2^-8 of sum |x||w| (+ |addend|): the reference's per-element bound
    linear = epilogue in ("none", "relu")
    check_matmul(result, x, deq(w, fmt) if linear else None, ref, tol, addend=add if linear else None, alpha=alpha if alpha is not None else 1.0)
  if np.array_equal(out, ref): assert np.array_equal(many, ref)
  return out, ref


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_exact_integers_pin_the_operand_layouts(rt, fmt):
  # small integers are exact in both formats and in fp32 sums: any misplaced row, column or k shows up
  rng = np.random.default_rng(1)
  x = rng.integers(-2, 3, (256, 128)).astype(np.float32)
  w = rng.integers(-1, 2, (128, 256)).astype(np.float32)
  got, ref = run(rt, x, w, fmt, dtype="fp32")
  assert np.array_equal(got, x @ w)
  eye = np.zeros((256, 256), np.float32)
  eye[np.arange(256), np.arange(256)] = 1
  xr = bf16(rng.uniform(-8, 8, (200, 256)))
  got, _ = run(rt, xr, eye, fmt)
  assert np.array_equal(got, xr)                                   # A @ I == A, with a ragged last block of rows


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m", [33, 128, 300, 512])
def test_rows(rt, fmt, m):
  rng = np.random.default_rng(m)
  x, w = acts(rng, m, 1024), weights(rng, 1024, 512)
  got, ref = run(rt, x, w, fmt)
  check_matmul(got, x, None, ref, 1e-2)
  got, ref = run(rt, x, w, fmt, "relu", dtype="fp32")
  check_matmul(got, x, None, ref, 1e-4)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_gate_up_pair(rt, fmt):
  rng = np.random.default_rng(4)
  x, w, w2 = acts(rng, 384, 512), weights(rng, 512, 640), weights(rng, 512, 640)
  got, ref = run(rt, x, w, fmt, "glu", w2)
  check_matmul(got, x, None, ref, 1e-2)


def test_config2_shapes_reduced_rows(rt):
  # the prefill configuration's weights at full size (4096 x 14336 gate/up in bfp8, 14336 x 4096 down in bfp4), 256 rows
  rng = np.random.default_rng(2)
  x = acts(rng, 256, 4096)
  wg, wu = weights(rng, 4096, 14336), weights(rng, 4096, 14336)
  got, ref = run(rt, x, wg, "bfp8", "glu", wu)
  check_matmul(got, x, None, ref, 1e-2)
  h = bf16(ref)
  wd = weights(rng, 14336, 4096)
  got, ref = run(rt, h, wd, "bfp4")
  check_matmul(got, h, None, ref, 1e-2)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_addend_and_scale(rt, fmt):
  # a bias row and a residual of M rows, added before the activation; a scale; fp32 results
  rng = np.random.default_rng(5)
  x, w = acts(rng, 300, 256), weights(rng, 256, 512)
  bias, resid = bf16(rng.normal(0, 1, (1, 512))), bf16(rng.normal(0, 1, (300, 512)))
  for add in (bias, resid):
    got, ref = run(rt, x, w, fmt, "relu", add=add)
    check_matmul(got, x, None, ref, 1e-2)
    got, ref = run(rt, x, w, fmt, "silu", add=add)
    check_matmul(got, x, None, ref, 1e-2)
  got, ref = run(rt, x, w, fmt, alpha=0.5, add=resid, dtype="fp32")
  check_matmul(got, x, None, ref, 1e-4)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("k,n", [(96, 96), (160, 1000), (1024, 416), (80, 130), (64, 32), (32, 4128)])
def test_shapes_that_are_not_whole_blocks(rt, fmt, k, n):
  # a last run of fewer than four tile columns, a block column with one run, an odd last tile row of K, and K and N
  # that are not whole tiles: all through the one kernel, exact on small integers and within tolerance on weights
  rng = np.random.default_rng(k * 7 + n)
  xi, wi = rng.integers(-2, 3, (70, k)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32)
  got, _ = run(rt, xi, wi, fmt, dtype="fp32")
  assert np.array_equal(got, xi @ wi)
  x, w, w2 = acts(rng, 300, k), weights(rng, k, n, stress=False), weights(rng, k, n, stress=False)
  add = bf16(rng.normal(0, 1, (300, n)))
  got, ref = run(rt, x, w, fmt, "relu", add=add)
  check_matmul(got, x, None, ref, 1e-2)
  got, ref = run(rt, x, w, fmt, "glu", w2)
  check_matmul(got, x, None, ref, 1e-2)


@pytest.mark.parametrize("epilogue", ["none", "glu"])
def test_without_room_for_parts_of_k(rt, monkeypatch, epilogue):
  # a device with room for x by rows but not for the parts: the matmul runs all the same, and one that has no room for x by
  # rows either says so. (The kernel for few rows, which this size takes, uses neither; test_parts_of_k_in_memory does the same where both are used.)
  rng = np.random.default_rng(5)
  m, k, n = 77, 2048, 544
  x, w, w2 = acts(rng, m, k), weights(rng, k, n), weights(rng, k, n)
  tx, tw, tw2 = upload(rt, x), upload(rt, w).cast("bfp8").columns(), upload(rt, w2).cast("bfp8").columns()
  asked, alloc = [], rt.dram_alloc
  def tight(size, limit=2 * m * k):
    asked.append(size)
    if size > limit: raise MemoryError(f"no {size} bytes free in DRAM")
    return alloc(size)
  def expression(): return (tx @ tw) if epilogue == "none" else (tx @ tw).silu() * (tx @ tw2)
  monkeypatch.setattr(rt, "dram_alloc", tight)
  y = expression().realize()
  assert asked[-2] > asked[-1] == 2 * m * k
  monkeypatch.setattr(rt, "dram_alloc", lambda size: tight(size, 2 * m * k - 1))
  with pytest.raises(MemoryError, match="bytes free"): expression().realize()
  monkeypatch.undo()
  ref = x @ o.dequant(w, "bfp8")
  if epilogue == "glu": ref = o.silu(ref) * (x @ o.dequant(w2, "bfp8"))
  check_matmul(y.numpy(), x, o.dequant(w, "bfp8") if epilogue == "none" else None, ref, 1e-2)


def test_results_stay_inside_their_tiles(rt):
  # the tensors either side of a result in device memory keep their bytes (ragged rows and columns included)
  from baretile_b200.tensor import Tensor
  from helpers import raw_tiles
  rng = np.random.default_rng(9)
  x, w = acts(rng, 70, 96), weights(rng, 96, 130, stress=False)
  tx, tw = upload(rt, x), upload(rt, w).cast("bfp8").columns()
  before = upload(rt, np.full((32, 32), 3.0, np.float32))
  y = (tx @ tw).realize()
  after = upload(rt, np.full((32, 32), 5.0, np.float32))
  y2 = (tx @ tw).relu().realize()
  assert np.all(before.numpy() == 3.0) and np.all(after.numpy() == 5.0)
  assert np.array_equal(np.maximum(y.numpy(), 0), y2.numpy())
  tiles = raw_tiles(rt, y).view(np.uint16).reshape(3, 5, 1024)
  full = o.untilize(tiles.reshape(15, 1024), 1, 96, 160)[0]
  assert not full[70:].any() and not full[:, 130:].any()            # rows past M and columns past N are zero


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m,k,n", [(33, 64, 32), (33, 4096, 64), (77, 2080, 330), (256, 1024, 128), (257, 2112, 96), (300, 8192, 288), (520, 1536, 1000)])
def test_shared_k_and_half_blocks(rt, fmt, m, k, n):
  # few blocks of 256 rows and an odd last tile row, every epilogue. The expression takes the kernel for few rows, whose clusters share K; `run` gives
  # the kernel for many rows no room for parts of K (test_parts_of_k_in_memory has sizes that take them)
  rng = np.random.default_rng(m + k + n)
  xi, wi = rng.integers(-2, 3, (m, k)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32)
  got, _ = run(rt, xi, wi, fmt, dtype="fp32")
  assert np.array_equal(got, xi @ wi)
  x, w, w2 = acts(rng, m, k), weights(rng, k, n, stress=False), weights(rng, k, n, stress=False)
  for add in (bf16(rng.normal(0, 1, (1, n))), bf16(rng.normal(0, 1, (m, n)))):
    got, ref = run(rt, x, w, fmt, "relu", add=add, alpha=0.5)
    check_matmul(got, x, None, ref, 1e-2)
  got, ref = run(rt, x, w, fmt, "silu", dtype="fp32")
  check_matmul(got, x, None, ref, 1e-4)
  got, ref = run(rt, x, w, fmt, "glu", w2)
  check_matmul(got, x, None, ref, 1e-2)


@pytest.mark.parametrize("fmt,m,k,n,pair", [("bfp8", 33, 18784, 70, True), ("bfp4", 300, 18016, 100, True), ("bfp8", 330, 23968, 58, True),
                                            ("bfp4", 400, 8992, 2900, False), ("bfp8", 300, 11040, 4000, False), ("bfp4", 1442, 12096, 1935, False)])
def test_parts_of_k_in_memory(rt, monkeypatch, fmt, m, k, n, pair):
  """Sizes at which pairs of CTAs share K through memory (gemm_kernel and reduce_kernel, after a launch that lays x out by rows): blocks of 256 and 512 rows, 2 to 16
  parts, an odd last tile row in the last part. And the same without room for the parts, and without any."""
  from baretile_b200 import _lib
  rng = np.random.default_rng(m + k + n)
  def launches():
    count = ctypes.c_uint64()
    _lib.call("bt_launch_count", ctypes.byref(count))
    return count.value
  def ints(a, b, *shape): return rng.integers(a, b, shape).astype(np.float32)
  w, v = ints(-1, 2, k, n), ints(-1, 2, k, n) if pair else None
  tw, tv = upload(rt, w).cast(fmt).columns(), upload(rt, v).cast(fmt).columns() if pair else None
  def split(expression):
    before = launches()
    y = expression.realize()
    assert launches() - before == 3
    return y.numpy()
  # small integers: fp32 sums are exact in any order, and so is a wide scale; values for the activations
  xi, x = ints(-2, 3, m, k), bf16(rng.normal(0, 1 / np.sqrt(k), (m, k)))
  ti, tx = upload(rt, xi), upload(rt, x)
  if pair:
    ref = o.silu(x @ w) * (x @ v)
    check_matmul(split(tx.matmul(tw, dtype="fp32").silu() * tx.matmul(tv, dtype="fp32")), x, None, ref, 1e-4)
    expression = lambda: (tx @ tw).silu() * (tx @ tv)
    check_matmul(split(expression()), x, None, ref, 1e-2)
  else:
    exact, bias, resid = xi @ w, ints(-9, 10, 1, n), ints(-9, 10, m, n)
    tb, tr = upload(rt, bias), upload(rt, resid)
    assert np.array_equal(split(ti.matmul(tw, dtype="fp32")), exact)
    assert np.array_equal(split((ti.matmul(tw, dtype="fp32") * 0.5 + tr).relu()), np.maximum(exact * 0.5 + resid, 0))
    assert np.array_equal(split(ti.matmul(tw, dtype="fp32") + tb), exact + bias)
    ref = o.silu(x @ w + bias)
    expression = lambda: ((tx @ tw) + tb).silu()
    check_matmul(split(expression()), x, None, ref, 1e-2)
  alloc = rt.dram_alloc
  def tight(size, limit=-(-2 * m * k // 256) * 256):
    if size > limit: raise MemoryError(f"no {size} bytes free in DRAM")
    return alloc(size)
  monkeypatch.setattr(rt, "dram_alloc", tight)
  before = launches()
  y = expression().realize()
  assert launches() - before <= 2
  monkeypatch.setattr(rt, "dram_alloc", lambda size: tight(size, 2 * m * k - 1))
  with pytest.raises(MemoryError, match="bytes free"): expression().realize()
  monkeypatch.undo()
  check_matmul(y.numpy(), x, None, ref, 1e-2)
