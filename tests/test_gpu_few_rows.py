"""The tensor-core matmul for few rows (weights expanded into tensor memory): edges of its token groups and blocks of rows, of sub-panels
of fewer than four tile columns, of stages and of the clusters that share K, against the oracle's dequantised weights; and the
rule that chooses it against the kernel for many rows."""
import numpy as np
import pytest
from oracle import bfp_oracle as o
from helpers import acts, bf16, check_matmul, upload, weights
from test_gpu_prefill import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m,k,n", [(33, 32, 32), (48, 64, 96), (49, 96, 128), (64, 128, 160), (65, 160, 320), (80, 1120, 64), (96, 288, 544), (97, 2048, 256),
                                   (112, 4128, 416), (113, 544, 1504), (127, 256, 2400), (128, 992, 4896), (128, 352, 9600), (129, 352, 544), (160, 1120, 96), (161, 544, 1504), (255, 96, 128), (256, 2080, 416)])
def test_edges(rt, fmt, m, k, n):
  # small integers are exact in both formats and in fp32 sums, whatever the order: any misplaced row, column or k shows up.
  # (All of these go to the kernel for few rows; `run` compares the other one with it.)
  rng = np.random.default_rng(m * 131 + k + n)
  xi, wi, vi = rng.integers(-2, 3, (m, k)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32)
  add = rng.integers(-9, 10, (m, n)).astype(np.float32)
  got, _ = run(rt, xi, wi, fmt, dtype="fp32")
  assert np.array_equal(got, xi @ wi)
  got, _ = run(rt, xi, wi, fmt, "relu", add=add, alpha=0.5, dtype="fp32")
  assert np.array_equal(got, np.maximum((xi @ wi) * 0.5 + add, 0))
  got, ref = run(rt, xi, wi, fmt, "glu", vi, dtype="fp32")
  check_matmul(got, xi, None, ref, 1e-4)


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m", [40, 128])
def test_same_bits_every_time(rt, fmt, m):
  # sums of parts of K are added in order: a result does not depend on timing, nor on what ran before it
  rng = np.random.default_rng(m)
  x, w, w2 = acts(rng, m, 1536), weights(rng, 1536, 640), weights(rng, 1536, 640)
  tx, tw, tw2 = upload(rt, x), upload(rt, w).cast(fmt).columns(), upload(rt, w2).cast(fmt).columns()
  first = ((tx @ tw).silu() * (tx @ tw2)).numpy()
  for _ in range(20):
    ys = [((tx @ tw).silu() * (tx @ tw2)).realize() for _ in range(3)]
    assert all(np.array_equal(y.numpy(), first) for y in ys)
  assert o.rel_err(first, o.silu(x @ o.dequant(w, fmt)) * (x @ o.dequant(w2, fmt))) <= 1e-2


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
def test_fp32_sums_are_no_further_from_64_bits(rt, fmt):
  # fp32 accumulation over K = 4096: an error of the sums of products within that of adding them one after the other,
  # K * 2^-24 of the sum of magnitudes (a bound; what is seen is a hundredth of it)
  rng = np.random.default_rng(11)
  x, w = acts(rng, 100, 4096), weights(rng, 4096, 256)
  got, _ = run(rt, x, w, fmt, dtype="fp32")
  wd = o.dequant(w, fmt).astype(np.float64)
  assert (np.abs(got - x.astype(np.float64) @ wd) <= 4096 * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(wd))).all()


def test_chain_and_recording(rt):
  # a gate/up pair and the matmul on its result back to back, live and replayed, between decode matmuls that read and write the same tensors
  rng = np.random.default_rng(3)
  x = upload(rt, acts(rng, 77, 512))
  wg, wu, wd = (upload(rt, weights(rng, *s)).cast("bfp8").columns() for s in ((512, 1408), (512, 1408), (1408, 512)))
  def mlp(x): return (((((x @ wg).silu() * (x @ wu)).realize() @ wd) + x).realize())
  want = mlp(mlp(x)).numpy()
  held = []
  with rt.record() as step:
    held.append(mlp(x)), held.append(mlp(held[-1]))
  for _ in range(3):
    step.replay()
    rt.wait()
    assert np.array_equal(held[-1].numpy(), want)
  step.close()


@pytest.mark.parametrize("fmt", ["bfp8", "bfp4"])
@pytest.mark.parametrize("m,k,n", [(33, 96, 130), (129, 544, 1000), (300, 4128, 96), (520, 352, 2080), (1000, 256, 4128), (2050, 1056, 9000)])
def test_the_same_as_the_kernel_for_many_rows(rt, fmt, m, k, n):
  # whichever kernel the rule takes: every epilogue, addend and result type, exactly as the other kernel has it on small integers
  from baretile_b200.tensor import FMT_CODE, Tensor
  rng = np.random.default_rng(m + k + n)
  x, w, v = rng.integers(-2, 3, (m, k)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32), rng.integers(-1, 2, (k, n)).astype(np.float32)
  tx, tw, tv = upload(rt, x), upload(rt, w).cast(fmt).columns(), upload(rt, v).cast(fmt).columns()
  adds = {0: None, 1: upload(rt, rng.integers(-9, 10, (1, n)).astype(np.float32)), m: upload(rt, rng.integers(-9, 10, (m, n)).astype(np.float32))}
  K = tx.tc * 32
  rows = rt.dram_alloc(2 * m * K)
  rt.launch("bt_untilize", (2, tx.addr, rows, 1, m, K), name="rows")
  for epilogue, add, dtype in (("none", 0, "fp32"), ("relu", m, "bf16"), ("none", 1, "bf16"), ("relu", 1, "fp32")):
    y = tx.matmul(tw, dtype=dtype)
    if add: y = y + adds[add]
    if epilogue == "relu": y = y.relu()
    want = Tensor(rt, m, n, dtype=dtype)
    a = adds[add]
    rt.launch("bt_gemm_bfp", (FMT_CODE[fmt], 1 if epilogue == "relu" else 0, m, K, n, rows, tw.addr, 0, a.addr if a is not None else 0, add, 1.0, want.addr, FMT_CODE[dtype], rt.work), name="many rows")
    assert np.array_equal(y.numpy(), want.numpy()), (epilogue, add, dtype)
  got = (tx.matmul(tw).silu() * tx.matmul(tv)).numpy()
  check_matmul(got, x, None, o.silu(x @ w) * (x @ v), 1e-2)
  rt.dram_free(rows)


@pytest.mark.parametrize("fmt,m", [("bfp8", 96), ("bfp8", 112), ("bfp4", 100)])
def test_first_call_on_new_weights(rt, fmt, m):
  # weights that come from memory for the first time arrive out of order: a warp must not take a place of the ring that has not been filled
  # yet for one that has
  rng = np.random.default_rng(m)
  x = upload(rt, acts(rng, m, 2048))
  raw = [upload(rt, weights(rng, 2048, 4160)) for _ in range(2)]
  for _ in range(40):
    wg, wu = (r.cast(fmt).columns() for r in raw)
    first, second = [((x @ wg).silu() * (x @ wu)).realize() for _ in range(2)]
    assert np.array_equal(first.numpy(), second.numpy())
