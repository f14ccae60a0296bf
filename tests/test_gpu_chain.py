"""Chains of small matmuls (chain_kernel): a list whose matmuls read one another through the exchange against one launch per
matmul, bit for bit, and against the oracle. Every size sits at an edge: sub-panels of 1, 2 and 4 tile columns, fewer tile rows
than warps, the last tile row of a warp's first and second batch, partial last columns, 1 to 8 tokens. (64 x 9600: its down projection is
not small, so that the list runs in the general kernel, and has to give the same bits.)"""
import ctypes
import numpy as np
import pytest
from oracle import bfp_oracle as o
from helpers import acts, bf16, check_matmul, upload, weights

pytestmark = pytest.mark.gpu


def layers(x, ws, steps):
  """steps of (projection, gate/up pair, down projection) with residuals, as a decoder has them; every result."""
  out = []
  for _ in range(steps):
    a = ((x @ ws[0]) + x).realize()
    h = ((a @ ws[1]).silu() * (a @ ws[2])).realize()
    x = ((h @ ws[3]) + a).realize()
    out += [a, h, x]
  return out


@pytest.mark.parametrize("m,d,f,fmt", [(1, 32, 32, "bfp8"), (1, 576, 1536, "bfp8"), (2, 256, 300, "bfp4"), (3, 700, 1500, "bfp4"), (5, 480, 1568, "bfp8"),
                                       (8, 576, 1536, "bfp8"), (4, 64, 5024, "bfp8"), (1, 96, 3072, "bfp4"), (2, 64, 9600, "bfp8"), (7, 1000, 1000, "bfp8"), (8, 640, 1160, "bfp4")])
def test_chain_equals_separate_launches(rt, m, d, f, fmt):
  rng = np.random.default_rng(m * d + f)
  shapes = (d, d), (d, f), (d, f), (f, d)
  host = [weights(rng, *s) for s in shapes]
  ws = [upload(rt, w).cast(fmt).columns() for w in host]
  hx = acts(rng, m, d)
  x = upload(rt, hx)
  separate = [t.numpy() for t in layers(x, ws, 4)]
  with rt.queue(): queued = layers(x, ws, 4)
  with rt.record() as step: held = layers(x, ws, 4)
  for _ in range(3): step.replay()
  rt.wait()
  for got, again, want in zip(queued, held, separate):
    assert np.array_equal(got.numpy(), want) and np.array_equal(again.numpy(), want)
  step.close()
  # and against the oracle: every matmul from the inputs that it had
  wd = [o.dequant(np.pad(w, ((0, 0), (0, -w.shape[1] % 16))), fmt)[:, :w.shape[1]] for w in host]
  a, h, y = separate[:3]
  check_matmul(a, hx, wd[0], hx @ wd[0] + hx, addend=hx)
  check_matmul(h, None, None, o.silu(a @ wd[1]) * (a @ wd[2]))
  check_matmul(y, h, wd[3], h @ wd[3] + a, addend=a)


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
@pytest.mark.parametrize("m", [1, 6])
def test_chain_with_breaks(rt, m, dtype):
  """A list in which some matmuls do not read the one before: other inputs, another activation, a bias row, fp32 results."""
  rng = np.random.default_rng(m)
  w, v = (upload(rt, weights(rng, 288, n)).cast("bfp8").columns() for n in (288, 160))
  x, z, bias = upload(rt, acts(rng, m, 288)), upload(rt, acts(rng, m, 288)), upload(rt, acts(rng, m, 288))
  def some():
    a = (x @ w).relu().realize()
    b = (z.matmul(v, dtype=dtype) * 0.5).realize()
    c = ((a @ w) + bias).realize()
    e = (c @ w).silu().realize()
    return [a, b, c, e, ((e @ w) + c).realize(), (e @ v).realize(), ((a @ w) + e).realize()]
  separate = [t.numpy() for t in some()]
  with rt.queue(): queued = some()
  rt.wait()
  for got, want in zip(queued, separate): assert np.array_equal(got.numpy(), want)


def test_chain_results_reuse_memory(rt):
  """Results freed as soon as they are used: their memory comes back as a later matmul's result of the same list."""
  rng = np.random.default_rng(3)
  w = upload(rt, weights(rng, 320, 320) * 3).cast("bfp8").columns()
  x = upload(rt, acts(rng, 2, 320))
  def chain():
    y = x
    for _ in range(40): y = ((y @ w) + y).relu().realize()
    return y
  want = chain().numpy()
  with rt.queue(): got = chain()
  assert np.array_equal(got.numpy(), want)


@pytest.mark.parametrize("m,d,f,up,down,wide", [(8, 1152, 1024, "bfp4", "bfp8", 0), (8, 1152, 1024, "bfp8", "bfp4", 0), (8, 1152, 1024, "bfp4", "bfp4", 9600),
                                                (8, 1344, 1024, "bfp4", "bfp8", 0), (3, 576, 1536, "bfp4", "bfp8", 9600), (1, 1152, 1024, "bfp8", "bfp4", 9500)])
def test_chain_of_stages_that_differ(rt, m, d, f, up, down, wide):
  """Both formats in a list, and sub-panels of four tile columns (`wide`) among narrow ones: stages of 18, 34 and 36 KB in a ring that may have no
  room for two of them."""
  rng = np.random.default_rng(m + d + wide)
  gate, lift, back, side = (upload(rt, weights(rng, *s, stress=False)).cast(fmt).columns() for s, fmt in (((d, f), up), ((d, f), up), ((f, d), down), ((96, wide or 32), "bfp4")))
  x, z = upload(rt, acts(rng, m, d)), upload(rt, acts(rng, m, 96))
  def run():
    y, out = x, []
    for _ in range(5):
      if wide: out.append((z @ side).realize())
      h = ((y @ gate).silu() * (y @ lift)).realize()
      y = ((h @ back) + y).realize()
      out += [h, y]
    return out
  separate = [t.numpy() for t in run()]
  with rt.queue(): queued = run()
  rt.wait()
  for got, want in zip(queued, separate): assert np.array_equal(got.numpy(), want)


def test_tags_start_over(rt):
  """The launch's number, a word of the workspace (kWsEpoch in csrc/gemv.cu), at its last value: the exchanges are cleared and it starts over."""
  rng = np.random.default_rng(4)
  w = upload(rt, weights(rng, 320, 320)).cast("bfp8").columns()
  x = upload(rt, acts(rng, 2, 320))
  def chain():
    y = x
    for _ in range(6): y = (y @ w).realize()
    return y
  want = chain().numpy()
  number = lambda: int.from_bytes(rt.download(rt.work + 148, 4), "little")
  rt.wait()
  rt.upload(rt.work + 148, ((1 << 26) - 2).to_bytes(4, "little"))
  for after in ((1 << 26) - 1, 0, 1, 2):
    with rt.queue(): got = chain()
    assert np.array_equal(got.numpy(), want)
    assert number() == after


def test_exact_weights(rt):
  """Weights near both ends of bf16's range, which the expansion holds exactly."""
  for scale in (2.0 ** 100, 2.0 ** -100):
    w = bf16(np.random.default_rng(5).integers(-60, 61, (64, 64)) * scale)
    x = bf16(np.random.default_rng(6).integers(-3, 4, (2, 64)))
    got = upload(rt, x).matmul(upload(rt, w).cast("bfp8").columns(), dtype="fp32").numpy()
    assert np.array_equal(got.astype(np.float64), x.astype(np.float64) @ o.dequant(w, "bfp8").astype(np.float64))


@pytest.mark.parametrize("m,k,n", [(1, 64, 96), (3, 96, 64), (8, 64, 4096)])
def test_addend_wider_than_the_matmul_before(rt, m, k, n):
  """x and the addend start at the same place, and the addend goes on past what the matmul before has written there."""
  from baretile_b200 import _lib
  from baretile_b200.tensor import Tensor
  rng = np.random.default_rng(m + n)
  w, v = (upload(rt, weights(rng, k, c, stress=False)).cast("bfp8").columns() for c in (k, n))
  x, wide = upload(rt, acts(rng, m, k)), acts(rng, m, max(k, n))
  def run(queued):
    y, z = upload(rt, wide), Tensor(rt, m, n)
    ops = [_lib.GemvOp(fmt=8, epilogue=0, M=m, K=k, N=c, out_dtype=0, alpha=1.0, x=a, w=b.addr, add=add, out=to)
           for c, a, b, add, to in ((k, x.addr, w, 0, y.addr), (n, y.addr, v, y.addr, z.addr))]
    for some in ([ops] if queued else [[o] for o in ops]): _lib.call("bt_gemv_queue", rt.device, len(some), (_lib.GemvOp * len(some))(*some), rt.work, rt.work_bytes, rt.stream)
    return z.numpy()
  assert np.array_equal(run(True), run(False))
