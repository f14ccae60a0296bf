"""The C-ABI boundary and the host-side mirror, without a GPU: the library loads and exports every symbol the header
declares, the Python bindings agree with the header, and argument checks run before anything touches a device."""
import ctypes, pathlib, random, re, subprocess, sys
import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
HEADER = (ROOT / "include" / "baretile_b200.h").read_text()


def declared():
  code = re.sub(r"/\*.*?\*/", "", HEADER, flags=re.S)
  return {m.group(2): m.group(3) for m in re.finditer(r"\b(int|const char \*)\s*(bt_\w+)\s*\(([^;]*)\)\s*;", code)}


@pytest.fixture(scope="module")
def built():
  so = ROOT / "baretile_b200" / "libbaretile_b200.so"
  if not so.exists():
    run = subprocess.run(["make", "-C", str(ROOT / "baretile_b200" / "csrc"), "-j4"], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
  return so


def test_library_exports_every_declared_symbol(built):
  lib, names = ctypes.CDLL(str(built)), declared()
  assert len(names) >= 25
  for name in names: assert hasattr(lib, name), f"{name} is declared in the header but not exported"


def test_bindings_match_header(built):
  from baretile_b200 import _lib
  names = declared()
  for name, argtypes in _lib.SIGNATURES.items():
    assert name in names, f"{name} is bound but not declared"
    params = [p for p in names[name].split(",") if p.strip() and p.strip() != "void"]
    assert len(params) == len(argtypes), (name, names[name])
  assert set(names) - set(_lib.SIGNATURES) == {"bt_last_error"}
  _lib.lib()


def test_argument_checks_need_no_device(built):
  from baretile_b200 import _lib
  n = ctypes.c_int(-1)
  _lib.call("bt_device_count", ctypes.byref(n))
  assert n.value >= 0
  with pytest.raises(ValueError, match="bfp8"): _lib.call("bt_pack_bfp", 0, 3, 256, 512, 1, 0)
  with pytest.raises(ValueError, match="1 to 32 rows"): _lib.call("bt_gemv_bfp", 0, 8, 0, 40, 64, 64, 256, 256, 0, 0, 1.0, 256, 0, 0, 0, 0, 256, 1 << 30, 0)
  with pytest.raises(ValueError, match="multiples of 32"): _lib.call("bt_gemv_bfp", 0, 8, 0, 8, 60, 64, 256, 256, 0, 0, 1.0, 256, 0, 0, 0, 0, 256, 1 << 30, 0)
  with pytest.raises(ValueError, match="GLU"): _lib.call("bt_gemv_bfp", 0, 8, 3, 8, 64, 64, 256, 256, 0, 0, 1.0, 256, 0, 0, 0, 0, 256, 1 << 30, 0)
  op = _lib.GemvOp(fmt=8, epilogue=0, M=8, K=64, N=60, out_dtype=0, alpha=1.0, x=256, w=256, out=256)
  with pytest.raises(ValueError, match="matmul 0: K and N"): _lib.call("bt_gemv_queue", 0, 1, ctypes.byref(op), 256, 1 << 30, 0)
  with pytest.raises(ValueError, match="at least one"): _lib.call("bt_gemv_queue", 0, 0, ctypes.byref(op), 256, 1 << 30, 0)
  assert b"at least one" in _lib.lib().bt_last_error()


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
  from baretile_b200 import _lib
  monkeypatch.setattr(_lib, "_lib", None)
  monkeypatch.setattr(_lib, "PATH", tmp_path / "libbaretile_b200.so")
  with pytest.raises(RuntimeError, match="no CPU fallback"): _lib.lib()


def test_tensor_checks_without_a_device():
  # bad calls raise ValueError before any allocation, also under python -O (reference: test/test_kernels.py:370-389)
  code = """
from baretile_b200.tensor import Tensor
class Runtime:
  def check(self): pass
  def dram_alloc(self, size): return 0
  def dram_free(self, addr): pass
rt = Runtime()
x, y = Tensor(rt, 2, 3), Tensor(rt, 2, 3)
for bad in (lambda: x @ y, lambda: x + Tensor(rt, 3, 2), lambda: Tensor.frombytes(rt, 1, 1, bytes(2), dtype="bfp8"),
            lambda: Tensor(rt, 0, 1), lambda: Tensor(rt, 1, 1, dtype="float64"), lambda: Tensor.of(rt, [[1, 2], [3]]),
            lambda: x.cast("int32") @ y, lambda: x.columns(), lambda: x.topk(1)):
  try: bad()
  except ValueError: continue
  raise SystemExit("no ValueError")
print("all raised")
"""
  run = subprocess.run([sys.executable, "-O", "-c", code], capture_output=True, text=True, timeout=120, cwd=ROOT)
  assert run.returncode == 0 and run.stdout.strip() == "all raised", run.stdout + run.stderr


class TightRuntime:
  """A runtime without a device that hands out addresses while there is room, and notes what is launched."""
  active, work, work_bytes, room = True, 1 << 40, 1 << 30, 1 << 62
  def __init__(self): self.used, self.launched, self.asked = {}, [], []
  def check(self):
    if not self.active: raise RuntimeError("runtime is closed or was replaced by an overlapping runtime")
  def dram_alloc(self, size):
    self.asked.append(size)
    if sum(self.used.values()) + size > self.room: raise MemoryError(f"no {size} bytes free in DRAM")
    addr = 1 << 20 | len(self.asked) << 32
    self.used[addr] = size
    return addr
  def dram_free(self, addr): del self.used[addr]
  def launch(self, kernel, args=(), units=None, name=""): self.launched.append((kernel, args))


def _many_rows(rt):
  from baretile_b200.tensor import Tensor
  x, w = Tensor(rt, 77, 2048), Tensor(rt, 2048, 544, dtype="bfp8")
  w.runs = (5, 64, 0)
  return x, w


def test_many_rows_run_without_room_for_parts_of_k():
  # scratch for x by rows is all that a matmul of many rows needs: with no room for parts of K beside it, it does without
  rt = TightRuntime()
  x, w = _many_rows(rt)
  y = (x @ w).realize()
  kernel, args = rt.launched.pop()
  assert kernel == "bt_gemm_tiles" and args[-2] > 2 * 77 * 2048 + 77 * 544 * 4 and len(rt.used) == 3
  rt.room = sum(rt.used.values()) + 3 * 17 * 2048 + 2 * 77 * 2048
  z = (x @ w).realize()
  kernel, args = rt.launched.pop()
  assert kernel == "bt_gemm_tiles" and args[-2] == 2 * 77 * 2048 and len(rt.used) == 4
  del z
  rt.room -= 1
  z = x @ w
  for _ in range(2):
    with pytest.raises(MemoryError, match="bytes free"): z.realize()
    assert not rt.launched and z.addr is None and len(rt.used) == 3     # an attempt that fails keeps nothing
  rt.room += 1
  assert z.realize().addr in rt.used


def test_expressions_on_a_closed_runtime_raise():
  # at once, as anything else on it does, not first when a result is asked for
  from baretile_b200.tensor import Tensor
  rt = TightRuntime()
  x, w = Tensor(rt, 4, 64), Tensor(rt, 64, 64, dtype="bfp8")
  y = x @ w
  rt.active = False
  for late in (lambda: x @ w, lambda: x.matmul(w, dtype="fp32"), lambda: y.relu(), lambda: y.silu(), lambda: y * 2, lambda: 0.5 * y, lambda: y * y,
               lambda: y + y, lambda: y.realize(), lambda: Tensor(rt, 1, 1)):
    with pytest.raises(RuntimeError, match="closed"): late()
  rt.active = True
  (x @ w).relu()


def test_hole_allocator_merges():
  from baretile_b200.runtime import _merge_holes
  holes = [(512, 256), (0, 256), (256, 256), (2048, 64)]
  _merge_holes(holes)
  assert holes == [(0, 768), (2048, 64)]


def test_queue_plan_follows_the_addresses(built):
  # which earlier matmul each one of a queue waits for: worked out on the host from the buffers, no device needed
  from baretile_b200 import _lib
  def op(x, out, m=8, k=512, n=1024, add=0, fmt=8, epilogue=0, w=0x100000, w2=0x200000):
    return _lib.GemvOp(fmt=fmt, epilogue=epilogue, M=m, K=k, N=n, out_dtype=0, alpha=1.0, x=x, w=w, w2=w2 if epilogue == 3 else 0, add=add, out=out)
  def plan(ops):
    arr, waits = (_lib.GemvOp * len(ops))(*ops), (ctypes.c_int * len(ops))()
    _lib.call("bt_gemv_queue_plan", len(ops), arr, waits)
    return list(waits)
  A, B, C, D, E = (0x1000000 * i for i in range(1, 6))
  # a chain: every matmul reads the one before it
  assert plan([op(A, B), op(B, C, k=1024), op(C, D, k=1024), op(D, E, k=1024)]) == [-1, 0, 1, 2]
  # independent matmuls: only the limit of two in flight holds them back
  assert plan([op(A, B), op(A, C), op(A, D), op(A, E)]) == [-1, -1, 0, 1]
  # the addend is read too; a result buffer is not overwritten while an earlier matmul may still read or write it
  assert plan([op(A, B), op(A, C, add=B)]) == [-1, 0]
  assert plan([op(A, B), op(C, A)]) == [-1, 0]                       # writes what the first one reads
  assert plan([op(A, B), op(C, B)]) == [-1, 0]                       # writes what the first one writes
  assert plan([op(A, B), op(A + 512 * 64, C, k=32)]) == [-1, -1]      # reads A's tiles past the first one's 16: no overlap with B
  assert plan([op(A, B), op(B + 2048 * 31, C, k=32)]) == [-1, 0]      # the last tile of B
  assert plan([op(A, B), op(B + 2048 * 32, C, k=32)]) == [-1, -1]     # just past B
  # a result in memory that held an earlier matmul's weights, whose last byte still counts, and just past them
  for fmt, size in ((8, 16 * 32 * 1088), (4, 16 * 32 * 576)):
    assert plan([op(A, B, fmt=fmt, w=D), op(C, D + size - 256)]) == [-1, 0]
    assert plan([op(A, B, fmt=fmt, w=D), op(C, D + size)]) == [-1, -1]
    assert plan([op(A, B, fmt=fmt, epilogue=3, w2=D), op(C, D + size - 256)]) == [-1, 0]
  # a list longer than one launch: the 33rd matmul starts a new launch and waits for all of the first
  many = [op(A, B + 0x10000 * i) for i in range(34)]
  waits = plan(many)
  assert waits[:3] == [-1, -1, 0] and waits[31] == 29 and waits[32] == -1 and waits[33] == -1
  with pytest.raises(ValueError, match="matmul 1: takes 1 to 32 rows"): plan([op(A, B), op(A, C, m=33)])


def _gates(ops):
  from baretile_b200 import _lib
  arr, gates = (_lib.GemvOp * len(ops))(*ops), (ctypes.c_int * (2 * len(ops)))()
  _lib.call("bt_gemv_queue_gates", len(ops), arr, gates)
  return [tuple(gates[2 * i:2 * i + 2]) for i in range(len(ops))]


def _links(ops, sms=148):
  from baretile_b200 import _lib
  arr, links = (_lib.GemvOp * len(ops))(*ops), (ctypes.c_int * len(ops))()
  _lib.call("bt_gemv_queue_links", sms, len(ops), arr, links)
  return list(links)


def test_chain_takes_from_the_matmul_before_what_that_one_has(built):
  from baretile_b200 import _lib
  def op(x, out, k=64, n=64, add=0, m=2, fp32=False):
    return _lib.GemvOp(fmt=8, epilogue=0, M=m, K=k, N=n, out_dtype=int(fp32), alpha=1.0, x=x, w=0x100000, add=add, out=out)
  A, B, C, D, *more = (0x1000000 * i for i in range(1, 12))
  def links(*ops):           # behind a chain of some matmuls, so that the list is one whatever these are
    m = ops[0].M
    lead = [op(a, b, m=m) for a, b in zip(more, more[1:])]
    got = _links(lead + list(ops))
    assert got[:len(lead)] in ([0] + [1] * (len(lead) - 1), [-1] * len(lead))
    return got[len(lead):]
  assert links(op(A, B), op(B, C), op(C, D)) == [0, 1, 1]
  assert links(op(A, B), op(B, C, add=B)) == [0, 1]
  assert links(op(A, B), op(B, C, n=32, add=B)) == [0, 1]
  # an addend of more columns than the matmul before has results: the columns past those come from memory
  assert links(op(A, B), op(B, C, n=96, add=B)) == [0, 0]
  assert links(op(A, B), op(B, C, n=8192, add=B)) == [0, 0]
  assert links(op(A, B), op(B, C, n=96, add=D)) == [0, 1]
  # another width or number of rows, an addend or a result that overlaps the result before, and fp32 results
  assert links(op(A, B, n=96), op(B, C)) == [0, 0] and links(op(A, B), op(B, C, m=1)) == [0, 0] and links(op(A, B, fp32=True), op(B, C)) == [0, 0]
  assert links(op(A, B), op(B, C, add=B + 2048)) == [0, 0] and links(op(A, B), op(B, B + 2048)) == [0, 0]
  # a matmul that is not small, or more rows: the general kernel
  assert links(op(A, B), op(B, C, n=32768)) == [-1, -1] and links(op(A, B, m=9), op(B, C, m=9)) == [-1, -1]


def test_chain_kernel_takes_lists_that_gain_by_it(built):
  # (k, n) of each matmul, read from the one before ("chain") or from inputs of their own ("apart")
  from baretile_b200 import _lib
  def takes(how, m, *shapes):
    at = [0x1000000 * (i + 1) for i in range(2 * len(shapes) + 1)]
    ops = [_lib.GemvOp(fmt=8, epilogue=0, M=m, K=-(-k // 32) * 32, N=-(-n // 32) * 32, out_dtype=0, alpha=1.0, w=0x100000, out=at[2 * i + 1],
                       x=at[2 * i - 1] if i and how == "chain" else at[2 * i]) for i, (k, n) in enumerate(shapes)]
    links = _links(ops)
    assert links[0] in (0, -1) and len(set(links[1:])) <= 1
    return links[0] == 0
  def back_and_forth(a, b, count): return [(a, b), (b, a)] * (count // 2) + [(a, b)] * (count % 2)
  for m in (1, 3, 8):
    assert takes("chain", m, *back_and_forth(576, 1536, 24)) and takes("chain", m, (576, 576), (576, 576)) and takes("chain", m, *back_and_forth(2048, 512, 24))
    assert takes("apart", m, *[(576, 1536)] * 4) and takes("apart", m, *[(576, 576)] * 24) and takes("apart", m, *[(100, 9000)] * 2)
    # one alone, some narrow ones, and many tile rows: the general kernel
    assert not takes("apart", m, (576, 1536)) and not takes("apart", m, *[(576, 576)] * 3)
    for k, n in ((1024, 768), (2048, 512), (4096, 256)): assert not takes("apart", m, *[(k, n)] * 24) and not takes("apart", m, (k, n))
    assert takes("chain", m, (2048, 256), (256, 2048)) == (m == 1) and not takes("chain", m, (4096, 256), (256, 4096)) and not takes("chain", m, (256, 4096), (4096, 256))
    assert takes("chain", m, *back_and_forth(8192, 64, 24)) == (m == 1) and not takes("chain", m, *back_and_forth(100, 9000, 24))
  assert takes("chain", 1, *back_and_forth(4096, 256, 24)) and takes("chain", 3, *back_and_forth(4096, 256, 24))


def test_chain_ring_takes_every_stage(built):
  """A chain's ring may be shorter than two stages. Whatever stood in it before, a stage asks for no more than an empty ring has: on no CTA
  would its copy wait for room that nobody frees."""
  from baretile_b200 import _lib
  def rooms(m, layers, *matmuls):
    """layers of (format, k, n, gate/up pair) matmuls, each reading the one before where that has k columns."""
    ops, out, columns = [], 0x1000000, 0
    for i in range(layers):
      for fmt, k, n, pair in matmuls:
        k, n, x = -(-k // 32) * 32, -(-n // 32) * 32, out
        if k != columns: x = 0x1000
        out, columns = out + 0x1000000, n
        ops.append(_lib.GemvOp(fmt=fmt, epilogue=3 if pair else 0, M=m, K=k, N=n, out_dtype=0, alpha=1.0, x=x, w=0x100000, w2=0x200000 if pair else 0, out=out))
    arr, got = (_lib.GemvOp * len(ops))(*ops), (ctypes.c_int * (2 * len(ops)))()
    _lib.call("bt_gemv_queue_rooms", 148, len(ops), arr, got)
    return [tuple(got[2 * i:2 * i + 2]) for i in range(len(ops))]
  short = 0
  def check(got):
    nonlocal short
    for ring, most in got:
      assert 0 < most <= ring or ring == most == 0
      short += 0 < ring < 2 * 34816
  for up, down in ((8, 8), (4, 8), (8, 4), (4, 4)):
    for m in (1, 3, 8):
      for d in (32, 96, 320, 576, 1024, 1152, 1344):
        for f in (64, 576, 1024, 1152, 1536, 3072, 9600):
          check(rooms(m, 8, (up, d, f, True), (down, f, d, False)))
        check(rooms(m, 8, (4, 96, 9600, False), (up, d, 1024, True), (down, 1024, d, False)))
  assert short
  # stages of 18432 and 34816 bytes in a ring of 50176: CTAs 20 to 31 take one of each
  assert rooms(8, 3, (4, 1152, 1024, True), (8, 1024, 1152, False))[5] == (50176, 50176)


def _complete(gates):
  """For each matmul, the earlier ones of its launch that are complete when it starts: those it looks at, and whatever was
  complete when those started. Nothing else: a matmul may be complete, or start, while one before it still runs."""
  seen = []
  for looks in gates: seen.append({j for g in looks if g >= 0 for j in (g, *seen[g])})
  return seen


def _must_be_complete(ops, i):
  """The earlier matmuls of ops[i]'s launch (of 32) that it may not overlap: users of its scratch (two sets, taken in
  turn) and those one of whose results it reads or overwrites, or that read what it writes."""
  def reads(o): return {o.x, o.add} - {0}
  def writes(o): return {o.arg_val, o.arg_idx} if o.epilogue == 4 else {o.out}
  o, first = ops[i], i // 32 * 32
  return {e for e in range(first, i) if (i - e) % 2 == 0 or writes(ops[e]) & (reads(o) | writes(o)) or reads(ops[e]) & writes(o)}


def test_queue_waits_cover_every_dependence(built):
  # a matmul looks at the counters of one or two earlier ones, each of which speaks for its own matmul only; what else must
  # be complete has to follow from those
  from baretile_b200 import _lib
  def op(x, out, k=32, n=32, add=0, pick=False):
    return _lib.GemvOp(fmt=8, epilogue=4 if pick else 0, M=1, K=k, N=n, out_dtype=0, alpha=1.0, x=x, w=0x100000, add=add, out=0 if pick else out,
                       arg_val=out if pick else 0, arg_idx=out + 0x100000 if pick else 0)
  A, B, C, D, E, F = (0x1000000 * i for i in range(1, 7))
  lists = {
    "a result read three places back": [op(A, B, k=8192), op(C, D), op(C, E), op(B, F)],
    "two dependences": [op(A, B, k=8192), op(C, D), op(D, E, add=B)],
    "scratch": [op(A, B, k=8192, pick=True), op(C, D), op(D, E, pick=True)],
    "memory used again": [op(A, B, k=8192), op(C, D), op(C, E), op(C, A, n=8192)],
  }
  for name, ops in lists.items():
    seen = _complete(_gates(ops))
    for i in range(len(ops)): assert _must_be_complete(ops, i) <= seen[i], (name, i, _gates(ops))
  # in a chain the one before it is all that a matmul looks at
  assert _gates([op(A, B), op(B, C), op(C, D), op(D, E)]) == [(-1, -1), (0, -1), (1, -1), (2, -1)]
  assert _gates([op(A, B), op(A, C), op(A, D), op(A, E)]) == [(-1, -1), (-1, -1), (0, -1), (1, 0)]
  rng = random.Random(3)
  for _ in range(300):
    places = [0x1000000 * i for i in range(1, rng.choice([4, 8, 40]))]
    ops = []
    for _ in range(rng.randint(1, 70)):
      x, out, add = (rng.choice(places) for _ in range(3))
      ops.append(op(x, out, add=add if rng.random() < 0.3 else 0, pick=rng.random() < 0.2))
    gates = _gates(ops)
    seen = _complete(gates)
    for i in range(len(ops)):
      assert _must_be_complete(ops, i) <= seen[i], (i, gates)
      assert all(g == -1 or i // 32 * 32 <= g < i for g in gates[i])     # the launch before it is complete as a whole


def test_queue_collects_matmuls_and_flushes_in_order(monkeypatch):
  # host logic of Runtime.queue(): matmuls are collected, anything else that needs the stream sends them first, the
  # block's end sends the rest; the C-ABI calls are captured instead of made, so no device is needed
  from baretile_b200 import _lib, runtime
  calls = []
  def fake_call(name, *args):
    if name == "bt_gemv_queue":
      n, arr = args[1], args[2]
      calls.append((name, [(arr[i].fmt, arr[i].epilogue, arr[i].M, arr[i].K, arr[i].N, arr[i].x, arr[i].w, arr[i].w2, arr[i].add, arr[i].out, arr[i].out_dtype,
                            arr[i].arg_val, arr[i].arg_idx, arr[i].arg_base, round(arr[i].alpha, 3)) for i in range(n)]))
    else: calls.append((name, args))
  monkeypatch.setattr(_lib, "call", fake_call)
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.launches, rt.sent, rt.log, rt.pending, rt.timing, rt.work, rt.work_bytes = True, 0, 7, 0, {}, None, None, False, 4096, 1 << 20
  rt.sides, rt.unjoined, rt.side = [], [], None
  def matmul(x, out, epilogue=0, w2=0, alpha=1.0):
    rt.launch("bt_gemv_bfp", (8, epilogue, 4, 512, 1024, x, 0x1000, w2, 0, ctypes.c_float(alpha), out, 0, 0, 0, 0, rt.work, rt.work_bytes), name="matmul")
  matmul(0x10, 0x20)                                                  # outside a queue: sent at once
  assert [c[0] for c in calls] == ["bt_gemv_bfp"]
  calls.clear()
  with rt.queue():
    matmul(0x10, 0x20)
    matmul(0x20, 0x30, epilogue=3, w2=0x2000, alpha=0.5)
    assert calls == []                                               # nothing has left yet
    rt.launch("bt_untilize", (2, 0x30, 0x40, 1, 4, 1024), name="readback")
    matmul(0x40, 0x50)
  assert [c[0] for c in calls] == ["bt_gemv_queue", "bt_untilize", "bt_gemv_queue"]
  assert calls[0][1] == [(8, 0, 4, 512, 1024, 0x10, 0x1000, 0, 0, 0x20, 0, 0, 0, 0, 1.0), (8, 3, 4, 512, 1024, 0x20, 0x1000, 0x2000, 0, 0x30, 0, 0, 0, 0, 0.5)]
  assert len(calls[2][1]) == 1 and calls[2][1][0][5] == 0x40
  assert rt.launches == 5 and rt.pending is None
  calls.clear()
  with pytest.raises(KeyError):
    with rt.queue():
      matmul(0x10, 0x20)
      raise KeyError("the block fails")
  assert calls == [] and rt.pending is None                          # a failed block sends nothing


def test_beside_blocks_fork_from_the_stream_and_join_it_again(monkeypatch):
  # host logic of Runtime.beside(): a block's copies go to a stream of its own that starts behind what the runtime has
  # queued; the runtime's later launches do not wait for it until join(); the C-ABI calls are captured, no device needed
  from baretile_b200 import _lib, runtime
  calls, made = [], iter(range(100, 200))
  def fake_call(name, *args):
    if name in ("bt_stream_create", "bt_event_create"): args[-1]._obj.value = next(made)
    calls.append((name, args))
  monkeypatch.setattr(_lib, "call", fake_call)
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.launches, rt.sent, rt.log, rt.pending, rt.timing, rt.work, rt.work_bytes = True, 0, 7, 0, {}, None, None, False, 4096, 1 << 20
  rt.sides, rt.unjoined, rt.side, rt.recording = [], [], None, None
  buf = (ctypes.c_char * 64)()
  with rt.beside(): rt.upload_async(0x1000, buf)
  with rt.beside(): rt.download_async(buf, 0x2000)
  rt.launch("bt_untilize", (2, 0x30, 0x40, 1, 4, 1024), name="readback")
  (s1, f1, d1), (s2, f2, d2) = rt.sides
  assert len({7, s1, s2}) == 3 and rt.stream == 7 and rt.unjoined == [d1, d2]
  order = [(n, a) for n, a in calls if n not in ("bt_stream_create", "bt_event_create")]
  assert [n for n, _ in order] == ["bt_event_record", "bt_stream_wait_event", "bt_h2d", "bt_event_record",
                                   "bt_event_record", "bt_stream_wait_event", "bt_d2h", "bt_event_record", "bt_untilize"]
  assert order[0][1] == (0, f1, 7) and order[1][1] == (0, s1, f1) and order[2][1][-1] == s1 and order[3][1] == (0, d1, s1)
  assert order[4][1] == (0, f2, 7) and order[5][1] == (0, s2, f2) and order[6][1][-1] == s2 and order[7][1] == (0, d2, s2)
  assert order[8][1][-1] == 7                                         # the runtime's own launch did not wait for either
  calls.clear()
  rt.join()
  assert calls == [("bt_stream_wait_event", (0, 7, d1)), ("bt_stream_wait_event", (0, 7, d2))] and rt.unjoined == []
  with pytest.raises(RuntimeError, match="own stream"):
    with rt.beside(): rt.launch("bt_gemv_bfp", (8, 0, 4, 512, 1024, 0x10, 0x1000, 0, 0, ctypes.c_float(1.0), 0x20, 0, 0, 0, 0, rt.work, rt.work_bytes))
  assert rt.stream == 7 and rt.side is None                           # the failed block gave the stream back
  rt.join()
  calls.clear()
  with rt.beside():
    with pytest.raises(RuntimeError, match="already open"):
      with rt.beside(): pass
    with pytest.raises(RuntimeError, match="inside a beside block"): rt.join()


def test_replay_runs_behind_the_matmuls_collected_before_it(monkeypatch):
  from baretile_b200 import _lib, runtime
  calls = []
  monkeypatch.setattr(_lib, "call", lambda name, *args: calls.append(name))
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.launches, rt.sent, rt.log, rt.pending, rt.timing, rt.work, rt.work_bytes = True, 0, 7, 0, {}, None, None, False, 4096, 1 << 20
  rt.sides, rt.unjoined, rt.side, rt.recording = [], [], None, None
  step = runtime.Recording(rt)
  step.graph, step.count, step.launches = 5, 3, [("bt_untilize", (2, 0x30, 0x40, 1, 4, 1024), None, "readback")]
  with rt.queue():
    rt.launch("bt_gemv_bfp", (8, 0, 4, 512, 1024, 0x10, 0x1000, 0, 0, 1.0, 0x20, 0, 0, 0, 0, rt.work, rt.work_bytes))
    step.replay()
  assert calls == ["bt_gemv_queue", "bt_graph_launch"]
  # and a recorded matmul stays out of beside blocks, as any other does
  rt.side, rt.stream = 7, 9
  step.replay()
  step.launches.append(("bt_gemm_tiles", (), None, ""))
  with pytest.raises(RuntimeError, match="own stream"): step.replay()
  assert calls == ["bt_gemv_queue", "bt_graph_launch", "bt_graph_launch"]
  rt.active = False


def test_memory_freed_behind_a_beside_block_is_not_reused_before_the_join(monkeypatch):
  # the block's stream may still read it, and the runtime's own stream, or another block's, does not wait for that
  from baretile_b200 import _lib, runtime
  calls, room, next_arena = [], [1], 1 << 32
  made = iter(range(100, 200))
  def fake_call(name, *args):
    nonlocal next_arena
    calls.append((name, args))
    if name in ("bt_stream_create", "bt_event_create"): args[-1]._obj.value = next(made)
    if name == "bt_malloc":
      if not room: raise MemoryError("no bytes free")
      room.pop()
      args[-1]._obj.value, next_arena = next_arena, next_arena + (1 << 40)
  monkeypatch.setattr(_lib, "call", fake_call)
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.recording, rt.pending, rt.log, rt.sent, rt.launches, rt.timing = True, 0, 7, None, None, None, {}, 0, False
  rt.sides, rt.unjoined, rt.side, rt.holes, rt.used, rt.arenas, rt.kept, rt.kept_count = [], [], None, [], {}, [], {}, 0
  a = rt.dram_alloc(4096)
  rt.dram_free(a)
  assert rt.dram_alloc(4096) == a                                     # nothing beside: reused at once
  with rt.beside():
    rt.dram_free(a)                                                   # what the block has queued may still use it
    b = rt.dram_alloc(4096)
    assert b != a
  rt.dram_free(b)
  c = rt.dram_alloc(4096)
  assert c not in (a, b)
  with rt.beside(): assert rt.dram_alloc(4096) not in (a, b, c)
  rt.join()
  assert {rt.dram_alloc(4096), rt.dram_alloc(4096)} == {a, b}
  # with no other memory left the host waits for the blocks' streams instead of giving up
  with rt.beside(): pass
  rest = rt.dram_alloc(rt.holes[0][1])
  rt.dram_free(c)
  calls.clear()
  assert rt.dram_alloc(4096) == c and [n for n, _ in calls] == ["bt_malloc", "bt_stream_sync", "bt_stream_sync"]
  assert {args[1] for n, args in calls if n == "bt_stream_sync"} == {s for s, _, _ in rt.sides}
  with pytest.raises(MemoryError, match="no 8192 bytes free"): rt.dram_alloc(8192)
  rt.dram_free(rest)
  rt.active = False


@pytest.mark.parametrize("size", [1, 4096, (256 << 10) - 1, 256 << 10])
def test_upload_returns_when_its_source_has_been_read(monkeypatch, size):
  # a copy that is only queued may still have page-locked memory to read: uploads go through the two entry points that
  # return when they have read it, whatever memory it is
  from baretile_b200 import _lib, runtime
  calls = []
  monkeypatch.setattr(_lib, "call", lambda name, *args: calls.append((name, args)))
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.pending, rt.recording, rt.stage = False, 0, 7, None, None, 99
  rt.check = lambda: None
  for data in (bytes(size), bytearray(size), memoryview(bytearray(size + 1))[1:], (ctypes.c_char * size)()):
    rt.upload(4096, data)
    name, args = calls.pop()
    assert (name, args[0], args[1], args[3:]) == (("bt_upload", 0, 4096, (size, 7)) if size < 256 << 10 else ("bt_stage_upload", 99, 4096, (size, 7))) and not calls


def test_large_copies_without_staging_buffers(monkeypatch):
  # a host with no page-locked memory or threads to spare still copies, as it does what is small
  from baretile_b200 import _lib, runtime
  calls = []
  def fake_call(name, *args):
    calls.append(name)
    if name == "bt_stage_create": raise MemoryError("no memory or threads for a staging object")
  monkeypatch.setattr(_lib, "call", fake_call)
  rt = runtime.Runtime.__new__(runtime.Runtime)
  rt.active, rt.device, rt.stream, rt.pending, rt.recording, rt.stage = False, 0, 7, None, None, 0
  rt.check = lambda: None
  rt.upload(4096, bytes(1 << 20))
  assert len(rt.download(4096, 1 << 20)) == 1 << 20
  assert calls == ["bt_stage_create", "bt_upload", "bt_stage_create", "bt_d2h", "bt_stream_sync"]


def test_newer_entry_points_refuse_bad_arguments_before_any_device_work(built):
  """Argument checks come first in every entry point: they raise ValueError on a box without a GPU too."""
  import ctypes
  from baretile_b200 import _lib
  f = ctypes.c_float(1.0)
  # prefill matmul: K in whole tiles, w2 only with the gate/up epilogue, an addend of 1 or M rows
  with pytest.raises(ValueError, match="multiple of 32"): _lib.call("bt_gemm_bfp", 0, 8, 0, 64, 40, 64, 256, 256, 0, 0, 0, f, 256, 0, 256, 0)
  with pytest.raises(ValueError, match="w2 goes with"): _lib.call("bt_gemm_bfp", 0, 8, 0, 64, 64, 64, 256, 256, 256, 0, 0, f, 256, 0, 256, 0)
  with pytest.raises(ValueError, match="1 or M rows"): _lib.call("bt_gemm_bfp", 0, 8, 0, 64, 64, 64, 256, 256, 0, 256, 7, f, 256, 0, 256, 0)
  # put: formats, distinct aligned tensors
  with pytest.raises(ValueError, match="unknown format"): _lib.call("bt_put", 0, 3, 256, 512, 768, 1, 1, 32, 32, 0, 0)
  with pytest.raises(ValueError, match="apart from dst"): _lib.call("bt_put", 0, 8, 256, 256, 768, 1, 1, 32, 32, 0, 0)
  # the streaming layout: one launch takes up to 65535 runs of 4 tile columns; and an event to wait for must exist
  with pytest.raises(ValueError, match="tile columns in one launch"): _lib.call("bt_relayout", 0, 8, 1, 1, 4 * 65535 + 1, 256, 512, 0)
  with pytest.raises(ValueError, match="null event"): _lib.call("bt_stream_wait_event", 0, 0, 0)
  with pytest.raises(ValueError, match="no bytes"): _lib.call("bt_upload", 0, 256, 256, 0, 0)
  # many small matrices: a table is needed
  with pytest.raises(ValueError, match="no matrices"): _lib.call("bt_tilize_many", 0, 2, 0, None, None, None, None, 0)
  with pytest.raises(ValueError, match="itemsize"): _lib.call("bt_untilize_many", 0, 3, 1, None, None, None, None, 0)
  # the exchange over peer memory: ranks of one box, one tile row of whole tiles, steps from 1
  peers = (ctypes.c_uint64 * 2)(256, 512)
  with pytest.raises(ValueError, match="rank"): _lib.call("bt_peer_allreduce_round", 0, 2, 2, peers, 0, 1, 4, 64, 256, 0)
  with pytest.raises(ValueError, match="step"): _lib.call("bt_peer_allreduce_round", 0, 0, 2, peers, 0, 0, 4, 64, 256, 0)
  with pytest.raises(ValueError, match="rows at offset"): _lib.call("bt_peer_allreduce_round", 0, 0, 2, peers, 0, 1, 33, 64, 256, 0)
  with pytest.raises(ValueError, match="up to 8 ranks"): _lib.call("bt_peer_open", 0, 1, 0, 9, 1024, peers, 0)
  with pytest.raises(ValueError, match="rows at offset"): _lib.call("bt_peer_argmax_combine", 0, 0, 2, peers, 0, 1, 40, 256, 256, 512, 0)
