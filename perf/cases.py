"""The work that a program on this framework has it do, as cases to time: the matmul on block-float weights as a single
call, as a recorded decode step, as a jit'd step from host values to host values, as a greedy pick and as a prefill; and
what surrounds it, loading weights from the host and keeping a block-float cache.

A case is a dict of plain values. Every kind of case has a range of sizes, given in `draw`; the listed ones are points
of these ranges. Weights are N(0, s) with 1% of the input channels scaled by 20 (the outlier channels that stress
shared exponents), s such that a matmul keeps its input's magnitude; activations are N(0, 1) in bf16."""
import math
import torch
from baretile_b200 import pci
from baretile_b200.chip import Chip
from baretile_b200.runtime import Runtime
from baretile_b200.tensor import Tensor, jit

VALUE_BYTES = {"bfp8": 17 / 16, "bfp4": 9 / 16}   # a value and its share of the exponent of its run of 16


def listed():
  return [
    # one fused call on a small model's MLP (SmolLM-135M): what a single expression costs
    {"name": "call_relu_576x1536", "kind": "call", "m": 32, "k": 576, "n": 1536, "fmt": "bfp8", "act": "relu", "bias": False, "out": "bf16"},
    # one fused call on odd sizes, bias and activation, a few rows (a small speculative batch)
    {"name": "call_silu_1000x4100", "kind": "call", "m": 5, "k": 1000, "n": 4100, "fmt": "bfp4", "act": "silu", "bias": True, "out": "bf16"},
    # a whole small model's layers for one token, host values in and host values out, through jit
    {"name": "token_576x1536", "kind": "token", "m": 1, "d": 576, "f": 1536, "layers": 30, "fmt": "bfp8"},
    # decode of single sequences: recorded layers of Llama-3-8B's shape, replayed
    {"name": "decode_4096x14336_m1", "kind": "decode", "m": 1, "d": 4096, "f": 14336, "layers": 4, "fmt": "bfp8"},
    # the same for a small batch, weights in four bits
    {"name": "decode_4096x14336_m8", "kind": "decode", "m": 8, "d": 4096, "f": 14336, "layers": 4, "fmt": "bfp4"},
    # a batch of 16 on a layer of Llama-3-70B's shape
    {"name": "decode_8192x28672_m16", "kind": "decode", "m": 16, "d": 8192, "f": 28672, "layers": 2, "fmt": "bfp4"},
    # matmuls that do not read one another's results in one recorded queue: the benchmark's sweep
    {"name": "sweep_4096x14336", "kind": "sweep", "d": 4096, "f": 14336},
    # greedy pick of the next token for 4 drafts, Llama-3-70B's head
    {"name": "pick_8192x128256", "kind": "pick", "m": 4, "k": 8192, "n": 128256, "fmt": "bfp8"},
    # prefill of a 2048-token prompt: gate/up pair in bfp8, down projection in bfp4
    {"name": "prefill_2048", "kind": "prefill", "m": 2048, "d": 4096, "f": 14336, "fmt": "bfp8", "down": "bfp4"},
    # prefill of a short prompt of an odd length
    {"name": "prefill_77", "kind": "prefill", "m": 77, "d": 2048, "f": 5632, "fmt": "bfp4", "down": "bfp8"},
    # loading a weight matrix from host memory: upload, cast, lay out by columns, and the first matmul on it
    {"name": "load_4096x14336", "kind": "load", "k": 4096, "n": 14336, "fmt": "bfp8"},
    # a step's new keys into a block-float cache (64 heads and sequences), and the cache decoded for its reader
    {"name": "cache_64x4096x128", "kind": "cache", "batch": 64, "rows": 4096, "cols": 128, "n": 16, "fmt": "bfp8"},
  ]


def draw(rng):
  """One more case of the ranges the listed ones stand for. A drawn case costs no more than the largest listed one of
  its kind."""
  def log(a, b): return max(a, min(b, round(math.exp(rng.uniform(math.log(a), math.log(b))))))
  def size(a, b):                                  # mostly whole tiles, as models have them; one in four is any number
    n = log(a, b)
    return n if rng.random() < 0.25 else max(32, n // 32 * 32)
  fmt, kind = rng.choice(["bfp8", "bfp4"]), rng.choice(["call", "token", "decode", "decode", "sweep", "pick", "prefill", "prefill", "load", "cache"])
  if kind == "call":
    return {"kind": kind, "m": log(1, 32), "k": size(64, 8192), "n": size(64, 14336), "fmt": fmt, "act": rng.choice(["none", "relu", "silu", "glu"]),
            "bias": rng.random() < 0.5, "out": rng.choice(["bf16", "bf16", "fp32"])}
  if kind == "token":
    d = size(256, 1024)
    return {"kind": kind, "m": log(1, 8), "d": d, "f": size(d, 3 * d), "layers": log(4, 30), "fmt": fmt}
  if kind == "decode":
    d = size(1024, 8192)
    f = size(2 * d, min(4 * d, 28672))
    return {"kind": kind, "m": log(1, 32), "d": d, "f": f, "layers": max(1, min(16, int(434e6 / (d * d + 3 * d * f)))), "fmt": fmt}
  if kind == "sweep":
    d = size(1024, 4096)
    return {"kind": kind, "d": d, "f": size(2 * d, min(4 * d, 14336))}
  if kind == "pick":
    return {"kind": kind, "m": log(1, 8), "k": size(512, 8192), "n": log(1000, 4008) * 32, "fmt": fmt}
  if kind == "prefill":
    d, m = size(512, 4096), log(33, 2048)
    return {"kind": kind, "m": m, "d": d, "f": size(2 * d, min(4 * d, 14336)), "fmt": fmt, "down": rng.choice(["bfp8", "bfp4"])}
  if kind == "load":
    return {"kind": kind, "k": size(256, 4096), "n": size(256, 14336), "fmt": fmt}
  cols = rng.choice([64, 80, 96, 128])
  return {"kind": "cache", "batch": log(1, 64), "rows": log(64, 4096), "cols": cols, "n": log(1, 64), "fmt": fmt}


# ---- the runtime, and values on the device -------------------------------------------------------------------------

_runtime, _views = None, {}


def runtime():
  """The program's one runtime."""
  global _runtime
  if _runtime is None: _runtime = Runtime(Chip(pci.open_device(0)))
  return _runtime


class _Memory:
  def __init__(self, addr, size): self.__cuda_array_interface__ = {"shape": (size,), "typestr": "|u1", "data": (addr, False), "version": 3}


def view(t):
  """A tensor's storage, whole tiles, as a torch tensor over the same memory (made once for a place and size)."""
  kind = {"bf16": torch.bfloat16, "fp32": torch.float32, "int32": torch.int32}.get(t.dtype, torch.uint8)
  size = t.tiles * {"bf16": 2048, "fp32": 4096, "int32": 4096, "bfp8": 1088, "bfp4": 576}[t.dtype]
  key = int(t.addr), size, kind
  if key not in _views:
    if len(_views) > 4096: _views.clear()
    _views[key] = torch.as_tensor(_Memory(int(t.addr), size), device="cuda").view(kind)
  return _views[key]


class State:
  """What a program holds between passes: tensors, steps, and the last pass's results."""
  def __init__(self, case, seed):
    self.held, self.step = None, None
    self.case, self.rt = case, runtime()
    self.gen = torch.Generator(device="cuda").manual_seed(seed)
  def __del__(self):
    if self.step is not None: self.step.close()

  def normal(self, rows, cols, scale=1.0, outliers=False):
    a = torch.randn((rows, cols), generator=self.gen, device="cuda", dtype=torch.bfloat16).mul_(scale)
    if outliers and rows >= 100: a[torch.randperm(rows, generator=self.gen, device="cuda")[:rows // 100]] *= 20
    return a
  def tensor(self, a, dtype="bf16"):
    """A tensor from values already on the device."""
    batch, rows, cols = (1, *a.shape) if a.dim() == 2 else a.shape
    torch.cuda.synchronize()
    t = Tensor(self.rt, rows, cols, batch=batch, dtype=dtype)
    self.rt.launch("bt_tilize", (a.element_size(), a.data_ptr(), t.addr, batch, rows, cols), name="upload")
    self.rt.wait()
    return t
  def weights(self, k, n, fmt, gain=1.0):
    return self.tensor(self.normal(k, n, gain / math.sqrt((5 if k >= 100 else 1) * k), outliers=True)).cast(fmt).columns()


def _layer(x, wo, wg, wu, wd):
  """A decoder layer's matmuls: a projection and an MLP, each with its residual."""
  x = ((x @ wo) + x).realize()
  h = ((x @ wg).silu() * (x @ wu)).realize()
  return ((h @ wd) + x).realize()


def _layers(s, d, f, fmt, count):
  return [(s.weights(d, d, fmt, 0.15), s.weights(d, f, fmt), s.weights(d, f, fmt), s.weights(f, d, fmt, 0.15)) for _ in range(count)]


def _sweep(case):
  """(k, n, format, rows, pair) of the sweep's matmuls, ordered so that a weight matrix comes up again only after all others."""
  d, f = case["d"], case["f"]
  return [(k, n, fmt, m, pair) for m in (1, 8, 32) for fmt in ("bfp8", "bfp4") for k, n, pair in ((d, d, False), (d, f, False), (f, d, False), (d, f, True))]


def prepare(case, seed):
  s = State(case, seed)
  rt, kind = s.rt, case["kind"]
  if kind == "call":
    s.x, s.w = s.tensor(s.normal(case["m"], case["k"])), s.weights(case["k"], case["n"], case["fmt"])
    s.w2 = s.weights(case["k"], case["n"], case["fmt"]) if case["act"] == "glu" else None
    s.bias = s.tensor(s.normal(1, case["n"])) if case["bias"] and case["act"] != "glu" else None
  elif kind == "token":
    layers = _layers(s, case["d"], case["f"], case["fmt"], case["layers"])
    def forward(x):
      for weights in layers: x = _layer(x, *weights)
      return x
    s.forward = jit(forward)
    s.host = s.normal(case["m"], case["d"]).view(torch.int16).cpu().numpy().tobytes()
    for _ in range(2): s.forward(Tensor.frombytes(rt, case["m"], case["d"], s.host))       # a call that runs, a call that records
  elif kind == "decode":
    s.layers, s.x = _layers(s, case["d"], case["f"], case["fmt"], case["layers"]), s.tensor(s.normal(case["m"], case["d"]))
    s.held = []                                    # every layer's result, which a replay writes again
    with rt.record() as s.step:
      for weights in s.layers: s.held.append(_layer(s.held[-1] if s.held else s.x, *weights))
  elif kind == "sweep":
    weights, s.work, s.held = {}, [], []
    def weight(*key):
      if key not in weights: weights[key] = s.weights(*key[:3])
      return weights[key]
    for k, n, fmt, m, pair in _sweep(case):
      x = s.tensor(s.normal(m, k))
      s.work.append((x, weight(k, n, fmt, "gate" if pair else "w"), weight(k, n, fmt, "up") if pair else None))
    with rt.record() as s.step:
      for x, w, w2 in s.work: s.held.append((((x @ w).silu() * (x @ w2)) if w2 else x @ w).realize())
  elif kind == "pick":
    s.x, s.w = s.tensor(s.normal(case["m"], case["k"])), s.weights(case["k"], case["n"], case["fmt"])
  elif kind == "prefill":
    d, f = case["d"], case["f"]
    s.x = s.tensor(s.normal(case["m"], d))
    s.wg, s.wu, s.wd = s.weights(d, f, case["fmt"]), s.weights(d, f, case["fmt"]), s.weights(f, d, case["down"])
  elif kind == "load":
    s.host = s.normal(case["k"], case["n"], 1 / math.sqrt(5 * case["k"]), outliers=True).view(torch.int16).cpu().numpy().tobytes()
    s.x = s.tensor(s.normal(1, case["k"]))
  else:
    shape = case["batch"], case["rows"], case["cols"]
    s.cache = s.tensor(s.normal(shape[0] * shape[1], shape[2]).view(shape)).cast(case["fmt"])
    n = min(case["n"], case["rows"])
    at = int(torch.randint(0, case["rows"] - n + 1, (1,), generator=s.gen, device="cuda"))
    s.ids = s.tensor(torch.arange(at, at + n, dtype=torch.int32, device="cuda").view(1, n), "int32")
    s.rows = s.tensor(s.normal(shape[0] * n, shape[2]).view(shape[0], n, shape[2]))
  rt.wait()
  return s


def run(s):
  case, rt, kind = s.case, s.rt, s.case["kind"]
  if kind == "call":
    y = s.x.matmul(s.w, dtype=case["out"])
    if s.bias is not None: y = y + s.bias
    if case["act"] == "relu": y = y.relu()
    elif case["act"] == "silu": y = y.silu()
    elif case["act"] == "glu": y = y.silu() * s.x.matmul(s.w2, dtype=case["out"])
    s.held = [y.realize()]
  elif kind == "token": return s.forward(Tensor.frombytes(rt, case["m"], case["d"], s.host)).numpy()
  elif kind in ("decode", "sweep"): s.step.replay()
  elif kind == "pick": s.held = list((s.x @ s.w).topk(1))
  elif kind == "prefill": s.held = [(((s.x @ s.wg).silu() * (s.x @ s.wu)) @ s.wd).realize()]
  elif kind == "load":
    packed = Tensor.frombytes(rt, case["k"], case["n"], s.host).cast(case["fmt"])
    s.w = packed.columns()
    s.held = [packed, (s.x @ s.w).realize()]
  else:
    s.cache.put(s.ids, s.rows)
    s.held = [s.cache, s.cache.cast("bf16")]
  return [view(t) for t in s.held]


def work(case):
  def matmul(m, k, n, fmt, matrices=1): return matrices * k * n * VALUE_BYTES[fmt] + 2 * m * (k + n), 2 * m * k * n * matrices
  kind = case["kind"]
  if kind in ("call", "pick"):
    parts = [matmul(case["m"], case["k"], case["n"], case["fmt"], 2 if case.get("act") == "glu" else 1)]
    if kind == "pick": parts = [(parts[0][0] - 2 * case["m"] * case["n"] + 8 * case["m"], parts[0][1])]
  elif kind in ("token", "decode"):                # the layers' weights, and the rows that go in and come out
    m, d, f = case["m"], case["d"], case["f"]
    values = case["layers"] * (d * d + 3 * d * f)
    parts = [(values * VALUE_BYTES[case["fmt"]] + 4 * m * d, 2 * m * values)]
  elif kind == "sweep": parts = [matmul(m, k, n, fmt, 2 if pair else 1) for k, n, fmt, m, pair in _sweep(case)]
  elif kind == "prefill":
    m, d, f = case["m"], case["d"], case["f"]
    up, down = matmul(m, d, f, case["fmt"], 2), matmul(m, f, d, case["down"])
    parts = [(up[0] - 2 * m * f, up[1]), (down[0] - 2 * m * f, down[1])]
  elif kind == "load":                             # the host's values once across, the packed values out
    k, n = case["k"], case["n"]
    parts = [(k * n * (2 + VALUE_BYTES[case["fmt"]]), 2 * k * n)]
  else:
    values = case["batch"] * case["cols"]
    parts = [(values * (case["rows"] * (VALUE_BYTES[case["fmt"]] + 2) + min(case["n"], case["rows"]) * (2 + VALUE_BYTES[case["fmt"]])), 0)]
  return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(o for _, o in parts))}


def tolerance(case):
  kind = case["kind"]
  if kind == "cache": return "exact"               # bytes of the cache and values it decodes to
  if kind == "pick": return {"rel": 1e-4}          # fp32 sums; the ids are whole numbers and stay the same
  if kind == "call" and case["out"] == "fp32": return {"rel": 1e-4}
  return {"rel": 1e-2}                             # bf16 results of fp32 sums, through several roundings in a chain; packed bytes stay the same
