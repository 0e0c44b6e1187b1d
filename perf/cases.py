"""The work that a program built on this package has it do on one GPU, as cases
with sizes: decode steps of the engine over the three cache kinds, prefill
attention, the hand-over of a prefix into a decode slot, and the weight-only int8
layers at decode and prefill row counts.

Kinds of cases and what they stand for:

  step      `KVCacheEngine.generate` over a few attention layers.  The engine owns
            the caches and the bookkeeping; the projections around the attention are
            the model's, so q, k, v of every layer and the logits stand ready.
  paged     one decode step over page pools: the page-table walk on the device, then
            append and paged attention of every layer.
  prefill   the attention layer of a prompt: causal mask tiled over the grouped
            query rows, the K/V of the prompt kept for the insert.
  insert    `KVCacheEngine.insert`: the prefix of all layers into one decode slot.
  pages     the same into reserved pages, and the pages given back.
  ffn       RMSNorm and the feed-forward block.
  linear    one weight-only int8 projection.

Head counts are (query heads, KV heads) per GPU: whole models, or one rank's share
of a model whose KV heads are sharded.
"""

import math

import numpy as np
import torch

from jetstream_pytorch_b200 import attention_kernel as ak
from jetstream_pytorch_b200 import insert as insert_ops
from jetstream_pytorch_b200 import layers
from jetstream_pytorch_b200.cache_manager import KVCachePrefill, PageKVCacheGenerate
from jetstream_pytorch_b200.engine import KVCacheEngine, Prefix
from jetstream_pytorch_b200.environment import JetEngineEnvironment, JetEngineEnvironmentData, QuantizationConfig
from jetstream_pytorch_b200.page_attention_manager import PageAttentionManager

DEV = "cuda"
D = 128  # head_dim of every configuration
VOCAB = 32000

# (query heads, KV heads): multi-head, grouped by 4 and by 8, and the shares of a GPU among 4 or 8
HEADS = ((32, 32), (32, 8), (64, 8), (16, 2), (8, 1), (4, 1))
# (dim, hidden_dim) of the feed-forward blocks
FFN = ((4096, 11008), (4096, 14336), (5120, 13824), (8192, 28672))
# (in, out) features of single projections
LINEAR = ((4096, 4096), (4096, 6144), (8192, 1280), (8192, 8192), (8192, 10240), (3584, 8192))


def listed():
  return [
      # a grouped-query model's int8 decode at the batch its cache is sized for: the package's main workload
      dict(name="step int8 b96 64/8", kind="step", cache="int8", ring=False, batch=96, hq=64, hkv=8, seq=2048, layers=2),
      # multi-head int8 decode over the ring buffer, the default engine mode (additive mask, shared position)
      dict(name="step int8 ring b8 32/32", kind="step", cache="int8", ring=True, batch=8, hq=32, hkv=32, seq=2048, layers=2),
      # one user: what a step costs when nothing is large
      dict(name="step int8 b1 32/8", kind="step", cache="int8", ring=False, batch=1, hq=32, hkv=8, seq=1024, layers=4),
      # unquantised cache, left aligned, odd batch
      dict(name="step bf16 b31 32/8", kind="step", cache="bf16", ring=False, batch=31, hq=32, hkv=8, seq=2048, layers=2),
      # paged bf16 pools as the engine's paged mode keeps them
      dict(name="paged bf16 b32 32/8", kind="paged", cache="bf16", batch=32, hq=32, hkv=8, low=1, high=2047, layers=2),
      # paged int8 pools with scale pools, long contexts
      dict(name="paged int8 b96 64/8", kind="paged", cache="int8", batch=96, hq=64, hkv=8, low=512, high=2047, layers=2),
      # prefill attention at the default maximal input length, int8 serving (unit scales during prefill)
      dict(name="prefill 1024 32/8", kind="prefill", quantized=True, hq=32, hkv=8, length=1024),
      # a prompt of 900 tokens, padded to 1024, into one slot of a stacked int8 cache
      dict(name="insert int8 l900 32 layers", kind="insert", cache="int8", batch=8, hkv=8, seq=2048, length=900, padded=1024, layers=32),
      # a prompt into pages of per-layer int8 pools
      dict(name="pages int8 l500 32 layers", kind="pages", cache="int8", hkv=8, length=500, stacked=False, layers=32),
      # the feed-forward block of a large model for a decode batch
      dict(name="ffn 8192/28672 b96", kind="ffn", dim=8192, hidden=28672, rows=96),
      # the same block of a smaller model for a whole prompt: the compute-bound end
      dict(name="ffn 4096/14336 l1024", kind="ffn", dim=4096, hidden=14336, rows=1024),
      # the fused q/k/v projection of a small decode batch
      dict(name="linear 4096/6144 b7", kind="linear", k=4096, n=6144, rows=7),
  ]


def _log(rng, low, high):
  return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
  kind = rng.choice(("step", "step", "paged", "prefill", "insert", "pages", "ffn", "linear"))
  if kind == "step":
    hq, hkv = rng.choice(HEADS)
    seq = rng.choice((512, 1024, 1280, 2048))
    cache = rng.choice(("int8", "int8", "bf16"))
    batch = min(_log(rng, 1, 96), 96 * 2048 * 8 // (seq * hkv * (1 if cache == "int8" else 2)))
    return dict(kind=kind, cache=cache, ring=rng.random() < 0.35, batch=batch, hq=hq, hkv=hkv, seq=seq,
                layers=rng.randint(1, 2) if batch > 24 else rng.randint(2, 6))
  if kind == "paged":
    hq, hkv = rng.choice(HEADS)
    cache = rng.choice(("int8", "bf16"))
    high = rng.randint(64, 2047)
    batch = min(_log(rng, 1, 96), 96 * 2048 * 8 // (2048 * hkv * (1 if cache == "int8" else 2)))
    return dict(kind=kind, cache=cache, batch=batch, hq=hq, hkv=hkv, low=rng.randint(1, high), high=high,
                layers=rng.randint(1, 2) if batch > 24 else rng.randint(2, 6))
  if kind == "prefill":
    hq, hkv = rng.choice(HEADS)
    longest = int(1024 * math.sqrt(32 / max(hq, 32)))
    return dict(kind=kind, quantized=rng.random() < 0.5, hq=hq, hkv=hkv, length=_log(rng, 16, longest))
  if kind in ("insert", "pages"):
    length = _log(rng, 5, 1900)
    nl = rng.randint(8, 32)
    hkv = rng.choice((1, 2, 8))
    cache = rng.choice(("int8", "bf16"))
    if kind == "pages":
      return dict(kind=kind, cache=cache, hkv=hkv, length=length, stacked=rng.random() < 0.4, layers=nl)
    padded = max(16, 1 << (length - 1).bit_length())  # prompts are padded to powers of two
    return dict(kind=kind, cache=cache, batch=rng.randint(1, 8), hkv=hkv, seq=2048, length=length, padded=padded, layers=nl)
  if kind == "ffn":
    dim, hidden = rng.choice(FFN)
    most = 1024 * 4096 * 14336 // (dim * hidden)
    return dict(kind=kind, dim=dim, hidden=hidden, rows=_log(rng, 1, most))
  k, n = rng.choice(LINEAR)
  return dict(kind=kind, k=k, n=n, rows=_log(rng, 1, 1024))


# --------------------------------------------------------------------- inputs


def _gen(seed):
  return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
  return torch.randn(shape, generator=g, device=DEV, dtype=torch.bfloat16)


def _heads_first(g, tokens, heads):
  """[1,H,T,D] as a model hands it over: the transposed view of its [1,T,H,D] projection."""
  return _randn(g, 1, tokens, heads, D).transpose(1, 2)


def _fill_cache(g, t):
  """N(0,1) keys or values in place; int8 caches hold their codes at about 127 for 3.5 deviations."""
  for part in (t if t.ndim == 5 else [t]):
    x = torch.randn(part.shape, generator=g, device=DEV, dtype=torch.bfloat16)
    part.copy_(x.mul_(36).round_().clamp_(-127, 127) if part.dtype == torch.int8 else x)


def _fill_scales(g, t):
  t.copy_((torch.rand(t.shape, generator=g, device=DEV) * 0.6 + 3.2) / 127)


def _lengths(seed, batch, low, high):
  """Lengths spread evenly over [low, high], in an order of the seed (every seed has the same sum)."""
  at = low + (np.arange(batch) + 0.5) / batch * (high - low)
  return np.random.RandomState(seed % (1 << 31)).permutation(np.round(at).astype(np.int64))


def _env(case, **more):
  quant = QuantizationConfig(enable_kv_quantization=case.get("cache") == "int8")
  return JetEngineEnvironment(JetEngineEnvironmentData(quant_config=quant, **more), device=DEV)


def _prepare_step(case, seed):
  g = _gen(seed)
  b, hq, hkv, s, nl = (case[k] for k in ("batch", "hq", "hkv", "seq", "layers"))
  env = _env(case, batch_size=b, cache_sequence_length=s, cache_shape=(b, hkv, s, D), num_layers=nl,
             ring_buffer=case["ring"])
  kernel = layers.Int8KVAttentionKernel if case["cache"] == "int8" else layers.AttentionKernel
  kernels = [kernel(env, i) for i in range(nl)]

  def model(params, tokens, input_pos, caches, mask, start, rbi, rbk):
    for i, attend in enumerate(kernels):
      q, k, v = params["qkv"][i]
      cache = caches[0] if env.generate_cache_stacked else caches[i]
      params["out"][i] = attend(q, k, v, mask, cache, start=start, end=input_pos, ragged_batch_index=rbi,
                                ragged_block_index=rbk)
    return params["logits"]

  engine = KVCacheEngine(env, model)
  ds = engine.init_decode_state()
  for pair in ds.caches:
    for t in pair:
      _fill_cache(g, t)
  for pair in ds.cache_scales:
    for t in pair:
      _fill_scales(g, t)
  lens = torch.from_numpy(_lengths(seed, b, 1, s - 1)).to(DEV)
  at = torch.arange(s, device=DEV)[None, :]
  if case["ring"]:
    ds.current_position = s // 3
    begin = (ds.current_position - lens) % s
    valid = (at - begin[:, None]) % s < lens[:, None]
  else:
    begin = torch.zeros_like(lens)
    valid = at < lens[:, None]
  ds.start.copy_(begin)
  ds.input_pos.copy_(lens)
  ds.lens.copy_(1 + lens[:, None] % 100)
  ds.mask.masked_fill_(valid, 0.0)
  ds.tokens.copy_(torch.randint(0, VOCAB, (b, 1), generator=g, device=DEV))
  params = {"qkv": [(_randn(g, b, hq, 1, D), _randn(g, b, hkv, 1, D), _randn(g, b, hkv, 1, D)) for _ in range(nl)],
            "logits": torch.randn((b, 1, VOCAB), generator=g, device=DEV), "out": [None] * nl}
  return dict(engine=engine, ds=ds, params=params)


def _run_step(st):
  new, data = st["engine"].generate(st["params"], st["ds"])
  return dict(out=list(st["params"]["out"]), data=data, tokens=new.tokens, caches=new.caches, scales=new.cache_scales,
              position=new.current_position, lens=new.lens, input_pos=new.input_pos, mask=new.mask)


PAGE = 64


def _prepare_paged(case, seed):
  g = _gen(seed)
  b, hq, hkv, nl = (case[k] for k in ("batch", "hq", "hkv", "layers"))
  int8 = case["cache"] == "int8"
  lens = _lengths(seed, b, case["low"], case["high"])
  most = 2048 // PAGE
  total = int(sum(n // PAGE + 1 for n in lens)) + 8
  order = np.random.RandomState(seed % (1 << 31)).permutation(total).tolist()
  pam = PageAttentionManager(b, total, PAGE, most, free_page_order=order)
  for slot in range(b):
    pam.reserve_pages_insert(slot, int(lens[slot]))
  pam.fill_new_pages(lens)
  env = _env(case, batch_size=b, cache_sequence_length=2048, num_layers=nl, ring_buffer=False,
             paged_attention_total_num_pages=total, paged_attention_page_size=PAGE)
  pools = []
  for _ in range(nl):
    k, v = (torch.empty((hkv, total, PAGE, D), dtype=torch.int8 if int8 else torch.bfloat16, device=DEV) for _ in range(2))
    _fill_cache(g, k)
    _fill_cache(g, v)
    ks = vs = None
    if int8:
      ks, vs = (torch.empty((1, total, PAGE, 1), dtype=torch.bfloat16, device=DEV) for _ in range(2))
      _fill_scales(g, ks)
      _fill_scales(g, vs)
    pools.append((k, v, ks, vs))
  table, _ = pam.device_tables(DEV)
  return dict(env=env, pam=pam, table=table, lens=torch.from_numpy(lens.astype(np.int32)).to(DEV), pools=pools,
              kernels=[layers.AttentionKernel(env, i) for i in range(nl)],
              qkv=[(_randn(g, b, hq, 1, D), _randn(g, b, hkv, 1, D), _randn(g, b, hkv, 1, D)) for _ in range(nl)])


def _run_paged(st):
  pam, env = st["pam"], st["env"]
  pti, active, lengths = pam.get_page_token_indices_device(st["lens"], st["table"])
  pam.lengths_device, pam.page_indices_device = lengths, st["table"]
  outs = []
  for i, (k, v, ks, vs) in enumerate(st["pools"]):
    q, xk, xv = st["qkv"][i]
    cache = PageKVCacheGenerate(k, v, pam, pti, None, env=env, k_scaler=ks, v_scaler=vs, n_active_dev=active)
    if ks is None:
      outs.append(st["kernels"][i](q, xk, xv, None, cache))
    else:
      cache.update(xk, xv, i)
      outs.append(ak.call_paged_attention(env, q.squeeze(2), k, v, lengths, st["table"], k_scaler=ks, v_scaler=vs))
  return dict(out=outs, pools=st["pools"], indices=pti, lengths=lengths)


def _prepare_prefill(case, seed):
  g = _gen(seed)
  hq, hkv, n = case["hq"], case["hkv"], case["length"]
  env = _env(case, batch_size=1, cache_sequence_length=2048, num_layers=1, ring_buffer=False)
  kernel = layers.Int8KVAttentionKernel if case["quantized"] else layers.AttentionKernel
  mask = torch.full((n, n), float("-inf"), dtype=torch.bfloat16, device=DEV).triu(1)
  return dict(kernel=kernel(env, 0), quantized=case["quantized"], mask=mask.repeat(hq // hkv, 1)[None, None],
              q=_heads_first(g, n, hq), k=_heads_first(g, n, hkv), v=_heads_first(g, n, hkv))


def _run_prefill(st):
  cache = KVCachePrefill(kv_quantize=st["quantized"])
  out = st["kernel"](st["q"], st["k"], st["v"], st["mask"], cache)
  return dict(out=out)


def _prepare_insert(case, seed):
  g = _gen(seed)
  b, hkv, s, nl = (case[k] for k in ("batch", "hkv", "seq", "layers"))
  env = _env(case, batch_size=b, cache_sequence_length=s, cache_shape=(b, hkv, s, D), num_layers=nl, ring_buffer=False)
  engine = KVCacheEngine(env)
  prefix = Prefix(torch.randint(0, VOCAB, (1, 1), generator=g, device=DEV),
                  [(_heads_first(g, case["padded"], hkv), _heads_first(g, case["padded"], hkv)) for _ in range(nl)],
                  case["length"])
  return dict(engine=engine, ds=engine.init_decode_state(), prefix=prefix, slot=b // 2)


def _run_insert(st):
  ds = st["engine"].insert(st["prefix"], st["ds"], st["slot"])
  return dict(caches=ds.caches, scales=ds.cache_scales, tokens=ds.tokens, mask=ds.mask, start=ds.start,
              input_pos=ds.input_pos, lens=ds.lens)


def _prepare_pages(case, seed):
  g = _gen(seed)
  hkv, nl, n = case["hkv"], case["layers"], case["length"]
  int8 = case.get("cache", "int8") == "int8"
  total = 8 * 2048 // PAGE
  rng = np.random.RandomState(seed % (1 << 31))
  pam = PageAttentionManager(8, total, PAGE, 2048 // PAGE, free_page_order=rng.permutation(total).tolist())
  pool_k, pool_v = (torch.zeros((nl, hkv, total, PAGE, D), dtype=torch.int8 if int8 else torch.bfloat16, device=DEV)
                    for _ in range(2))
  scale_k, scale_v = ((torch.ones((nl, 1, total, PAGE, 1), dtype=torch.bfloat16, device=DEV) for _ in range(2))
                      if int8 else (None, None))
  if case["stacked"]:
    at = list(range(nl))
    pk, pv = _randn(g, nl, 1, hkv, n, D), _randn(g, nl, 1, hkv, n, D)
    prefix = [(pk[i], pv[i]) for i in range(nl)]
  else:  # every layer's pools and prefix lie where they happened to be allocated
    at = rng.permutation(nl).tolist()
    prefix = [(_heads_first(g, n, hkv), _heads_first(g, n, hkv)) for _ in range(nl)]
  return dict(pam=pam, prefix=prefix, length=n, pools=[(pool_k[i], pool_v[i]) for i in at],
              scales=[(scale_k[i], scale_v[i]) for i in at] if int8 else None, whole=(pool_k, pool_v, scale_k, scale_v))


def _run_pages(st):
  insert_ops.insert_page_attention_with_reservation(st["pam"], st["prefix"], st["length"], st["pools"], 3,
                                                    cache_scales=st["scales"])
  st["pam"].free_pages_resource(3)  # the sequence is done
  return dict(pools=st["whole"])


def _linear(g, k, n):
  m = layers.WeightOnlyPerChannelQuantizedLinear(k, n, device=DEV)
  m.quantize_weight_from_nn_linear(torch.randn((n, k), generator=g, device=DEV) / math.sqrt(k))
  return m


def _prepare_ffn(case, seed):
  g = _gen(seed)
  dim, hidden = case["dim"], case["hidden"]
  norm = layers.RMSNorm(dim, device=DEV)
  norm.weight.data.copy_(1 + 0.1 * _randn(g, dim))
  block = layers.FeedForward(dim, hidden, device="meta")
  block.w1, block.w2, block.w3 = _linear(g, dim, hidden), _linear(g, hidden, dim), _linear(g, dim, hidden)
  return dict(norm=norm, block=block, x=_randn(g, case["rows"], dim))


def _run_ffn(st):
  x = st["x"]
  if layers.ActivationLevels.fits(x):
    y, levels = st["norm"](x, with_levels=True)
    return dict(out=st["block"](y, levels=levels), normed=y)
  y = st["norm"](x)
  return dict(out=st["block"](y), normed=y)


def _prepare_linear(case, seed):
  g = _gen(seed)
  return dict(layer=_linear(g, case["k"], case["n"]), x=_randn(g, case["rows"], case["k"]))


def _run_linear(st):
  return dict(out=st["layer"](st["x"]))


_PREPARE = {"step": _prepare_step, "paged": _prepare_paged, "prefill": _prepare_prefill, "insert": _prepare_insert,
            "pages": _prepare_pages, "ffn": _prepare_ffn, "linear": _prepare_linear}
_RUN = {"step": _run_step, "paged": _run_paged, "prefill": _run_prefill, "insert": _run_insert, "pages": _run_pages,
        "ffn": _run_ffn, "linear": _run_linear}


def prepare(case, seed):
  return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
  return _RUN[state["kind"]](state)


# ------------------------------------------------------------- work, tolerance


def work(case):
  kind = case["kind"]
  if kind in ("step", "paged"):
    b, hq, hkv, nl = (case[k] for k in ("batch", "hq", "hkv", "layers"))
    e, scale = (1, 2) if case["cache"] == "int8" else (2, 0)
    low, high = (1, case["seq"] - 1) if kind == "step" else (case["low"], case["high"])
    tokens = b * ((low + high) / 2 + 1)  # with the step's own
    out = 4 if kind == "step" and not case["ring"] else 2  # the lazy forms return float32
    layer = tokens * 2 * (hkv * D * e + scale)  # the cache, read once
    layer += b * D * (hq * (2 + out) + hkv * 2 * 2) + b * 2 * (hkv * D * e + scale)  # q, o, the new token in, its row out
    other = b * 40
    if kind == "step":
      other += b * VOCAB * 4
      if case["ring"]:
        layer += b * case["seq"] * 2  # the mask selects the tokens
    return {"bytes": nl * layer + other, "flops": nl * 4 * tokens * hq * D}
  if kind == "prefill":
    hq, hkv, n = case["hq"], case["hkv"], case["length"]
    # the mask is an input of the call like the others; its zeros select half of the scores
    return {"bytes": 2 * n * D * 2 * (hq + hkv) + 2 * (hq // hkv) * n * n, "flops": 4 * hq * D * n * (n + 1) / 2}
  if kind in ("insert", "pages"):
    hkv, nl = case["hkv"], case["layers"]
    e, scale = (1, 2) if case.get("cache", "int8") == "int8" else (2, 0)
    tokens = case["padded"] if kind == "insert" else case["length"]
    rows = tokens if kind == "insert" else -(-tokens // PAGE) * PAGE
    return {"bytes": nl * 2 * (tokens * hkv * D * 2 + rows * (hkv * D * e + scale)), "flops": 0}
  if kind == "ffn":
    d, h, m = case["dim"], case["hidden"], case["rows"]
    return {"bytes": 3 * d * h + 2 * (2 * h + d) + 2 * d + 3 * 2 * m * d, "flops": 6 * m * d * h}
  k, n, m = case["k"], case["n"], case["rows"]
  return {"bytes": k * n + 2 * n + 2 * m * (k + n), "flops": 2 * m * k * n}


def tolerance(case):
  if case["kind"] in ("insert", "pages"):
    return "exact"  # codes, scales and rows follow from the inputs bit for bit
  return {"rel": 1e-2}  # bf16 results (attention rows, linear layers); codes and tables are whole numbers: none may differ
