"""The performance cases of the serving hot path, through its public entry points.

Three kinds of work, at the sizes of the configurations that this repository measures (Llama-3.1-8B,
Qwen2.5-32B at tensor parallel 2, Qwen2.5-0.5B heads):

  attn_decode   one decode step of one attention layer: `RadixAttention.forward` in DECODE mode, which writes
                the new token's K/V to the paged pool and attends over the cached tokens.
  attn_extend   one prefill (extend) of one attention layer over an already cached prefix, EXTEND mode.
  linear        the four linear layers of a decoder layer (qkv, o, gate_up, down), each called on its own
                16-bit activation: unquantised, FP8 per channel, FP8 128x128 blocks, AWQ / GPTQ int4.
  step          whole decode forward over a short stack of unquantised decoder layers with embedding, final norm
                and vocabulary head; returns the logits.  (FP8 layers requantise their activations: a change of
                rounding in one moves the logits by 7e-2, which would hide mistakes.)

Decode-sized calls are replayed from a CUDA graph, as a serving engine runs them ("graph": True); prefill-sized
ones are called directly.  Cached keys and values are N(0, 1) rows at slots in random order, weights are random in
their storage types with scales that keep the outputs near 1.
"""
import math
from types import SimpleNamespace

import torch

from sglang_security_b200.layers.attention.b200_backend import B200AttnBackend
from sglang_security_b200.layers.dense_kernel import gemm_16bit
from sglang_security_b200.layers.linear import ColumnParallelLinear
from sglang_security_b200.layers.quantization.awq import AWQConfig
from sglang_security_b200.layers.quantization.fp8 import Fp8Config
from sglang_security_b200.layers.quantization.gptq import GPTQConfig
from sglang_security_b200.layers.quantization.w8a8_fp8 import W8A8Fp8Config
from sglang_security_b200.layers.radix_attention import RadixAttention
from sglang_security_b200.mem_cache.memory_pool import MHATokenToKVPool, ReqToTokenPool
from sglang_security_b200.model_executor.decode_step import GEOMETRIES, B200DecodeStep
from sglang_security_b200.model_executor.forward_batch_info import ForwardBatch, ForwardMode

DEV = "cuda"
FP8 = torch.float8_e4m3fn
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}

# (query heads, kv heads, head dim): Llama-3.1-8B on one GPU and its shards at tensor parallel 4, Qwen2.5-32B at
# tensor parallel 2, Qwen2.5-0.5B
HEADS = {"llama8b": (32, 8, 128), "llama8b-tp4": (8, 2, 128), "qwen32b-tp2": (20, 4, 128), "qwen0.5b": (14, 2, 64)}

# (N, K) of qkv, o, gate_up, down
LINEARS = {
    "llama8b": ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)),
    "llama8b-tp4": ((1536, 4096), (4096, 1024), (7168, 4096), (4096, 3584)),
    "qwen32b-tp2": ((3584, 5120), (5120, 2560), (27648, 5120), (5120, 13824)),
}


def listed():
    return [
        # one user's chat: a single short request, where launches and latency count
        {"name": "decode_one", "kind": "attn_decode", "heads": "llama8b", "kv": "bf16", "bs": 1, "ctx": 1500,
         "ragged": False, "seed": 1},
        # the headline decode batch: 64 requests of 4k tokens
        {"name": "decode_64x4k", "kind": "attn_decode", "heads": "llama8b", "kv": "bf16", "bs": 64, "ctx": 4096,
         "ragged": False, "seed": 2},
        # a running batch of unequal requests over an FP8 cache
        {"name": "decode_fp8kv_ragged", "kind": "attn_decode", "heads": "llama8b", "kv": "fp8", "bs": 27, "ctx": 6000,
         "ragged": True, "seed": 3},
        # new turns of several chats behind a shared cached prefix (radix hits)
        {"name": "extend_turns", "kind": "attn_extend", "heads": "llama8b", "kv": "bf16", "bs": 8, "prefix": 1536,
         "ext": 512, "ragged": True, "seed": 4},
        # two long fresh prompts
        {"name": "extend_2x8k", "kind": "attn_extend", "heads": "llama8b", "kv": "bf16", "bs": 2, "prefix": 0,
         "ext": 8192, "ragged": False, "seed": 5},
        # an unquantised model's prefill chunk, odd token count
        {"name": "linear_bf16_m777", "kind": "linear", "shape": "llama8b", "quant": "none", "dtype": "bf16", "m": 777},
        # FP8 linears of the headline decode batch
        {"name": "linear_fp8_m64", "kind": "linear", "shape": "llama8b", "quant": "fp8", "dtype": "bf16", "m": 64},
        # FP8 linears of a prefill chunk
        {"name": "linear_fp8_m2048", "kind": "linear", "shape": "llama8b", "quant": "fp8", "dtype": "bf16", "m": 2048},
        # block-scaled FP8 linears of a large prefill chunk, odd token count
        {"name": "linear_block_m3001", "kind": "linear", "shape": "llama8b", "quant": "fp8_block", "dtype": "bf16",
         "m": 3001},
        # int4 linears, one user decoding
        {"name": "linear_awq_m1", "kind": "linear", "shape": "qwen32b-tp2", "quant": "awq", "dtype": "f16", "m": 1},
        # int4 linears of a prefill chunk
        {"name": "linear_awq_m2048", "kind": "linear", "shape": "qwen32b-tp2", "quant": "awq", "dtype": "f16",
         "m": 2048},
        # whole decode forward of a small running batch with the vocabulary head
        {"name": "step_bf16_b16", "kind": "step", "layers": 2, "bs": 16, "ctx": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn_decode", "attn_extend", "attn_extend", "linear", "linear", "linear", "step"])
    if kind == "attn_decode":
        bs = _log(rng, 1, 64)
        return {"kind": kind, "heads": rng.choice(sorted(HEADS)), "kv": rng.choice(["bf16", "f16", "fp8"]), "bs": bs,
                "ctx": _log(rng, 64, min(16384, 262144 // bs)), "ragged": rng.random() < 0.7,
                "seed": rng.randrange(1 << 20)}
    if kind == "attn_extend":
        bs = rng.randint(1, 8)
        ext = _log(rng, 16, 8192 // bs)
        prefix = _log(rng, 16, 8192) if rng.random() < 0.6 else 0
        prefix = min(prefix, max(0, (1 << 26) // (bs * ext) - ext))  # no more score elements than the largest case
        return {"kind": kind, "heads": rng.choice(sorted(HEADS)), "kv": rng.choice(["bf16", "bf16", "f16", "fp8"]),
                "bs": bs, "prefix": prefix, "ext": ext, "ragged": rng.random() < 0.7, "seed": rng.randrange(1 << 20)}
    if kind == "linear":
        return {"kind": kind, "shape": rng.choice(sorted(LINEARS)),
                "quant": rng.choice(["none", "fp8", "fp8", "fp8_block", "fp8_block", "awq", "awq", "gptq"]),
                "dtype": rng.choice(["bf16", "f16"]), "m": _log(rng, 1, 2048)}
    return {"kind": kind, "layers": rng.randint(1, 2), "bs": _log(rng, 1, 64), "ctx": _log(rng, 64, 2048)}


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _lengths(case, most, least):
    """Per-request lengths: a function of the case, so that work() knows them without inputs."""
    if not case["ragged"]:
        return [most] * case["bs"]
    g = torch.Generator().manual_seed(case["seed"])
    u = torch.rand(case["bs"], generator=g).tolist()
    return [max(least, int(most * (0.25 + 0.75 * x))) for x in u]


def _sizes(case):
    """-> (cached prefix lengths, new token counts) of the requests."""
    if case["kind"] == "attn_decode":
        return [n - 1 for n in _lengths(case, case["ctx"], 1)], [1] * case["bs"]
    return [case["prefix"]] * case["bs"], _lengths(case, case["ext"], 1)


def _attention_state(case, seed):
    hq, hkv, d = HEADS[case["heads"]]
    prefix, new = _sizes(case)
    bs, total = case["bs"], sum(prefix) + sum(new)
    act = torch.float16 if case["kv"] == "f16" else torch.bfloat16
    g = _gen(seed)
    longest = max(p + n for p, n in zip(prefix, new))
    pool_dtype = FP8 if case["kv"] == "fp8" else act
    rtp = ReqToTokenPool(bs + 1, (longest + 8) // 4 * 4 + 4, DEV)
    kvp = MHATokenToKVPool(total + 16, 1, pool_dtype, hkv, d, 1, DEV)
    for buf in (kvp.k_buffer[0], kvp.v_buffer[0]):
        rows = torch.randn(buf.shape, device=DEV, generator=g)
        buf.copy_(rows.to(pool_dtype).view(torch.uint8) if pool_dtype == FP8 else rows)
    slots = torch.randperm(total, device=DEV, generator=g) + 1   # page size 1: any slot, in any order
    loc, at = [], 0
    for b in range(bs):
        n = prefix[b] + new[b]
        rtp.req_to_token[b, :n] = slots[at:at + n].to(torch.int32)
        loc.append(slots[at + prefix[b]:at + n])
        at += n
    t = sum(new)
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device=DEV, generator=g).to(act)
    cfg = SimpleNamespace(num_attention_heads=hq, context_len=rtp.max_context_len, get_num_kv_heads=lambda tp: hkv)
    backend = B200AttnBackend(SimpleNamespace(device=DEV, req_to_token_pool=rtp, token_to_kv_pool=kvp,
                                              model_config=cfg, tp_size=1, server_args=SimpleNamespace()))
    lens = torch.tensor([p + n for p, n in zip(prefix, new)], dtype=torch.int64)
    extend = {}
    if case["kind"] == "attn_extend":
        extend = dict(extend_seq_lens=torch.tensor(new, dtype=torch.int32, device=DEV),
                      extend_prefix_lens=torch.tensor(prefix, dtype=torch.int32, device=DEV),
                      extend_seq_lens_cpu=list(new), extend_prefix_lens_cpu=list(prefix), extend_num_tokens=t)
    fb = ForwardBatch(forward_mode=ForwardMode.EXTEND if extend else ForwardMode.DECODE, batch_size=bs,
                      req_pool_indices=torch.arange(bs, dtype=torch.int64, device=DEV), seq_lens=lens.to(DEV),
                      out_cache_loc=torch.cat(loc), seq_lens_sum=total, seq_lens_cpu=lens, req_to_token_pool=rtp,
                      token_to_kv_pool=kvp, attn_backend=backend, **extend)
    layer = RadixAttention(hq, d, d ** -0.5, hkv, 0)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=-1)
    return {"layer": layer, "q": q, "k": k, "v": v, "fb": fb, "pool": kvp}


def _linear_layers(case, g):
    """The four layers with random weights in their storage types, ready after loading."""
    quant, dtype = case["quant"], DTYPES[case["dtype"]]
    cfg = {"none": lambda: None, "fp8": lambda: W8A8Fp8Config(True),
           "fp8_block": lambda: Fp8Config(True, "dynamic", weight_block_size=[128, 128]),
           "awq": lambda: AWQConfig(4, 128, True),
           "gptq": lambda: GPTQConfig(4, 128, False, False, {})}[quant]()
    layers = []
    for n, k in LINEARS[case["shape"]]:
        lin = ColumnParallelLinear(k, n, bias=False, params_dtype=dtype, quant_config=cfg, tp_rank=0,
                                   tp_size=1).to(DEV)
        for name, p in lin.named_parameters(recurse=False):
            if p.dtype == FP8:
                p.data.copy_((torch.randn(p.shape, device=DEV, generator=g) * 0.5).to(FP8))
            elif name == "g_idx":
                p.data.copy_(torch.arange(k, device=DEV) // 128)
            elif p.dtype == torch.int32:
                p.data.copy_(torch.randint(-2 ** 31, 2 ** 31, p.shape, device=DEV, generator=g, dtype=torch.int64)
                             if "zeros" not in name else torch.full(p.shape, 0x77777777, device=DEV))
            elif "scale" in name:
                p.data.copy_((torch.rand(p.shape, device=DEV, generator=g) + 0.5) * (0.002 if p.dtype != torch.float32
                                                                                    else 0.02))
            else:
                p.data.copy_(torch.randn(p.shape, device=DEV, generator=g) * 0.02)
        raw = {name: p.data for name, p in lin.named_parameters(recurse=False)}
        if cfg is not None:
            lin.quant_method.process_weights_after_loading(lin)
        layers.append((lin, raw))
    return layers


def _linear_inputs(case, g):
    return [torch.randn(case["m"], k, device=DEV, generator=g).to(DTYPES[case["dtype"]])
            for _, k in LINEARS[case["shape"]]]


def _step_state(case, seed):
    bs, ctx = case["bs"], case["ctx"]
    step = B200DecodeStep(GEOMETRIES["llama3.1-8b"], None, DEV, max_bs=bs, max_ctx=ctx, layers=case["layers"],
                          seed=seed % (1 << 30), fill_kv=False)
    g = _gen(seed)
    for buf in step.token_to_kv_pool.k_buffer + step.token_to_kv_pool.v_buffer:
        buf.copy_(torch.randn(buf.shape, device=DEV, generator=g))
    slots = (torch.randperm(bs * ctx, device=DEV, generator=g) + 1).view(bs, ctx)
    step.req_to_token_pool.req_to_token[:bs, :ctx] = slots.to(torch.int32)
    fb = step.make_forward_batch(bs, torch.arange(bs, dtype=torch.int64, device=DEV),
                                 torch.full((bs,), ctx, dtype=torch.int64, device=DEV),
                                 slots[:, ctx - 1].contiguous(), bs * ctx)
    return {"step": step, "fb": fb, "positions": torch.full((bs,), ctx - 1, dtype=torch.int64, device=DEV),
            "ids": torch.randint(0, step.g.vocab, (bs,), device=DEV, generator=g)}


def _call(s):
    kind = s["case"]["kind"]
    if kind in ("attn_decode", "attn_extend"):
        s["fb"].attn_backend.init_forward_metadata(s["fb"])
        return s["layer"](s["q"], s["k"], s["v"], s["fb"])
    if kind == "linear":
        return [lin(x)[0] for (lin, _), x in zip(s["layers"], s["x"])]
    step, fb = s["step"], s["fb"]
    step.attn_backend.init_forward_metadata(fb)
    h, residual = step.embed[s["ids"]], None
    for layer in step.layers:
        h, residual = layer(s["positions"], h, fb, residual)
    h, _ = step.final_norm(h, residual)
    return gemm_16bit(h, step.lm_head)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        g = _gen(seed)
        s = {"layers": _linear_layers(case, g), "x": _linear_inputs(case, g)}
    elif kind == "step":
        s = _step_state(case, seed)
    else:
        s = _attention_state(case, seed)
    s["case"] = case
    if kind in ("attn_decode", "step") or (kind == "linear" and case["m"] <= 256):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _call(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["out"] = _call(s)
        s["graph"] = graph
    return s


def run(s):
    if "graph" in s:
        s["graph"].replay()
        out = s["out"]
    else:
        out = _call(s)
    if "pool" in s:     # the cache with the new tokens' rows is an output too
        return {"o": out, "k": s["pool"].k_buffer[0], "v": s["pool"].v_buffer[0]}
    return out


# ---------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind in ("attn_decode", "attn_extend"):
        hq, hkv, d = HEADS[case["heads"]]
        prefix, new = _sizes(case)
        pool = 1 if case["kv"] == "fp8" else 2
        cached, t = sum(prefix), sum(new)
        pairs = sum(n * p + n * (n + 1) // 2 for p, n in zip(prefix, new))
        return {"bytes": 2 * hkv * d * (cached * pool + t * (2 + pool)) + 4 * (cached + t) + 2 * t * hq * d * 2,
                "flops": 4 * hq * d * pairs}
    if kind == "linear":
        m, per_weight = case["m"], {"none": 2, "fp8": 1, "fp8_block": 1, "awq": 0.53, "gptq": 0.53}[case["quant"]]
        nk = LINEARS[case["shape"]]
        return {"bytes": int(sum(n * k * per_weight + 2 * m * (n + k) for n, k in nk)),
                "flops": sum(2 * m * n * k for n, k in nk)}
    g, bs, ctx, layers = GEOMETRIES["llama3.1-8b"], case["bs"], case["ctx"], case["layers"]
    weights = layers * sum(n * k for n, k in LINEARS["llama8b"])
    kv = layers * bs * ctx * 2 * g.kv_heads * g.head_dim
    return {"bytes": 2 * (weights + kv + g.vocab * (g.hidden + bs)),
            "flops": 2 * bs * (weights + g.vocab * g.hidden) + 4 * layers * g.heads * g.head_dim * bs * ctx}


def tolerance(case):
    """Two correct implementations differ by the rounding of the 16-bit result (and of the probabilities), 2.4e-3
    in bf16 and 3e-4 in f16 (up to 1e-3 where a sum tips an FP8 quantiser): four times that.  Through two whole
    layers and the head, other split counts of the attention alone change the logits by 9e-3 (largest 0.05 of
    their root mean square)."""
    if case["kind"] == "step":
        return {"rel": 3e-2, "max": 0.2}
    if case.get("kv") == "f16" or case.get("dtype") == "f16":
        return {"rel": 4e-3}
    return {"rel": 1e-2}


# ---------------------------------------------------------------------------------------------- in 64 bits
def _exact_attention(case, seed):
    s = _attention_state(case, seed)
    hq, hkv, d = HEADS[case["heads"]]
    prefix, new = _sizes(case)
    fb, pool = s["fb"], s["pool"]
    pool_dtype = FP8 if case["kv"] == "fp8" else s["q"].dtype
    caches = []
    for buf, rows in ((pool.k_buffer[0], s["k"]), (pool.v_buffer[0], s["v"])):
        full = buf.view(pool_dtype) if pool_dtype == FP8 else buf
        full = full.to(torch.float32)
        full[fb.out_cache_loc] = rows.reshape(-1, hkv, d).to(pool_dtype).to(torch.float32)
        caches.append(full)
    q = s["q"].reshape(-1, hq, d).double()
    out = torch.empty(q.shape[0], hq * d, dtype=torch.float64, device=DEV)
    at = 0
    for b, (p, n) in enumerate(zip(prefix, new)):
        idx = fb.req_to_token_pool.req_to_token[b, :p + n].long()
        kb, vb = (c[idx].double() for c in caches)
        for lo in range(0, n, 1024):
            hi = min(n, lo + 1024)
            seen = torch.arange(p + n, device=DEV)[None, :] > torch.arange(p + lo, p + hi, device=DEV)[:, None]
            for h in range(hq):
                sc = q[at + lo:at + hi, h] @ kb[:, h // (hq // hkv)].T * d ** -0.5
                sc = sc.masked_fill_(seen, float("-inf")).softmax(-1)
                out[at + lo:at + hi, h * d:(h + 1) * d] = sc @ vb[:, h // (hq // hkv)]
        at += n
    return out


def _dequantised(case, raw, n, k):
    """The weight as [N, K] in 64 bits."""
    quant = case["quant"]
    if quant == "none":
        return raw["weight"].double()
    if quant == "fp8":
        return raw["weight"].double() * raw["weight_scale"].double()
    if quant == "fp8_block":
        sc = raw["weight_scale_inv"].double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
        return raw["weight"].double() * sc
    sc = raw["scales"].repeat_interleave(128, 0)
    if quant == "awq":      # nibble order of the format: 0 4 1 5 2 6 3 7
        shift = torch.tensor([0, 16, 4, 20, 8, 24, 12, 28], device=DEV)
        w = ((raw["qweight"][:, :, None] >> shift) & 15).reshape(k, n)
        return ((w - 7).double() * sc.double()).t()
    shift = torch.arange(0, 32, 4, device=DEV)
    w = ((raw["qweight"][:, None, :] >> shift[None, :, None]) & 15).reshape(k, n)
    return ((w - 8).double() * sc.double()).t()    # the format stores the zero point less one


def _exact_activation(case, x):
    """The activation as the quantiser of the scheme leaves it, in 64 bits."""
    if case["quant"] == "fp8":          # per token: scale = amax / 448, multiply by its reciprocal
        f = x.float()
        s = f.abs().amax(-1, keepdim=True) / 448.0
        return (f * (1.0 / s)).clamp(-448, 448).to(FP8).double() * s.double()
    if case["quant"] == "fp8_block":    # per token and 128 columns
        f = x.float().view(x.shape[0], -1, 128)
        s = f.abs().amax(-1, keepdim=True).clamp(min=1e-10) / 448.0
        return ((f / s).clamp(-448, 448).to(FP8).double() * s.double()).view(x.shape)
    return x.double()


def exact(case, seed):
    if case["kind"] in ("attn_decode", "attn_extend"):
        return {"o": _exact_attention(case, seed), "k": None, "v": None}
    if case["kind"] == "linear":
        g = _gen(seed)
        layers = _linear_layers(case, g)
        return [_exact_activation(case, x) @ _dequantised(case, raw, lin.output_size, lin.input_size).t()
                for (lin, raw), x in zip(layers, _linear_inputs(case, g))]
    return None     # the activations are requantised between layers: a rounding travels through all that follow
