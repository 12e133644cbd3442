"""What is timed: calls that a user of this package makes, from one small matrix-vector product to whole prompts.

kind           entry points                                             what it stands for
gemv           bpd_qmatmul_q4k_q8k_cuda, bpd_qmatmul_q4k_gpu_st,        one product of a decode loop that calls operator by operator
               bpd_qmatmul_q8_0_cuda
dequant        bpd_dequant_q4k_gpu_st                                   a tensor unpacked to fp32
gemm           bpd_qmm_q4k_q8k_cuda                                     a few tokens at once (batched decoding, speculative drafts)
layer_set      bpdq_gemv_stream_run, bpdq_gemm_rg16_stream_run          all products of a decode step as persistent launches
llama          bpd_llama_forward_tiles_cuda                             a Q8_0 Llama: a prompt, or a token against a filled cache
hybrid,        Engine.feed / Engine.end over DeviceHybrid               the two hybrid decoders: a prompt from an empty sequence, or a
vuzelix                                                                 token against a filled one

Shapes are Mistral-7B's, Llama-3-8B's (fewer layers, a vocabulary of 32000) and those of measure.py's hybrid decoders.  Weights of
the quantized products are drawn per seed; a hybrid decoder is loaded once per process and shape, as a server does, and the
sequences' tokens are drawn per seed.
"""
import ctypes as C
import math

import numpy as np
import torch

from bpd_substrate_b200 import capi, hybrid, synth, vuzelix
from bpd_substrate_b200.engine import Engine
from bpd_substrate_b200.llama import LAYER_FIELDS, make_config

LAYER = tuple((rows, cols) for _, rows, cols in synth.MISTRAL_LAYER)
F64 = torch.float64


def listed():
    return [
        # latency: the smallest matrix of a layer (wk / wv) as one call
        {"name": "gemv_q4k_1024x4096", "kind": "gemv", "format": "q4k_q8k", "rows": 1024, "cols": 4096},
        # the Q8_0 product of the reference's benchmark
        {"name": "gemv_q8_0_4096x4096", "kind": "gemv", "format": "q8_0", "rows": 4096, "cols": 4096},
        # the reference's own GPU operator: fp32 activations, a feed-forward matrix
        {"name": "gemv_q4k_f32_14336x4096", "kind": "gemv", "format": "q4k_f32", "rows": 14336, "cols": 4096},
        # one feed-forward tensor unpacked
        {"name": "dequant_14336x4096", "kind": "dequant", "blocks": 229376},
        # batched decoding: 16 sequences through a feed-forward matrix
        {"name": "gemm_q4k_16x14336x4096", "kind": "gemm", "tokens": 16, "rows": 14336, "cols": 4096},
        # a larger, ragged batch through the matrix of long rows
        {"name": "gemm_q4k_61x4096x14336", "kind": "gemm", "tokens": 61, "rows": 4096, "cols": 14336},
        # every product of a token through 32 layers: the headline workload
        {"name": "layer_set_32", "kind": "layer_set", "layers": 32, "tokens": 1},
        # a decoded token late in a conversation
        {"name": "llama_decode_4000", "kind": "llama", "layers": 4, "heads": 32, "kv_heads": 8, "dim": 128, "ff": 14336, "tokens": 1, "context": 4000, "f16": True},
        # a prompt of a page or two
        {"name": "llama_prefill_1000", "kind": "llama", "layers": 4, "heads": 32, "kv_heads": 8, "dim": 128, "ff": 14336, "tokens": 1000, "context": 0, "f16": True},
        {"name": "hybrid_decode_4000", "kind": "hybrid", "width": 2048, "layers": 4, "tokens": 1, "context": 4000, "dtype": "bfloat16"},
        {"name": "hybrid_prefill_2048", "kind": "hybrid", "width": 2048, "layers": 4, "tokens": 2048, "context": 0, "dtype": "bfloat16"},
        {"name": "vuzelix_prefill_700", "kind": "vuzelix", "width": 2048, "layers": 4, "tokens": 700, "context": 0, "dtype": "bfloat16"},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "dequant", "gemm", "gemm", "layer_set", "llama", "llama", "hybrid", "hybrid", "vuzelix", "vuzelix"])
    if kind == "gemv":
        cols = 256 * _spread(rng, 4, 56)
        return {"kind": kind, "format": rng.choice(["q4k_q8k", "q4k_f32", "q8_0"]), "rows": _spread(rng, 500, 14336 * 4096 // cols), "cols": cols}
    if kind == "dequant":
        return {"kind": kind, "blocks": _spread(rng, 3000, 229376)}
    if kind == "gemm":
        cols = 256 * _spread(rng, 4, 56)
        return {"kind": kind, "tokens": _spread(rng, 2, 64), "rows": _spread(rng, 500, 14336 * 4096 // cols), "cols": cols}
    if kind == "layer_set":
        return {"kind": kind, "layers": _spread(rng, 1, 31), "tokens": rng.choice([1, 1, 1, 8])}
    one = rng.random() < 0.5
    context = _spread(rng, 40, 4000) if one else 0
    if kind == "llama":
        heads, kv_heads, dim, ff = rng.choice([(32, 8, 128, 14336), (32, 8, 128, 11008), (32, 32, 64, 5632), (16, 4, 64, 4096)])
        return {"kind": kind, "layers": rng.randint(1, 4), "heads": heads, "kv_heads": kv_heads, "dim": dim, "ff": ff,
                "tokens": 1 if one else _spread(rng, 3, 999), "context": context, "f16": rng.random() < 0.75}
    dtype = "float32" if rng.random() < 0.2 else "bfloat16"
    return {"kind": kind, "width": rng.choice([1024, 1536, 2048]), "layers": rng.randint(2, 4),
            "tokens": 1 if one else _spread(rng, 12, 2047 if dtype == "bfloat16" else 300), "context": context, "dtype": dtype}


# ---- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _normal(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _q4k(g, rows, cols):
    """Q4_K rows: fp16 |N(0, 0.02)| scales, everything else uniform bytes (6-bit scales and mins, nibbles)."""
    blocks = rows * cols // 256
    raw = torch.randint(0, 256, (blocks, 144), device="cuda", generator=g, dtype=torch.uint8)
    raw[:, :4] = (0.02 * _normal(g, blocks, 2)).abs().half().view(torch.uint8)
    return raw.view(rows, cols // 256, 144)


def _q8_0(g, rows, cols, sigma):
    """Q8_0 rows: fp16 |N(0, sigma)| scales, int8 uniform on [-127, 127]."""
    blocks = rows * cols // 32
    raw = torch.empty(blocks, 34, device="cuda", dtype=torch.uint8)
    raw[:, :2] = (sigma * _normal(g, blocks, 1)).abs().half().view(torch.uint8)
    raw[:, 2:] = torch.randint(-127, 128, (blocks, 32), device="cuda", generator=g, dtype=torch.int8).view(torch.uint8)
    return raw.view(rows, cols // 32, 34)


def _stream():
    return torch.cuda.current_stream().cuda_stream


class State(dict):
    """A case's state: named tensors and handles; `free` gives handles back."""
    free = None

    def __del__(self):
        if self.free is not None:
            self.free()


def prepare(case, seed):
    return {"gemv": _prepare_gemv, "dequant": _prepare_dequant, "gemm": _prepare_gemm, "layer_set": _prepare_layer_set,
            "llama": _prepare_llama, "hybrid": _prepare_decoder, "vuzelix": _prepare_decoder}[case["kind"]](case, seed)


def run(state):
    return {"llama": _run_llama, "hybrid": _run_decoder, "vuzelix": _run_decoder}.get(state["case"]["kind"], _run_call)(state)


def _prepare_gemv(case, seed):
    g, rows, cols = _gen(seed), case["rows"], case["cols"]
    w = _q8_0(g, rows, cols, 0.01) if case["format"] == "q8_0" else _q4k(g, rows, cols)
    lib, s = capi.load(), State(case=case, w=w, x=_normal(g, cols), out=torch.empty(rows, device="cuda"))
    entry = {"q4k_q8k": lib.bpd_qmatmul_q4k_q8k_cuda, "q4k_f32": lib.bpd_qmatmul_q4k_gpu_st, "q8_0": lib.bpd_qmatmul_q8_0_cuda}[case["format"]]
    sizes = (1, rows, cols) if case["format"] == "q8_0" else (rows, cols)
    s["call"] = entry, (w.data_ptr(), s["x"].data_ptr(), s["out"].data_ptr(), *sizes, _stream())
    return s


def _run_call(s):
    entry, args = s["call"]
    capi.check(entry(*args))
    return s["out"]


def _prepare_dequant(case, seed):
    s = State(case=case, w=_q4k(_gen(seed), case["blocks"], 256), out=torch.empty(case["blocks"], 256, device="cuda"))
    s["call"] = capi.load().bpd_dequant_q4k_gpu_st, (s["w"].data_ptr(), s["out"].data_ptr(), case["blocks"], 0, _stream())
    return s


def _prepare_gemm(case, seed):
    g, n, rows, cols = _gen(seed), case["tokens"], case["rows"], case["cols"]
    s = State(case=case, w=_q4k(g, rows, cols), x=_normal(g, n, cols), out=torch.empty(n, rows, device="cuda"))
    s["call"] = capi.load().bpd_qmm_q4k_q8k_cuda, (s["w"].data_ptr(), s["x"].data_ptr(), s["out"].data_ptr(), n, rows, cols, 0, 0, None, _stream())
    return s


def _prepare_layer_set(case, seed):
    """Weights resident, one arena of activations and one of outputs, and the plan of the persistent launches; with several
    tokens the weights are held re-tiled."""
    lib, g, layers, n = capi.load(), _gen(seed), case["layers"], case["tokens"]
    shapes = LAYER * layers
    s = State(case=case, x=_normal(g, n * sum(k for _, k in shapes)), out=torch.empty(n * sum(m for m, _ in shapes), device="cuda"), w=[])
    descs, xo, oo = (capi.GemvDesc * len(shapes))(), 0, 0
    for j, (m, k) in enumerate(shapes):
        w = _q4k(g, m, k)
        if n > 1:
            tiles = torch.empty(lib.bpd_q4k_rg16_bytes(m, k), device="cuda", dtype=torch.uint8)
            capi.check(lib.bpd_repack_q4k_rg16_cuda(w.data_ptr(), tiles.data_ptr(), m, k, _stream()))
            w = tiles
        s["w"].append(w)
        descs[j] = capi.GemvDesc(w.data_ptr(), s["x"].data_ptr() + 4 * xo, s["out"].data_ptr() + 4 * oo, m, k)
        xo, oo = xo + n * k, oo + n * m
    if n > 1:
        size = lib.bpdq_gemm_rg16_stream_workspace_bytes(len(descs), descs, n)
        s["ws"] = torch.empty(size, device="cuda", dtype=torch.uint8)
        plan, destroy = lib.bpdq_gemm_rg16_stream_create(len(descs), descs, n, s["ws"].data_ptr(), size), lib.bpdq_gemm_rg16_stream_destroy
    else:
        size = lib.bpdq_batch_workspace_bytes(len(descs), descs)
        s["ws"] = torch.empty(size, device="cuda", dtype=torch.uint8)
        plan, destroy = lib.bpdq_gemv_stream_create(len(descs), descs, s["ws"].data_ptr(), size), lib.bpdq_gemv_stream_destroy
    if not plan:
        raise capi.BpdqError("the plan was refused")
    s["call"] = (lib.bpdq_gemm_rg16_stream_run if n > 1 else lib.bpdq_gemv_stream_run), (plan, _stream())
    s.free = lambda: destroy(plan)
    return s


VOCAB = 32000


def _llama_shapes(case):
    e, kv, f = case["heads"] * case["dim"], case["kv_heads"] * case["dim"], case["ff"]
    return {"w_q": (e, e), "w_k": (kv, e), "w_v": (kv, e), "w_o": (e, e), "w_gate": (f, e), "w_up": (f, e), "w_down": (e, f)}


def _llama_tensors(case, seed):
    """Weights (rows of unit norm on average), a cache filled up to `context`, token ids."""
    g, e, n = _gen(seed), case["heads"] * case["dim"], case["tokens"]

    def mat(rows, cols):
        return _q8_0(g, rows, cols, 1.0 / (73.0 * math.sqrt(cols)))

    def norm():
        return 1.0 + 0.1 * _normal(g, e)

    t = {"embed": _q8_0(g, VOCAB, e, 1.0 / 73.0), "out_norm": norm(), "layers": []}
    t["head"] = t["embed"]      # one table for both, as in a file without a head of its own: the greedy choice has a margin
    for _ in range(case["layers"]):
        t["layers"].append({f: norm() if f.endswith("norm_w") else mat(*_llama_shapes(case)[f]) for f in LAYER_FIELDS})
    shape = (case["layers"], case["context"] + n, case["kv_heads"] * case["dim"])
    kind = torch.float16 if case["f16"] else torch.float32
    t["k"], t["v"] = _normal(g, *shape, dtype=kind), _normal(g, *shape, dtype=kind)
    t["k"][:, case["context"]:] = 0
    t["v"][:, case["context"]:] = 0
    t["tokens"] = torch.randint(0, VOCAB, (n,), device="cuda", generator=g, dtype=torch.int32)
    t["pos"] = torch.arange(case["context"], case["context"] + n, device="cuda", dtype=torch.int32)
    return t


def _llama_structs(t, layers):
    arr = (capi.LlamaLayerWeights * len(layers))()
    for i, layer in enumerate(layers):
        for f, v in layer.items():
            setattr(arr[i], f, v.data_ptr())
    return capi.LlamaWeights(t["embed"].data_ptr(), arr, t["out_norm"].data_ptr(), t["head"].data_ptr(), None)


def _prepare_llama(case, seed):
    """A prompt runs on the re-tiled copies of the matrices, as DeviceLlama.retile makes them."""
    lib, t, n = capi.load(), _llama_tensors(case, seed), case["tokens"]
    s = State(t, case=case, logits=torch.empty(n, VOCAB, device="cuda"), picked=torch.empty(n, device="cuda", dtype=torch.int64))
    cfg = make_config(case["layers"], case["heads"], case["kv_heads"], case["dim"], case["ff"], VOCAB, case["context"] + n,
                      kv_cache_f16=int(case["f16"]))
    tiles = None
    if n > 1:
        def tile(w, rows, cols):
            out = torch.empty(lib.bpd_q8_0_tiles_bytes(rows, cols), device="cuda", dtype=torch.uint8)
            capi.check(lib.bpd_repack_q8_0_tiles_cuda(w.data_ptr(), out.data_ptr(), rows, cols, _stream()))
            return out
        e = case["heads"] * case["dim"]
        s["tiled"] = dict(t, layers=[{f: tile(layer[f], *shape) for f, shape in _llama_shapes(case).items()} for layer in t["layers"]],
                          head=tile(t["head"], VOCAB, e))
        tiles = C.byref(_llama_structs(s["tiled"], s["tiled"]["layers"]))
    s["call"] = lib.bpd_llama_forward_tiles_cuda, (t["tokens"].data_ptr(), n, C.byref(_llama_structs(t, t["layers"])), tiles, C.byref(cfg),
                                                   t["pos"].data_ptr(), case["context"], t["k"].data_ptr(), t["v"].data_ptr(),
                                                   s["logits"].data_ptr(), s["picked"].data_ptr(), _stream())
    return s


def _run_llama(s):
    entry, args = s["call"]
    capi.check(entry(*args))
    return {"logits": s["logits"], "picked": s["picked"], "k": s["k"], "v": s["v"]}


def _decoder_config(case):
    """The layers of measure.py's two decoders: every mixer in turn, the last attention layer on an earlier one's cache."""
    w, n = case["width"], case["layers"]
    h = w // 128
    if case["kind"] == "hybrid":
        r = w // 256
        latent = {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 3 * w // 8, "scale": 192 ** -0.5,
                  "rot": {"dims": 64, "base": 500000.0}}
        mixers = [("retention", {"heads": r, "dim": 256, "vdim": 256, "rot": {"dims": 256, "base": 10000.0},
                                 "decay": [1.0 - 2.0 ** (-5 - i * 7.0 / max(1, r - 1)) for i in range(r)]}),
                  ("mamba2", {"heads": w // 32, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}),
                  ("latent_attention", latent), ("latent_attention", dict(latent, kv_from=2))]
        return {"architecture": "Gurusun", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-6},
                "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": w * 7 // 2}} for t, m in mixers[:n]]}
    delta = {"heads": h, "kv_heads": h, "dim": 128, "vdim": 128, "conv": 4}
    grouped = {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5 * 4, "softcap": 50.0, "mask": {"size": 8192}}
    mixers = [("channel_delta", delta), ("attention", grouped), ("channel_delta", delta), ("attention", dict(grouped, kv_from=1))]
    return {"architecture": "Vuzelix", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-6}, "embedding": {"scale": w ** 0.5}, "streams": 4,
            "residual_mult": 0.5, "logit_softcap": 30.0,
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": w * 21 // 4}} for t, m in mixers[:n]]}


def _decoder_spec(case):
    config = _decoder_config(case)
    if case["kind"] == "hybrid":
        return hybrid.HybridSpec(config)
    spec = vuzelix.VuzelixSpec(config)
    spec.ranks = {i: (128, 128) for i, la in enumerate(config["layers"]) if la["type"] == "channel_delta"}
    return spec


def _decoder_tensors(spec):
    """A checkpoint's tensors as bf16 bits: matrices that keep activations O(1), the package's own values for the rest."""
    g, rng, out = _gen(1), np.random.default_rng(1), {}
    for name, shape in spec.tensor_shapes().items():
        if name == "embed":
            v = _normal(g, *shape) * (1.0 / spec.embed_scale if hasattr(spec, "embed_scale") else 1.0)
        else:
            v = spec.synthetic_value(name, name.rsplit(".", 1)[-1], shape, rng)
            v = _normal(g, *shape) / math.sqrt(shape[1]) if v is None else torch.from_numpy(np.array(v, np.float32))
        out[name] = v.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)
    if "head" in out:
        out["head"] = out["embed"]      # equal tables: the greedy choice has a margin, as a trained model's has
    return out


CAPACITY = 4096
_loaded = {}        # the decoder that this process serves


def _decoder(case):
    key = (case["kind"], case["width"], case["layers"], case["dtype"])
    if key not in _loaded:
        while _loaded:
            _loaded.popitem()[1].close()
        spec = _decoder_spec(case)
        _loaded[key] = hybrid.DeviceHybrid(spec, hybrid.ArrayTensors(_decoder_tensors(spec)), dtype=case["dtype"], capacity=CAPACITY)
    return _loaded[key]


def _token_ids(case, seed):
    return np.random.default_rng(seed).integers(0, VOCAB, case["context"] + case["tokens"]).astype(np.int32)


def _prepare_decoder(case, seed):
    ids = _token_ids(case, seed)
    engine = Engine(_decoder(case), slots=1, portion=2048)
    s = State(case=case, engine=engine, ids=ids[case["context"]:])
    s.free = engine.close
    if case["context"]:
        engine.feed("sequence", ids[:case["context"]], logits=False)
    return s


def _run_decoder(s):
    engine, c = s["engine"], s["case"]
    logits, picked = engine.feed("sequence", s["ids"], [c["tokens"] - 1])
    if c["context"]:
        engine.live["sequence"].length = c["context"]     # the next pass decodes at this position again
    else:
        engine.end("sequence")                             # the next pass is a new request
    return {"logits": logits, "picked": picked}


# ---- what a pass cannot do without

def _matrix_elements(shapes):
    return sum(s[0] * s[1] for s in shapes if len(s) == 2)


def work(case):
    kind = case["kind"]
    if kind == "gemv":
        m, k = case["rows"], case["cols"]
        return {"bytes": (synth.gemv_bytes_q8_0 if case["format"] == "q8_0" else synth.gemv_bytes_q4k)(m, k), "flops": 2 * m * k}
    if kind == "dequant":
        return {"bytes": case["blocks"] * (144 + 1024), "flops": 0}
    if kind == "gemm":
        n, m, k = case["tokens"], case["rows"], case["cols"]
        return {"bytes": synth.gemv_bytes_q4k(m, k, n), "flops": 2 * n * m * k}
    if kind == "layer_set":
        n, size = case["tokens"], sum(m * k for m, k in LAYER)
        return {"bytes": case["layers"] * sum(synth.gemv_bytes_q4k(m, k, n) for m, k in LAYER), "flops": 2 * n * case["layers"] * size}
    n, ctx, layers = case["tokens"], case["context"], case["layers"]
    seen = n * ctx + n * (n + 1) // 2               # pairs of a query and a key it sees
    if kind == "llama":
        e, row = case["heads"] * case["dim"], case["kv_heads"] * case["dim"] * (2 if case["f16"] else 4)
        weights = layers * _matrix_elements(_llama_shapes(case).values()) + VOCAB * e
        moved = weights // 32 * 34 + n * e // 32 * 34 + 2 * layers * (ctx + n) * row + 2 * layers * n * row + n * (4 * VOCAB + 8)
        return {"bytes": moved, "flops": 2 * n * weights + 4 * layers * seen * e}
    spec, a = _decoder_spec(case), 2 if case["dtype"] == "bfloat16" else 4
    shapes, flops, moved = spec.tensor_shapes(), 0, 0
    matrices = {k: s for k, s in shapes.items() if len(s) == 2 and not any(t in k for t in ("conv", "hc")) and k not in ("embed", "head")}
    moved += 2 * _matrix_elements(matrices.values()) + 2 * VOCAB * case["width"] + n * 4 + 4 * VOCAB + 8
    flops += 2 * n * _matrix_elements(matrices.values()) + 2 * VOCAB * case["width"]
    for la in spec.layers:
        m, h = la["mixer"], la["mixer"]["heads"]
        if la["type"] in ("latent_attention", "attention"):
            latent = la["type"] == "latent_attention"
            row = m["kv_rank"] + m["rot_dim"] if latent else m["kv_heads"] * (m["dim"] + m["vdim"])
            moved += a * row * ((ctx + n) + (n if m.get("kv_from") is None else 0))
            flops += 2 * seen * h * (m["dim"] + m["vdim"] + (m["rot_dim"] if latent else 0))
        else:
            state = h * m["vdim"] * (m["state"] if la["type"] == "mamba2" else m["dim"])
            moved += 8 * state
            flops += (6 if la["type"] == "channel_delta" else 4) * n * state
    return {"bytes": moved, "flops": flops}


# About four times the largest distance from 64-bit sums seen over the ranges.  Quantized products add exact integers with fp32
# scales (2e-7); a Llama forward re-quantizes activations to int8 at every product, so a last-bit difference now and then becomes
# one of a whole step (1.3e-2 in the logits of a prompt); bf16 decoders round every activation to 8 bits (3e-3).
def tolerance(case):
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    if kind in ("gemv", "gemm", "layer_set"):
        return {"rel": 8e-7, "max": 1e-5}
    if kind == "llama":
        return {"rel": 3e-2, "max": 0.4, "differ": 0.01}
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5, "max": 6e-5}
    return {"rel": 1.2e-2, "max": 0.06}


# ---- the same results in 64 bits, in plain torch

def _unpack_q4k(raw):
    """[..., blocks, 144] -> [..., blocks, 8, 32] weights; scale and minimum products as exact fp32 numbers in 64 bits."""
    d, dmin = raw[..., 0:2].contiguous().view(torch.float16).to(F64), raw[..., 2:4].contiguous().view(torch.float16).to(F64)
    s = raw[..., 4:16].to(torch.int32)
    lo, mid, hi = s[..., 0:4], s[..., 4:8], s[..., 8:12]
    scale = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], -1).to(F64)
    low = torch.cat([mid & 63, (hi >> 4) | ((mid >> 6) << 4)], -1).to(F64)
    q = raw[..., 16:]
    q = q.reshape(*q.shape[:-1], 8, 16)
    nib = torch.cat([q & 15, q >> 4], -1).to(F64)                    # byte i of a sub-block holds its values i and 16 + i
    return (d * scale)[..., None] * nib - (dmin * low)[..., None]


def _quantized(x, block, half):
    """Activations as int8 blocks give them back: the scale rounded to fp16 (Q8_0) or fp32 (Q8_K)."""
    b = x.float().reshape(*x.shape[:-1], -1, block)
    top = b.abs().amax(-1, keepdim=True)
    limit = torch.full_like(top, 127.0)       # tensors on both sides: a division by or of a number is a product with a reciprocal
    d = top / limit
    q = torch.round(b * torch.where(top > 0, limit / top, 0.0))
    d = d.half() if half else d
    return (q.to(F64) * d.to(F64)).reshape(x.shape)


def _unpack_q8_0(raw):
    return (raw[..., :2].contiguous().view(torch.float16).to(F64) * raw[..., 2:].contiguous().view(torch.int8).to(F64)).flatten(-2)


def _rows_product(raw, x, unpack):
    """x [n, K] times every row, in slices of about 64 million weights."""
    step, out = max(1, (1 << 26) // x.shape[-1]), []
    for at in range(0, raw.shape[0], step):
        w = unpack(raw[at:at + step])
        out.append(x @ w.reshape(w.shape[0], -1).T)
    return torch.cat(out, -1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hybrid", "vuzelix"):
        return _exact_decoder(case, seed)
    if kind == "llama":
        return _exact_llama(case, seed)
    if kind == "layer_set":
        g, n, shapes = _gen(seed), case["tokens"], LAYER * case["layers"]
        x, at, out = _normal(g, n * sum(k for _, k in shapes)), 0, []
        for m, k in shapes:
            out.append(_rows_product(_q4k(g, m, k), _quantized(x[at:at + n * k].view(n, k), 256, False), _unpack_q4k).flatten())
            at += n * k
        return torch.cat(out)
    s = prepare(case, seed)
    if kind == "dequant":
        return _unpack_q4k(s["w"]).reshape(case["blocks"], 256)
    x = s["x"].view(-1, case["cols"])
    if case.get("format") == "q8_0":
        out = _rows_product(s["w"], _quantized(x, 32, True), _unpack_q8_0)
    else:
        out = _rows_product(s["w"], x.to(F64) if case.get("format") == "q4k_f32" else _quantized(x, 256, False), _unpack_q4k)
    return out if kind == "gemm" else out[0]


def _exact_llama(case, seed):
    # One rounding's difference in a product's int8 input is a difference of 1e-3 behind it.  A prompt of 64 tokens or more has
    # hundreds of these on any path, and its distance from 64 bits is steady (1.3e-2); with a few tokens it is 1e-7 or 1e-2 by
    # chance, whatever computed it, and says nothing.
    if case["tokens"] < 64:
        return None
    t, n, ctx = _llama_tensors(case, seed), case["tokens"], case["context"]
    heads, kv_heads, dim = case["heads"], case["kv_heads"], case["dim"]
    kind, eps = t["k"].dtype, 1e-5
    # the angles are defined by fp32 steps: pos, times a constant once per pair
    angle, step = [t["pos"].float()], torch.tensor(np.float32(500000.0) ** np.float32(-2.0 / dim), device="cuda", dtype=torch.float32)
    for _ in range(dim // 2 - 1):
        angle.append(angle[-1] * step)
    angle = torch.stack(angle, -1).to(F64)[:, None]

    def norm(x, w):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F64)

    def product(w, x):
        return _rows_product(w, _quantized(x, 32, True), _unpack_q8_0)

    def turn(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()], -1).flatten(-2)

    x, ks, vs = _unpack_q8_0(t["embed"][t["tokens"].long()]), t["k"].to(F64), t["v"].to(F64)
    for i, la in enumerate(t["layers"]):
        h = norm(x, la["attn_norm_w"])
        q = turn(product(la["w_q"], h).view(n, heads, dim))
        ks[i, ctx:] = turn(product(la["w_k"], h).view(n, kv_heads, dim)).flatten(1)
        vs[i, ctx:] = product(la["w_v"], h)
        k, v = (c[i].to(kind).to(F64).view(-1, kv_heads, dim) for c in (ks, vs))
        seen = torch.arange(ctx + n, device="cuda")[None] <= t["pos"][:, None]
        out = torch.empty(n, heads, dim, device="cuda", dtype=F64)
        for j in range(heads):
            m = j // (heads // kv_heads)
            p = torch.softmax((q[:, j] @ k[:, m].T * dim ** -0.5).masked_fill(~seen, -math.inf), -1)
            out[:, j] = p @ v[:, m]
        x = x + product(la["w_o"], out.flatten(1))
        h = norm(x, la["ffn_norm_w"])
        x = x + product(la["w_down"], torch.nn.functional.silu(product(la["w_gate"], h)) * product(la["w_up"], h))
    logits = product(t["head"], norm(x, t["out_norm"]))
    return {"logits": logits, "picked": None, "k": ks, "v": vs}


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn_pairs(x, base, interleaved):
    """Rotary embedding of x [T, heads, dims] at positions 0, 1, ..."""
    d = x.shape[-1]
    a = torch.arange(x.shape[0], device="cuda", dtype=F64)[:, None, None] * float(base) ** (-2.0 * torch.arange(d // 2, device="cuda", dtype=F64) / d)
    u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :d // 2], x[..., d // 2:])
    y = (u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin())
    return torch.stack(y, -1).flatten(-2) if interleaved else torch.cat(y, -1)


def _conv(x, w):
    """Causal convolution of every channel, x [T, C], w [C, taps] with the newest tap last."""
    taps = w.shape[1]
    x = torch.cat([torch.zeros(taps - 1, x.shape[1], device="cuda", dtype=F64), x])
    return sum(x[j:x.shape[0] - taps + 1 + j] * w[:, j] for j in range(taps))


def _decayed(q, k, v, log_decay):
    """sum over j <= i of exp(log_decay_{j+1} + ... + log_decay_i) (q_i . k_j) v_j for one head; log_decay [T]."""
    c = torch.cumsum(log_decay, 0)
    mask = torch.ones(len(c), len(c), device="cuda", dtype=torch.bool).tril()
    return ((q @ k.T) * (c[:, None] - c[None]).masked_fill(~mask, -math.inf).exp()) @ v


def _exact_decoder(case, seed):
    spec = _decoder_spec(case)
    w = {k: torch.from_numpy(v.view(np.int16).copy()).cuda().view(torch.bfloat16).to(F64) for k, v in _decoder_tensors(spec).items()}
    ids = torch.from_numpy(_token_ids(case, seed).astype(np.int64)).cuda()
    logits = (_exact_hybrid if case["kind"] == "hybrid" else _exact_vuzelix)(spec.config, w, ids)
    return {"logits": logits[None], "picked": None}


def _exact_hybrid(cfg, w, ids):
    silu, T, eps = torch.nn.functional.silu, len(ids), cfg["norm"]["eps"]
    causal = torch.ones(T, T, device="cuda", dtype=torch.bool).tril()
    caches = {}

    def norm(x, name):
        return torch.tanh(w[name + ".alpha"] * x) * w[name] + w[name + ".b"]

    def mixer(i, la, h):
        m, p = la["mixer"], f"l{i}.mix."
        H = m["heads"]
        if la["type"] == "retention":
            q, k = ((h @ w[p + n].T).view(T, H, m["dim"]) for n in "qk")
            v = (h @ w[p + "v"].T).view(T, H, m["vdim"])
            q, k = (_turn_pairs(z, m["rot"]["base"], False) for z in (q, k))
            o = torch.stack([_decayed(q[:, n], k[:, n] * m["dim"] ** -0.5, v[:, n],
                                      torch.full((T,), math.log(m["decay"][n]), device="cuda", dtype=F64)) for n in range(H)], 1)
            return (_rms(o, eps).flatten(1) * silu(h @ w[p + "g"].T)) @ w[p + "o"].T
        if la["type"] == "mamba2":
            V, N, G = m["vdim"], m["state"], m["groups"]
            inner = H * V
            z, xbc, dt = torch.split(h @ w[p + "in"].T, [inner, inner + 2 * G * N, H], 1)
            xbc = silu(_conv(xbc, w[p + "conv"]) + w[p + "conv.b"])
            x, b, c = torch.split(xbc, [inner, G * N, G * N], 1)
            x, b, c = x.view(T, H, V), b.view(T, G, N), c.view(T, G, N)
            dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"], threshold=100.0)
            log_decay = -torch.exp(w[p + "A_log"]) * dt
            y = torch.stack([_decayed(c[:, n * G // H], b[:, n * G // H] * dt[:, n:n + 1], x[:, n], log_decay[:, n]) + w[p + "D"][n] * x[:, n]
                             for n in range(H)], 1)
            y = y.flatten(1) * silu(z)
            return (_rms(y.view(T, m["norm_groups"], -1), eps).flatten(1) * w[p + "norm"]) @ w[p + "o"].T
        D, r, R = m["dim"], m["rot_dim"], m["kv_rank"]
        if m.get("kv_from") is None:
            u = h @ w[p + "dkv"].T
            caches[i] = (_rms(u[:, :R], eps) * w[p + "dkv.norm"], _turn_pairs(u[:, None, R:], m["rot"]["base"], True)[:, 0])
        c, kr = caches[i if m.get("kv_from") is None else m["kv_from"]]
        q = ((_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T).view(T, H, D + r)
        qr = _turn_pairs(q[..., D:], m["rot"]["base"], True)
        o = []
        for n in range(H):
            s = q[:, n, :D] @ (c @ w[p + "uk"][n * D:(n + 1) * D].T).T + qr[:, n] @ kr.T
            o.append(torch.softmax((s * m["scale"]).masked_fill(~causal, -math.inf), -1) @ (c @ w[p + "uv"].view(H, m["vdim"], R)[n].T))
        return torch.cat(o, 1) @ w[p + "o"].T

    x = w["embed"][ids]
    for i, la in enumerate(cfg["layers"]):
        x = x + norm(mixer(i, la, norm(x, f"l{i}.norm1")), f"l{i}.norm1b")
        h = norm(x, f"l{i}.norm2")
        x = x + norm((silu(h @ w[f"l{i}.mlp.gate"].T) * (h @ w[f"l{i}.mlp.up"].T)) @ w[f"l{i}.mlp.down"].T, f"l{i}.norm2b")
    return w["embed"] @ norm(x[-1], "final.norm")


def _exact_vuzelix(cfg, w, ids):
    silu, T, eps = torch.nn.functional.silu, len(ids), cfg["norm"]["eps"]
    at = torch.arange(T, device="cuda")
    caches = {}

    def delta(m, p, h):
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (silu(_conv(h @ w[p + n].T, w[f"{p}{n}.conv"])) for n in "qkv")
        q, k, v = q.view(T, G, D), k.view(T, G, D), v.view(T, H, V)
        q, k = ((z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for z in (q, k))
        q, beta = q * D ** -0.5, torch.sigmoid(h @ w[p + "b"].T)
        step = torch.nn.functional.softplus((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"], threshold=100.0).view(T, H, D)
        decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * step)
        s, o = torch.zeros(H, D, V, device="cuda", dtype=F64), torch.empty(T, H, V, device="cuda", dtype=F64)
        for i in range(T):
            s = s * decay[i, :, :, None]
            u = beta[i, :, None] * (v[i] - torch.einsum("hdv,hd->hv", s, k[i]))
            s = s + k[i, :, :, None] * u[:, None]
            o[i] = torch.einsum("hdv,hd->hv", s, q[i])
        gate = torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T).view(T, H, V)
        return (_rms(o, eps) * w[p + "norm"] * gate).flatten(1) @ w[p + "o"].T

    def attention(i, m, p, h):
        H, G = m["heads"], m["kv_heads"]
        if m.get("kv_from") is None:
            caches[i] = _rms((h @ w[p + "k"].T).view(T, G, -1), eps), (h @ w[p + "v"].T).view(T, G, -1)
        k, v = caches[i if m.get("kv_from") is None else m["kv_from"]]
        q = _rms((h @ w[p + "q"].T).view(T, H, -1), eps)
        sees = (at[None] <= at[:, None]) & (at[None] // m["mask"]["size"] == at[:, None] // m["mask"]["size"])
        o = []
        for n in range(H):
            s = m["softcap"] * torch.tanh(q[:, n] @ k[:, n * G // H].T * m["scale"] / m["softcap"])
            s = torch.cat([s.masked_fill(~sees, -math.inf), torch.zeros(T, 1, device="cuda", dtype=F64)], 1)      # the sink
            o.append(torch.softmax(s, -1)[:, :-1] @ v[:, n * G // H])
        return torch.cat(o, 1) @ w[p + "o"].T

    x = (w["embed"][ids] * cfg["embedding"]["scale"])[:, None].repeat(1, cfg["streams"], 1)
    for i, la in enumerate(cfg["layers"]):
        for sub in (1, 2):
            hc = f"l{i}.hc{sub}."
            h = _rms(torch.einsum("s,tsw->tw", w[hc + "in"], x), eps) * w[f"l{i}.norm{sub}"]
            if sub == 2:
                y = torch.nn.functional.gelu(h @ w[f"l{i}.mlp.up"].T, approximate="tanh") @ w[f"l{i}.mlp.down"].T
            else:
                y = (delta(la["mixer"], f"l{i}.mix.", h) if la["type"] == "channel_delta" else attention(i, la["mixer"], f"l{i}.mix.", h))
            x = torch.einsum("su,tsw->tuw", w[hc + "mix"], x) + cfg["residual_mult"] * w[hc + "out"][:, None] * y[:, None]
    out = w["head"] @ (_rms(x[-1].sum(0), eps) * w["final.norm"])
    return cfg["logit_softcap"] * torch.tanh(out / cfg["logit_softcap"])
