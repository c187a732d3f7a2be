"""Timed workloads of the W8A8 linear path and the decoder stack around it, called through the package's public entry points.

Five kinds of work, each over the range in which a text-to-speech engine meets it:

  linear    one eager ``Context.linear`` over a weight that the loader packed and registered: a head at decode time
  dropin    decoder layers through the C++ drop-in functions with the reference's own signatures, eager, row-major
            weights nobody packed: what an engine that only re-links against the library runs, for one token or a prompt
  decode    one token for every sequence of a batch through the slow-AR stack (36 layers), replayed from a CUDA graph
  frame     one frame of the fast-AR codebook decoder (ten codebook steps of a 4-layer stack and the codebook head), one graph
  prefill   the linear path of one decoder layer over a prompt, through the fused calls of the C ABI, eager

Sizes are the repository's own: hidden 2560, 32 query / 8 kv heads of 128, SwiGLU 9728, groups of 64, 128 or 256,
vocabulary 155776 with 4097 sampled rows, codebooks of 4096, prompts of up to 8192 tokens, at most 2048 tokens of decode
context. Weights are int8 uniform with fp16 group scales. The scales of the stacks are set so that a layer's contribution
is small against the residual stream, as in a trained network: with every layer dwarfing the stream, a last-bit difference
would grow from layer to layer and outputs of two correct implementations could not be compared.
"""
import importlib.util
import math
import sys
from pathlib import Path

import torch

PACKAGE = "fish_audio_cpp_b200"
DIM, HEADS, KV_HEADS, HEAD_DIM, INTER = 2560, 32, 8, 128, 9728
QKV, ATTN = (HEADS + 2 * KV_HEADS) * HEAD_DIM, HEADS * HEAD_DIM
CODEBOOKS, CODEBOOK_SIZE, VOCAB, SAMPLED_ROWS = 10, 4096, 155776, 4097
EPS = 1e-6
# Gains on the weight scales (see above): projections that read a normed row, and w2, which reads a SwiGLU product.
IN_GAIN, DOWN_GAIN = 1.0 / 12, 1.0 / 16


def _package():
    """The package directory carries a hyphen, so it is imported under an explicit module name."""
    if PACKAGE not in sys.modules:
        root = Path.cwd() / "fish-audio-cpp_b200"
        spec = importlib.util.spec_from_file_location(PACKAGE, root / "__init__.py", submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[PACKAGE] = mod
        spec.loader.exec_module(mod)
    return sys.modules[PACKAGE]


_CTX = []


def _context():
    """The program's one library context (one per stream; everything here runs on the current stream)."""
    if not _CTX:
        torch.cuda.set_device(0)
        _CTX.append(_package().Context(0))
    return _CTX[0]


# ---- the cases -----------------------------------------------------------------------------------------------------


def listed():
    return [
        # The rows the decode sampler reads, three sequences in flight: the smallest call, a row count that no tile divides.
        {"name": "sampled_head_m3", "kind": "linear", "tokens": 3, "rows": SAMPLED_ROWS, "k": DIM, "group": 256},
        # The whole vocabulary for a batch of eight: the largest weight there is.
        {"name": "lm_head_m8", "kind": "linear", "tokens": 8, "rows": VOCAB, "k": DIM, "group": 256},
        # An engine that only re-linked: one new token through four layers, groups of 64 (the exporter's default).
        {"name": "dropin_decode_m1_g64", "kind": "dropin", "tokens": 1, "layers": 4, "group": 64, "smooth": False},
        # The same engine over a prompt of odd length, with the exporter's smoothing vectors.
        {"name": "dropin_prompt_m613_g64", "kind": "dropin", "tokens": 613, "layers": 1, "group": 64, "smooth": True},
        # The headline: eight sequences at a context of 1024.
        {"name": "decode_b8_ctx1024_g256", "kind": "decode", "batch": 8, "context": 1024, "group": 256},
        # One listener, near the end of the context window, at a length that no block divides.
        {"name": "decode_b1_ctx1937_g256", "kind": "decode", "batch": 1, "context": 1937, "group": 256},
        # A busy server early in its utterances, groups of 64.
        {"name": "decode_b16_ctx350_g64", "kind": "decode", "batch": 16, "context": 350, "group": 64},
        # A frame of ten codebooks for the headline's batch.
        {"name": "frame_b8_g64", "kind": "frame", "batch": 8, "group": 64},
        # A sentence without a reference voice.
        {"name": "prefill_m150_g64", "kind": "prefill", "tokens": 150, "group": 64},
        # A sentence with a reference voice.
        {"name": "prefill_m2048_g256", "kind": "prefill", "tokens": 2048, "group": 256},
        # A long prompt of odd length, groups of 64.
        {"name": "prefill_m4001_g64", "kind": "prefill", "tokens": 4001, "group": 64},
        # The longest prompt, groups of 256.
        {"name": "prefill_m8192_g256", "kind": "prefill", "tokens": 8192, "group": 256},
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "dropin", "decode", "frame", "prefill", "decode", "prefill"])
    group = rng.choice([64, 64, 128, 256, 256])
    if kind == "linear":
        return {"kind": kind, "tokens": _log_int(rng, 1, 32), "rows": _log_int(rng, 2000, VOCAB),
                "k": rng.choice([1024, DIM, ATTN, INTER]) if rng.random() < 0.5 else DIM, "group": group}
    if kind == "dropin":
        tokens = _log_int(rng, 1, 2048)
        return {"kind": kind, "tokens": tokens, "layers": 4 if tokens <= 32 else 1, "group": group, "smooth": rng.random() < 0.5}
    if kind == "decode":
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "context": _log_int(rng, 20, 2040), "group": group}
    if kind == "frame":
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "group": group}
    return {"kind": kind, "tokens": _log_int(rng, 40, 8192), "group": group}


# ---- inputs --------------------------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _weight(gen, n, k, group, gain=1.0):
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=gen)
    s = (torch.empty((n, k // group), device="cuda").uniform_(1e-3, 5e-3, generator=gen) * gain).half()
    return w, s


def _rows(gen, m, k, gain=1.0):
    """fp16 N(0, 1) rows with one channel in two hundred twenty times larger, the outliers of transformer activations."""
    x = torch.randn((m, k), device="cuda", generator=gen) * gain
    out = torch.randperm(k, device="cuda", generator=gen)[: max(1, k // 200)]
    x[:, out] *= 20
    return x.half()


def _norm(gen, n):
    return torch.empty((n,), device="cuda").uniform_(0.8, 1.2, generator=gen).half()


def _packed(ctx, w, s, group):
    n, k = w.shape
    p = torch.empty((ctx.packed_weight_bytes(n, k, group),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(w, s, n, k, group, p)
    ctx.register_packed_weight(w, p, n, k, group)
    return p


class _State:
    """What the user's program holds; gives its registrations back when it goes."""

    def __init__(self, ctx, kind):
        self.ctx, self.kind, self.registered, self.stack, self.graph = ctx, kind, [], None, None

    def __del__(self):
        try:
            self.graph = None
            if self.stack is not None:
                self.stack.close()
                self.stack.__dict__.clear()  # (the stack refers to itself)
            for w in self.registered:
                self.ctx.register_packed_weight(w, None)
        except Exception:
            pass


def _stack(ctx, layers, batch, context, group, qk_norm, seed, out_gain):
    """A SlowARStack with its scales brought to the gains above (and packed again)."""
    from fish_audio_cpp_b200 import stack as S

    st = S.SlowARStack(torch, ctx, S.SlowARConfig(n_layer=layers, group=group, qk_norm=qk_norm), batch, context, max_new=16,
                       seed=seed)
    for lw in st.layers:
        for w, s, gain in (("wqkv", "sqkv", IN_GAIN), ("wo", "so", out_gain), ("w13", "s13", IN_GAIN), ("w2", "s2", DOWN_GAIN)):
            lw[s].mul_(gain)
            n, k = lw[w].shape
            ctx.pack_weight(lw[w], lw[s], n, k, group, lw[w + "_packed"])
    return st


def _capture(body):
    body()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        body()
    return graph


def prepare(case, seed):
    ctx = _context()
    st = _State(ctx, case["kind"])
    gen = _generator(seed)
    g = case["group"]
    st.group = g
    kind = case["kind"]
    if kind == "linear":
        st.m, st.n, st.k = case["tokens"], case["rows"], case["k"]
        st.w, st.s = _weight(gen, st.n, st.k, g)
        st.packed = _packed(ctx, st.w, st.s, g)
        st.registered.append(st.w)
        st.x = _rows(gen, st.m, st.k)
        st.y = torch.empty((st.m, st.n), dtype=torch.float16, device="cuda")
    elif kind == "dropin":
        m = st.m = case["tokens"]
        st.layers = []
        for _ in range(case["layers"]):
            lw = {"attn_norm": _norm(gen, DIM), "ffn_norm": _norm(gen, DIM)}
            for name, n, k, gain in (("wqkv", QKV, DIM, IN_GAIN), ("wo", DIM, ATTN, IN_GAIN), ("w1", INTER, DIM, IN_GAIN),
                                     ("w3", INTER, DIM, IN_GAIN), ("w2", DIM, INTER, DOWN_GAIN)):
                lw[name], lw["s_" + name] = _weight(gen, n, k, g, gain)
            for name in ("wqkv", "w1", "w3"):  # the projections that the exporter smooths
                lw["smooth_" + name] = torch.empty((DIM,), device="cuda").uniform_(0.5, 2.0, generator=gen).half() if case["smooth"] else None
            st.layers.append(lw)
        half = dict(dtype=torch.float16, device="cuda")
        st.x0, st.attn = _rows(gen, m, DIM, 4.0), (torch.randn((m, ATTN), device="cuda", generator=gen) * 0.2).half()
        st.x, st.h, st.delta = (torch.empty((m, DIM), **half) for _ in range(3))
        st.qkv = torch.empty((case["layers"], m, QKV), **half)
        st.gate, st.up = torch.empty((m, INTER), **half), torch.empty((m, INTER), **half)
    elif kind == "decode":
        st.x = (torch.randn((case["batch"], DIM), device="cuda", generator=gen) * 12).half()
        st.stack = stack = _stack(ctx, 36, case["batch"], case["context"], g, True, seed, 1.0)

        def step():
            stack.reset_positions()
            stack.decode_step(st.x)
        st.graph = _capture(step)
        del step
    elif kind == "frame":
        b = case["batch"]
        st.x = (torch.randn((CODEBOOKS, b, DIM), device="cuda", generator=gen) * 12).half()
        st.head, st.s_head = _weight(gen, CODEBOOK_SIZE, DIM, g)
        st.packed = _packed(ctx, st.head, st.s_head, g)
        st.registered.append(st.head)
        st.logits = torch.empty((CODEBOOKS, b, CODEBOOK_SIZE), dtype=torch.float16, device="cuda")
        st.stack = stack = _stack(ctx, 4, b, 0, g, False, seed, 1.0 / 8)

        def frame():
            stack.reset_positions()
            for c in range(CODEBOOKS):
                hidden = stack.decode_step(st.x[c])
                ctx.linear(st.head, st.s_head, g, hidden, st.logits[c], b, CODEBOOK_SIZE, DIM)
        st.graph = _capture(frame)
        del frame
    else:
        m = st.m = case["tokens"]
        st.attn_norm, st.ffn_norm = _norm(gen, DIM), _norm(gen, DIM)
        for name, n, k, gain in (("wqkv", QKV, DIM, IN_GAIN), ("wo", DIM, ATTN, IN_GAIN), ("w2", DIM, INTER, DOWN_GAIN)):
            setattr(st, name, _weight(gen, n, k, g, gain))
        w1, s1 = _weight(gen, INTER, DIM, g, IN_GAIN)
        w3, s3 = _weight(gen, INTER, DIM, g, IN_GAIN)
        w13 = torch.empty((2 * INTER, DIM), dtype=torch.int8, device="cuda")
        s13 = torch.empty((2 * INTER, DIM // g), dtype=torch.float16, device="cuda")
        ctx.pack_gate_up(w1, s1, w3, s3, INTER, DIM, DIM // g, w13, s13)
        st.w13 = (w13, s13)
        st.x0, st.attn = _rows(gen, m, DIM, 4.0), (torch.randn((m, ATTN), device="cuda", generator=gen) * 0.2).half()
        for name, n, dtype in (("x", DIM, torch.float16), ("qkv", QKV, torch.float16), ("act", INTER, torch.float16),
                               ("xq", DIM, torch.int8), ("aq", ATTN, torch.int8), ("actq", INTER, torch.int8),
                               ("xs", DIM // g, torch.float32), ("a_s", ATTN // g, torch.float32),
                               ("acts", INTER // g, torch.float32)):
            setattr(st, name, torch.empty((m, n), dtype=dtype, device="cuda"))
    torch.cuda.synchronize()  # temporaries of the packing above are done with
    return st


# ---- one pass ------------------------------------------------------------------------------------------------------


def run(st):
    ctx, g = st.ctx, st.group
    if st.kind == "linear":
        ctx.linear(st.w, st.s, g, st.x, st.y, st.m, st.n, st.k)
        return st.y
    if st.kind == "dropin":
        m = st.m
        st.x.copy_(st.x0)  # the embeddings arrive
        for l, lw in enumerate(st.layers):
            ctx.shim_rms_norm(st.x, lw["attn_norm"], st.h, m, DIM, EPS)
            ctx.shim_int8_dequant_gemm_fp16(lw["wqkv"], lw["s_wqkv"], g, None, lw["smooth_wqkv"], st.h, st.qkv[l], QKV, m, DIM)
            # (the engine's own attention runs here)
            ctx.shim_int8_dequant_gemm_fp16(lw["wo"], lw["s_wo"], g, None, None, st.attn, st.delta, DIM, m, ATTN)
            ctx.shim_residual_add(st.x, st.delta, m * DIM)
            ctx.shim_rms_norm(st.x, lw["ffn_norm"], st.h, m, DIM, EPS)
            ctx.shim_int8_dequant_gemm_fp16(lw["w1"], lw["s_w1"], g, None, lw["smooth_w1"], st.h, st.gate, INTER, m, DIM)
            ctx.shim_silu_forward(st.gate, m * INTER)
            ctx.shim_int8_dequant_gemm_fp16(lw["w3"], lw["s_w3"], g, None, lw["smooth_w3"], st.h, st.up, INTER, m, DIM)
            ctx.shim_mul_forward(st.gate, st.up, m * INTER)
            ctx.shim_int8_dequant_gemm_fp16(lw["w2"], lw["s_w2"], g, None, None, st.gate, st.delta, DIM, m, INTER)
            ctx.shim_residual_add(st.x, st.delta, m * DIM)
        return {"x": st.x, "qkv": st.qkv}
    if st.kind == "decode":
        st.graph.replay()
        return {"hidden": st.stack.out, "k_cache": st.stack.k_cache, "v_cache": st.stack.v_cache}
    if st.kind == "frame":
        st.graph.replay()
        return {"logits": st.logits, "k_cache": st.stack.k_cache, "v_cache": st.stack.v_cache}
    pkg, m = _package(), st.m
    st.x.copy_(st.x0)
    ctx.rmsnorm_quantize(st.x, st.attn_norm, EPS, m, DIM, g, st.xq, st.xs)
    ctx.linear_q(*st.wqkv, g, st.xq, st.xs, st.qkv, m, QKV, DIM)
    # (the engine's own prefill attention runs here)
    ctx.quantize(st.attn, m, ATTN, g, st.aq, st.a_s)
    ctx.linear_q(*st.wo, g, st.aq, st.a_s, st.x, m, DIM, ATTN, epilogue=pkg.EPI_RESIDUAL, residual=st.x)
    ctx.rmsnorm_quantize(st.x, st.ffn_norm, EPS, m, DIM, g, st.xq, st.xs)
    ctx.linear_q(*st.w13, g, st.xq, st.xs, st.act, m, 2 * INTER, DIM, epilogue=pkg.EPI_SWIGLU)
    ctx.quantize(st.act, m, INTER, g, st.actq, st.acts)
    ctx.linear_q(*st.w2, g, st.actq, st.acts, st.x, m, DIM, INTER, epilogue=pkg.EPI_RESIDUAL, residual=st.x)
    return {"x": st.x, "qkv": st.qkv, "act": st.act}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

LAYER_WEIGHTS = QKV * DIM + DIM * ATTN + 2 * INTER * DIM + DIM * INTER


def work(case):
    g, kind = case["group"], case["kind"]
    per_weight = 1 + 2 / g  # an int8 code and its share of an fp16 scale
    if kind == "linear":
        m, n, k = case["tokens"], case["rows"], case["k"]
        return {"bytes": n * k * per_weight + 2 * m * (k + n), "flops": 2 * m * n * k}
    if kind == "dropin":
        m, layers = case["tokens"], case["layers"]
        return {"bytes": layers * (LAYER_WEIGHTS * per_weight + 2 * m * QKV) + 2 * m * (ATTN + 2 * DIM),
                "flops": 2 * m * layers * LAYER_WEIGHTS}
    if kind == "decode":
        b, layers, tokens = case["batch"], 36, case["context"] + 1
        kv = 2 * b * tokens * layers * KV_HEADS * HEAD_DIM * 2
        return {"bytes": layers * LAYER_WEIGHTS * per_weight + kv + 4 * b * DIM,
                "flops": layers * b * (2 * LAYER_WEIGHTS + 4 * tokens * ATTN)}
    if kind == "frame":
        # A codebook step depends on the one before it, and its 0.4 GB of weights do not fit on the chip: ten reads.
        b, layers = case["batch"], 4
        weights = layers * LAYER_WEIGHTS + CODEBOOK_SIZE * DIM
        return {"bytes": CODEBOOKS * (weights * per_weight + 2 * b * (DIM + CODEBOOK_SIZE)), "flops": 2 * b * CODEBOOKS * weights}
    m = case["tokens"]
    return {"bytes": LAYER_WEIGHTS * per_weight + 2 * m * (ATTN + 2 * DIM + QKV + INTER), "flops": 2 * m * LAYER_WEIGHTS}


def tolerance(case):
    """Outputs are fp16 of fp32 sums. One linear: a sum in another order moves an output by at most its last bits. Where a
    quantiser follows such an output, a last-bit difference moves an int8 code by one step of the group's absmax / 127 now
    and then; through the 36 layers of a stack (or the four of a frame, ten times) those steps add up to the size of the
    quantisation noise itself."""
    if case["kind"] == "linear":
        return {"rel": 1e-3, "max": 1e-2}
    if case["kind"] in ("decode", "frame"):
        return {"rel": 2.5e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.3}
