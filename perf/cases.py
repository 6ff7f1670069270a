"""The calls that a user of this backend makes, as cases to be timed: prompts, chats, sampled and long conversations,
frame input, many sequences at once and the bare quantised product, on the model shapes of the benchmark
(`gguf_synth.SPECS`), random weights N(0, 0.02), prompts of uniform-random token ids.

A case is one pass: what `run` does for one prepared state.  Every pass starts its sequences anew (start_pos 0), so a
pass can be repeated and leaves nothing for the next one."""
import functools
import math
import os
import tempfile

import numpy as np
import torch

from wick_b200 import gguf_synth as gs
from wick_b200 import ops
from wick_b200.model import CudaLfm2Model, InferenceState

BLOCK_BYTES = {"q4_0": 18, "q8_0": 34}


def listed():
    return [
        # time to the first token of a one-line prompt: the smallest call, launches and latency
        dict(name="prompt_350m_q4_9", kind="prefill", model="lfm2-350m", qtype="q4_0", n=9, ubatch=512, mode="exact"),
        # an audio front end: frames in, then frame by frame (the embedding-input calls), a ragged count under one chunk
        dict(name="frames_350m_q8_137", kind="frames", model="lfm2-350m", qtype="q8_0", n=137, steps=32),
        # a page of text, not a multiple of the 512-token chunk
        dict(name="prompt_1p6b_q4_1000", kind="prefill", model="lfm2.5-1.6b", qtype="q4_0", n=1000, ubatch=512, mode="exact"),
        # the benchmark's long prompt, in the 512-token chunks that a session uses
        dict(name="prompt_1p6b_q4_4096", kind="prefill", model="lfm2.5-1.6b", qtype="q4_0", n=4096, ubatch=512, mode="exact"),
        # the same with the GEMM that a user may choose for throughput instead of the CPU path's bits
        dict(name="prompt_1p6b_q4_2048_tensor", kind="prefill", model="lfm2.5-1.6b", qtype="q4_0", n=2048, ubatch=512, mode="tensor"),
        # the headline: 128-token prompt, 128 greedy tokens with the loop on the GPU
        dict(name="chat_1p6b_q4_128_128", kind="chat", model="lfm2.5-1.6b", qtype="q4_0", n=128, steps=128, how="generate"),
        # the session's own loop: one call per token, the small model
        dict(name="chat_350m_q4_128_128_calls", kind="chat", model="lfm2-350m", qtype="q4_0", n=128, steps=128, how="calls"),
        # a sampled reply: temperature, top-k and top-p on the GPU, one call per token, 8-bit weights
        dict(name="chat_1p6b_q8_128_64_sampled", kind="chat", model="lfm2.5-1.6b", qtype="q8_0", n=128, steps=64, how="sample"),
        # long context: 4096-token prompt, then 512 tokens against it
        dict(name="chat_350m_q8_4096_512", kind="chat", model="lfm2-350m", qtype="q8_0", n=4096, steps=512, how="generate"),
        # a serving loop's full batch: each sequence has a prompt of its own (half to one and a half times n)
        dict(name="serve_1p6b_q4_64", kind="serve", model="lfm2.5-1.6b", qtype="q4_0", rows=64, n=96, steps=96),
        # and a nearly empty one
        dict(name="serve_350m_q8_6", kind="serve", model="lfm2-350m", qtype="q8_0", rows=6, n=200, steps=64),
        # the bare product of the benchmark's matmul sweep
        dict(name="matmul_q4_6912x2048_2002", kind="matmul", qtype="q4_0", m=6912, k=2048, n=2002),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["prefill", "prefill", "prefill", "chat", "chat", "chat", "serve", "serve", "frames", "matmul"])
    c = dict(kind=kind, qtype=rng.choice(["q4_0", "q8_0"]))
    if kind == "matmul":
        m, k = rng.choice([(6912, 2048), (2048, 6912), (6144, 2048), (2048, 2048), (4608, 1024), (1024, 4608), (3072, 1024)])
        return dict(c, m=m, k=k, n=logu(1, 4096))
    c["model"] = rng.choice(["lfm2-350m", "lfm2.5-1.6b"])
    if kind == "prefill":
        return dict(c, n=logu(1, 4096), ubatch=rng.choice([512, 512, 0]), mode=rng.choice(["exact", "exact", "exact", "tensor"]))
    if kind == "frames":
        return dict(c, n=logu(8, 1024), steps=logu(4, 64))
    if kind == "chat":
        return dict(c, n=logu(4, 3000), steps=logu(16, 192), how=rng.choice(["generate", "calls", "sample"]))
    return dict(c, rows=logu(2, 64), n=logu(16, 96), steps=logu(16, 80))


# ── models: weights are a user's file, loaded once per process and kept ────────────────────────────
def _blocks(x, qtype):
    """f32 [rows, k] -> uint8 [rows, k/32 * block bytes], the rounding of gguf_synth.quantize_q4_0 / quantize_q8_0."""
    b = x.reshape(-1, 32)
    big = b.gather(1, b.abs().argmax(1, keepdim=True))
    d = big / -8.0 if qtype == "q4_0" else big.abs() / 127.0
    v = b * torch.where(d == 0, torch.zeros_like(d), 1.0 / d)
    head = d.half().view(torch.uint8)
    if qtype == "q4_0":
        q = (v + 8.5).clamp_(0, 15).to(torch.uint8)
        body = q[:, :16] | (q[:, 16:] << 4)
    else:
        body = torch.copysign((v.abs() + 0.5).floor(), v).to(torch.int8).view(torch.uint8)
    return torch.cat([head, body], 1).reshape(x.shape[0], -1)


def _write_model(path, spec, qtype):
    tensors = gs._tensor_list(spec)
    kind = gs.QUANTIZERS[qtype][1]
    plan = [(n, s, kind, s[0] * (s[1] // 32) * BLOCK_BYTES[qtype]) if t == "quant" else (n, s, gs.GGML_F32, 4 * math.prod(s))
            for n, s, t in tensors]
    kvs = [gs.kv_str("general.architecture", "lfm2"), gs.kv_u32("general.alignment", gs.GGUF_ALIGNMENT),
           gs.kv_u32("lfm2.block_count", spec.n_layers), gs.kv_u32("lfm2.embedding_length", spec.hidden),
           gs.kv_u32("lfm2.feed_forward_length", spec.ffn), gs.kv_u32("lfm2.attention.head_count", spec.n_heads),
           gs.kv_i32_array("lfm2.attention.head_count_kv", [spec.n_kv_heads if i in spec.attn_layers else 0 for i in range(spec.n_layers)]),
           gs.kv_u32("lfm2.vocab_size", spec.vocab), gs.kv_u32("lfm2.context_length", spec.context_length),
           gs.kv_u32("lfm2.shortconv.l_cache", spec.conv_kernel), gs.kv_f32("lfm2.rope.freq_base", spec.rope_theta),
           gs.kv_f32("lfm2.attention.layer_norm_rms_epsilon", spec.rms_eps)]
    g = torch.Generator("cuda").manual_seed(0)
    w = gs.GgufWriter(path, kvs, plan)
    for name, shape, t in tensors:
        if t == "norm":
            w.write_tensor(name, np.ones(shape, np.float32))
            continue
        x = torch.randn(shape, generator=g, device="cuda") * 0.02
        w.write_tensor(name, (_blocks(x, qtype) if t == "quant" else x).cpu().numpy())
    w.close()


@functools.lru_cache(maxsize=None)
def _model(name, qtype, mode="exact"):
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "model.gguf")
        _write_model(path, gs.SPECS[name], qtype)
        m = CudaLfm2Model(path, 8192)
    m.set_prefill_mode(mode)
    torch.cuda.empty_cache()
    return m


class _Slots:
    """Sequence slots of a model, given back with the state that holds them."""

    def __init__(self, m, n):
        self.m, self.ids = m, [m.seq_create() for _ in range(n)]

    def __del__(self):
        for i in self.ids:
            self.m.seq_destroy(i)


# ── one state, one pass ─────────────────────────────────────────────────────────────────────────────
def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng([seed, 77])
    if kind == "matmul":
        g = torch.Generator("cuda").manual_seed(seed)
        raw = _blocks(torch.randn(case["m"], case["k"], generator=g, device="cuda") * 0.02, case["qtype"])
        w = ops.QuantWeight(ops.QTYPE_ID[case["qtype"]], raw.cpu().numpy(), case["m"], case["k"])
        xs, xq = ops.quantize_f32_to_q8_0(torch.randn(case["n"], case["k"], generator=g, device="cuda"))
        return dict(kind=kind, w=w, xs=xs, xq=xq)
    spec, m = gs.SPECS[case["model"]], _model(case["model"], case["qtype"], case.get("mode", "exact"))
    s = dict(case, m=m, st=InferenceState())
    if kind == "frames":
        s["frames"] = (rng.standard_normal((case["n"] + case["steps"], spec.hidden)) * 0.02).astype(np.float32)
    elif kind == "serve":
        lens = rng.integers(case["n"] // 2, case["n"] + case["n"] // 2, size=case["rows"], endpoint=True)
        s["prompts"] = [rng.integers(0, spec.vocab, size=n, dtype=np.uint32) for n in lens]
        s["slots"] = _Slots(m, case["rows"])
    else:
        s["prompt"] = rng.integers(0, spec.vocab, size=case["n"], dtype=np.uint32)
        s["r"] = rng.random(case.get("steps", 0), dtype=np.float32)  # the sampler's uniform draws
    return s


def run(s):
    kind = s["kind"]
    if kind == "matmul":
        if s["xq"].shape[0] == 1:
            return ops.gemv_q8(s["w"], s["xs"], s["xq"])
        return ops.gemm_q8(s["w"], s["xs"], s["xq"])
    m, st = s["m"], s["st"]
    if kind == "prefill":
        return m.forward_prefill_chunked(s["prompt"], 0, st, s["ubatch"])[1]
    if kind == "frames":
        n, f = s["n"], s["frames"]
        rows = [m.forward_prefill_from_embeddings(f[:n], n, 0, st)]
        rows += [m.forward_from_embedding(f[n + i], n + i, st) for i in range(s["steps"])]
        return np.stack(rows)
    if kind == "serve":
        ids = s["slots"].ids
        logits = [m.seq_prefill(i, p, 0) for i, p in zip(ids, s["prompts"])]
        first = [int(np.argmax(v)) for v in logits]
        return m.decode_batch_steps(first, ids, s["steps"]), np.stack(logits)
    logits = m.forward_prefill_chunked(s["prompt"], 0, st, 512)[1]
    tok = int(np.argmax(logits))
    if s["how"] == "generate":
        return logits, m.generate_greedy(tok, s["steps"], st)
    out = []
    for i in range(s["steps"]):
        if s["how"] == "calls":
            tok = m.forward_greedy([tok], s["n"] + i, st)
        else:
            tok = m.forward_sample([tok], s["n"] + i, st, 0.8, 40, 0.95, float(s["r"][i]))
        out.append(tok)
    return logits, np.array(out, np.int64)


# ── what a pass cannot do without ───────────────────────────────────────────────────────────────────
def work(case):
    if case["kind"] == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * (k // 32) * BLOCK_BYTES[case["qtype"]] + n * (k + k // 8) + 4 * n * m, "flops": 2 * n * m * k}
    spec, steps, n, rows = gs.SPECS[case["model"]], case.get("steps", 0), case["n"], case.get("rows", 1)
    wb = spec.quant_bytes(case["qtype"])
    head = 2 * spec.vocab * spec.hidden
    layers = 2 * wb // BLOCK_BYTES[case["qtype"]] * 32 - head
    na = len(spec.attn_layers)
    # weights once for a prompt (for all of a batch's prompts: they are there together) and once for each step, the keys
    # and values written once and read once by each step; a frame's logits, a prompt's last logits
    kv = rows * na * 2 * spec.kv_dim * 4
    steps_kv = sum(n + i for i in range(steps)) * kv
    pairs = n * (n + 1) // 2 + sum(n + i for i in range(steps))
    return {"bytes": (1 + steps) * wb + kv * (n + steps) + steps_kv + 4 * spec.vocab * rows,
            "flops": rows * ((n + steps) * layers + (1 + steps) * head + 4 * na * spec.hidden * pairs)}


def tolerance(case):
    # The default path promises the CPU path's own bits: integer block sums, then a fixed order of float operations.
    # The "tensor" mode rounds differently, which moves single 8-bit activations by one step: a few 1e-2 on logits.
    return {"rel": 3e-2} if case.get("mode") == "tensor" else "exact"
