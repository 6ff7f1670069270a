"""Attention of a KV head's query heads together, with the quantised result handed to the exact GEMM in its operand order: against
the oracle at the edges of the 64-key tiles, for every split of 1 to 8 heads over the threads, and with rows whose last pipeline
stage is half empty (12 and 20 blocks)."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("qtype", ["q4_0", "q8_0"])
@pytest.mark.parametrize("hidden,heads,n_kv,ffn", [(256, 4, 4, 512), (384, 6, 2, 640), (384, 6, 1, 640), (512, 8, 1, 1152)])
def test_prompts_and_batched_steps_at_tile_edges(cuda_lib, orc, model_dir, monkeypatch, qtype, hidden, heads, n_kv, ffn):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import gguf_synth as gs
    from wick_b200.model import CudaLfm2Model
    name = f"group-{hidden}-{heads}-{n_kv}"
    monkeypatch.setitem(gs.SPECS, name, dataclasses.replace(gs.SPECS["tiny"], name=name, hidden=hidden, n_heads=heads, n_kv_heads=n_kv, ffn=ffn))
    path = gs.cached_model(name, qtype, 0, cache_dir=model_dir, norm_jitter=0.2, weight_std=0.05)
    m = CudaLfm2Model(path, 512)
    ids, nxt, oracles = [], [], []
    for n in (200, 1, 2, 63, 64, 65, 127, 129):  # (the first one makes the copies of the weights)
        o = orc.OracleModel(path, 512)
        toks = gs.random_prompt(n, m.config().vocab_size, seed=n)
        sid = m.seq_create()
        want = o.forward_prefill(toks, 0)
        assert np.array_equal(bits(m.seq_prefill(sid, toks, 0)), bits(want)), n
        ids.append(sid)
        nxt.append(orc.argmax(want))
        oracles.append(o)
    for rows in (len(ids), 3):
        got = m.decode_batch_logits(nxt[:rows], ids[:rows])
        for i in range(rows):
            want = oracles[i].forward(int(nxt[i]))
            assert np.array_equal(bits(got[i]), bits(want)), (rows, i)
            nxt[i] = orc.argmax(want)


@pytest.mark.parametrize("heads,n_kv,rows", [(8, 1, 33), (12, 2, 17)])
def test_many_heads_to_a_kv_head_in_small_batches(cuda_lib, orc, model_dir, monkeypatch, heads, n_kv, rows):
    """More than four heads and at most 32 (row, KV head) pairs: the kernels of one head to a CTA, with a quantiser of their own; one row more: this one."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import gguf_synth as gs
    from wick_b200.model import CudaLfm2Model
    spec = dataclasses.replace(gs.SPECS["tiny"], name=f"small-batch-{heads}-{n_kv}", hidden=64 * heads, n_heads=heads, n_kv_heads=n_kv)
    monkeypatch.setitem(gs.SPECS, spec.name, spec)
    path = gs.cached_model(spec.name, "q4_0", 0, cache_dir=model_dir, norm_jitter=0.2, weight_std=0.05)
    m, ids, oracles, toks = CudaLfm2Model(path, 128), [], [], []
    for i in range(rows):
        ids.append(m.seq_create())
        oracles.append(orc.OracleModel(path, 128))
        prompt = gs.random_prompt(9 + 3 * i, spec.vocab, seed=i)
        m.seq_prefill(ids[i], prompt, 0)
        toks.append(orc.argmax(oracles[i].forward_prefill(prompt, 0)))
    kernels = []
    for step in range(2):  # (the first one of each size makes buffers)
        for n in (rows - 1, rows):
            before = m.kernel_launches()
            got = m.decode_batch_logits(toks[:n], ids[:n])
            kernels.append(m.kernel_launches() - before)
            for i in range(n):
                want = oracles[i].forward(int(toks[i]))
                assert np.array_equal(bits(got[i]), bits(want)), (step, n, i)
                toks[i] = orc.argmax(want)
    assert kernels[2] == kernels[3] + len(spec.attn_layers)


@pytest.mark.parametrize("heads,n_kv", [(1, 8), (2, 3), (3, 2), (4, 8), (5, 1), (6, 3), (7, 1), (8, 2)])
@pytest.mark.parametrize("n,start", [(33, 0), (40, 31), (34, 64), (36, 1000), (33, 4003)])
def test_kernel_against_the_per_head_one(cuda_lib, heads, n_kv, n, start):
    """Every split of 1 to 8 heads over the threads, contexts of one tile to many, against attention_prefill (itself compared with the oracle) and
    the quantiser; and the result's place among other rows: nothing is written behind the last one."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(heads * 10 + n)
    nh, kv = heads * n_kv, n_kv * 64
    q = torch.randn((n, nh * 64), generator=g, device="cuda")
    k, v = (torch.randn((start + n, kv), generator=g, device="cuda") for _ in range(2))
    want_s, want_q = ops.quantize_f32_to_q8_0(ops.attention_prefill(q, k, v, n, start, nh, n_kv, 64, False))
    s, b = torch.full((n + 1, nh * 2), 7.0, device="cuda"), torch.full((n + 1, nh * 64), 7, dtype=torch.int8, device="cuda")
    _lib.check(cuda_lib.wick_cuda_debug_attention_group(q.data_ptr(), k.data_ptr(), v.data_ptr(), s.data_ptr(), b.data_ptr(), n, start, nh, n_kv, 64,
                                                        torch.cuda.current_stream().cuda_stream))
    assert torch.equal(s[:n].view(torch.int32), want_s.view(torch.int32)) and torch.equal(b[:n], want_q)
    assert (s[n] == 7).all() and (b[n] == 7).all()


@pytest.mark.parametrize("dim", [32, 1024, 4064, 4096, 4128, 8160, 8192, 8224, 12320, 16384, 16416])
def test_add_rmsnorm_quant_by_row_length(cuda_lib, dim):
    """One, two and four quads to a thread and the edges between them, against the operators one by one; longer rows are refused."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(dim)
    n = 3
    h, add = (torch.randn((n, dim), generator=g, device="cuda") * 3 for _ in range(2))
    w = torch.rand(dim, generator=g, device="cuda") + 0.5
    for a in (add, None):
        hidden, normed = h.clone(), torch.empty_like(h)
        s, b = torch.empty((n, dim // 32), device="cuda"), torch.empty((n, dim), dtype=torch.int8, device="cuda")
        r = cuda_lib.wick_cuda_debug_add_rmsnorm_quant(hidden.data_ptr(), a.data_ptr() if a is not None else None, w.data_ptr(), n, dim, 1e-5,
                                                       normed.data_ptr(), s.data_ptr(), b.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if dim > 16384:
            assert r == _lib.ERR_CUDA
            continue
        _lib.check(r)
        total = h + a if a is not None else h
        assert torch.equal(hidden, total)
        want = ops.rmsnorm_(total.clone(), w, 1e-5)
        # (the f64 sums are added in different fixed orders: at most the last bit of the factor, so of a value, may differ)
        assert (normed.view(torch.int32) - want.view(torch.int32)).abs().max() <= 1
        want_s, want_q = ops.quantize_f32_to_q8_0(normed)
        assert torch.equal(s, want_s) and torch.equal(b, want_q)


def test_rows_wider_than_a_thread_per_four_elements(cuda_lib, orc, model_dir, monkeypatch):
    """Hidden rows above 4096 elements: the add + RMSNorm + quantise kernel has more than four of them per thread."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import gguf_synth as gs
    from wick_b200.model import CudaLfm2Model
    spec = dataclasses.replace(gs.SPECS["tiny"], name="wide-rows", hidden=4352, n_layers=2, attn_layers=(1,), n_heads=68, n_kv_heads=17, ffn=256, vocab=256)
    monkeypatch.setitem(gs.SPECS, spec.name, spec)
    path = gs.cached_model(spec.name, "q4_0", 0, cache_dir=model_dir, norm_jitter=0.2)
    m, o = CudaLfm2Model(path, 64), orc.OracleModel(path, 64)
    sid = m.seq_create()
    toks = gs.random_prompt(17, spec.vocab, seed=3)
    want = o.forward_prefill(toks, 0)
    assert np.array_equal(bits(m.seq_prefill(sid, toks, 0)), bits(want))
    assert np.array_equal(bits(m.decode_batch_logits([orc.argmax(want)], [sid])[0]), bits(o.forward(orc.argmax(want))))


@pytest.mark.parametrize("hidden", [16384, 16416, 1 << 20])
def test_hidden_rows_that_no_kernel_holds_are_refused_at_load(cuda_lib, model_dir, hidden):
    """A launch with such rows is refused, and the captured decode step was left without it: all logits 0, and no error.  (16384 itself is
    a length that the kernel takes: this file is turned down for its head size.)"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import _lib, gguf_synth as gs
    from wick_b200.model import CudaLfm2Model
    data = bytearray(open(gs.cached_model("tiny", "q4_0", 0, cache_dir=model_dir), "rb").read())
    key = b"lfm2.embedding_length" + (gs.T_UINT32).to_bytes(4, "little")
    at = data.index(key) + len(key)
    data[at:at + 4] = hidden.to_bytes(4, "little")
    with pytest.raises(_lib.WickCudaError) as e:
        CudaLfm2Model.from_bytes(bytes(data), 64)
    assert e.value.code == _lib.ERR_BAD_GGUF and ("16384" in str(e.value)) == (hidden > 16384)
