"""Edges of the kernels' dispatch rules: tile widths and extreme scales of the exact tensor-core GEMM, the operator GEMM's
switch to it, the split of attention items over warps, the sampler's small top-k path, one-row prefills and the decode
ring with few slots.  Everything is compared bit for bit with the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.fixture(scope="module")
def ops(cuda_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import ops
    return ops


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def assert_bits(got, want, what):
    got = got.detach().cpu().numpy() if isinstance(got, torch.Tensor) else got
    assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want, F32).view(np.uint32)), what


@pytest.mark.parametrize("dtype", ["q4_0", "q8_0"])
@pytest.mark.parametrize("scales", ["smallest", "largest", "mixed"])
def test_exact_gemm_keeps_every_f16_scale(ops, orc, dtype, scales):
    """f16 scales from the smallest subnormal to the largest value, and zero, in weights and activations."""
    rng = np.random.default_rng(3)
    m, k, n = 130, 384, 19
    bb = 18 if dtype == "q4_0" else 34
    raw = rng.integers(0, 256, size=(m, k // 32, bb), dtype=np.uint8)
    pick = {"smallest": [6e-8, 1.2e-7, 0.0], "largest": [65504.0, -60000.0, 32768.0], "mixed": [6e-8, 65504.0, 0.02, -1.0, 0.0]}[scales]
    raw[:, :, :2] = rng.choice(np.array(pick, np.float16), size=(m, k // 32, 1)).view(np.uint8).reshape(m, k // 32, 2)
    bs = rng.choice(np.abs(np.array(pick, np.float16)), size=(n, k // 32)).astype(F32)
    bq = rng.integers(-127, 128, size=(n, k), dtype=np.int8)
    w = ops.QuantWeight(ops.QTYPE_ID[dtype], raw.reshape(-1), m, k)
    want = np.stack([orc.gemv(orc.QTYPE_ID[dtype], raw.reshape(m, -1), bs[j], bq[j], m, k) for j in range(n)])
    assert_bits(ops.gemm_q8_tc_exact(w, dev(bs), dev(bq)), want, f"{dtype} {scales}")


@pytest.mark.parametrize("dtype", ["q4_0", "q8_0"])
@pytest.mark.parametrize("where", ["weights", "activations", "both"])
@pytest.mark.parametrize("m,k,n", [(130, 384, 19), (6144, 128, 90), (6144, 128, 130)])  # tiles of 16 x 8; two rounds of 64 x 32; six of 64 x 16
def test_exact_gemm_with_infinite_scales(ops, orc, dtype, where, m, k, n):
    """Scales beyond f16 (a block of activations above 8.3 million; an infinity or NaN in a file): the reference's infinities and
    NaNs, not NaN throughout.  Only the sign and payload of a NaN are free."""
    rng = np.random.default_rng(5)
    raw = rng.integers(0, 256, size=(m, k // 32, 18 if dtype == "q4_0" else 34), dtype=np.uint8)
    d = rng.uniform(0.01, 0.02, size=(m, k // 32)).astype(np.float16)
    bs = rng.uniform(0.01, 0.02, size=(n, k // 32)).astype(np.float16)
    if where != "activations":
        d[1, 0], d[2, 1], d[m - 1, 2], d[7, 0] = np.inf, -np.inf, np.inf, np.nan
    if where != "weights":
        bs[0, 0], bs[3, 1], bs[n - 1, 2], bs[5, 1:3] = np.inf, np.inf, np.inf, np.inf
        bs[6, 0] = 0.0
    raw[:, :, :2] = d.view(np.uint8).reshape(m, k // 32, 2)
    bs = bs.astype(F32)
    bq = rng.integers(1, 128, size=(n, k), dtype=np.int8) * rng.choice(np.array([-1, 1], np.int8), size=(n, 1))
    if dtype == "q8_0":
        raw[:, :, 2:] = rng.integers(1, 128, size=raw[:, :, 2:].shape)  # lane partials without a zero: infinities survive
    bq[n // 2, :32] = 0                                                   # and a block with nothing but zeros
    w = ops.QuantWeight(ops.QTYPE_ID[dtype], raw.reshape(-1), m, k)
    got = ops.gemm_q8_tc_exact(w, dev(bs), dev(bq)).cpu().numpy()
    want = np.stack([orc.gemv(orc.QTYPE_ID[dtype], raw.reshape(m, -1), bs[j], bq[j], m, k) for j in range(n)])
    assert np.isinf(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert_bits(np.where(np.isnan(got), F32(0), got), np.where(np.isnan(want), F32(0), want), f"{dtype} {where}")


def test_model_with_infinite_weight_scales(cuda_lib, orc, model_dir, tmp_path):
    """Infinite scales in rows of the vocabulary matrix: a batched step's logits are the CPU path's infinities and NaNs."""
    import wick_b200.model as wick
    from wick_b200 import gguf_synth as gs
    clean = gs.cached_model("tiny-wide", "q4_0", 0, cache_dir=model_dir, norm_jitter=0.2, weight_std=0.05)
    (k, vocab), _, off = orc.GgufFile(clean).tensors["token_embd.weight"]
    data = bytearray(open(clean, "rb").read())
    for r in range(vocab - 100, vocab):
        at = off + (r * (k // 32) + r % (k // 32)) * 18
        data[at:at + 2] = np.array([np.inf if r % 2 else -np.inf], np.float16).tobytes()
    path = tmp_path / "inf.gguf"
    path.write_bytes(bytes(data))
    cm, rows = wick.CudaLfm2Model(str(path), 256), 10
    ids, oms = [cm.seq_create() for _ in range(rows)], [orc.OracleModel(str(path), 256) for _ in range(rows)]
    for i in range(rows):
        toks = gs.random_prompt(9 + i, vocab - 100, seed=i)
        cm.seq_prefill(ids[i], toks, 0), oms[i].forward_prefill(toks, 0)
    for step in range(2):
        got = cm.decode_batch_logits([3 * i + step for i in range(rows)], ids)
        want = np.stack([oms[i].forward(3 * i + step) for i in range(rows)])
        assert np.isinf(want).any() and np.isnan(want).any() and np.isfinite(want[:, :vocab - 100]).all()
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert_bits(np.where(np.isnan(got), F32(0), got), np.where(np.isnan(want), F32(0), want), f"step {step}")


@pytest.mark.parametrize("m,k,n", [(130, 384, 19), (6144, 128, 90), (6144, 128, 130)])  # tiles of 16 x 8; two rounds of 64 x 32; six of 64 x 16
def test_operator_gemm_with_scales_that_are_not_f16(ops, orc, m, k, n):
    """A caller's own quantiser need not round its scales to f16: tiny, subnormal and huge ones, alone and beside ordinary ones."""
    from wick_b200 import gguf_synth as gs
    rng = np.random.default_rng(9)
    raw = gs.quantize_q4_0((rng.standard_normal((m, k)) * 0.02).astype(F32))
    bs = (10.0 ** rng.uniform(-4, 0, size=(n, k // 32))).astype(F32)
    bs[2] = 10.0 ** rng.uniform(-44, -8, size=k // 32)
    bs[4, 1], bs[5, 2], bs[6, 3], bs[n - 1, 0] = 1e-12, 3e-39, 1e13, 1e30
    bs[7], bs[8, 1:] = 2.0 ** -49, np.nextafter(F32(2.0 ** -49), F32(0))   # the last inside and the first outside
    bs[9], bs[10, 0] = np.nextafter(F32(2.0 ** 16), F32(0)), 2.0 ** 16
    bq = rng.integers(-127, 128, size=(n, k), dtype=np.int8)
    w = ops.QuantWeight(ops.DT_Q4_0, raw, m, k)
    want = np.stack([orc.gemv(orc.DT_Q4_0, raw, bs[j], bq[j], m, k) for j in range(n)])
    assert np.isfinite(want).all()
    assert_bits(ops.gemm_q8(w, dev(bs), dev(bq)), want, f"{m} x {k}")


@pytest.mark.parametrize("m,k,n", [(128, 128, 2), (128, 128, 7), (256, 256, 8), (256, 256, 9), (384, 128, 15), (2048, 128, 73), (6144, 128, 64),
                                   (2048, 128, 600), (100, 160, 40)])
def test_operator_gemm_on_either_path(ops, orc, m, k, n):
    """Around the switch to the tensor cores (more than 8 columns, k a multiple of 128) and the choice of tile width."""
    from wick_b200 import gguf_synth as gs
    rng = np.random.default_rng(m + n)
    raw = gs.quantize_q4_0((rng.standard_normal((m, k)) * 0.02).astype(F32))
    w = ops.QuantWeight(ops.DT_Q4_0, raw, m, k)
    bs, bq = orc.quantize_q8_0(rng.standard_normal((n, k), dtype=F32))
    out = ops.gemm_q8(w, dev(bs), dev(bq))
    for j in sorted({0, n // 2, n - 1}):
        assert_bits(out[j], orc.gemv(orc.DT_Q4_0, raw, bs[j], bq[j], m, k), f"column {j}")


@pytest.mark.parametrize("n,start,nh,nkv,hd", [(512, 100, 32, 8, 64), (300, 0, 7, 1, 64), (257, 31, 5, 1, 32), (7, 0, 1, 1, 64)])
def test_attention_items_over_warps(ops, orc, n, start, nh, nkv, hd):
    """Lists of (query run, head) items that the warps of a CTA do not divide evenly."""
    rng = np.random.default_rng(n)
    group, kv_dim = nh // nkv, nkv * hd
    q = rng.standard_normal((n, nh * hd), dtype=F32)
    kc, vc = (rng.standard_normal((start + n, kv_dim), dtype=F32) for _ in range(2))
    out = ops.attention_prefill(dev(q), dev(kc), dev(vc), n, start, nh, nkv, hd, True).cpu().numpy()
    for kv_h in range(nkv):
        fl = orc.flash_attention_gqa(np.ascontiguousarray(q.T), kc, vc, kv_h * group, group, n, n, kv_dim, kv_h * hd, hd, F32(1.0) / np.sqrt(F32(hd)), start)
        for g in range(group):
            h = kv_h * group + g
            assert_bits(np.ascontiguousarray(out[:, h * hd:(h + 1) * hd]), fl[g], f"head {h}")


@pytest.mark.parametrize("n,top_k", [(65536, 255), (65536, 256), (65536, 257), (1023, 200), (5000, 3)])
def test_sampler_around_its_small_top_k_path(ops, orc, n, top_k):
    """Few distinct values (ties at the threshold, more candidates than the small path takes) and ordinary logits."""
    rng = np.random.default_rng(top_k)
    for logits in ((rng.standard_normal(n) * 3).astype(F32), rng.integers(-40, 0, size=n).astype(F32), np.repeat(F32(1.5), n),
                   np.sort(rng.standard_normal(n)).astype(F32)):
        for r in (0.0, 0.37, 0.999):
            assert ops.sample_logits(dev(logits), 0.8, top_k, 1.0, r) == orc.sample(logits, 0.8, top_k, 1.0, r)


@pytest.mark.parametrize("qtype", ["q4_0", "q8_0"])
def test_decode_with_a_short_ring_and_one_row_prefills(cuda_lib, orc, model_dir, qtype):
    """A context that leaves the ring five slots (gate and up share one), steps through the persistent kernel by every entry
    point that takes a single row."""
    import wick_b200.model as wick
    from wick_b200 import gguf_synth as gs
    path = gs.cached_model("tiny-longctx", qtype, 0, cache_dir=model_dir, norm_jitter=0.2, weight_std=0.05)
    cm, om = wick.CudaLfm2Model(path, 24000), orc.OracleModel(path, 24000)
    st = wick.InferenceState()
    assert cm.decode_path() == "persistent"
    toks = gs.random_prompt(30, cm.config().vocab_size, seed=3)
    assert_bits(cm.forward_prefill(toks, 0, st), om.forward_prefill(toks, 0), "prompt")
    assert list(cm.generate_greedy(5, 12, st)) == list(om.generate_greedy(5, 12))
    assert_bits(cm.forward_prefill(toks[:1], 42, st), om.forward_prefill(toks[:1], 42), "one-token prefill")
    emb = np.random.default_rng(1).standard_normal(cm.config().hidden_size).astype(F32) * F32(0.1)
    assert_bits(cm.forward_from_embedding(emb, 43, st), om.forward_from_embedding(emb), "one frame")
    assert_bits(cm.forward_embedding([int(toks[2])], 44, st), om.forward_embedding(int(toks[2])), "hidden row")
    assert list(cm.generate_greedy(6, 4, st)) == list(om.generate_greedy(6, 4))
    assert_bits(cm.forward_prefill(toks[:1], 0, st), om.forward_prefill(toks[:1], 0), "one-token prompt")


def test_attention_whose_scores_just_fit_the_default_shared_memory(cuda_lib, orc, model_dir):
    """8100 keys of 64: 47.9 KB of dynamic shared memory and the kernel's static 384 bytes are more than the 48 KB that need no opt-in.  (A
    process of its own: one larger call before would have raised the limit.)"""
    import os, subprocess, sys
    from wick_b200 import gguf_synth as gs
    code = """
import os, sys
os.environ["WICK_CUDA_DECODE"] = "graph"
import numpy as np, torch
from oracle import oracle as orc
from wick_b200 import ops
import wick_b200.model as wick
cm, om = wick.CudaLfm2Model(sys.argv[1], 8100), orc.OracleModel(sys.argv[1], 8100)
st, toks = wick.InferenceState(), list(range(5, 35))
first = orc.argmax(om.forward_prefill(toks, 0))
assert orc.argmax(cm.forward_prefill(toks, 0, st)) == first
assert list(cm.generate_greedy(first, 8, st)) == list(om.generate_greedy(first, 8))
q, k, v = (torch.randn(n, 64, device="cuda") for n in (1, 8100, 8100))
short = ops.attention_decode(q, k[:8000], v[:8000], 1, 1, 64, 8000)
v[8000:], k[8000:] = 0, -100 * torch.sign(q)   # the last hundred keys count for nothing
assert torch.equal(ops.attention_decode(q, k, v, 1, 1, 64, 8100), short)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code, gs.cached_model("tiny-longctx", "q4_0", 0, cache_dir=model_dir, norm_jitter=0.2, weight_std=0.05)],
                   check=True, cwd=root, timeout=300)
