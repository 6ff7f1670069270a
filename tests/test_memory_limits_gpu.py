"""Calls that can do without a weight copy still work where there is no memory for one: the copy is a matter of speed."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
F32 = np.float32


class Filled:
    """All device memory but `left` bytes taken."""

    def __init__(self, left):
        self.left, self.hold = left, []

    def __enter__(self):
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        for _ in range(4):
            take = torch.cuda.mem_get_info()[0] - self.left
            if take > (1 << 21):
                self.hold.append(torch.empty(take >> 21 << 21, dtype=torch.uint8, device="cuda"))

    def __exit__(self, *exc):
        self.hold.clear()
        torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def ops(cuda_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wick_b200 import ops
    return ops


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_operator_product_without_memory_for_the_copy(ops, orc):
    m, k, n = 65536, 1024, 9                             # a copy of 75 MB
    rng = np.random.default_rng(0)
    raw = rng.integers(0, 256, size=(m, k // 32, 18), dtype=np.uint8)
    raw[:, :, :2] = np.full((m, k // 32, 1), 0.01, np.float16).view(np.uint8).reshape(m, k // 32, 2)
    w = ops.QuantWeight(ops.DT_Q4_0, raw.reshape(-1), m, k)
    bs, bq = orc.quantize_q8_0(rng.standard_normal((n, k), dtype=F32))
    dbs, dbq, out = dev(bs), dev(bq), torch.zeros((n, m), device="cuda")  # (loads what zero_ needs, too)
    want = orc.gemv(orc.DT_Q4_0, raw.reshape(m, -1), bs[n - 1], bq[n - 1], m, k)
    with Filled(48 << 20):
        for _ in range(2):
            out.zero_()
            ops.gemm_q8(w, dbs, dbq, out)
            assert np.array_equal(out[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))
    out.zero_()
    ops.gemm_q8(w, dbs, dbq, out)                        # with memory again: the tensor cores
    assert np.array_equal(out[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_operator_weight_with_one_copy_and_no_memory_for_the_other(ops, orc):
    m, k, n = 65536, 1024, 20                            # copies of 75 MB
    rng = np.random.default_rng(1)
    raw = rng.integers(0, 256, size=(m, k // 32, 18), dtype=np.uint8)
    raw[:, :, :2] = np.full((m, k // 32, 1), 0.01, np.float16).view(np.uint8).reshape(m, k // 32, 2)
    w = ops.QuantWeight(ops.DT_Q4_0, raw.reshape(-1), m, k)
    bs, bq = orc.quantize_q8_0(rng.standard_normal((n, k), dtype=F32))
    dbs, dbq = dev(bs), dev(bq)
    ops.gemm_q8_tc(w, dbs, dbq)
    want = orc.gemv(orc.DT_Q4_0, raw.reshape(m, -1), bs[n - 1], bq[n - 1], m, k)
    with Filled(48 << 20):
        got = ops.gemm_q8_tc_exact(w, dbs, dbq)          # (its output: 5 MB)
        assert np.array_equal(got[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_few_rows_without_memory_for_the_copies(ops, orc, model_dir):
    """9 to 15 rows: served by the CUDA cores, bit for bit the same; nothing stays allocated; more rows are refused as ever."""
    import wick_b200.model as wick
    from wick_b200 import _lib, gguf_synth as gs
    cm = wick.CudaLfm2Model(gs.cached_model("lfm2-350m", "q4_0", 0, cache_dir=model_dir), 256)
    st, toks = wick.InferenceState(), gs.random_prompt(16, cm.config().vocab_size)
    ids = [cm.seq_create() for _ in range(2)]
    cm.decode_batch_logits([1, 2], ids)                  # the batch's own buffers
    cm.set_prefill_mode("exact-cuda-cores")
    want = cm.forward_prefill(toks[:15], 0, st)
    cm.set_prefill_mode("exact")
    before = cm.gpu_memory_bytes()
    with Filled(48 << 20):
        for _ in range(2):
            assert np.array_equal(cm.forward_prefill(toks[:15], 0, st).view(np.uint32), want.view(np.uint32))
        assert cm.gpu_memory_bytes() == before
        with pytest.raises(_lib.WickCudaError) as e:
            cm.forward_prefill(toks, 0, st)
        assert e.value.code == _lib.ERR_OOM and cm.gpu_memory_bytes() == before
    assert np.array_equal(cm.forward_prefill(toks[:15], 0, st).view(np.uint32), want.view(np.uint32))
    with_copies = cm.gpu_memory_bytes()
    assert with_copies > before                          # the copies are there now; that of the vocabulary matrix is not yet
    with Filled(48 << 20):
        first = cm.decode_batch_logits([3, 4], ids)
        assert cm.gpu_memory_bytes() == with_copies
    alone = []
    for tok in (1, 2):
        s = wick.InferenceState()
        cm.forward_prefill([tok], 0, s)
        alone.append(cm.forward([tok + 2], 1, s))
    assert np.array_equal(first.view(np.uint32), np.stack(alone).view(np.uint32))


def test_both_gemms_of_a_model_share_the_memory_of_its_copies(ops, model_dir):
    """Switching the mode of a live model needs no memory, whichever came first, and the new mode's GEMM runs at once."""
    import wick_b200.model as wick
    from wick_b200 import gguf_synth as gs
    path = gs.cached_model("lfm2-350m", "q4_0", 0, cache_dir=model_dir)
    toks = gs.random_prompt(40, gs.SPECS["lfm2-350m"].vocab)

    def step(m, ids):
        """Kernels of a step of two rows, and its logits."""
        before = m.kernel_launches()
        return m.decode_batch_logits([3, 4], ids), m.kernel_launches() - before

    def fresh(mode):
        m = wick.CudaLfm2Model(path, 256)
        m.set_prefill_mode(mode)
        logits = m.forward_prefill(toks, 0, wick.InferenceState())
        ids = [m.seq_create() for _ in range(2)]
        return m, logits, ids, step(m, ids)[0]
    exact, exact_logits, exact_ids, exact_first = fresh("exact")
    kernels = step(exact, exact_ids)[1]
    tensor, tensor_logits, tensor_ids, tensor_first = fresh("tensor")
    assert exact_ids == tensor_ids
    assert np.array_equal(tensor_first.view(np.uint32), exact_first.view(np.uint32))  # (two rows are exact in either mode)
    size = exact.gpu_memory_bytes()
    assert tensor.gpu_memory_bytes() == size
    tensor.set_prefill_mode("exact")
    step(tensor, tensor_ids)
    assert step(tensor, tensor_ids)[1] == kernels         # two rows are enough to go over to the exact GEMM
    with Filled(48 << 20):
        for m in (exact, tensor):
            for mode, want in (("tensor", tensor_logits), ("exact", exact_logits), ("tensor", tensor_logits)):
                m.set_prefill_mode(mode)
                assert np.array_equal(m.forward_prefill(toks, 0, wick.InferenceState()).view(np.uint32), want.view(np.uint32)), mode
            m.set_prefill_mode("exact")
            for i in exact_ids:
                m.seq_destroy(i)
                assert m.seq_create() == i
            assert np.array_equal(step(m, exact_ids)[0].view(np.uint32), exact_first.view(np.uint32))
            assert step(m, exact_ids)[1] == kernels and m.gpu_memory_bytes() == size
