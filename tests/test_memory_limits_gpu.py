"""Calls that need no int8 weight copy still work where there is no memory for one: the copy is a matter of speed."""
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
