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
    dbs, dbq, out = dev(bs), dev(bq), torch.empty((n, m), device="cuda")
    want = orc.gemv(orc.DT_Q4_0, raw.reshape(m, -1), bs[n - 1], bq[n - 1], m, k)
    with Filled(48 << 20):
        for _ in range(2):
            out.zero_()
            ops.gemm_q8(w, dbs, dbq, out)
            assert np.array_equal(out[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))
    out.zero_()
    ops.gemm_q8(w, dbs, dbq, out)                        # with memory again: the tensor cores
    assert np.array_equal(out[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))
