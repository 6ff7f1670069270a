"""Operator-API weights around the tensor-core product: reports of expired waits, captures of
other streams, and weights that are to stay at their packed size."""
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


def make(ops, orc, m=128, k=128, n=9, seed=0):
    """A weight, its raw blocks, and n quantised columns."""
    from wick_b200 import gguf_synth as gs
    rng = np.random.default_rng(seed)
    raw = gs.quantize_q4_0((rng.standard_normal((m, k)) * 0.02).astype(F32))
    bs, bq = orc.quantize_q8_0(rng.standard_normal((n, k), dtype=F32))
    return ops.QuantWeight(ops.DT_Q4_0, raw, m, k), raw, bs, bq


def check_product(ops, orc, w, raw, bs, bq):
    out = ops.gemm_q8(w, dev(bs), dev(bq)).cpu().numpy()
    for j in (0, len(bq) - 1):
        assert np.array_equal(out[j].view(np.uint32), orc.gemv(orc.DT_Q4_0, raw, bs[j], bq[j], w.m, w.k).view(np.uint32))


def plant(w, code=6):
    """What a kernel does whose wait has expired, done by the host."""
    return w._lib.wick_cuda_debug_weight_error(w._h, code)


def test_expired_wait_of_the_last_product_is_reported(ops, orc):
    from wick_b200 import _lib
    w, *args = make(ops, orc)
    w.check_products()                                   # nothing has run
    assert plant(w) == _lib.ERR_BAD_ARG                  # no word yet
    check_product(ops, orc, w, *args)
    w.check_products()
    assert plant(w) == _lib.OK
    with pytest.raises(_lib.WickCudaError) as e:
        w.check_products()
    assert e.value.code == _lib.ERR_TIMEOUT and "code 6" in e.value.message
    w.check_products()                                   # reported once
    assert plant(w) == _lib.OK
    with pytest.raises(_lib.WickCudaError) as e:         # or by the next product
        ops.gemm_q8(w, dev(args[1]), dev(args[2]))
    assert e.value.code == _lib.ERR_TIMEOUT
    check_product(ops, orc, w, *args)


def test_a_report_names_its_own_weight(ops, orc):
    """More weights than a page of error words: none takes another's report."""
    from wick_b200 import _lib
    ws, args = [], None
    for _ in range(1030):
        w, *args = make(ops, orc, m=4)
        ops.gemm_q8(w, dev(args[1]), dev(args[2]))
        ws.append(w)
    assert plant(ws[-1]) == _lib.OK
    for w in ws[:-1]:
        w.check_products()
    with pytest.raises(_lib.WickCudaError):
        ws[-1].check_products()
    for w in ws[5:]:
        w.close()
    check_product(ops, orc, ws[0], *args)


def test_first_product_beside_a_capture(ops, orc):
    """A weight's first product on one stream while another stream is captured (in torch's default, global mode) disturbs neither."""
    w, raw, bs, bq = make(ops, orc)
    x, dbs, dbq = torch.zeros(4, device="cuda"), dev(bs), dev(bq)
    out, side = torch.empty((len(bq), w.m), device="cuda"), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        x += 1
        with torch.cuda.stream(side):
            ops.gemm_q8(w, dbs, dbq, out)
    side.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    assert np.array_equal(out[8].cpu().numpy().view(np.uint32), orc.gemv(orc.DT_Q4_0, raw, bs[8], bq[8], w.m, w.k).view(np.uint32))


def test_captured_products(ops, orc):
    """Captured before and after the weight has its copy; replayed on new columns."""
    for warm in (False, True):
        w, raw, bs, bq = make(ops, orc, n=20)
        xs, xq, out = dev(bs), dev(bq), torch.empty((20, w.m), device="cuda")
        if warm:
            ops.gemm_q8(w, xs, xq, out)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ops.gemm_q8(w, xs, xq, out)
        _, _, bs, bq = make(ops, orc, n=20, seed=1)
        xs.copy_(dev(bs)), xq.copy_(dev(bq))
        g.replay()
        torch.cuda.synchronize()
        w.check_products()
        for j in (0, 19):
            assert np.array_equal(out[j].cpu().numpy().view(np.uint32), orc.gemv(orc.DT_Q4_0, raw, bs[j], bq[j], w.m, w.k).view(np.uint32))


def test_captured_product_of_a_weight_with_the_other_copy(ops, orc):
    """A weight that gemm_q8_tc has used runs on the tensor cores from a capture on, too: its copy for them is made beside the capture."""
    w, raw, bs, bq = make(ops, orc, m=16384, k=1024, n=20)
    xs, xq, out = dev(bs), dev(bq), torch.empty((20, w.m), device="cuda")
    ops.gemm_q8_tc(w, xs, xq)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ops.gemm_q8(w, xs, xq, out)
    assert torch.cuda.mem_get_info()[0] < free - (16 << 20)                 # 18.9 MB
    _, _, bs, bq = make(ops, orc, n=20, k=1024, seed=1)
    xs.copy_(dev(bs)), xq.copy_(dev(bq))
    g.replay()
    w.check_products()
    for j in (0, 19):
        assert np.array_equal(out[j].cpu().numpy().view(np.uint32), orc.gemv(orc.DT_Q4_0, raw, bs[j], bq[j], w.m, w.k).view(np.uint32))


def test_weight_that_stays_on_the_cuda_cores(ops, orc, monkeypatch):
    """The environment switch of the models, for operator weights: no copy, the same bits."""
    from wick_b200 import _lib
    monkeypatch.setenv("WICK_CUDA_PREFILL", "exact-cuda-cores")
    w, *args = make(ops, orc, m=16384, k=1024, n=40)
    monkeypatch.delenv("WICK_CUDA_PREFILL")
    x = dev(args[1]), dev(args[2])
    out = torch.empty((40, w.m), device="cuda")
    ops.gemm_q8(make(ops, orc)[0], *(dev(a) for a in make(ops, orc)[2:]))   # (loads the kernels)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ops.gemm_q8(w, *x, out)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > free - (8 << 20)                  # the copy would take 18.9 MB
    assert plant(w) == _lib.ERR_BAD_ARG
    check_product(ops, orc, w, *args)
    same, *_ = make(ops, orc, m=16384, k=1024, n=40)
    assert torch.equal(out.view(torch.int32), ops.gemm_q8(same, *x).view(torch.int32))
