"""The bit-exact GEMM on the tensor cores at the edges of its tiles, stages and rounds, against the CUDA-core kernel (itself
compared with the oracle) for every output and the oracle for sampled ones."""
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


# On 148 SMs the rule takes tiles of 16 x 8, 64 x 8, 64 x 16 and 96 x 32 for these, one round and several; stages of 256 elements, the last
# one half there (k = 128, 384).  Every shape, and more tiles than SMs with fewer stages to a tile than producer groups: test_every_tile_shape.
@pytest.mark.parametrize("dtype", ["q4_0", "q8_0"])
@pytest.mark.parametrize("m,k,n", [(1, 128, 1), (16, 256, 8), (17, 384, 9), (95, 640, 16), (97, 1024, 33), (2400, 128, 7), (4808, 128, 65),
                                   (1000, 384, 24), (9600, 256, 31), (96 * 160, 128, 40), (2048, 1152, 200), (520, 2304, 97)])
def test_exact_gemm_at_its_edges(ops, orc, cuda_core_weight, dtype, m, k, n):
    rng = np.random.default_rng(m + k + n)
    raw = rng.integers(0, 256, size=(m, k // 32, 18 if dtype == "q4_0" else 34), dtype=np.uint8)  # every int8, -128 too
    raw[:, :, :2] = rng.uniform(-0.02, 0.02, size=(m, k // 32)).astype(np.float16).view(np.uint8).reshape(m, k // 32, 2)
    bq = rng.integers(-128, 128, size=(n, k), dtype=np.int8)
    bs = rng.uniform(0.0, 0.1, size=(n, k // 32)).astype(np.float16).astype(F32)
    dt = ops.QTYPE_ID[dtype]
    got = ops.gemm_q8_tc_exact(ops.QuantWeight(dt, raw.reshape(-1), m, k), dev(bs), dev(bq))
    assert torch.equal(got.view(torch.int32), ops.gemm_q8(cuda_core_weight(dt, raw.reshape(-1), m, k), dev(bs), dev(bq)).view(torch.int32))
    for j in {0, n - 1}:
        want = orc.gemv(dt, raw.reshape(m, -1), bs[j], bq[j], m, k)
        assert np.array_equal(got[j].cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("m,k,n,off", [(130, 256, 20, 4), (97, 384, 33, 8), (16, 640, 9, 12), (9600, 384, 31, 4), (2400, 128, 40, 12), (2048, 1152, 200, 4)])
def test_columns_that_are_not_16_byte_aligned(ops, orc, cuda_core_weight, m, k, n, off):
    """A caller's 4-byte aligned columns run on the tensor cores, too."""
    from wick_b200 import _lib, gguf_synth as gs
    rng = np.random.default_rng(m + n)
    raw = gs.quantize_q4_0((rng.standard_normal((m, k)) * 0.02).astype(F32))
    bs, bq = orc.quantize_q8_0(rng.standard_normal((n, k), dtype=F32))
    room = torch.zeros(n * k + off, dtype=torch.int8, device="cuda")
    room[off:] = dev(bq).flatten()
    want = ops.gemm_q8(cuda_core_weight(ops.DT_Q4_0, raw, m, k), dev(bs), dev(bq))
    assert np.array_equal(want[n - 1].cpu().numpy().view(np.uint32), orc.gemv(orc.DT_Q4_0, raw, bs[n - 1], bq[n - 1], m, k).view(np.uint32))
    for f in (ops.gemm_q8, ops.gemm_q8_tc_exact):
        w = ops.QuantWeight(ops.DT_Q4_0, raw, m, k)
        got = f(w, dev(bs), room[off:].view(n, k))
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
        assert w._lib.wick_cuda_debug_weight_error(w._h, 0) == _lib.OK  # (BAD_ARG where no product has used the tensor cores)


# Rows and tokens of the tile shapes: of the form with activations in operand order, which every prompt and batched step of a model
# takes, and of that with int8 columns (gemm_q8).
TILES = {True: [(96, 32), (96, 16), (64, 24), (64, 16), (64, 8), (32, 8), (16, 8)],
         False: [(96, 32), (64, 32), (64, 16), (64, 8), (32, 8), (16, 16), (16, 8)]}


def gemm_rows(w, x, ready, tile=-1):
    """The product of f32 rows by a tile shape (-1: the rule's) and the shape that ran."""
    import ctypes as C
    from wick_b200 import _lib
    out, t = torch.empty((x.shape[0], w.m), device="cuda"), (C.c_int32 * 3)(tile, 0, 0)
    _lib.check(w._lib.wick_cuda_debug_gemm_rows(w._h, x.data_ptr(), x.shape[0], int(ready), t, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return out, (t[1], t[2])


@pytest.mark.parametrize("dtype", ["q4_0", "q8_0"])
@pytest.mark.parametrize("ready", [True, False])
@pytest.mark.parametrize("tile", range(7))
def test_every_tile_shape(ops, orc, cuda_core_weight, dtype, ready, tile):
    """A row and a token more than a tile, fewer than three of each, and more tiles than SMs; k = 128 * odd leaves half of the last stage empty."""
    rows, tokens = TILES[ready][tile]
    for m, k, n in ((rows + 1, 128, tokens + 1), (3 * rows - 5, 384, 2 * tokens - 1), (rows * 150 + 7, 640, 3 * tokens + 2), (1, 1152, 1)):
        rng = np.random.default_rng(m + k + n)
        raw = rng.integers(0, 256, size=(m, k // 32, 18 if dtype == "q4_0" else 34), dtype=np.uint8)  # every int8, -128 too
        raw[:, :, :2] = rng.uniform(-0.02, 0.02, size=(m, k // 32)).astype(np.float16).view(np.uint8).reshape(m, k // 32, 2)
        dt = ops.QTYPE_ID[dtype]
        x = dev(rng.standard_normal((n, k), dtype=F32) * np.exp(rng.standard_normal((n, 1), dtype=F32)))
        x[n // 2, :32] = 0
        got, ran = gemm_rows(ops.QuantWeight(dt, raw.reshape(-1), m, k), x, ready, tile)
        assert ran == (rows, tokens)
        bs, bq = ops.quantize_f32_to_q8_0(x)
        assert torch.equal(got.view(torch.int32), ops.gemm_q8(cuda_core_weight(dt, raw.reshape(-1), m, k), bs, bq).view(torch.int32)), (m, k, n)
        want = orc.gemv(dt, raw.reshape(m, -1), bs[n - 1].cpu().numpy(), bq[n - 1].cpu().numpy(), m, k)
        assert np.array_equal(got[n - 1].cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("ready,m,n,tile", [(True, 6144, 512, 0), (True, 2048, 96, 1), (True, 65536, 24, 2), (True, 2048, 64, 3), (True, 1024, 33, 4),
                                            (True, 65536, 6, 5), (True, 2048, 6, 6), (False, 6912, 2002, 0), (False, 2048, 96, 1), (False, 2048, 64, 2),
                                            (False, 1024, 33, 3), (False, 2048, 9, 6)])
def test_tile_shapes_of_ordinary_sizes(ops, ready, m, n, tile):
    """What the rule takes on 148 SMs."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule goes by the device's SMs")
    w = ops.QuantWeight(ops.DT_Q4_0, np.zeros(m * 4 * 18, np.uint8), m, 128)
    assert gemm_rows(w, torch.ones((n, 128), device="cuda"), ready)[1] == TILES[ready][tile]
