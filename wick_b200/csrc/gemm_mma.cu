// Bit-exact integer GEMM for sm_100a: Q4_0 / Q8_0 weights x Q8_0 activations with the arithmetic of gemm_q*_q8_0_neon
// (simd.rs:696-1019) in its order.  Per output there are eight chains
//     acc[parity of the block][lane group] = acc + RN(float(p) * (f16(d_w) * d_x)),   blocks in ascending order,
// p = the integer dot product of the 8 elements of a NEON lane group (words l and 4 + l of a block), combined at the end as
// ((a0 + a1) + (a2 + a3)) per parity, even + odd.
//
// A lane group's eight elements are the K of one mma.sync m16n8k8 (f16 in, f32 out: products and sums of integers below 2^18 are
// exact), so the dot products arrive in the registers of the warp that owns the outputs, as floats, and no sums are wasted on
// other lane groups.  What is left is packed f32x2 arithmetic, two tokens per instruction: per 16 x 8 outputs and block 4 mma,
// 8 products, 8 additions and 2 scale products.
//
// Bound: the MMAs and the packed arithmetic one after the other.  In loops of their own an mma with a zero C takes 4.5 cycles of a
// scheduler, a packed operation 2 to 2.4, and both together the sum (they share something, the registers' read ports by
// guess): 54 cycles per (16 x 8, block) with every operand in shared memory, a ceiling of 170 TFLOP/s.  The whole kernel
// reaches 134 (6144 x 2048 at 512 tokens 96 us; by ncu FMA pipe 60 %, MMAs 27, issue 54, 3.2 warps per scheduler: the rest
// is latency) with activations that arrive as operands and 127 (101 us; 6912 x 2048 at 2002 433) where it converts
// them: there four warps have 5 % of the issue slots, and in small tiles a chain of their own.
// tcgen05 was here before (int8, lane groups as zero-padded columns, sums handed over through tensor memory): 115 and 463 us
// for those, 17 us for 1024 x 4608 at 9 tokens (now 7) and 23 for 2048 x 6912 at 16 (9.8): a hand-over per stage bound it, a round of
// release, issue, MMAs and wait that small tiles cannot hide at all, and that no order of loads or number of units shortened
// (next block loaded across stages 110, four smaller units 134).
// Taken back here: stages of 128 elements (147 against 101 us); more warps to the schedulers (R = 7: 104, R = 8: 142 against
// 96, for want of registers) and wider tiles with fewer (64 x 48: 114, 64 x 64: 161).
#include <cuda_fp16.h>
#include <algorithm>
#include <climits>
#include <cstring>

#include "gemm_mma.cuh"

namespace wick {

namespace {

constexpr int KB = MMA_STAGE_BLOCKS;  // blocks per pipeline stage (256 elements of K)
constexpr uint32_t MMA_SPIN_LIMIT = 1u << 18;  // try_wait itself suspends for a while, so this is of the order of a second

// R x 16 rows, NT x 8 tokens; a warp takes 16 rows, the blocks of one parity and 4 / LS of the lane groups: 2 R LS consumer warps.  READY: the activations are
// there in operand order (MmaInput) and come by bulk copies like the weights, issued by one warp; otherwise (operators: int8 columns
// of the caller) four warps convert them.
template <int R, int NT, bool READY, int LS>
struct MmaShape {
    static constexpr int CONSUMERS = 2 * R * LS, LG = 4 / LS, PRODUCERS = READY ? 1 : 4;
    static constexpr int THREADS = 32 * (CONSUMERS + PRODUCERS);
    static constexpr int TOKENS = 8 * NT;
    static constexpr int CTAS = R >= 4 ? 1 : 2;  // per SM
    static constexpr int W_BYTES = KB * MMA_CHUNK, X_BYTES = KB * MMA_X_CHUNK;  // of a row tile / token tile in a stage
    // As many stages as fit (up to 12): with five of them the small tiles had too few bytes of weights in flight.
    static constexpr int STAGE_BYTES = R * W_BYTES + NT * X_BYTES;
    static constexpr int FIT = (220000 / CTAS - R * (2 * LS - 1) * NT * 512) / STAGE_BYTES, STAGES = FIT < 12 ? FIT : 12;
    static constexpr int XW = READY ? 1 : NT, GROUPS = PRODUCERS / XW;  // producer warps to a stage; stages in the works at a time
};

template <int R, int NT, bool READY, int LS>
struct MmaSmem {
    using S = MmaShape<R, NT, READY, LS>;
    struct Stage {
        alignas(16) uint8_t a[R][KB][MMA_CHUNK];      // as in memory
        alignas(16) uint8_t b[NT][KB][MMA_X_CHUNK];   // as in an MmaInput: lane (token g, c)'s f16 pairs of the lane groups, scales
    };
    Stage stage[S::STAGES];
    alignas(16) float part[R][2 * LS - 1][NT][32][4];  // sums of a row tile's other warps, handed to its first one
    unsigned long long full[S::STAGES];               // weights and activations are there
    unsigned long long empty[S::STAGES];              // all consumer warps have read the stage
    unsigned long long part_full[R], part_empty[R];
    volatile uint32_t abort;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {  // asks once, never suspends
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of a whole warp.  False once the limit is hit or another warp has already given up.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t* err, uint32_t code) {
    for (uint32_t i = 0; i < MMA_SPIN_LIMIT; i++) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if ((i & 1023u) == 1023u && __any_sync(0xffffffffu, *abort)) return false;
    }
    *abort = 1;
    if ((threadIdx.x & 31) == 0) atomicCAS(err, 0u, code);
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t* err, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_test(bar, parity)) || mbar_wait_slow(bar, parity, abort, err, code);
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}

template <int N>
__device__ __forceinline__ void lds_words(uint32_t (&v)[N], uint32_t a) {
    if constexpr (N == 4)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
    else if constexpr (N == 2)
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(a));
    else
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[0]) : "r"(a));
}
__device__ __forceinline__ f32x2 lds64(uint32_t a) {
    f32x2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// D = A (16 x 8) * B (8 x 8): the dot products of one lane group, exact in f32.
__device__ __forceinline__ void mma_16x8x8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}

struct MmaTile {
    int mat, row_tile0, n0;
};
template <int R, int TOKENS>
__device__ __forceinline__ MmaTile mma_decode_tile(const MmaJob& job, int t, int tiles_n) {
    MmaTile r;
    r.mat = (t >= job.tile_start[1] ? 1 : 0) + (t >= job.tile_start[2] ? 1 : 0);
    const int local = t - job.tile_start[r.mat];
    r.row_tile0 = (local / tiles_n) * R;
    r.n0 = (local % tiles_n) * TOKENS;
    return r;
}

// WIDE: the columns are 16-byte aligned.  (A form of its own: as a branch it cost the aligned ones 2 of 440 us, 6912 x 2048 at 2002.)
template <int R, int NT, bool Q8, bool READY, int LS, bool WIDE>
__global__ void __launch_bounds__(MmaShape<R, NT, READY, LS>::THREADS, MmaShape<R, NT, READY, LS>::CTAS)
k_gemm_mma(const __grid_constant__ MmaJob job, const __grid_constant__ f32x2 minus_zero, uint32_t* err) {
    using S = MmaShape<R, NT, READY, LS>;
    using Stage = typename MmaSmem<R, NT, READY, LS>::Stage;
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t mma_smem_raw[];
    MmaSmem<R, NT, READY, LS>* sm = reinterpret_cast<MmaSmem<R, NT, READY, LS>*>(mma_smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = job.k / QK, k_stages = (nb + KB - 1) / KB;
    const int tiles_n = (job.n + S::TOKENS - 1) / S::TOKENS;
    const int tiles = job.tile_start[3];
    const uint32_t g_total = (uint32_t)((tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * (uint32_t)k_stages;
    const uint32_t fbar0 = smem_u32(&sm->full[0]), ebar0 = smem_u32(&sm->empty[0]);

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::STAGES; s++) {
            mbar_init(smem_u32(&sm->full[s]), READY ? 1 : 1 + S::XW);  // the bulk copies' (with their bytes) + every converting warp's
            mbar_init(smem_u32(&sm->empty[s]), S::CONSUMERS);
        }
        for (int r = 0; r < R; r++) {
            mbar_init(smem_u32(&sm->part_full[r]), 2 * LS - 1);
            mbar_init(smem_u32(&sm->part_empty[r]), 1);
        }
        sm->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    if (READY && warp >= S::CONSUMERS) {
        // ── producer: lane i < R copies row tile i of a stage, lane R + i token tile i (past the end: the last one again) ──
        int wt = blockIdx.x, wks = 0, xt = blockIdx.x, xks = 0;  // tile and stage of it that is copied next
        const int x_tiles = (job.n + MMA_X_ROWS - 1) / MMA_X_ROWS, x_item = min(max(lane - R, 0), NT - 1);
        const uint8_t *wsrc = nullptr, *xsrc = nullptr;
        const uint8_t* x = job.x;
        auto copy_weights = [&](uint32_t s) {
            if (wks == 0) {
                const MmaTile tl = mma_decode_tile<R, S::TOKENS>(job, wt, tiles_n);
                const int row_tiles = (job.m[tl.mat] + MMA_ROWS - 1) / MMA_ROWS;
                wsrc = job.w[tl.mat] + (size_t)min(tl.row_tile0 + min(lane, R - 1), row_tiles - 1) * k_stages * S::W_BYTES;
                wt += gridDim.x;
            }
            const uint32_t bar = fbar0 + s * 8;
            if (lane == 0) mbar_arrive_expect_tx(bar, S::STAGE_BYTES);
            __syncwarp();
            if (lane < R) bulk_load(smem_u32(sm->stage[0].a[lane]) + s * (uint32_t)sizeof(Stage), wsrc, S::W_BYTES, bar);
            wsrc += S::W_BYTES;
            if (++wks == k_stages) wks = 0;
        };
        auto copy_activations = [&](uint32_t s) {
            if (xks == 0) {
                const int n0 = mma_decode_tile<R, S::TOKENS>(job, xt, tiles_n).n0;
                xsrc = x + (size_t)min(n0 / MMA_X_ROWS + x_item, x_tiles - 1) * k_stages * S::X_BYTES;
                xt += gridDim.x;
            }
            if (lane >= R && lane < R + NT) bulk_load(smem_u32(sm->stage[0].b[x_item]) + s * (uint32_t)sizeof(Stage), xsrc, S::X_BYTES, fbar0 + s * 8);
            xsrc += S::X_BYTES;
            if (++xks == k_stages) xks = 0;
        };
        const uint32_t ahead = min(g_total, (uint32_t)S::STAGES);  // stages whose weights are asked for before the activations are there
        for (uint32_t g = 0; g < ahead; g++) copy_weights(g);
        pdl_wait();
        asm volatile("" : "+l"(x) : : "memory");
        for (uint32_t g = 0; g < ahead; g++) copy_activations(g);
        uint32_t s = 0, par = 0;
        for (uint32_t g = ahead; g < g_total; g++) {
            if (!mbar_wait(ebar0 + s * 8, par, &sm->abort, err, 1)) break;
            copy_weights(s);
            copy_activations(s);
            if (++s == S::STAGES) {
                s = 0;
                par ^= 1;
            }
        }
    } else if (warp >= S::CONSUMERS) {
        // ── producers: weights by bulk copies, activations converted to f16 in operand order ──
        // A stage belongs to XW warps (as many as there are token tiles), the stages go round the groups.  A warp takes four cycles and
        // more from one instruction to the next: with all four on every stage, ~150 instructions each, small tiles took 0.4 us a
        // stage for 0.15 of work (2048 x 6912 at 8 columns: 14.7 us), and any division here shows in the large ones too.
        const int pw = warp - S::CONSUMERS, grp = pw / S::XW, xw = pw % S::XW;
        // A task is 16 bytes of a token (half a block): lane bits 0, 1, 3, 4 are half and block, bit 2 the token, so that a token's 256
        // bytes are read together and the eight lanes of a store's quarter hit different banks (the two pieces of a
        // lane's 32 bytes are written in the order that its block's parity gives).
        const int half = lane & 1, blk = ((lane >> 1) & 1) | ((lane >> 2) & 6), piece = blk & 1, tok1 = (lane >> 2) & 1;
        constexpr int TASKS = 4, SCALES = 2, DEPTH = NT == 1 ? 1 : 2;  // of a lane in a stage; own stages read ahead
        struct Fetched {
            uint4 q[TASKS];
            float s[SCALES];
        };
        const int8_t* xq = job.xq;
        const float* xs = job.xs;
        int xt = blockIdx.x, xks = grp;  // tile and stage of it that is read next
        const int8_t* qsrc[TASKS];
        const float* ssrc[SCALES];
        auto seek = [&]() {  // (tokens past the last one repeat it; their outputs are not stored)
            for (; xks >= k_stages; xks -= k_stages) xt += gridDim.x;
            const int n0 = mma_decode_tile<R, S::TOKENS>(job, min(xt, tiles - 1), tiles_n).n0;  // (behind the last tile: it is read again, for nothing)
#pragma unroll
            for (int i = 0; i < TASKS; i++)
                qsrc[i] = xq + (size_t)min(n0 + (i * S::XW + xw) * 2 + tok1, job.n - 1) * job.k + (xks * KB + blk) * QK + half * 16;
#pragma unroll
            for (int i = 0; i < SCALES; i++)
                ssrc[i] = xs + (size_t)min(n0 + ((i * S::XW + xw) * 32 + lane) / KB, job.n - 1) * nb + xks * KB + lane % KB;
        };
        auto fetch = [&](Fetched& f) {
            // (a last stage that is only partly there: zeros, like the weights' padding)
            const int in_q = xks * KB + blk < nb, in_s = xks * KB + lane % KB < nb;
            if constexpr (WIDE) {
#pragma unroll
                for (int i = 0; i < TASKS; i++)
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                        "@p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                        : "=&r"(f.q[i].x), "=&r"(f.q[i].y), "=&r"(f.q[i].z), "=&r"(f.q[i].w)
                        : "l"(qsrc[i]), "r"(in_q));
            } else {  // (rows are multiples of 128 bytes: all of them are off by the same)
#pragma unroll
                for (int i = 0; i < TASKS; i++)
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                        "@p ld.global.u32 %0, [%4];\n\t@p ld.global.u32 %1, [%4 + 4];\n\t@p ld.global.u32 %2, [%4 + 8];\n\t"
                        "@p ld.global.u32 %3, [%4 + 12];\n\t}"
                        : "=&r"(f.q[i].x), "=&r"(f.q[i].y), "=&r"(f.q[i].z), "=&r"(f.q[i].w)
                        : "l"(qsrc[i]), "r"(in_q));
            }
#pragma unroll
            for (int i = 0; i < TASKS; i++) qsrc[i] += S::GROUPS * KB * QK;
#pragma unroll
            for (int i = 0; i < SCALES; i++) {
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.f32 %0, [%1];\n\t}"
                             : "=&f"(f.s[i])
                             : "l"(ssrc[i]), "r"(in_s));
                ssrc[i] += S::GROUPS * KB;
            }
            xks += S::GROUPS;
            if (xks >= k_stages) seek();
        };
        // Weights of one stage, by the group's first warp: lane i < R copies row tile i (past the end: the last one again).
        int wt = blockIdx.x, wks = grp;
        const uint8_t* wsrc = nullptr;
        auto seek_w = [&]() {
            for (; wks >= k_stages; wks -= k_stages) wt += gridDim.x;
            const MmaTile tl = mma_decode_tile<R, S::TOKENS>(job, min(wt, tiles - 1), tiles_n);
            const int row_tiles = (job.m[tl.mat] + MMA_ROWS - 1) / MMA_ROWS;
            wsrc = job.w[tl.mat] + ((size_t)min(tl.row_tile0 + lane, row_tiles - 1) * k_stages + wks) * S::W_BYTES;
        };
        auto fetch_weights = [&](uint32_t s) {
            const uint32_t bar = fbar0 + s * 8;
            if (lane == 0) mbar_arrive_expect_tx(bar, R * S::W_BYTES);
            __syncwarp();
            if (lane < R) bulk_load(smem_u32(sm->stage[0].a[lane]) + s * (uint32_t)sizeof(Stage), wsrc, S::W_BYTES, bar);
            wsrc += S::GROUPS * S::W_BYTES;
            wks += S::GROUPS;
            if (wks >= k_stages) seek_w();
        };
        const uint32_t ahead = min(g_total, (uint32_t)S::STAGES);  // stages whose weights are asked for before the activations are there
        if (xw == 0) {
            seek_w();
            for (uint32_t g = grp; g < ahead; g += S::GROUPS) fetch_weights(g);
        }
        pdl_wait();
        asm volatile("" : "+l"(xq), "+l"(xs) : : "memory");
        seek();
        Fetched f[DEPTH];
#pragma unroll
        for (int d = 0; d < DEPTH; d++) fetch(f[d]);
        const uint32_t b_dst = smem_u32(sm->stage[0].b[0][blk]) + (tok1 * 4 + 2 * half) * 16;
        // the piece that is written first holds the bytes 0, 1 of the words in even blocks, 2, 3 in odd ones
        const uint32_t sel0 = piece ? 0x4342 : 0x4140, sel1 = piece ? 0x4140 : 0x4342;
        uint32_t s = grp, par = 1;
        bool ok = true;
        for (uint32_t g0 = grp; g0 < g_total && ok; g0 += DEPTH * S::GROUPS) {
#pragma unroll
            for (int d = 0; d < DEPTH; d++) {
                const uint32_t g = g0 + d * S::GROUPS;
                if (g >= g_total) break;
                ok = mbar_wait(ebar0 + s * 8, par, &sm->abort, err, 1);
                if (!ok) break;
                if (xw == 0 && g >= ahead) fetch_weights(s);
                const uint32_t st = s * (uint32_t)sizeof(Stage);
#pragma unroll
                for (int i = 0; i < TASKS; i++) {
                    const uint32_t w[4] = {f[d].q[i].x ^ 0x80808080u, f[d].q[i].y ^ 0x80808080u, f[d].q[i].z ^ 0x80808080u, f[d].q[i].w ^ 0x80808080u};
                    uint32_t u[4], v[4];
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        u[l] = mma_hsub_1152(__byte_perm(w[l], 0x64646464u, sel0));
                        v[l] = mma_hsub_1152(__byte_perm(w[l], 0x64646464u, sel1));
                    }
                    const int pair = i * S::XW + xw;  // tokens 2 * pair, 2 * pair + 1
                    const uint32_t dst = b_dst + st + (pair >> 2) * S::X_BYTES + (pair & 3) * 128;
                    sts128(dst + piece * 16, u[0], u[1], u[2], u[3]);
                    sts128(dst + (piece ^ 1) * 16, v[0], v[1], v[2], v[3]);
                }
#pragma unroll
                for (int i = 0; i < SCALES; i++) {
                    const int tok = ((i * S::XW + xw) * 32 + lane) / KB;
                    reinterpret_cast<float*>(sm->stage[s].b[tok / MMA_X_ROWS][lane % KB] + 512)[tok % MMA_X_ROWS] = f[d].s[i];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(fbar0 + s * 8);
                fetch(f[d]);
                s += S::GROUPS;
                if (s >= S::STAGES) {
                    s -= S::STAGES;
                    par ^= 1;
                }
            }
        }
    } else {
        // ── consumers ──
        constexpr int LG = S::LG;
        const int rt = warp / (2 * LS), role = warp % (2 * LS), parity = role & 1, part = role >> 1, gid = lane >> 2, c = lane & 3;
        pdl_wait();  // (the outputs may still be read by the predecessor)
        struct Frag {
            uint32_t a[LG];
            f32x2 sw;  // rows gid, gid + 8
            uint32_t b[NT][LG];
            f32x2 sx[NT];
        };
        const uint32_t a_off = smem_u32(sm->stage[0].a[rt][parity]) + lane * 16 + part * (4 * LG), s_off = smem_u32(sm->stage[0].a[rt][parity]) + 512 + gid * 8;
        const uint32_t b_off = smem_u32(sm->stage[0].b[0][parity]) + lane * 16 + part * (4 * LG), x_off = smem_u32(sm->stage[0].b[0][parity]) + 512 + c * 8;
        auto load = [&](Frag& f, uint32_t st, int j) {  // j: which of the stage's blocks of this parity
            lds_words(f.a, a_off + st + j * (2 * MMA_CHUNK));
            f.sw = lds64(s_off + st + j * (2 * MMA_CHUNK));
#pragma unroll
            for (int n = 0; n < NT; n++) {
                lds_words(f.b[n], b_off + st + j * (2 * MMA_X_CHUNK) + n * S::X_BYTES);
                f.sx[n] = lds64(x_off + st + j * (2 * MMA_X_CHUNK) + n * S::X_BYTES);
            }
        };
        f32x2 acc[NT][2][LG];  // [token tile][row gid / gid + 8][lane group], halves = tokens 2c, 2c + 1
        auto chains = [&](const Frag& f) {
            uint32_t a0[LG], a1[LG];
#pragma unroll
            for (int l = 0; l < LG; l++) {
                a0[l] = Q8 ? f16_pair_lo(f.a[l]) : __byte_perm(f.a[l], 0, 0x1404);
                a1[l] = Q8 ? f16_pair_hi(f.a[l]) : __byte_perm(f.a[l], 0, 0x3424);
            }
            float s0, s1;
            unpack2(f.sw, s0, s1);
            const f32x2 sw[2] = {pack2(s0, s0), pack2(s1, s1)};
#pragma unroll
            for (int n = 0; n < NT; n++) {
                float p[LG][4];
#pragma unroll
                for (int l = 0; l < LG; l++) mma_16x8x8(p[l], a0[l], a1[l], f.b[n][l]);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const f32x2 d = mul2(sw[h], f.sx[n]);
#pragma unroll
                    for (int l = 0; l < LG; l++)  // (+ -0: the product alone, which a packed mul + add would not stay)
                        acc[n][h][l] = add2(acc[n][h][l], fma2(pack2(p[l][2 * h], p[l][2 * h + 1]), d, minus_zero));
                }
            }
        };
        uint32_t g = 0, tile_no = 0, s = 0, par = 0;
        bool ok = g_total == 0 || mbar_wait(fbar0, 0, &sm->abort, err, 2);
        // A warp that is alone on its scheduler, or nearly, waits for its own loads: the next block's operands are loaded under the
        // chains of one, across stages too.  From two token tiles on a block has work enough to hide them, and the registers
        // are better left to the compiler (64 x 16 tiles: 2048 x 6912 at 64 tokens 19.0 against 17.6 us, at 512 121 against
        // 108; R = 6, NT = 4: 103 against 96 us for 6144 x 2048).  Where converting warps share the schedulers, NT = 2 wants it too.
        constexpr bool AHEAD = NT == 1 || (NT == 2 && !READY);
        Frag f0, f1;
        if (AHEAD) load(f0, 0, 0);
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, tile_no++) {
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int l = 0; l < LG; l++) acc[n][0][l] = acc[n][1][l] = pack2(0.f, 0.f);
#pragma unroll 1
            for (int ks = 0; ks < k_stages; ks++, g++) {
                const uint32_t s1 = s + 1 == S::STAGES ? 0 : s + 1, npar = s1 ? par : par ^ 1;
                const uint32_t st = s * (uint32_t)sizeof(Stage);
                const bool more = g + 1 < g_total;
                const bool q = more && mbar_test(fbar0 + s1 * 8, npar);
                if constexpr (AHEAD) {
#pragma unroll
                    for (int j = 0; j < KB / 2; j += 2) {
                        load(f1, st, j + 1);
                        chains(f0);
                        if (j + 2 < KB / 2) {
                            load(f0, st, j + 2);
                        } else {
                            if (more && !__all_sync(0xffffffffu, q)) {
                                ok = mbar_wait_slow(fbar0 + s1 * 8, npar, &sm->abort, err, 2);
                                if (!ok) break;
                            }
                            load(f0, (more ? s1 : s) * (uint32_t)sizeof(Stage), 0);
                        }
                        chains(f1);
                    }
                    if (!ok) break;
                } else {
#pragma unroll
                    for (int j = 0; j < KB / 2; j++) {
                        load(f0, st, j);
                        chains(f0);
                    }
                    if (more && !__all_sync(0xffffffffu, q)) {
                        ok = mbar_wait_slow(fbar0 + s1 * 8, npar, &sm->abort, err, 2);
                        if (!ok) break;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(ebar0 + s * 8);
                s = s1;
                par = npar;
            }
            if (!ok) break;
            f32x2 sum[NT][2];  // of this warp's lane groups
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    sum[n][h] = acc[n][h][0];
                    if constexpr (LG >= 2) sum[n][h] = add2(sum[n][h], acc[n][h][1]);
                    if constexpr (LG == 4) sum[n][h] = add2(sum[n][h], add2(acc[n][h][2], acc[n][h][3]));
                }
            if (role) {
                ok = mbar_wait(smem_u32(&sm->part_empty[rt]), (tile_no & 1) ^ 1, &sm->abort, err, 3);
                if (!ok) break;
                float* ex = &sm->part[rt][role - 1][0][lane][0];
#pragma unroll
                for (int n = 0; n < NT; n++) *reinterpret_cast<ulonglong2*>(ex + n * 128) = make_ulonglong2(sum[n][0], sum[n][1]);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sm->part_full[rt]));
            } else {
                ok = mbar_wait(smem_u32(&sm->part_full[rt]), tile_no & 1, &sm->abort, err, 4);
                if (!ok) break;
                auto other = [&](int n, int r) { return *reinterpret_cast<const ulonglong2*>(&sm->part[rt][r - 1][n][lane][0]); };
#pragma unroll
                for (int n = 0; n < NT; n++) {  // ((a0 + a1) + (a2 + a3)) of a parity from its parts, then even + odd
                    ulonglong2 v[2];
#pragma unroll
                    for (int par2 = 0; par2 < 2; par2++) {
                        ulonglong2 q[LS];
#pragma unroll
                        for (int i = 0; i < LS; i++) q[i] = i == 0 && par2 == 0 ? make_ulonglong2(sum[n][0], sum[n][1]) : other(n, 2 * i + par2);
#pragma unroll
                        for (int w = LS; w > 1; w /= 2)
#pragma unroll
                            for (int i = 0; i < w / 2; i++) q[i] = make_ulonglong2(add2(q[2 * i].x, q[2 * i + 1].x), add2(q[2 * i].y, q[2 * i + 1].y));
                        v[par2] = q[0];
                    }
                    sum[n][0] = add2(v[0].x, v[1].x);
                    sum[n][1] = add2(v[0].y, v[1].y);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sm->part_empty[rt]));
                const MmaTile tl = mma_decode_tile<R, S::TOKENS>(job, t, tiles_n);
                const int m = job.m[tl.mat], row = (tl.row_tile0 + rt) * MMA_ROWS + gid;
                float* out = job.out[tl.mat];
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int tok = tl.n0 + n * 8 + 2 * c;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        float v0, v1;
                        unpack2(sum[n][h], v0, v1);
                        if (row + 8 * h < m) {
                            if (tok < job.n) out[(size_t)tok * m + row + 8 * h] = v0;
                            if (tok + 1 < job.n) out[(size_t)(tok + 1) * m + row + 8 * h] = v1;
                        }
                    }
                }
            }
        }
    }
    if (sm->abort)  // copies issued before the failure may still be landing in this CTA's shared memory
        for (int i = 0; i < 64; i++) __nanosleep(1000);
}

// One thread per (chunk, lane).
__global__ void k_mma_pack(DevWeight w, uint8_t* __restrict__ out) {
    const int nb = w.k / QK, nb_pad = (nb + KB - 1) / KB * KB, row_tiles = (w.m + MMA_ROWS - 1) / MMA_ROWS;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)row_tiles * nb_pad * 32) return;
    const int lane = (int)(idx & 31), gid = lane >> 2, c = lane & 3;
    const size_t chunk = idx >> 5;
    const int b = (int)(chunk % nb_pad), row0 = (int)(chunk / nb_pad) * MMA_ROWS + gid;
    uint32_t o[4];
    float sc[2];
#pragma unroll
    for (int l = 0; l < 4; l++) o[l] = w.dtype == DT_Q4_0 ? 0u : 0x80808080u;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int row = row0 + 8 * h;
        sc[h] = 0.f;
        if (row >= w.m || b >= nb) continue;
        const int g = row >> 2, r = row & 3;
        sc[h] = __half2float(w.d[(size_t)g * nb * 4 + b * 4 + r]);
        const uint32_t* qg = reinterpret_cast<const uint32_t*>(w.q + (size_t)g * w.q_group_bytes());
#pragma unroll
        for (int l = 0; l < 4; l++) {
            uint32_t two;  // elements 2c, 2c + 1 of lane group l
            if (w.dtype == DT_Q4_0) {
                // bytes of the word: elements 4l.. in the low nibbles, 16 + 4l.. in the high ones
                const uint32_t v = (qg[q4_word(b, r, l)] >> (c & 2 ? 4 : 0)) >> (c & 1 ? 16 : 0);
                two = 0;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const __half f = __int2half_rn((int)((v >> (8 * i)) & 15u) - 8);  // three significant bits: its low byte is 0
                    two |= (uint32_t)(__half_as_ushort(f) >> 8) << (8 * i);
                }
            } else {
                two = ((qg[q8_word(b, c >> 1, r, l)] >> (c & 1 ? 16 : 0)) & 0xFFFFu) ^ 0x8080u;
            }
            o[l] = h ? (o[l] & 0x0000FFFFu) | two << 16 : (o[l] & 0xFFFF0000u) | two;
        }
    }
    uint8_t* dst = out + chunk * MMA_CHUNK;
    reinterpret_cast<uint4*>(dst)[lane] = make_uint4(o[0], o[1], o[2], o[3]);
    if (c == 0) reinterpret_cast<float2*>(dst + 512)[gid] = make_float2(sc[0], sc[1]);
}

cudaError_t device_sm_count(int* sms) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e != cudaSuccess ? e : cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
}

template <int R, int NT, bool Q8, bool READY, int LS, bool WIDE>
cudaError_t launch_kernel(cudaStream_t st, const MmaJob& job, int sms, uint32_t* err) {
    using S = MmaShape<R, NT, READY, LS>;
    const size_t smem = sizeof(MmaSmem<R, NT, READY, LS>);
    static RaisedPerDevice limit;
    const cudaError_t e = raise_dynamic_smem(limit, (const void*)k_gemm_mma<R, NT, Q8, READY, LS, WIDE>, smem);
    if (e != cudaSuccess) return e;
    g_kernel_launches++;
    const f32x2 minus_zero = 0x8000000080000000ull;
    return launch_pdl(st, k_gemm_mma<R, NT, Q8, READY, LS, WIDE>, dim3(std::min(job.tile_start[3], sms * S::CTAS)), dim3(S::THREADS), smem, job, minus_zero, err);
}
template <int R, int NT, bool READY, int LS = 1>
cudaError_t launch_shape(cudaStream_t st, const MmaJob& job, bool q8, int sms, uint32_t* err) {
    if constexpr (!READY)
        if ((uintptr_t)job.xq & 15)
            return q8 ? launch_kernel<R, NT, true, READY, LS, false>(st, job, sms, err) : launch_kernel<R, NT, false, READY, LS, false>(st, job, sms, err);
    return q8 ? launch_kernel<R, NT, true, READY, LS, true>(st, job, sms, err) : launch_kernel<R, NT, false, READY, LS, true>(st, job, sms, err);
}

}  // namespace

bool mma_gemm_supported(int m, int k) { return m > 0 && k > 0 && k % 128 == 0; }

cudaError_t mma_weight_fill(cudaStream_t st, const DevWeight& w, uint8_t* p) {
    MmaWeight t;
    t.m = w.m;
    t.k = w.k;
    const size_t threads = t.bytes() / MMA_CHUNK * 32;
    g_kernel_launches++;
    k_mma_pack<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(w, p);
    return cudaGetLastError();
}

cudaError_t launch_gemm_mma(cudaStream_t st, const MmaWeight* const* w, float* const* out, int count, const uint8_t* x, const int8_t* xq,
                            const float* xs, int n, uint32_t* err, MmaTileShape* tile) {
    if (n <= 0 || count <= 0) return cudaSuccess;
    if (count > 3) return cudaErrorInvalidValue;
    for (int i = 1; i < count; i++) {
        if (w[i]->k != w[0]->k) return cudaErrorInvalidValue;
        if (w[i]->dtype != w[0]->dtype) {  // mixed types: a launch each
            for (int j = 0; j < count; j++) {
                const cudaError_t e = launch_gemm_mma(st, w + j, out + j, 1, x, xq, xs, n, err, tile);
                if (e != cudaSuccess) return e;
            }
            return cudaSuccess;
        }
    }
    int sms = 0;
    cudaError_t e = device_sm_count(&sms);
    if (e != cudaSuccess) return e;
    MmaJob job;
    memset(&job, 0, sizeof(job));
    job.x = x;
    job.xq = xq;
    job.xs = xs;
    job.n = n;
    job.k = w[0]->k;
    auto tiles = [&](int rows, int tokens) {
        int t = 0;
        for (int i = 0; i < count; i++) t += (w[i]->m + rows - 1) / rows * ((n + tokens - 1) / tokens);
        return t;
    };
    // The shape that needs least time: rounds of tiles times what a stage of one takes, in 1/100 us, measured with one CTA of it on an
    // SM and with all that fit.  Wide tiles do a little more per stage (96 x 32 outputs in 1.56 us, 64 x 16 in 0.54, 16 x 8 in 0.28),
    // narrow ones end sooner where there are few: 2048 x 6912 at 64 tokens 45.1 us as 96 x 32 and 17.6 as 64 x 16, at 96 tokens
    // 32.3 as 64 x 16 (two rounds, the second with a third of the SMs) and 24.7 as 64 x 24, at 6 tokens 12.4 as 64 x 8 and 9.5 as
    // 16 x 8, where two warps share a row tile's lane groups (11.3 with one).
    struct Shape {
        int r, nt, ctas, one, all;
    };
    static constexpr Shape READY_SHAPES[MMA_SHAPES] = {{6, 4, 1, 156, 156}, {6, 2, 1, 78, 78}, {4, 3, 1, 80, 80}, {4, 2, 1, 53, 54},
                                                     {4, 1, 1, 38, 42},   {2, 1, 2, 36, 38}, {1, 1, 2, 27, 28}};
    // (with the converting warps: two lane-group warps bring nothing, 1024 x 4608 at 9 tokens 8.4 against 8.1 us.  32 x 8 and 16 x 16 are
    // for narrow matrices with many columns: 96 x 6912 at 600 16.8 us as 32 x 8, without the two 22.6; 16 x 2048 at 2400 8.7 and 10.2)
    static constexpr Shape CONVERT_SHAPES[MMA_SHAPES] = {{6, 4, 1, 176, 176}, {4, 4, 1, 120, 120}, {4, 2, 1, 67, 67}, {4, 1, 1, 41, 41},
                                                       {2, 1, 2, 42, 46},   {1, 2, 2, 46, 51},   {1, 1, 2, 32, 40}};
    const Shape* shapes = x ? READY_SHAPES : CONVERT_SHAPES;
    int best = 0, best_cost = INT_MAX;
    for (int i = 0; i < MMA_SHAPES; i++) {
        const Shape& s = shapes[i];
        const int t = tiles(s.r * MMA_ROWS, s.nt * 8), slots = sms * s.ctas, rest = t % slots;
        const int cost = t / slots * s.all + (rest == 0 ? 0 : rest <= sms ? s.one : s.all);
        if (cost < best_cost) best = i, best_cost = cost;
    }
    if (tile && tile->index >= 0 && tile->index < MMA_SHAPES) best = tile->index;
    const int rows = shapes[best].r * MMA_ROWS, tokens = shapes[best].nt * 8;
    if (tile) *tile = MmaTileShape{best, rows, tokens};
    int t = 0;
    for (int i = 0; i < 3; i++) {
        job.tile_start[i] = t;
        if (i >= count) continue;  // (matrices that are not there own no tiles)
        job.w[i] = w[i]->p;
        job.out[i] = out[i];
        job.m[i] = w[i]->m;
        t += (w[i]->m + rows - 1) / rows * ((n + tokens - 1) / tokens);
    }
    job.tile_start[3] = t;
    const bool q8 = w[0]->dtype == DT_Q8_0;
    if (x) switch (best) {
            case 0: return launch_shape<6, 4, true>(st, job, q8, sms, err);
            case 1: return launch_shape<6, 2, true>(st, job, q8, sms, err);
            case 2: return launch_shape<4, 3, true>(st, job, q8, sms, err);
            case 3: return launch_shape<4, 2, true>(st, job, q8, sms, err);
            case 4: return launch_shape<4, 1, true>(st, job, q8, sms, err);
            case 5: return launch_shape<2, 1, true>(st, job, q8, sms, err);
            default: return launch_shape<1, 1, true, 2>(st, job, q8, sms, err);
        }
    switch (best) {
        case 0: return launch_shape<6, 4, false>(st, job, q8, sms, err);
        case 1: return launch_shape<4, 4, false>(st, job, q8, sms, err);
        case 2: return launch_shape<4, 2, false>(st, job, q8, sms, err);
        case 3: return launch_shape<4, 1, false>(st, job, q8, sms, err);
        case 4: return launch_shape<2, 1, false>(st, job, q8, sms, err);
        case 5: return launch_shape<1, 2, false>(st, job, q8, sms, err);
        default: return launch_shape<1, 1, false>(st, job, q8, sms, err);
    }
}

}  // namespace wick
