// Matrix product of float32 operands for more than a few rows, C[M, N] = A[M, K] W[N, K]^T with float32's precision, on the
// 5th-generation tensor cores.
//
// A float32 number is the sum of three bfloat16 numbers, x = x0 + x1 + x2 (each the nearest to what is left: 3 x 8 bits hold
// the 24 bits of the mantissa).  Both operands are split times 2^24, which loses nothing: the third part has room in bfloat16's
// exponents down to the smallest subnormal number (unscaled, numbers below 2^-109 would lose it), and sums are scaled back, exactly,
// in the epilogue.  A product of two such sums has nine terms; the six whose orders of magnitude add up to 2 or less (a2 w0, a0 w2,
// a1 w1, a1 w0, a0 w1, a0 w0) are multiplied, exactly, by the bfloat16 tensor cores; of the three left out a1 w2 and a2 w1 reach
// 2^-25 of the product, all together 2^-24, a float32 multiply-add's own rounding.  What costs precision on tensor cores is the
// accumulation, whose additions are truncated: so an accumulator in tensor memory lives for 64 elements of K only (its small
// terms first, its four large additions last) and is then added, rounded to nearest, into float32 registers.  A sum of K products so has K / 64
// ordinary float32 additions where the plain kernel's chain of multiply-adds has K.
//
// The weights take the M side of the instruction (128 rows of W a tile), tokens the N side (tiles of 64 or 128).  The
// weights stay float32 in memory: a tile is fetched by TMA, eight warps split it in registers and put the three parts into
// tensor memory, from where the MMA reads them (its A operand).  The tokens are split beforehand by a small kernel of
// their own into three bfloat16 planes, since every tile of W reads them again.
//
// Roles (640 threads, one CTA an SM):
//   warp 0, one lane   TMA of the tokens' three planes, 64 elements of K a stage
//   warp 1, one lane   MMA: 24 instructions a stage, then commits onto the stage's barriers
//   warp 2, one lane   TMA of the weights (two boxes of 32 columns a stage); they are weights, so the first stages are asked
//                      for before the dependency wait
//   warps 4..11        split: a thread owns a row of the tile and half of a stage
//   warps 12..19       sums: a thread owns a row of W and half of the tokens; epilogue (lanes are neighbouring columns of
//                      C, so every store is one run of 128 bytes)
// Few tiles (few tokens or a narrow output): K is cut into spans, one CTA each, which form a cluster; their sums meet in
// distributed shared memory and are added in span order.
//
// What is not finite: the split of an infinity or of a number that rounds to one (from 2^104 on) leaves NaN where the plain sum may be
// finite or infinite, and scaled sums are infinite from 2^80 on.  A sum that comes out not finite is therefore formed again from the
// float32 operands with plain multiply-adds.
//
// Bound: six bfloat16 products per float32 product under the power limit, i.e. a sixth of the 1,375 TFLOP/s that bfloat16
// products sustain (229), or the stream of the weights for few tokens.  Measured: 2,048 x 16,384 x 2,048 in 0.69 ms = 200 TFLOP/s
// (plain kernel 3.40 ms = 40; the MMAs alone, nothing waited for, 0.44 ms), 2,048 x 2,048 x 8,192 in 0.38 ms (1.94), 64 x 2,048 x
// 8,192 in 39 us (634).  Error against 64 bits, of the norm: 1.3e-7 at K = 2,048 and 2.2e-7 at 8,192 (plain kernel 8.1e-7 and 1.6e-6).
// Tried and not faster: three stages of tokens, one lane alone polling, a barrier per consumer (3 % slower).
#include "tcgen05.cuh"

namespace b200 {

constexpr int kF32Threads = 640;
constexpr int kF32SplitWarp = 4, kF32SumWarp = 12;   // the first of eight warps each (multiples of 4: tensor memory lanes go by warp % 4)
constexpr int kF32Rows = 128;        // rows of W per tile
constexpr int kF32MaxSpans = 8;
constexpr int TS = 2;                // stages of tokens, of parts and accumulators: one barrier tells all of a stage's MMAs' end

__device__ int g_gemm_f32_status = 0;  // 0 ok; else (role << 8 | stage) of the wait that gave up

template <int BN, int WS>
struct F32Smem {
    alignas(1024) __nv_bfloat16 tok[TS][3][BN * BK];
    alignas(1024) float w[WS][2][kF32Rows * 32];
    alignas(8) uint64_t tok_full[TS];
    uint64_t w_full[WS];
    uint64_t w_empty[WS];
    uint64_t part_full[2];    // split warps -> MMA: the three parts of a stage's weights lie in tensor memory
    uint64_t done[2];         // MMA -> all the others: the stage's MMAs are complete (its tokens and parts are read, its sums are there)
    uint64_t acc_empty[2];    // sum warps -> MMA
    uint32_t tmem_base;
    int abort_flag;
};

struct F32Args {
    const float* A;      // [M][lda], for sums that are formed again
    const float* W;      // [N][ldw]
    float* C;            // [M][ldc]
    const float* bias;   // [N] or null
    int lda, ldw, ldc, M, N, K;
    int epilogue;        // 0 store, 1 residual add, 2 gated SiLU, 3 gated GELU (tanh form), 4 gated and clamped
    int silu_cols;
    float gate_limit, gate_slope;
    int blocks_per_span; // of 64 elements of K
};

__device__ __forceinline__ void mbar_arrive_f32(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// whether three phases have all ended, without waiting
__device__ __forceinline__ bool mbar_test3(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, uint64_t* c, uint32_t pc) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p, q, r;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n"
        "and.pred p, p, q;\nand.pred p, p, r;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(smem_u32(a)), "r"(pa), "r"(smem_u32(b)), "r"(pb), "r"(smem_u32(c)), "r"(pc) : "memory");
    return done != 0;
}
// D[tmem] (+)= A[tmem] B[smem]: A's row i lies in lane i, its K elements as bfloat16 pairs along the columns
__device__ __forceinline__ void umma_bf16_from_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, int accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

constexpr float kF32Up = 16777216.f;                        // operands are split times 2^24 ...
constexpr float kF32Down = 1.f / (kF32Up * kF32Up);         // ... and sums carry 2^48

// x, y -> the three bfloat16 parts of 2^24 x and 2^24 y as pairs (x in the low half)
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    unsigned long long xy, up;
    asm("mov.b64 %0, {%1, %2};" : "=l"(xy) : "f"(x), "f"(y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(up) : "f"(kF32Up));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(xy) : "l"(up));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(xy));
    __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    p0 = *reinterpret_cast<uint32_t*>(&h);
    x -= __uint_as_float(p0 << 16);
    y -= __uint_as_float(p0 & 0xffff0000u);
    h = __floats2bfloat162_rn(x, y);
    p1 = *reinterpret_cast<uint32_t*>(&h);
    x -= __uint_as_float(p1 << 16);
    y -= __uint_as_float(p1 & 0xffff0000u);
    h = __floats2bfloat162_rn(x, y);
    p2 = *reinterpret_cast<uint32_t*>(&h);
}

// the tokens' planes: planes[p][row][0 .. padded - 1], zeros from K on (padded: K rounded up to a multiple of 8).
// Bound by its bytes (4 read, 6 written per element): a thread takes 8 elements.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ A, int lda, __nv_bfloat16* __restrict__ planes, int M, int K, int padded) {
    pdl_wait();
    pdl_launch_dependents();   // (not before the wait: what the next kernel reads ahead of its own wait is then older than this kernel)
    const int per_row = padded / 8;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)M * per_row) return;
    const int row = (int)(i / per_row), k = (int)(i - (long long)row * per_row) * 8;
    const float* src = A + (size_t)row * lda + k;
    float v[8];
    if (k + 8 <= K && ((uintptr_t)src & 15) == 0) {
        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = k + j < K ? src[j] : 0.f;
    }
    uint32_t p[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split_pair(v[2 * j], v[2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        *reinterpret_cast<uint4*>(planes + ((size_t)q * M + row) * padded + k) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
}

// one sum from the float32 operands, in order of k (a NaN stays one: a row that holds NaN throughout costs nothing)
__device__ __noinline__ float plain_sum(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.f;
    for (int k = 0; k < K && !isnan(s); ++k) s = fmaf(a[k], w[k], s);
    return s;
}

// (a call, not inlined: the epilogue is unrolled over a thread's sums)
__device__ __noinline__ float gated_f32(float gate, float up, int epilogue, float limit, float slope) {
    if (epilogue == 4) {
        const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
        return g / (1.0f + expf(-slope * g)) * (u + 1.0f);
    }
    if (epilogue == 3) return 0.5f * gate * (1.0f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) * up;
    return (gate / (1.0f + expf(-gate))) * up;
}
__device__ __noinline__ float silu_f32(float s) { return s / (1.0f + expf(-s)); }

// One sum (times 2^48) per lane, lanes being neighbouring columns n of row m of C (n - lane a multiple of 32): epilogue and store.  All
// lanes of the warp call it.  EPI: 0 store, 1 residual add, 2 the gated ones.
template <int EPI>
__device__ __forceinline__ void finish_sum(float s, int m, int n, const F32Args& p) {
    const bool live = m < p.M && n < p.N;
    s *= kF32Down;
    if (live && !isfinite(s)) s = plain_sum(p.A + (size_t)m * p.lda, p.W + (size_t)n * p.ldw, p.K);
    if (p.bias != nullptr && live) s += p.bias[n];
    if (EPI == 2) {
        const float up = __shfl_down_sync(0xffffffffu, s, 1);   // even lanes hold gates, the next lane the up value
        if (live && (n & 1) == 0)                               // (N is even: n + 1 < N)
            p.C[(size_t)m * p.ldc + (n >> 1)] = gated_f32(s, up, p.epilogue, p.gate_limit, p.gate_slope);
        return;
    }
    if (!live) return;
    float* c = p.C + (size_t)m * p.ldc + n;
    if (EPI == 1) *c += s;
    else *c = n < p.silu_cols ? silu_f32(s) : s;
}

template <int BN, int WS, int EPI>
__global__ void __launch_bounds__(kF32Threads, 1)
gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_tok, const __grid_constant__ CUtensorMap map_w, const F32Args p) {
    using Smem = F32Smem<BN, WS>;
    constexpr int kHalf = BN / 2;            // tokens a sum thread owns
    constexpr uint32_t kTmemCols = 512;      // two accumulators of BN columns, two stages of 3 x 32 columns of weights
    constexpr int kPitch = kF32Rows + 1;     // floats per token of the partial tile that spans exchange
    static_assert(sizeof(float) * BN * kPitch <= sizeof(Smem::tok), "the partial tile fits where the tokens' stages were");
    extern __shared__ uint8_t smem_raw[];
    auto& sm = *reinterpret_cast<Smem*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = (p.M + BN - 1) / BN, tiles_n = (p.N + kF32Rows - 1) / kF32Rows, n_tiles = tiles_m * tiles_n;
    const int n_spans = gridDim.y, span = blockIdx.y;    // (with spans the grid has one CTA per tile and span)
    const int kb_total = (p.K + BK - 1) / BK;
    const int kb0 = span * p.blocks_per_span, k_iters = max(0, min(kb_total, kb0 + p.blocks_per_span) - kb0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < TS; ++s) mbar_init(&sm.tok_full[s], 1);
        for (int s = 0; s < WS; ++s) { mbar_init(&sm.w_full[s], 1); mbar_init(&sm.w_empty[s], 8); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm.part_full[b], 8); mbar_init(&sm.done[b], 1);
            mbar_init(&sm.acc_empty[b], 8);
        }
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_tok) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem_base;
    const uint32_t tmem_parts = tmem + 2 * BN;
    volatile int* abort_flag = &sm.abort_flag;
    // tiles run down the tokens first: the CTAs at work at one time share a few blocks of W
    auto fetch_weights = [&](int it, int tile, int k) {
        const int s = it % WS, n0 = (tile / tiles_m) * kF32Rows;
        mbar_expect_tx(&sm.w_full[s], kF32Rows * BK * 4);
        tma_load_2d(sm.w[s][0], &map_w, (kb0 + k) * BK, n0, &sm.w_full[s]);
        tma_load_2d(sm.w[s][1], &map_w, (kb0 + k) * BK + 32, n0, &sm.w_full[s]);
    };
    const bool weights_lane = warp == 2 && lane == 0;
    const int early = min(WS, k_iters);      // stages of the first tile that are asked for ahead of the wait
    if (weights_lane && (int)blockIdx.x < n_tiles)
        for (int k = 0; k < early; ++k) fetch_weights(k, blockIdx.x, k);
    pdl_launch_dependents();
    pdl_wait();

    if (warp == 0 && lane == 0) {
        // ---- tokens
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const int m0 = (tile % tiles_m) * BN;
            for (int k = 0; k < k_iters; ++k, ++it) {
                const int s = it % TS;
                if (it >= TS && !mbar_wait(&sm.done[s], ((it / TS) - 1) & 1, abort_flag)) {
                    *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (1 << 8) | s); ok = false; break;
                }
                mbar_expect_tx(&sm.tok_full[s], 3 * BN * BK * 2);
                // (a box may reach from one plane into the next, or past the last: those columns are never stored)
                for (int q = 0; q < 3; ++q) tma_load_2d(sm.tok[s][q], &map_tok, (kb0 + k) * BK, q * p.M + m0, &sm.tok_full[s]);
            }
        }
    } else if (weights_lane) {
        // ---- weights
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            for (int k = 0; k < k_iters; ++k, ++it) {
                if (it < early) continue;
                const int s = it % WS;
                if (it >= WS && !mbar_wait(&sm.w_empty[s], ((it / WS) - 1) & 1, abort_flag)) {
                    *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (2 << 8) | s); ok = false; break;
                }
                fetch_weights(it, tile, k);
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA.  An instruction is issued when the tensor core has taken the one before, so the thread is busy for as long
        // as they run, and a wait, even for what is there already, costs 120 cycles: the next stage's barriers are asked for
        // (all three at once) while the last instructions of this one are still queued.
        constexpr uint32_t idesc = umma_idesc_bf16(kF32Rows, BN);
        const int total = (int)blockIdx.x < n_tiles ? ((n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * k_iters : 0;
        auto ready = [&](int it) {
            const int s = it % TS, b = it & 1;
            const uint32_t half = (it >> 1) & 1;   // (a fresh barrier passes a wait for parity 1)
            if (mbar_test3(&sm.acc_empty[b], half ^ 1, &sm.tok_full[s], (it / TS) & 1, &sm.part_full[b], half)) return true;
            if (mbar_wait(&sm.acc_empty[b], half ^ 1, abort_flag) && mbar_wait(&sm.tok_full[s], (it / TS) & 1, abort_flag) &&
                mbar_wait(&sm.part_full[b], half, abort_flag)) return true;
            *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (3 << 8) | s);
            return false;
        };
        bool ok = total > 0 && ready(0);
        for (int it = 0; it < total && ok; ++it) {
            const int s = it % TS, b = it & 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + b * BN;
            // the terms in order of growing size: an accumulator's truncated additions then cost least
            constexpr int part_w[6] = {2, 0, 1, 1, 0, 0}, part_t[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                if (q == 4 && it + 1 < total) ok = ready(it + 1);
                const uint32_t a = tmem_parts + b * 96 + part_w[q] * 32;
                const uint64_t bd = umma_desc(sm.tok[s][part_t[q]]);
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) umma_bf16_from_tmem(acc, a + 8 * kk, bd + 2 * kk, idesc, (q | kk) != 0);
            }
            umma_commit(&sm.done[b]);
        }
    } else if (warp >= kF32SplitWarp && warp < kF32SumWarp) {
        // ---- split: this thread's row of the tile, 32 of a stage's 64 elements.  The parts are made before the wait for
        // their place in tensor memory: only the stores lie between two stages' MMAs.
        const int quarter = warp & 3, h = (warp - kF32SplitWarp) >> 2, row = quarter * 32 + lane;
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            for (int k = 0; k < k_iters; ++k, ++it) {
                const int s = it % WS, b = it & 1;
                ok = mbar_wait(&sm.w_full[s], (it / WS) & 1, abort_flag);
                if (!ok && lane == 0) { *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (4 << 8) | s); }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) break;
                const float* src = sm.w[s][h] + row * 32;   // eight 16-byte pieces, at piece ^ (row % 8)
                uint32_t p0[16], p1[16], p2[16];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(src + ((j ^ (row & 7)) << 2));
                    split_pair(v.x, v.y, p0[2 * j], p1[2 * j], p2[2 * j]);
                    split_pair(v.z, v.w, p0[2 * j + 1], p1[2 * j + 1], p2[2 * j + 1]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_f32(&sm.w_empty[s]);
                ok = it < 2 || mbar_wait(&sm.done[b], ((it >> 1) & 1) ^ 1, abort_flag);
                if (!ok && lane == 0) { *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (6 << 8) | b); }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t dst = tmem_parts + b * 96 + h * 16 + ((uint32_t)(quarter * 32) << 16);
                tmem_st_x16(dst, p0);
                tmem_st_x16(dst + 32, p1);
                tmem_st_x16(dst + 64, p2);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_f32(&sm.part_full[b]);
            }
        }
    } else if (warp >= kF32SumWarp) {
        // ---- sums: row n0 + 32 quarter + lane of W, tokens kHalf * half .. of the tile
        const int quarter = warp & 3, half = (warp - kF32SumWarp) >> 2;
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const int m0 = (tile % tiles_m) * BN + half * kHalf, n = (tile / tiles_m) * kF32Rows + quarter * 32 + lane;
            float sum[kHalf];
#pragma unroll
            for (int j = 0; j < kHalf; ++j) sum[j] = 0.f;
#pragma unroll 1
            for (int k = 0; k < k_iters; ++k, ++it) {
                const int b = it & 1;
                ok = mbar_wait(&sm.done[b], (it >> 1) & 1, abort_flag);
                if (!ok && lane == 0) { *abort_flag = 1; atomicCAS(&g_gemm_f32_status, 0, (5 << 8) | b); }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < kHalf; c += 16) {
                    float v[16];
                    tmem_ld_x16(tmem + b * BN + half * kHalf + c + ((uint32_t)(quarter * 32) << 16), v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c + j] += v[j];
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_f32(&sm.acc_empty[b]);
            }
            if (!ok) break;
            if (n_spans == 1) {
#pragma unroll
                for (int j = 0; j < kHalf; ++j) if (m0 + j < p.M) finish_sum<EPI>(sum[j], m0 + j, n, p);
            } else {
                // (every stage of tokens has been read: the last accumulator is complete)
                float* partial = reinterpret_cast<float*>(sm.tok);
#pragma unroll
                for (int j = 0; j < kHalf; ++j) partial[(half * kHalf + j) * kPitch + quarter * 32 + lane] = sum[j];
            }
        }
    }
    __syncthreads();
    if (n_spans > 1) {
        cluster_sync_all();   // every span's sums are in its CTA's shared memory
        // token span, span + n_spans, ... of the tile: four warps a token, lanes along the columns of C
        const int tile = blockIdx.x, m0 = (tile % tiles_m) * BN, col = (warp & 3) * 32 + lane, n = (tile / tiles_m) * kF32Rows + col;
        if (!*abort_flag) {
            for (int j = span + (warp >> 2) * n_spans; j < BN && m0 + j < p.M; j += (kF32Threads / 128) * n_spans) {
                const float* mine = reinterpret_cast<const float*>(sm.tok) + j * kPitch + col;
                float part[kF32MaxSpans];
#pragma unroll
                for (int sp = 0; sp < kF32MaxSpans; ++sp) part[sp] = sp < n_spans ? cluster_load_f32(cluster_peer_address(mine, sp)) : 0.f;
                float s = 0.f;
#pragma unroll
                for (int sp = 0; sp < kF32MaxSpans; ++sp) s += part[sp];
                finish_sum<EPI>(s, m0 + j, n, p);
            }
        }
        cluster_sync_all();   // no CTA leaves while a peer may still read its shared memory
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// float32 [rows, K] with row stride ld; boxes of box_rows x 32 elements, 128-byte swizzle
static bool make_map_f32(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {32, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int WS, int EPI>
static int launch_f32(const __nv_bfloat16* planes, int padded, F32Args p, int n_spans_asked, cudaStream_t stream) {
    CUtensorMap mt, mw;
    if (!make_map(&mt, planes, 3 * p.M, padded, padded, BN) || !make_map_f32(&mw, p.W, p.N, p.K, p.ldw, kF32Rows)) return kErrUnsupportedSize;
    const size_t smem = sizeof(F32Smem<BN, WS>) + 1024;
    auto kernel = gemm_f32_tcgen05_kernel<BN, WS, EPI>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return (int)cudaGetLastError();
        configured = true;
    }
    static int known[kF32MaxSpans + 1] = {0};   // clusters of so many CTAs that can run at once, plus one; 0: not asked yet
    auto resident = [&](int s) {
        if (known[s] == 0) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(device_sm_count(), s);
            cfg.blockDim = dim3(kF32Threads);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = s; attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
            known[s] = n + 1;
        }
        return known[s] - 1;
    };
    const int kb = (p.K + BK - 1) / BK;
    const long long tiles = (long long)((p.M + BN - 1) / BN) * ((p.N + kF32Rows - 1) / kF32Rows);
    // as many spans as can all run at once, as long as each keeps four stages of K
    int spans = 1;
    for (int s = kF32MaxSpans; s > 1 && spans == 1; --s)
        if (tiles * s <= device_sm_count() && kb / s >= 4 && tiles <= resident(s)) spans = s;
    if (n_spans_asked > 0) spans = n_spans_asked <= kF32MaxSpans && n_spans_asked <= kb ? n_spans_asked : 1;
    p.blocks_per_span = (kb + spans - 1) / spans;
    spans = (kb + p.blocks_per_span - 1) / p.blocks_per_span;   // (no span is left empty)
    const unsigned grid_x = spans > 1 ? (unsigned)tiles : (unsigned)(tiles < device_sm_count() ? tiles : device_sm_count());
    return launch_pdl_cluster(kernel, dim3(grid_x, spans), dim3(kF32Threads), smem, stream, dim3(1, spans, 1), true, mt, mw, p);
}

}  // namespace b200

// Whether (and with how many bfloat16 elements of scratch) the product goes to the tensor cores: 0, no.
// Left to the plain kernels: few rows (they stream the weights as fast), rows that TMA cannot address, and products so
// small that the second launch costs more than it saves.
extern "C" long long b200_gemm_f32_scratch(int M, int N, int K, int lda, int ldw) {
    if (M <= 16 || K < 64 || K % 4 != 0 || ldw % 4 != 0 || lda < K || N < 64 || (long long)N * K < 65536) return 0;
    if (3ll * M > 0x7fffffffll) return 0;
    return 3ll * M * ((K + 7) / 8 * 8);
}

// Reads and clears the status word (0 = every wait completed).  Synchronises.
extern "C" int b200_gemm_f32_tcgen05_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, b200::g_gemm_f32_status, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(b200::g_gemm_f32_status, &zero, sizeof(int));
    return v;
}

// A, W, C float32.  scratch: b200_gemm_f32_scratch bfloat16 elements, 16-byte aligned.  epilogue 0 store (the first
// silu_cols columns as silu(sum)), 1 residual add, 2 gated SiLU, 3 gated GELU (tanh form), 4 gated and clamped; bias
// float32 [N] or null.  n_spans: cuts of K, 0 lets the shape decide.
extern "C" int b200_gemm_f32_tcgen05(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K,
                                     int epilogue, float gate_limit, float gate_slope, const float* bias, int silu_cols,
                                     void* scratch, int n_spans, cudaStream_t stream) {
    using namespace b200;
    if (M <= 0 || N <= 0) return 0;
    if (epilogue < 0 || epilogue > 4 || (epilogue >= 2 && (N & 1)) || scratch == nullptr) return kErrBadArgument;
    if (b200_gemm_f32_scratch(M, N, K, lda, ldw) == 0 || ((uintptr_t)W & 15) || ((uintptr_t)scratch & 15)) return kErrUnsupportedSize;
    const int padded = (K + 7) / 8 * 8;
    const long long pieces = (long long)M * (padded / 8);
    int st = launch_pdl(split_rows_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, stream, (const float*)A, lda,
                        (__nv_bfloat16*)scratch, M, K, padded);
    if (st != 0) return st;
    F32Args p = {};
    p.A = (const float*)A; p.W = (const float*)W; p.C = (float*)C; p.bias = bias;
    p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.epilogue = epilogue; p.silu_cols = silu_cols; p.gate_limit = gate_limit; p.gate_slope = gate_slope;
    const auto planes = (const __nv_bfloat16*)scratch;
    // Tiles of 64 tokens also for 65 to 127 over a short K, where the epilogue is most of the time: 2,048 columns, K = 64: 9.2 us (13.7 in
    // tiles of 128, plain kernel 8.0 with twice the error); 512 columns, K = 128: 10.3 (14.9, 12.8).
    if (M <= 64 || (M < 128 && K <= 192))
        return epilogue == 0 ? launch_f32<64, 4, 0>(planes, padded, p, n_spans, stream)
             : epilogue == 1 ? launch_f32<64, 4, 1>(planes, padded, p, n_spans, stream)
                             : launch_f32<64, 4, 2>(planes, padded, p, n_spans, stream);
    return epilogue == 0 ? launch_f32<128, 3, 0>(planes, padded, p, n_spans, stream)
         : epilogue == 1 ? launch_f32<128, 3, 1>(planes, padded, p, n_spans, stream)
                         : launch_f32<128, 3, 2>(planes, padded, p, n_spans, stream);
}
