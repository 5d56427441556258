// Plain matrix product C = A W^T with 32-bit FMA accumulation, any storage types, any sizes.
//
// A is [M, K] (activations, row-major, row stride lda), W is [N, K] (a weight as the reference
// stores it: one row per output, core/model/tensor/FloatTensor.java:98-100 of the reference
// project).  Three kernels: tiles of 128 x 128 for prompts, of 64 x 64 for fewer than 128 rows, and a weight-streaming one for a decode step's few rows
// (further down).  These are the kernels of the true 32-bit path for few rows and for small products
// (gemm_f32_tcgen05.cu has the rest) and the fallback of the bfloat16 path for sizes or storage types the tensor-core
// kernels refuse.  Epilogues:
//   0  store         C[M, N] = acc                       (C of type TC)
//   1  residual add  C[M, N] += acc                      (C is the 32-bit residual stream)
//   2  gated SiLU    C[M, N/2] = silu(acc[2j]) * acc[2j+1]   (W holds gate and up rows interleaved;
//                    silu(g) = g / (1 + exp(-g)), inference/InferenceCore.java:163-166)
//   3  gated GELU    the same with gelu(g) = 0.5 g (1 + tanh(sqrt(2/pi) (g + 0.044715 g^3))), the tanh form
//   4  gated, clamped  with g = min(acc[2j], limit), u = clamp(acc[2j+1], -limit, limit):
//                    C[M, N/2] = g sigmoid(slope g) (u + 1); limit and slope are arguments
// A bias (float32 [N]) joins every sum before the epilogue.  The store epilogue may pass its first `silu_cols` columns through
// SiLU (projections that are used activated).
#include "common.cuh"

namespace b200 {

// the gated epilogues: activation of the gate value times the up value
__device__ __forceinline__ float gated_pair(float gate, float up, int epilogue, float limit, float slope) {
    if (epilogue == 4) {
        const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
        return g / (1.0f + expf(-slope * g)) * (u + 1.0f);
    }
    if (epilogue == 3) return 0.5f * gate * (1.0f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) * up;
    return (gate / (1.0f + expf(-gate))) * up;
}

// Several products of one shape side by side (gridDim.z of them): product z reads A + z a, W + z w and writes C + z c
// (elements).  One head's small product after another, for mixers that carry every head through a matrix of its own.
struct ProductExtras {
    long long a, w, c;
    float gate_limit, gate_slope;   // epilogue 4 alone reads these
    const float* bias;              // [N] or null
    int silu_cols;                  // epilogue 0: columns below this one are stored as silu(sum)
};
__device__ __forceinline__ float stored(const ProductExtras& x, int n, float sum) { return n < x.silu_cols ? sum / (1.0f + expf(-sum)) : sum; }
__device__ __forceinline__ float bias_of(const ProductExtras& x, int n) { return x.bias ? x.bias[n] : 0.f; }

constexpr int kTileM = 64, kTileN = 64, kTileK = 16, kGemmThreads = 256;

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(kGemmThreads)
gemm_generic_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, TC* __restrict__ C, int ldc,
                    int M, int N, int K, int epilogue, ProductExtras batch) {
    A += (size_t)blockIdx.z * batch.a;
    W += (size_t)blockIdx.z * batch.w;
    C += (size_t)blockIdx.z * batch.c;
    __shared__ float As[kTileK][kTileM + 4];
    __shared__ float Ws[kTileK][kTileN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
    const int tx = tid % 16, ty = tid / 16;  // thread owns rows ty*4..+3, columns tx*4..+3
    float acc[4][4] = {};

    for (int k0 = 0; k0 < K; k0 += kTileK) {
        // 64 x 16 elements of each operand, 4 per thread; consecutive threads read along K
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * kGemmThreads;
            const int r = e / kTileK, c = e % kTileK;
            const int k = k0 + c;
            As[c][r] = (m0 + r < M && k < K) ? to_f32<TA>(A[(size_t)(m0 + r) * lda + k]) : 0.f;
            Ws[c][r] = (n0 + r < N && k < K) ? to_f32<TW>(W[(size_t)(n0 + r) * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTileK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[i] = As[k][ty * 4 + i]; w[i] = Ws[k][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
        if (epilogue >= 2) {
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int n = n0 + tx * 4 + j;
                if (n + 1 < N) {
                    const float gate = acc[i][j] + bias_of(batch, n), up = acc[i][j + 1] + bias_of(batch, n + 1);
                    C[(size_t)m * ldc + n / 2] = from_f32<TC>(gated_pair(gate, up, epilogue, batch.gate_limit, batch.gate_slope));
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n = n0 + tx * 4 + j;
                if (n >= N) continue;
                TC* c = C + (size_t)m * ldc + n;
                const float sum = acc[i][j] + bias_of(batch, n);
                if (epilogue == 1) *c = from_f32<TC>(to_f32<TC>(*c) + sum);
                else *c = from_f32<TC>(stored(batch, n, sum));
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The same product for prompts (M >= 128): tiles of 128 x 128, a thread owns 8 x 8 sums, so that a k-step costs four
// 16-byte shared-memory loads per 64 multiply-adds instead of eight 4-byte loads per 16; the next tile's operands are
// fetched into registers while the current one is multiplied.  Still plain 32-bit FMA in a fixed order of k.
constexpr int kBigM = 128, kBigN = 128, kBigK = 16, kBigThreads = 256;

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(kBigThreads)
gemm_generic_big_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, TC* __restrict__ C, int ldc,
                        int M, int N, int K, int epilogue, ProductExtras batch) {
    A += (size_t)blockIdx.z * batch.a;
    W += (size_t)blockIdx.z * batch.w;
    C += (size_t)blockIdx.z * batch.c;
    __shared__ __align__(16) float As[kBigK][kBigM + 4];
    __shared__ __align__(16) float Ws[kBigK][kBigN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * kBigM, n0 = blockIdx.x * kBigN;
    const int tx = tid % 16, ty = tid / 16;   // rows ty * 8 .. + 7, columns tx * 8 .. + 7
    float acc[8][8] = {};
    float ra[8], rw[8];                        // this thread's share of the next tile: 8 elements of each operand
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tid + i * kBigThreads, r = e / kBigK, k = k0 + e % kBigK;   // 16 lanes read along k
            ra[i] = (m0 + r < M && k < K) ? to_f32<TA>(A[(size_t)(m0 + r) * lda + k]) : 0.f;
            rw[i] = (n0 + r < N && k < K) ? to_f32<TW>(W[(size_t)(n0 + r) * ldw + k]) : 0.f;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += kBigK) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tid + i * kBigThreads, r = e / kBigK, c = e % kBigK;
            As[c][r] = ra[i];
            Ws[c][r] = rw[i];
        }
        __syncthreads();
        if (k0 + kBigK < K) fetch(k0 + kBigK);
#pragma unroll
        for (int k = 0; k < kBigK; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As[k][ty * 8]), a1 = *reinterpret_cast<const float4*>(&As[k][ty * 8 + 4]);
            const float4 w0 = *reinterpret_cast<const float4*>(&Ws[k][tx * 8]), w1 = *reinterpret_cast<const float4*>(&Ws[k][tx * 8 + 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        if (m >= M) continue;
        if (epilogue >= 2) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const int n = n0 + tx * 8 + j;
                if (n + 1 < N) {
                    const float gate = acc[i][j] + bias_of(batch, n), up = acc[i][j + 1] + bias_of(batch, n + 1);
                    C[(size_t)m * ldc + n / 2] = from_f32<TC>(gated_pair(gate, up, epilogue, batch.gate_limit, batch.gate_slope));
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + tx * 8 + j;
                if (n >= N) continue;
                TC* c = C + (size_t)m * ldc + n;
                const float sum = acc[i][j] + bias_of(batch, n);
                if (epilogue == 1) *c = from_f32<TC>(to_f32<TC>(*c) + sum);
                else *c = from_f32<TC>(stored(batch, n, sum));
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The same product for a decode step's few rows (M <= 16): tiles of 64 tokens would leave the FMA units idle and
// read every weight through shared memory for nothing.  Here the weight rows are streamed 16 bytes per lane, every
// element meeting all M tokens' activations, which a lane holds in registers (gemm_fewrows_kernel) or fetches from L1
// (gemm_fourrows_kernel).
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}

// a weight is read once: not kept in L1, which holds the activations
template <typename T> __device__ __forceinline__ float4 load4_once(const T* p);
template <> __device__ __forceinline__ float4 load4_once<float>(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
template <> __device__ __forceinline__ float4 load4_once<__nv_bfloat16>(const __nv_bfloat16* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}

constexpr int kFewWarps = 8, kFewThreads = kFewWarps * 32;
constexpr int kFewRows = 8;               // weight rows of a CTA, in two groups of four
constexpr int kFewSlice = kFewWarps * 128;   // elements of K that the CTA's warps take at a time, 128 each

// Sums over the lanes of a warp of NV numbers by halving: afterwards lane l has the sum number l / (32 / NV) (31 exchanges
// for 32 numbers, where a butterfly per number would need 160).
template <int NV>
__device__ __forceinline__ float reduce_by_halving(float (&v)[NV], int lane) {
#pragma unroll
    for (int half = NV / 2, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
        const bool upper = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = upper ? v[i] : v[i + half];
            const float keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    }
#pragma unroll
    for (int bit = 16 / NV; bit >= 1; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
    return v[0];
}

// four products, the first two and the last two side by side in packed pairs of multiply-adds
__device__ __forceinline__ float dot4_pairs(const float4& w, const float4& x) {
    unsigned long long w01, w23, x01, x23;
    float even, odd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(w01) : "f"(w.x), "f"(w.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(w23) : "f"(w.z), "f"(w.w));
    asm("mov.b64 %0, {%1, %2};" : "=l"(x01) : "f"(x.x), "f"(x.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(x23) : "f"(x.z), "f"(x.w));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(w01) : "l"(x01));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(w01) : "l"(w23), "l"(x23));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(w01));
    return even + odd;
}

// A CTA owns eight consecutive weight rows (four gate/up pairs of the gated epilogue); its eight warps take 128 elements of
// every 1024 of K each.  A lane holds its four elements of all MT tokens in registers and carries the eight weight rows past
// them, four rows at a time: 4 x MT sums of four products per lane, summed over the lanes by halving, over the slices of K
// in a register and over the warps in shared memory in warp order.  Nine to sixteen tokens go in four parts (NH) past the same
// weights.  Still plain 32-bit FMA.
// Bound by the stream of the weights for up to four tokens (134 MB: 28 us, 4.7 TB/s; 43.5 us when every lane fetched the
// activations again for every four rows), from eight on by the instructions of the products and the exchanges (134 MB at 8
// tokens: 36 us against 46; at 16 tokens: 53 against 78; parts of 8 tokens there spill and take 65).  A slice of the eight rows (32 KB
// of float32 a CTA) is asked for before the dependency wait, and a group's next slice as soon as its registers are free.  (Sums kept over
// all slices, so that the lanes exchange once a CTA, need the activations again for the second group: 48 us at 8 tokens.)
template <typename TA, typename TW, typename TC, int MT, int NH>
__global__ void __launch_bounds__(kFewThreads, 2)
gemm_fewrows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, TC* __restrict__ C, int ldc,
                    int M, int N, int K, int epilogue, ProductExtras batch) {
    constexpr int NV = 4 * MT;
    A += (size_t)blockIdx.z * batch.a;
    W += (size_t)blockIdx.z * batch.w;
    C += (size_t)blockIdx.z * batch.c;
    __shared__ float part[kFewWarps][NH * kFewRows * MT];   // of a warp: [half][row][token]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * kFewRows;
    float4 wv[2][4];
    auto load_group = [&](int g, int k) {   // rows beyond N are clamped: read, never stored
#pragma unroll
        for (int r = 0; r < 4; ++r)
            wv[g][r] = k < K ? load4_once<TW>(W + (size_t)min(n0 + 4 * g + r, N - 1) * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const int first = (warp * 32 + lane) * 4;
    load_group(0, first);
    load_group(1, first);
    pdl_launch_dependents();
    pdl_wait();
    float total[NH][2];
#pragma unroll
    for (int h = 0; h < NH; ++h) total[h][0] = total[h][1] = 0.f;
    for (int k = first; k - first < K; k += kFewSlice) {   // (all lanes alike: the exchanges need the whole warp)
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            float4 x[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m)
                x[m] = k < K && h * MT + m < M ? load4<TA>(A + (size_t)(h * MT + m) * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                float v[NV];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        v[r * MT + m] = NH == 1 ? dot4_pairs(wv[g][r], x[m])
                                                : fmaf(wv[g][r].w, x[m].w, fmaf(wv[g][r].z, x[m].z, fmaf(wv[g][r].y, x[m].y, wv[g][r].x * x[m].x)));
                if (h == NH - 1) load_group(g, k + kFewSlice);
                total[h][g] += reduce_by_halving<NV>(v, lane);
            }
        }
    }
    if (lane % (32 / NV) == 0) {
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int g = 0; g < 2; ++g) part[warp][(h * 2 + g) * NV + lane / (32 / NV)] = total[h][g];
    }
    __syncthreads();
    // thread i: half, row and token of sum number i; the warps' sums are added in warp order
    const int i = threadIdx.x;
    if (i >= NH * kFewRows * MT) return;
    const int r = i / MT % kFewRows, m = i / (MT * kFewRows) * MT + i % MT, n = n0 + r;
    float sum = 0.f;
#pragma unroll
    for (int wp = 0; wp < kFewWarps; ++wp) sum += part[wp][i];
    if (batch.bias && n < N) sum += batch.bias[n];
    if (epilogue >= 2) {
        float up = 0.f;   // the gate row's thread also adds up the up row (the next row of the CTA)
        if ((r & 1) == 0) {
#pragma unroll
            for (int wp = 0; wp < kFewWarps; ++wp) up += part[wp][i + MT];
            if (batch.bias && n + 1 < N) up += batch.bias[n + 1];
            if (m < M && n + 1 < N) C[(size_t)m * ldc + n / 2] = from_f32<TC>(gated_pair(sum, up, epilogue, batch.gate_limit, batch.gate_slope));
        }
    } else if (m < M && n < N) {
        TC* c = C + (size_t)m * ldc + n;
        if (epilogue == 1) *c = from_f32<TC>(to_f32<TC>(*c) + sum);
        else *c = from_f32<TC>(stored(batch, n, sum));
    }
}

// The same for at most eight tokens with half as many rows a CTA and the activations fetched from L1 for every four weight rows: sums are
// kept over all of K and exchanged once, and tokens that are not there cost nothing.  Faster where the kernel above has fewer CTAs than
// the GPU has SMs and K is long (an SM's share is then one CTA's chain of slices: 8 tokens, 128 x 2,048 in float32: 3.2 us against 4.2), and
// for bfloat16 weights, whose multiply-adds and exchanges take longer than their stream (5 tokens, 16,384 x 2,048: 33 us against 44);
// fourrows_wins draws the line.  Four rows of sums for up to eight tokens are the 32 numbers that a warp sums by halving.
constexpr int kFourRows = 4, kFourTokens = 8;

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(kFewThreads)
gemm_fourrows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, TC* __restrict__ C, int ldc,
                     int M, int N, int K, int epilogue, ProductExtras batch) {
    constexpr int MT = kFourTokens;
    pdl_launch_dependents();
    pdl_wait();
    A += (size_t)blockIdx.z * batch.a;
    W += (size_t)blockIdx.z * batch.w;
    C += (size_t)blockIdx.z * batch.c;
    __shared__ float part[kFewWarps][kFourRows * MT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * kFourRows;
    const TW* w[kFourRows];
#pragma unroll
    for (int r = 0; r < kFourRows; ++r) w[r] = W + (size_t)min(n0 + r, N - 1) * ldw;   // clamped: read, never stored
    float acc[kFourRows * MT];
#pragma unroll
    for (int i = 0; i < kFourRows * MT; ++i) acc[i] = 0.f;
#pragma unroll 2
    for (int k = (warp * 32 + lane) * 4; k < K; k += kFewSlice) {
        float4 wv[kFourRows];
#pragma unroll
        for (int r = 0; r < kFourRows; ++r) wv[r] = load4<TW>(w[r] + k);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < M) {
                const float4 x = load4<TA>(A + (size_t)m * lda + k);
#pragma unroll
                for (int r = 0; r < kFourRows; ++r) {
                    // (32-bit weights: four products by themselves, then one addition, as the kernel above; 16-bit ones, whose products are
                    // exact, are bound by the instructions)
                    if constexpr (sizeof(TW) == 4) acc[r * MT + m] += dot4_pairs(wv[r], x);
                    else acc[r * MT + m] = fmaf(wv[r].w, x.w, fmaf(wv[r].z, x.z, fmaf(wv[r].y, x.y, fmaf(wv[r].x, x.x, acc[r * MT + m]))));
                }
            }
        }
    }
    part[warp][lane] = reduce_by_halving<kFourRows * MT>(acc, lane);   // lane l: sum number l
    __syncthreads();
    // thread i < 32: row i / MT, token i % MT; the warps' sums are added in warp order
    const int i = threadIdx.x;
    if (i >= kFourRows * MT) return;
    const int r = i / MT, m = i % MT, n = n0 + r;
    float sum = 0.f;
#pragma unroll
    for (int wp = 0; wp < kFewWarps; ++wp) sum += part[wp][i];
    if (batch.bias && n < N) sum += batch.bias[n];
    if (epilogue >= 2) {
        float up = 0.f;   // the gate row's thread also adds up the up row (the next row of the CTA)
        if ((r & 1) == 0) {
#pragma unroll
            for (int wp = 0; wp < kFewWarps; ++wp) up += part[wp][i + MT];
            if (batch.bias && n + 1 < N) up += batch.bias[n + 1];
            if (m < M && n + 1 < N) C[(size_t)m * ldc + n / 2] = from_f32<TC>(gated_pair(sum, up, epilogue, batch.gate_limit, batch.gate_slope));
        }
    } else if (m < M && n < N) {
        TC* c = C + (size_t)m * ldc + n;
        if (epilogue == 1) *c = from_f32<TC>(to_f32<TC>(*c) + sum);
        else *c = from_f32<TC>(stored(batch, n, sum));
    }
}

// Measured with weights from memory, M 1 to 16, N 32 to 28,672, K 64 to 14,336.  Up to one slice of K the kernel of eight rows is never
// slower.  float32 weights: four rows win below 384 weight rows (1.3 times at 128 x 2,048), from five tokens on as long as eight rows make
// fewer CTAs than there are SMs (1.14 times at 1,024 x 2,048; 0.75 at 2,048 x 2,048).  bfloat16 weights: four rows win (1.1 to 1.5 times)
// except for four tokens, which fill the other kernel's registers, where eight rows make one round of CTAs (0.7 at 2,048 x 2,048), and for
// three or eight tokens over a long K (0.8 at 4,096 x 14,336).
static bool fourrows_wins(int M, int N, int K, bool bf16_weights) {
    if (M > kFourTokens || K <= kFewSlice) return false;
    const int ctas = (N + kFewRows - 1) / kFewRows, sms = device_sm_count();
    if (!bf16_weights) return M <= 4 ? N < 384 : ctas <= sms;
    return M != 4 && !(ctas > sms && ctas <= 2 * sms) && !(K >= 8192 && (M == 3 || M >= 7));
}

template <typename TA, typename TW, typename TC>
static int launch_fewrows(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K, int epilogue,
                          int n_batch, ProductExtras batch, cudaStream_t stream) {
    if (fourrows_wins(M, N, K, sizeof(TW) == 2)) {
        // (an early start for grids that leave room on the SMs: about one round of CTAs would settle unevenly beside the predecessor's, 8 tokens,
        // 4,096 x 4,096: 26.0 us instead of 22.5)
        const dim3 grid((N + kFourRows - 1) / kFourRows, 1, n_batch);
        return launch_pdl_cluster(gemm_fourrows_kernel<TA, TW, TC>, grid, dim3(kFewThreads), 0, stream, dim3(1, 1, 1), (long long)grid.x * n_batch <= 2 * device_sm_count(),
                                  (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, epilogue, batch);
    }
    const dim3 grid((N + kFewRows - 1) / kFewRows, 1, n_batch);
    LaunchForm form;
    if (N >= kHeadRows) form.shared_percent = kStreamingSharedPercent;
    auto go = [&](auto kernel) {
        return launch_pdl_as(kernel, grid, dim3(kFewThreads), 0, stream, form, (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, epilogue, batch);
    };
    return M <= 4 ? go(gemm_fewrows_kernel<TA, TW, TC, 4, 1>) : M <= 8 ? go(gemm_fewrows_kernel<TA, TW, TC, 8, 1>) : go(gemm_fewrows_kernel<TA, TW, TC, 4, 4>);
}

}  // namespace b200

static int gemm_generic_launch(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw, void* C,
                               int c_dtype, int ldc, int M, int N, int K, int epilogue, int n_batch,
                               b200::ProductExtras batch, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || n_batch <= 0) return 0;
    if (n_batch > 65535) return b200::kErrUnsupportedSize;
    if (K <= 0 || epilogue < 0 || epilogue > 4) return b200::kErrBadArgument;
    if (epilogue == 1 && c_dtype != b200::kF32) return b200::kErrBadArgument;
    if (epilogue >= 2 && (N & 1)) return b200::kErrBadArgument;
    // a decode step's few rows: rows of 4 elements at a time, when the rows start on such a boundary
    const size_t a_el = a_dtype == b200::kF32 ? 4 : 2, w_el = w_dtype == b200::kF32 ? 4 : 2;
    if (M <= 16 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch.a % 4 == 0 && batch.w % 4 == 0 && ((uintptr_t)A % (4 * a_el)) == 0 && ((uintptr_t)W % (4 * w_el)) == 0) {
        B200_DISPATCH_DTYPE(a_dtype, TA, B200_DISPATCH_DTYPE2(w_dtype, TW, B200_DISPATCH_DTYPE3(c_dtype, TC,
            return b200::launch_fewrows<TA, TW, TC>(A, lda, W, ldw, C, ldc, M, N, K, epilogue, n_batch, batch, stream))));
    }
    if (M >= b200::kBigM && (M + b200::kBigM - 1) / b200::kBigM <= 65535) {
        dim3 big((N + b200::kBigN - 1) / b200::kBigN, (M + b200::kBigM - 1) / b200::kBigM, n_batch);
        B200_DISPATCH_DTYPE(a_dtype, TA, B200_DISPATCH_DTYPE2(w_dtype, TW, B200_DISPATCH_DTYPE3(c_dtype, TC,
            b200::gemm_generic_big_kernel<TA, TW, TC><<<big, b200::kBigThreads, 0, stream>>>(
                (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, epilogue, batch))));
        return b200::launch_status();
    }
    dim3 grid((N + b200::kTileN - 1) / b200::kTileN, (M + b200::kTileM - 1) / b200::kTileM, n_batch);
    if (grid.y > 65535) return b200::kErrUnsupportedSize;
    B200_DISPATCH_DTYPE(a_dtype, TA, B200_DISPATCH_DTYPE2(w_dtype, TW, B200_DISPATCH_DTYPE3(c_dtype, TC,
        b200::gemm_generic_kernel<TA, TW, TC><<<grid, b200::kGemmThreads, 0, stream>>>(
            (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, epilogue, batch))));
    return b200::launch_status();
}

extern "C" int b200_gemm_generic(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw, void* C,
                                 int c_dtype, int ldc, int M, int N, int K, int epilogue, float gate_limit,
                                 float gate_slope, const float* bias, int silu_cols, cudaStream_t stream) {
    return gemm_generic_launch(A, a_dtype, lda, W, w_dtype, ldw, C, c_dtype, ldc, M, N, K, epilogue, 1,
                               b200::ProductExtras{0, 0, 0, gate_limit, gate_slope, bias, silu_cols}, stream);
}

// n_batch products of the same shape: product z uses A + z a_step, W + z w_step, C + z c_step (steps in elements).
extern "C" int b200_gemm_generic_batched(const void* A, int a_dtype, int lda, long long a_step, const void* W, int w_dtype,
                                         int ldw, long long w_step, void* C, int c_dtype, int ldc, long long c_step, int M,
                                         int N, int K, int n_batch, cudaStream_t stream) {
    return gemm_generic_launch(A, a_dtype, lda, W, w_dtype, ldw, C, c_dtype, ldc, M, N, K, 0, n_batch,
                               b200::ProductExtras{a_step, w_step, c_step, 0.f, 0.f, nullptr, 0}, stream);
}
