// Several residual streams side by side (hyper-connections).
//
// The residual stream of a token is S rows of `width` 32-bit numbers, [T, S, width].  A sublayer reads one
// weighted sum of the streams, and its result y goes back into every stream while the streams are mixed
// among themselves:
//     u      = sum_a  read[a] x_a                            (streams_read_norm: u is normalised at once)
//     x_j  <-  sum_a  mix[a, j] x_a  +  write[j] y           (streams_combine, in place, all j from the old x)
// streams_combine is also what opens the streams (S_in = 1, mix = ones: every stream starts as the embedding)
// and what closes them (S_out = 1, mix = ones: the model's output is their sum).  All sums are 32-bit.
#include "tcgen05.cuh"

namespace b200 {

constexpr int kMaxStreams = 8;
constexpr int kStreamThreads = 256;

// out[t, j, c] = sum_a mix[a * s_out + j] * x[t, a, c]  (+ write[j] * y[t, c]).  `out` may be `x` itself when
// s_in == s_out: a thread reads the s_in numbers of its (t, c) before it writes the s_out.
template <int VEC>
__global__ void __launch_bounds__(kStreamThreads)
streams_combine_kernel(const float* __restrict__ x, float* out, const float* __restrict__ mix,
                       const float* __restrict__ write, const float* __restrict__ y, int s_in, int s_out, int width,
                       size_t n_units) {   // units of VEC numbers: T * width / VEC
    __shared__ float m_s[kMaxStreams * kMaxStreams], w_s[kMaxStreams];
    for (int i = threadIdx.x; i < s_in * s_out; i += kStreamThreads) m_s[i] = mix[i];
    for (int i = threadIdx.x; i < s_out; i += kStreamThreads) w_s[i] = (write != nullptr) ? write[i] : 0.f;
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    const int wv = width / VEC;
    for (size_t u = (size_t)blockIdx.x * kStreamThreads + threadIdx.x; u < n_units; u += (size_t)gridDim.x * kStreamThreads) {
        const size_t t = u / wv;
        const int c = (int)(u % wv) * VEC;
        float in[kMaxStreams][VEC];
#pragma unroll
        for (int a = 0; a < kMaxStreams; ++a) {
            if (a >= s_in) break;
            const float* p = x + (t * s_in + a) * width + c;
            if (VEC == 4) {
                const float4 v = *reinterpret_cast<const float4*>(p);
                in[a][0] = v.x; in[a][1] = v.y; in[a][2] = v.z; in[a][3] = v.w;
            } else {
                in[a][0] = p[0];
            }
        }
        float yv[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) yv[e] = 0.f;
        if (y != nullptr) {
            const float* p = y + t * width + c;
            if (VEC == 4) {
                const float4 v = *reinterpret_cast<const float4*>(p);
                yv[0] = v.x; yv[1] = v.y; yv[2] = v.z; yv[3] = v.w;
            } else {
                yv[0] = p[0];
            }
        }
#pragma unroll
        for (int j = 0; j < kMaxStreams; ++j) {
            if (j >= s_out) break;
            float acc[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
#pragma unroll
            for (int a = 0; a < kMaxStreams; ++a) {
                if (a >= s_in) break;
                const float m = m_s[a * s_out + j];
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += m * in[a][e];
            }
            if (y != nullptr) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += w_s[j] * yv[e];
            }
            float* o = out + (t * s_out + j) * width + c;
            if (VEC == 4) *reinterpret_cast<float4*>(o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            else o[0] = acc[0];
        }
    }
}

// out[r] = w * u / sqrt(mean(u^2) + eps) with u = sum_a read[a] x[row(r), a, :]: the read of a sublayer and its
// norm in one pass.  `rows` (optional) selects tokens, as in rmsnorm.  A CTA per row; u stays in registers for
// widths up to kStreamKeep * 256 and is formed again from x beyond that.
constexpr int kStreamKeep = 8;

template <typename TO>
__global__ void __launch_bounds__(kStreamThreads)
streams_read_norm_kernel(const float* __restrict__ x, const float* __restrict__ read, const float* __restrict__ w,
                         TO* __restrict__ out, const int* __restrict__ rows, int n_streams, int width, float eps) {
    __shared__ float scratch[33];
    __shared__ float r_s[kMaxStreams];
    if (threadIdx.x < n_streams) r_s[threadIdx.x] = read[threadIdx.x];
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    const int r = blockIdx.x;
    const float* xr = x + (size_t)(rows ? rows[r] : r) * n_streams * width;
    float keep[kStreamKeep];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < kStreamKeep; ++k) {
        const int c = k * kStreamThreads + threadIdx.x;
        float u = 0.f;
        if (c < width)
            for (int a = 0; a < n_streams; ++a) u += r_s[a] * xr[(size_t)a * width + c];
        keep[k] = u;
        ss += u * u;
    }
    for (int c = kStreamKeep * kStreamThreads + threadIdx.x; c < width; c += kStreamThreads) {
        float u = 0.f;
        for (int a = 0; a < n_streams; ++a) u += r_s[a] * xr[(size_t)a * width + c];
        ss += u * u;
    }
    ss = block_sum(ss, scratch);
    const float scale = 1.0f / sqrtf(ss / (float)width + eps);
    TO* o = out + (size_t)r * width;
#pragma unroll
    for (int k = 0; k < kStreamKeep; ++k) {
        const int c = k * kStreamThreads + threadIdx.x;
        if (c < width) o[c] = from_f32<TO>(w[c] * (scale * keep[k]));
    }
    for (int c = kStreamKeep * kStreamThreads + threadIdx.x; c < width; c += kStreamThreads) {
        float u = 0.f;
        for (int a = 0; a < n_streams; ++a) u += r_s[a] * xr[(size_t)a * width + c];
        o[c] = from_f32<TO>(w[c] * (scale * u));
    }
}

// The write-back of one sublayer and the read of the next in one pass over a token's streams (a CTA per token):
//     x_j <- sum_a mix[a, j] x_a + write[j] y      (in place)
//     y   <- 0                                     (the next sublayer's last product adds into it again)
//     out  = w * u / sqrt(mean(u^2) + eps),  u = sum_j read[j] x_j     (only when `read` is given)
// so the new streams are not read again for the norm, and nothing else has to clear y.
template <int VEC> struct StreamVec;
template <> struct StreamVec<4> {
    __device__ static void load(const float* p, float (&f)[4]) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    }
    __device__ static void store(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
    __device__ static void store(__nv_bfloat16* p, const float (&f)[4]) {
        __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    }
};
template <> struct StreamVec<1> {
    __device__ static void load(const float* p, float (&f)[1]) { f[0] = p[0]; }
    __device__ static void store(float* p, const float (&f)[1]) { p[0] = f[0]; }
    __device__ static void store(__nv_bfloat16* p, const float (&f)[1]) { p[0] = __float2bfloat16_rn(f[0]); }
};

// A CTA of up to kStepThreads threads per token, VEC columns per access (4 when the width and the pointers allow).  A thread
// asks for everything it reads of up to kStepKeep accesses before it writes anything (x is read and written through one pointer,
// so the compiler cannot), keeps their u in registers (widths up to kStepKeep * VEC * kStepThreads) and forms u again from
// the new streams beyond that.  S: the number of streams, or 0 for a number given at run time.
// Bound by its bytes (2,048 tokens, three streams of 2,048: 142 MB in 29.5 us, launches back to back; 1.4 times as long with 256 threads
// whose loads waited for the stores before them).
constexpr int kStepKeep = 2, kStepThreads = 512;

template <typename TO, int VEC, int S>
__global__ void __launch_bounds__(kStepThreads)
streams_step_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ write,
                    float* __restrict__ y, const float* __restrict__ read, const float* __restrict__ w,
                    TO* __restrict__ out, int streams, int width, float eps) {
    constexpr int MAXS = S > 0 ? S : kMaxStreams;
    const int n_streams = S > 0 ? S : streams, threads = blockDim.x;
    __shared__ float scratch[33];
    __shared__ float m_s[kMaxStreams * kMaxStreams], w_s[kMaxStreams], r_s[kMaxStreams];
    for (int i = threadIdx.x; i < n_streams * n_streams; i += threads) m_s[i] = mix[i];   // (weights: before the wait)
    if (threadIdx.x < n_streams) {
        w_s[threadIdx.x] = write[threadIdx.x];
        r_s[threadIdx.x] = read != nullptr ? read[threadIdx.x] : 0.f;
    }
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    const size_t t = blockIdx.x;
    float* xr = x + t * n_streams * width;
    float* yr = y + t * width;
    const int units = width / VEC;
    float ss = 0.f;
    auto fetch = [&](int c, float (&in)[MAXS][VEC], float (&yv)[VEC]) {
#pragma unroll
        for (int a = 0; a < MAXS; ++a)
            if (a < n_streams) StreamVec<VEC>::load(xr + (size_t)a * width + c, in[a]);
        StreamVec<VEC>::load(yr + c, yv);
    };
    auto mixed = [&](int c, const float (&in)[MAXS][VEC], const float (&yv)[VEC], float (&u)[VEC]) {
        float zero[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) zero[e] = u[e] = 0.f;
        StreamVec<VEC>::store(yr + c, zero);
#pragma unroll
        for (int j = 0; j < MAXS; ++j) {
            if (j >= n_streams) break;
            float acc[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
#pragma unroll
            for (int a = 0; a < MAXS; ++a) {
                if (a >= n_streams) break;
                const float m = m_s[a * n_streams + j];
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += m * in[a][e];
            }
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                acc[e] += w_s[j] * yv[e];
                u[e] += r_s[j] * acc[e];
            }
            StreamVec<VEC>::store(xr + (size_t)j * width + c, acc);
        }
    };
    float in[kStepKeep][MAXS][VEC], yv[kStepKeep][VEC], wv[kStepKeep][VEC], keep[kStepKeep][VEC];
#pragma unroll
    for (int k = 0; k < kStepKeep; ++k) {
        const int unit = k * threads + threadIdx.x;
        if (unit < units) {
            fetch(unit * VEC, in[k], yv[k]);
            if (read != nullptr) StreamVec<VEC>::load(w + unit * VEC, wv[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < kStepKeep; ++k) {
        const int unit = k * threads + threadIdx.x;
#pragma unroll
        for (int e = 0; e < VEC; ++e) keep[k][e] = 0.f;
        if (unit < units) mixed(unit * VEC, in[k], yv[k], keep[k]);
#pragma unroll
        for (int e = 0; e < VEC; ++e) ss += keep[k][e] * keep[k][e];
    }
    for (int unit = kStepKeep * threads + threadIdx.x; unit < units; unit += threads) {
        float u[VEC];
        fetch(unit * VEC, in[0], yv[0]);
        mixed(unit * VEC, in[0], yv[0], u);
#pragma unroll
        for (int e = 0; e < VEC; ++e) ss += u[e] * u[e];
    }
    if (read == nullptr) return;
    ss = block_sum(ss, scratch);
    const float scale = 1.0f / sqrtf(ss / (float)width + eps);
    TO* o = out + t * width;
#pragma unroll
    for (int k = 0; k < kStepKeep; ++k) {
        const int unit = k * threads + threadIdx.x;
        if (unit < units) {
            float res[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) res[e] = wv[k][e] * (scale * keep[k][e]);
            StreamVec<VEC>::store(o + unit * VEC, res);
        }
    }
    for (int unit = kStepKeep * threads + threadIdx.x; unit < units; unit += threads) {
        float wb[VEC], res[VEC];   // beyond the kept columns u is formed again from the new streams (this thread wrote them)
        StreamVec<VEC>::load(w + unit * VEC, wb);
#pragma unroll
        for (int e = 0; e < VEC; ++e) res[e] = 0.f;
        for (int j = 0; j < n_streams; ++j) {
            float xv[VEC];
            StreamVec<VEC>::load(xr + (size_t)j * width + unit * VEC, xv);
#pragma unroll
            for (int e = 0; e < VEC; ++e) res[e] += r_s[j] * xv[e];
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) res[e] = wb[e] * (scale * res[e]);
        StreamVec<VEC>::store(o + unit * VEC, res);
    }
}

// The same for prompts: persistent CTAs, two an SM, whose tokens arrive through a ring of shared-memory stages (bulk copies, up to
// kRingStages tokens ahead), so that an SM's loads never wait for the stores before them.  A thread keeps its u in registers
// (widths up to kStepKeep * 4 * kStepThreads); one barrier a token, behind which its stage is filled again.  2,048 tokens, three streams of
// 2,048 (142 MB, a part of them in L2), launches back to back: 29.5 us as above, 18.2 so.  For prompts of four tokens a CTA and more;
// fewer leave nothing to run ahead.  A copy that does not arrive within mbar_wait's two seconds is recorded in g_streams_status, with the
// step's streams half updated.
constexpr int kRingStages = 4, kRingBytes = 112 * 1024;

__device__ int g_streams_status = 0;

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <typename TO, int S>
__global__ void __launch_bounds__(kStepThreads)
streams_step_ring_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ write,
                         float* __restrict__ y, const float* __restrict__ read, const float* __restrict__ w,
                         TO* __restrict__ out, int n_tokens, int streams, int width, float eps, int stages) {
    constexpr int MAXS = S > 0 ? S : kMaxStreams;
    const int n_streams = S > 0 ? S : streams, threads = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    extern __shared__ __align__(128) float ring[];         // [stages][n_streams + 1][width]: a token's streams, then its y
    __shared__ uint64_t full[kRingStages];
    __shared__ float scratch[2][kStepThreads / 32];
    __shared__ float m_s[kMaxStreams * kMaxStreams], w_s[kMaxStreams], r_s[kMaxStreams];
    __shared__ int gave_up;
    const size_t stage = (size_t)(n_streams + 1) * width;
    for (int i = threadIdx.x; i < n_streams * n_streams; i += threads) m_s[i] = mix[i];   // (weights: before the wait)
    if (threadIdx.x < n_streams) {
        w_s[threadIdx.x] = write[threadIdx.x];
        r_s[threadIdx.x] = read != nullptr ? read[threadIdx.x] : 0.f;
    }
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    const uint32_t x_bytes = (uint32_t)(n_streams * width) * 4, y_bytes = (uint32_t)width * 4;
    auto fetch = [&](int i) {   // (one thread) this CTA's i-th token into its stage
        const size_t t = blockIdx.x + (size_t)i * gridDim.x;
        if (t >= (size_t)n_tokens) return;
        float* to = ring + (size_t)(i % stages) * stage;
        mbar_expect_tx(&full[i % stages], x_bytes + y_bytes);
        bulk_load(to, x + t * n_streams * width, x_bytes, &full[i % stages]);
        bulk_load(to + (size_t)n_streams * width, y + t * width, y_bytes, &full[i % stages]);
    };
    if (threadIdx.x == 0)
        for (int i = 0; i < stages; ++i) fetch(i);
    const int units = width / 4;
    float wv[kStepKeep][4];
#pragma unroll
    for (int k = 0; k < kStepKeep; ++k)
        if (read != nullptr && k * threads + (int)threadIdx.x < units) StreamVec<4>::load(w + (k * threads + threadIdx.x) * 4, wv[k]);
    for (int i = 0; blockIdx.x + (size_t)i * gridDim.x < (size_t)n_tokens; ++i) {
        const size_t t = blockIdx.x + (size_t)i * gridDim.x;
        const bool ok = mbar_wait(&full[i % stages], (i / stages) & 1, &gave_up);
        const float* in_s = ring + (size_t)(i % stages) * stage;
        float* xr = x + t * n_streams * width;
        float keep[kStepKeep][4], ss = 0.f;
#pragma unroll
        for (int k = 0; k < kStepKeep; ++k) {
#pragma unroll
            for (int e = 0; e < 4; ++e) keep[k][e] = 0.f;
            const int unit = k * threads + threadIdx.x, c = unit * 4;
            if (!ok || unit >= units) continue;
            float in[MAXS][4], yv[4];
            const float zero[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int a = 0; a < MAXS; ++a)
                if (a < n_streams) StreamVec<4>::load(in_s + (size_t)a * width + c, in[a]);
            StreamVec<4>::load(in_s + (size_t)n_streams * width + c, yv);
            StreamVec<4>::store(y + t * width + c, zero);
#pragma unroll
            for (int j = 0; j < MAXS; ++j) {
                if (j >= n_streams) break;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int a = 0; a < MAXS; ++a) {
                    if (a >= n_streams) break;
                    const float m = m_s[a * n_streams + j];
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[e] += m * in[a][e];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[e] += w_s[j] * yv[e];
                    keep[k][e] += r_s[j] * acc[e];
                }
                StreamVec<4>::store(xr + (size_t)j * width + c, acc);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) ss += keep[k][e] * keep[k][e];
        }
        ss = warp_sum(ss);
        if (lane == 0) scratch[i & 1][warp] = ss;
        if (__syncthreads_or(!ok)) {   // a copy did not arrive: say so, give the others another chance to land, and return
            if (threadIdx.x == 0) {
                atomicExch(&g_streams_status, 1);
                for (int k = i; k < i + stages && blockIdx.x + (size_t)k * gridDim.x < (size_t)n_tokens; ++k)
                    mbar_wait(&full[k % stages], (k / stages) & 1, &gave_up);
            }
            return;
        }
        if (threadIdx.x == 0) fetch(i + stages);     // (every thread has read the stage)
        if (read == nullptr) continue;
        ss = warp_sum(lane < (threads + 31) / 32 ? scratch[i & 1][lane] : 0.f);
        const float scale = 1.0f / sqrtf(ss / (float)width + eps);
#pragma unroll
        for (int k = 0; k < kStepKeep; ++k) {
            const int unit = k * threads + threadIdx.x;
            if (unit < units) {
                float res[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) res[e] = wv[k][e] * (scale * keep[k][e]);
                StreamVec<4>::store(out + t * width + unit * 4, res);
            }
        }
    }
}

template <typename TO, int VEC, int S>
static int launch_streams_step(float* x, const float* mix, const float* write, float* y, const float* read, const float* w, void* out,
                               int n_tokens, int n_streams, int width, float eps, cudaStream_t stream) {
    const int units = (width / VEC + 31) / 32 * 32, threads = units < kStepThreads ? units : kStepThreads;
    const size_t stage = (size_t)(n_streams + 1) * width * 4;
    const int stages = (int)(kRingBytes / stage) < kRingStages ? (int)(kRingBytes / stage) : kRingStages;
    if (VEC == 4 && n_tokens >= 4 * device_sm_count() && stages >= 2 && width <= 4 * kStepKeep * kStepThreads) {
        auto kernel = streams_step_ring_kernel<TO, S>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingBytes) != cudaSuccess) return (int)cudaGetLastError();
        return launch_pdl(kernel, dim3(2 * device_sm_count()), dim3(threads), stages * stage, stream, x, mix, write, y, read, w, (TO*)out,
                          n_tokens, n_streams, width, eps, stages);
    }
    return launch_pdl(streams_step_kernel<TO, VEC, S>, dim3(n_tokens), dim3(threads), 0, stream, x, mix, write, y, read, w, (TO*)out,
                      n_streams, width, eps);
}

}  // namespace b200

extern "C" int b200_streams_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, b200::g_streams_status, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(b200::g_streams_status, &zero, sizeof(int));
    return v;
}

extern "C" int b200_streams_step(float* x, const float* mix, const float* write, float* y, const float* read,
                                 const float* w, void* out, int out_dtype, int n_tokens, int n_streams, int width,
                                 float eps, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (n_streams < 1 || n_streams > b200::kMaxStreams || width < 1) return b200::kErrUnsupportedSize;
    if (read != nullptr && (w == nullptr || out == nullptr)) return b200::kErrBadArgument;
    const bool vec = width % 4 == 0 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (uintptr_t)out) & 15) == 0;
    B200_DISPATCH_DTYPE(out_dtype, TO,
        auto go = [&](auto launch) { return launch(x, mix, write, y, read, w, out, n_tokens, n_streams, width, eps, stream); };
        if (!vec) return go(b200::launch_streams_step<TO, 1, 0>);
        switch (n_streams) {
            case 1: return go(b200::launch_streams_step<TO, 4, 1>);
            case 2: return go(b200::launch_streams_step<TO, 4, 2>);
            case 3: return go(b200::launch_streams_step<TO, 4, 3>);
            case 4: return go(b200::launch_streams_step<TO, 4, 4>);
            default: return go(b200::launch_streams_step<TO, 4, 0>);
        });
}

extern "C" int b200_streams_combine(const float* x, float* out, const float* mix, const float* write, const float* y,
                                    int n_tokens, int s_in, int s_out, int width, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (s_in < 1 || s_out < 1 || s_in > b200::kMaxStreams || s_out > b200::kMaxStreams || width < 1) return b200::kErrUnsupportedSize;
    if (x == out && s_in != s_out) return b200::kErrBadArgument;
    const bool vec = width % 4 == 0 && (((uintptr_t)x | (uintptr_t)out | (uintptr_t)y) & 15) == 0;
    const size_t units = (size_t)n_tokens * width / (vec ? 4 : 1);
    const int grid = (int)((units + b200::kStreamThreads - 1) / b200::kStreamThreads < 148 * 16
                               ? (units + b200::kStreamThreads - 1) / b200::kStreamThreads : 148 * 16);
    return b200::launch_pdl(vec ? b200::streams_combine_kernel<4> : b200::streams_combine_kernel<1>, dim3(grid), dim3(b200::kStreamThreads), 0,
                            stream, x, out, mix, write, y, s_in, s_out, width, units);
}

extern "C" int b200_streams_read_norm(const float* x, const float* read, const float* w, void* out, int out_dtype,
                                      const int* rows, int n_rows, int n_streams, int width, float eps,
                                      cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (n_streams < 1 || n_streams > b200::kMaxStreams || width < 1) return b200::kErrUnsupportedSize;
    B200_DISPATCH_DTYPE(out_dtype, TO,
        return b200::launch_pdl(b200::streams_read_norm_kernel<TO>, dim3(n_rows), dim3(b200::kStreamThreads), 0, stream, x, read, w, (TO*)out,
                                rows, n_streams, width, eps));
}
