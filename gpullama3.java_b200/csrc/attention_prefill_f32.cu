// Causal grouped-query attention of prompt tokens over the paged cache in float32, a tile of queries at a time.
//
// The same sums as the plain kernel (attention_generic.cu: one CTA per token and query head, which reads every key for every
// query), for queries that share keys: a CTA owns BQ rows, a row being a (token, query head) of one kv
// head, so that a page of keys and values fetched once serves all of them.  Scores, softmax and sums stay 32-bit
// multiply-adds (inference/InferenceCore.java:106-145 of the reference project).
//
// 128 threads as 8 groups of 16 lanes; a group owns RT rows.  Both products are dot products along what is contiguous in
// the cache (a key's dimensions; a dimension's 64 tokens), four elements at a time by packed pairs of multiply-adds:
//   scores  thread: its RT rows x keys tx, tx + 16, tx + 32, tx + 48
//   output  thread: its RT rows x dimensions tx, tx + 16, ...
// The probabilities go through shared memory between the two, within their group of lanes.  Rows of shared memory are
// padded by four floats, so that 16 lanes that read 16 rows meet no bank twice.  Keys and values have one buffer each, refilled
// (cp.async) as soon as they are read: the next page's keys arrive during the softmax and the output, its values during
// the next scores.  Two or three CTAs share an SM and fill each other's waits.
// Bound by the multiply-add units and their operands from shared memory: 2,048 tokens, 32 heads of 64: 0.57 ms = 30 TFLOP/s of
// needed work (the plain kernel: 4.32 ms; 0.73 with the tiles of one head after those of another, an SM's share of the work then 0.74 to
// 1.36 of the mean); eight prompts of 256: 115 us (763).
// Sums are kept short, a score's over 16 dimensions, then two such sums, then 32 dimensions after 32, an output's over 32 keys, then a page
// (half as long with heads of 32), and what a page's addition into a row's output rounds off joins the next.  The error is then below the
// plain kernel's, which adds trees of 32 (200 tokens behind 1,600, heads of 64: 1.61e-7 of the norm against 1.89e-7).  Sums over 32 dimensions
// and 64 keys with nothing kept are 8 % faster and leave 2.1e-7, one chain over all keys 7e-7.
//
// Few queries: one, two or four rows a group, and the pages of a tile cut into spans, merged by a second kernel (the plan that picks both is
// with the caller).  8 sequences of 500 keys decoded, 32 heads of 64: 12 us (25 with the plain kernel in spans of a tile); 2 tokens
// behind 2,000 keys: 10 us, 16 tokens: 21 (plain 37 and 110; a single tile of 64 rows without spans: 251 and 252).
//
// Terms as in the plain kernel (window, chunk, slopes, sinks, gate, softcap; not keep_first).  Values of keys past a
// sequence's end are read as zeros.  A key that some row of the tile must not see has probability 0 there, and 0 times a value that is
// not finite is not 0: a page with such keys and such values is summed key by key, over the keys each row sees.
#include "common.cuh"

namespace b200 {

constexpr int kPfThreads = 128;
constexpr int kPfPitch = kPageTokens + 4;

struct PrefillF32Args {
    const float* q;
    float* out;             // [T][n_heads D]
    const int* cu_seqlens;  // [n_seqs + 1]
    const int* kv_lens;     // [n_seqs]
    const int* page_table;
    const float* k_pool;    // [page][kv_head][64][D]
    const float* v_pool;    // [page][kv_head][D][64]
    const float* slopes;
    const float* sinks;
    const float* gate;
    int q_row_stride, table_stride, n_heads, n_kv_heads, window, chunk, ld_gate;
    float softcap;
    float* part_o;          // with spans: [row][span][D] sums, row = token * n_heads + head
    float* part_ml;         // with spans: [row][span][2] maximum and sum of exponentials
};

__device__ __forceinline__ void fma_pair(float2& acc, float ax, float ay, float bx, float by) {
    unsigned long long a, b, &c = reinterpret_cast<unsigned long long&>(acc);
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(ax), "f"(ay));
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(bx), "f"(by));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
// 16 bytes into shared memory, the bytes from `valid` on as zeros
__device__ __forceinline__ void copy16_async(float* dst, const float* src, int valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid) : "memory");
}

template <int D, int RT>
struct PrefillF32Smem {
    float q[8 * RT][D + 4];
    float k[kPageTokens][D + 4];
    float v[D][kPfPitch];
    float p[8 * RT][kPfPitch];
};

// gridDim.z > 1: a tile's pages are shared out among so many CTAs, which leave unnormalised results.
template <int D, int RT>
__global__ void __launch_bounds__(kPfThreads, RT <= 2 ? 4 : D <= 64 ? 3 : 2)
attention_prefill_f32_kernel(const PrefillF32Args a) {
    constexpr int BQ = 8 * RT, DJ = D / 16;
    constexpr int DIMS = D <= 32 ? 8 : 16, KEYS = D <= 32 ? 16 : 32;   // dimensions and keys whose products are added up by themselves
    extern __shared__ __align__(16) float smem_f[];
    auto& sm = *reinterpret_cast<PrefillF32Smem<D, RT>*>(smem_f);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    // tiles in order of falling length over all kv heads: the long ones start together and the short ones fill the end
    const int g = blockIdx.x % a.n_kv_heads, seq = blockIdx.y, group = a.n_heads / a.n_kv_heads;
    pdl_launch_dependents();
    pdl_wait();
    const int begin = a.cu_seqlens[seq], q_len = a.cu_seqlens[seq + 1] - begin, kv_len = a.kv_lens[seq];
    const int n_rows = q_len * group;
    const int row0 = ((int)gridDim.x / a.n_kv_heads - 1 - (int)blockIdx.x / a.n_kv_heads) * BQ;
    if (row0 >= n_rows) return;
    const int pos0 = kv_len - q_len;                             // position of the sequence's first token of the pass
    const int* pages = a.page_table + (size_t)seq * a.table_stride;
    const size_t page_stride = (size_t)a.n_kv_heads * kPageTokens * D, head_off = (size_t)g * kPageTokens * D;
    auto first_of = [&](int pos) { return a.chunk > 0 ? pos - pos % a.chunk : a.window > 0 ? max(0, pos - a.window + 1) : 0; };
    const int pos_lo = pos0 + row0 / group, pos_hi = pos0 + min(row0 + BQ - 1, n_rows - 1) / group;
    const int first_lo = first_of(pos_lo), first_hi = first_of(pos_hi);
    int page = first_lo / kPageTokens, page_end = pos_hi / kPageTokens + 1;
    const int span = blockIdx.z, n_spans = gridDim.z;
    if (n_spans > 1) {
        const int each = (page_end - page + n_spans - 1) / n_spans;
        page += span * each;
        page_end = min(page_end, page + each);     // (a span may be empty)
    }

    auto fetch_keys = [&](int page) {
        const float* src = a.k_pool + (size_t)pages[page] * page_stride + head_off;
        for (int c = tid; c < kPageTokens * D / 4; c += kPfThreads)
            copy16_async(&sm.k[c / (D / 4)][c % (D / 4) * 4], src + (size_t)c * 4, 16);
    };
    auto fetch_values = [&](int page) {
        const float* src = a.v_pool + (size_t)pages[page] * page_stride + head_off;
        for (int c = tid; c < kPageTokens * D / 4; c += kPfThreads) {
            const int key = c % 16 * 4;
            copy16_async(&sm.v[c / 16][key], src + (size_t)c * 4, 4 * min(4, max(0, kv_len - page * kPageTokens - key)));
        }
    };
    if (page < page_end) fetch_keys(page);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (page < page_end) fetch_values(page);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int c = tid; c < BQ * D / 4; c += kPfThreads) {
        const int r = min(row0 + c / (D / 4), n_rows - 1), d = c % (D / 4) * 4;
        *reinterpret_cast<float4*>(&sm.q[c / (D / 4)][d]) = *reinterpret_cast<const float4*>(
            a.q + (size_t)(begin + r / group) * a.q_row_stride + (size_t)(g * group + r % group) * D + d);
    }
    float m_run[RT], l_run[RT];      // l_run: this lane's share of the row's sum
    float o[RT][DJ], rest[RT][DJ];   // rest: what the additions into o have rounded off
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = min(row0 + ty * RT + i, n_rows - 1);
        m_run[i] = a.sinks && span == 0 ? a.sinks[g * group + r % group] : -INFINITY;
        l_run[i] = a.sinks && span == 0 && tx == 0 ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < DJ; ++j) o[i][j] = rest[i][j] = 0.f;
    }
    const float sqrt_d = sqrtf((float)D);

    for (; page < page_end; ++page) {
        const int base = page * kPageTokens;
        const bool masked = base + kPageTokens - 1 > pos_lo || base < first_hi;    // some row must not see some key
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        // ---- scores: sums over even and odd dimensions of DIMS side by side, then of 32 dimensions, then of 32 after 32
        float sc[RT][4];
#pragma unroll
        for (int d0 = 0; d0 < D; d0 += 32) {
            float sum[RT][4];
#pragma unroll
            for (int part = 0; part < 32 / DIMS; ++part) {
                float2 s2[RT][4];
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s2[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
                for (int d = d0 + DIMS * part; d < d0 + DIMS * (part + 1); d += 4) {
                    float4 kv[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(&sm.k[tx + 16 * j][d]);
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        const float4 qv = *reinterpret_cast<const float4*>(&sm.q[ty * RT + i][d]);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            fma_pair(s2[i][j], qv.x, qv.y, kv[j].x, kv[j].y);
                            fma_pair(s2[i][j], qv.z, qv.w, kv[j].z, kv[j].w);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float both = s2[i][j].x + s2[i][j].y;
                        sum[i][j] = part == 0 ? both : sum[i][j] + both;
                    }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sc[i][j] = d0 == 0 ? sum[i][j] : sc[i][j] + sum[i][j];
        }
        __syncthreads();
        if (page + 1 < page_end) fetch_keys(page + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        // ---- softmax
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int r = min(row0 + ty * RT + i, n_rows - 1), pos = pos0 + r / group;
            const float slope = a.slopes ? a.slopes[g * group + r % group] : 0.f;
            const int first = masked ? first_of(pos) : 0;
            float s[4], m_new = m_run[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = base + tx + 16 * j;
                s[j] = D == 64 ? sc[i][j] * 0.125f : sc[i][j] / sqrt_d;
                if (a.softcap > 0.f) s[j] = soft_capped(s[j], a.softcap);
                if (a.slopes) s[j] -= slope * (float)(pos - key);
                if (masked && (key > pos || key < first)) s[j] = -INFINITY;
                m_new = fmaxf(m_new, s[j]);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, off));
            const float m_use = m_new == -INFINITY ? 0.f : m_new;    // (no key seen yet: every probability is 0)
            const float corr = expf(m_run[i] - m_use);
            m_run[i] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[j] = expf(s[j] - m_use);
                sum += s[j];
                sm.p[ty * RT + i][tx + 16 * j] = s[j];
            }
            l_run[i] = l_run[i] * corr + sum;
#pragma unroll
            for (int j = 0; j < DJ; ++j) { o[i][j] *= corr; rest[i][j] *= corr; }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        // ---- output
        int odd_values = 0;
        if (min(base + kPageTokens, kv_len) - 1 > pos_lo || base < first_hi) {   // keys of the sequence that some row must not see
            bool bad = false;
            for (int c = tid; c < D * kPageTokens; c += kPfThreads) bad |= !isfinite(sm.v[c / kPageTokens][c % kPageTokens]);
            odd_values = __syncthreads_or(bad);
        }
        if (odd_values) {
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int pos = pos0 + min(row0 + ty * RT + i, n_rows - 1) / group;
                const int from = max(0, first_of(pos) - base), to = min(kPageTokens - 1, pos - base);
                for (int key = from; key <= to; ++key) {
                    const float p = sm.p[ty * RT + i][key];
#pragma unroll
                    for (int j = 0; j < DJ; ++j) o[i][j] = fmaf(p, sm.v[tx + 16 * j][key], o[i][j]);
                }
            }
        } else {   // a page's sums by themselves, KEYS keys at a time, then into the row's with what that rounds off kept (Kahan, 1965)
            float sum[RT][DJ];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < DJ; ++j) sum[i][j] = 0.f;
#pragma unroll 1
            for (int key0 = 0; key0 < kPageTokens; key0 += KEYS) {
                float2 o2[RT][DJ];
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < DJ; ++j) o2[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
                for (int key = key0; key < key0 + KEYS; key += 4) {
                    float4 vv[DJ];
#pragma unroll
                    for (int j = 0; j < DJ; ++j) vv[j] = *reinterpret_cast<const float4*>(&sm.v[tx + 16 * j][key]);
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        const float4 pv = *reinterpret_cast<const float4*>(&sm.p[ty * RT + i][key]);
#pragma unroll
                        for (int j = 0; j < DJ; ++j) {
                            fma_pair(o2[i][j], pv.x, pv.y, vv[j].x, vv[j].y);
                            fma_pair(o2[i][j], pv.z, pv.w, vv[j].z, vv[j].w);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < DJ; ++j) sum[i][j] += o2[i][j].x + o2[i][j].y;
            }
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < DJ; ++j) {
                    const float add = sum[i][j] + rest[i][j], total = o[i][j] + add, lost = add - (total - o[i][j]);
                    o[i][j] = total;
                    rest[i][j] = lost == lost ? lost : 0.f;   // (nothing is kept of an infinite sum)
                }
        }
        __syncthreads();
        if (page + 1 < page_end) fetch_values(page + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        float l = l_run[i];
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
        const int r = row0 + ty * RT + i;
        if (r >= n_rows) continue;
        const int t = begin + r / group, h = g * group + r % group;
        if (n_spans > 1) {
            const size_t part = ((size_t)t * a.n_heads + h) * n_spans + span;
#pragma unroll
            for (int j = 0; j < DJ; ++j) a.part_o[part * D + tx + 16 * j] = o[i][j];
            if (tx == 0) { a.part_ml[part * 2] = m_run[i]; a.part_ml[part * 2 + 1] = l; }
            continue;
        }
        const float gate = a.gate ? 1.0f / (1.0f + expf(-a.gate[(size_t)t * a.ld_gate + h])) : 1.f;
        float* dst = a.out + ((size_t)t * a.n_heads + h) * D;
#pragma unroll
        for (int j = 0; j < DJ; ++j) dst[tx + 16 * j] = o[i][j] / l * gate;
    }
}

// out[row] = sum_s o_s exp(m_s - m) / sum_s l_s exp(m_s - m) over the spans of a (token, head) row, in span order; a thread per
// dimension, everything asked for at once
constexpr int kMostSpans = 16;

__global__ void __launch_bounds__(128)
attention_spans_merge_f32_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, float* __restrict__ out,
                                 int n_spans, int head_dim, int n_heads, const float* __restrict__ gate, int ld_gate) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = blockIdx.x;
    const int d = threadIdx.x;
    if (d >= head_dim) return;
    const float* ml = part_ml + row * n_spans * 2;
    float ms[kMostSpans], ls[kMostSpans], po[kMostSpans];
#pragma unroll
    for (int s = 0; s < kMostSpans; ++s) {
        const bool in = s < n_spans;
        ms[s] = in ? ml[2 * s] : -INFINITY;
        ls[s] = in ? ml[2 * s + 1] : 0.f;
        po[s] = in ? part_o[(row * n_spans + s) * head_dim + d] : 0.f;
    }
    const float gv = gate ? 1.0f / (1.0f + expf(-gate[(row / n_heads) * ld_gate + row % n_heads])) : 1.f;
    float m = -INFINITY;
#pragma unroll
    for (int s = 0; s < kMostSpans; ++s) m = fmaxf(m, ms[s]);
    float l = 0.f, acc = 0.f;
#pragma unroll
    for (int s = 0; s < kMostSpans; ++s) {
        if (s >= n_spans) break;
        const float f = ms[s] == -INFINITY ? 0.f : expf(ms[s] - m);
        l += ls[s] * f;
        acc += po[s] * f;
    }
    out[row * head_dim + d] = acc / l * gv;
}

template <int D, int RT>
static int launch_prefill_f32(PrefillF32Args a, int n_seqs, int max_q_len, int n_tokens, int n_spans, float* scratch, cudaStream_t stream) {
    constexpr int BQ = 8 * RT;
    const size_t smem = sizeof(PrefillF32Smem<D, RT>);
    auto kernel = attention_prefill_f32_kernel<D, RT>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return (int)cudaGetLastError();
        configured = true;
    }
    a.part_o = scratch;
    a.part_ml = n_spans > 1 ? scratch + (size_t)n_tokens * a.n_heads * n_spans * D : nullptr;
    const long long rows = (long long)max_q_len * (a.n_heads / a.n_kv_heads);
    const int st = launch_pdl(kernel, dim3((unsigned)((rows + BQ - 1) / BQ) * a.n_kv_heads, n_seqs, n_spans), dim3(kPfThreads), smem, stream, a);
    if (st != 0 || n_spans == 1) return st;
    return launch_pdl(attention_spans_merge_f32_kernel, dim3((unsigned)(n_tokens * a.n_heads)), dim3(D <= 64 ? 64 : 128), 0, stream, a.part_o, a.part_ml,
                      a.out, n_spans, D, a.n_heads, a.gate, a.ld_gate);
}

template <int D>
static int prefill_f32_of(const PrefillF32Args& a, int n_seqs, int max_q_len, int n_tokens, int tile, int n_spans, float* scratch, cudaStream_t stream) {
    switch (tile) {
        case 8: return launch_prefill_f32<D, 1>(a, n_seqs, max_q_len, n_tokens, n_spans, scratch, stream);
        case 16: return launch_prefill_f32<D, 2>(a, n_seqs, max_q_len, n_tokens, n_spans, scratch, stream);
        case 32: return launch_prefill_f32<D, 4>(a, n_seqs, max_q_len, n_tokens, n_spans, scratch, stream);
    }
    return kErrBadArgument;
}

}  // namespace b200

// Queries: the first n_heads head_dim elements of rows of q_row_stride elements, packed sequence after sequence
// (cu_seqlens); kv_lens counts each sequence's keys with this pass's.  head_dim 32, 64, 96 or 128; other sizes, rows off the 16-byte
// grid and more than 65,535 sequences are left to the plain kernel (kErrUnsupportedSize).  tile: rows of a tile, 8, 16 or 32.
// n_spans > 1: every tile's keys are cut into so many spans (at most 16; scratch: n_tokens n_heads n_spans (head_dim + 2) floats).
extern "C" int b200_attention_prefill_f32(const void* q, int q_row_stride, void* out, const int* cu_seqlens, const int* kv_lens,
                                          const int* page_table, int table_stride, const void* k_pool, const void* v_pool,
                                          int n_seqs, int max_q_len, int n_tokens, int n_heads, int n_kv_heads, int head_dim, int window,
                                          int chunk, const float* slopes, const float* sinks, const void* gate, int ld_gate,
                                          float softcap, int tile, int n_spans, float* scratch, cudaStream_t stream) {
    using namespace b200;
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if (!(softcap >= 0.f) || chunk < 0 || (chunk > 0 && window > 0)) return kErrBadArgument;
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return kErrBadArgument;
    if (q_row_stride % 4 != 0 || (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15)) return kErrUnsupportedSize;
    if (n_seqs > 65535 || (long long)max_q_len * n_heads > 0x7fffff00ll) return kErrUnsupportedSize;
    PrefillF32Args a = {};
    a.q = (const float*)q; a.out = (float*)out; a.cu_seqlens = cu_seqlens; a.kv_lens = kv_lens; a.page_table = page_table;
    a.k_pool = (const float*)k_pool; a.v_pool = (const float*)v_pool; a.slopes = slopes; a.sinks = sinks; a.gate = (const float*)gate;
    a.q_row_stride = q_row_stride; a.table_stride = table_stride; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads;
    a.window = window; a.chunk = chunk; a.ld_gate = ld_gate; a.softcap = softcap;
    if (n_spans < 1 || n_spans > kMostSpans || (n_spans > 1 && scratch == nullptr)) return kErrBadArgument;
    switch (head_dim) {
        case 32: return prefill_f32_of<32>(a, n_seqs, max_q_len, n_tokens, tile, n_spans, scratch, stream);
        case 64: return prefill_f32_of<64>(a, n_seqs, max_q_len, n_tokens, tile, n_spans, scratch, stream);
        case 96: return prefill_f32_of<96>(a, n_seqs, max_q_len, n_tokens, tile, n_spans, scratch, stream);
        case 128: return prefill_f32_of<128>(a, n_seqs, max_q_len, n_tokens, tile, n_spans, scratch, stream);
        default: return kErrUnsupportedSize;
    }
}
