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
#include <type_traits>

#include "tcgen05.cuh"

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
    const int* only_if;     // a word that must not be 0 for the kernel to do anything (null: no such word)
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
    if (a.only_if != nullptr && *a.only_if == 0) return;
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

// ---------------------------------------------------------------------------------------------
// The same on the tensor cores, for prompts (head_dim 64, an even number of query heads to a kv head, causal and nothing more).  Heads of
// 128 are not taken: the parts of two tiles of queries alone would fill 192 of the 227 KB of shared memory, and one tile leaves nothing to run
// during its softmax.
//
// A float32 number is the sum of three bfloat16 numbers exactly: x0 = bf16(x), x1 = bf16(x - x0), x2 = x - x0 - x1.  A product of
// two such sums is formed as six of its nine products (those left out are below 2^-24 of it), smallest first, by tcgen05.mma with
// float32 accumulators.  The accumulators cut off what does not fit where an addition rounds, so sums stay short: a score's over 32
// dimensions, an output's over 32 keys, two of each added in registers, and a page's output then to its row's with what that rounds
// off kept (sums of 64: 172 us in place of 240, errors a fifth above the kernel's above).  Keys and values are split once a launch
// (split_pages_kernel, into scratch memory, values times 2^24 so that the parts of small ones keep their bits), queries by the softmax
// threads, probabilities in registers.
// Probabilities are in [0, 1] and keys within the mask only.  A query or key of 2^60 or more (a score of 64 such products would reach
// 2^126), a value of 2^72 or more, or one that is not finite raises a flag, and the kernel above then does the launch over.  2^72: a row's
// sums are kept unnormalised, up to one value times 2^24 for each of its keys, and the launch takes fewer than 2^29 keys a sequence:
// 2^72 2^24 2^29 = 2^125 is finite.
//
// A CTA owns two tiles of 128 rows, the same tokens of two neighbouring heads, so that a page's parts serve both; warps 0 to 3 and 4
// to 7 are their softmax threads (a row each), one warp fetches, one issues each tile's products.  A tile's next scores are formed
// behind its outputs' products, while the other's softmax runs.  CTAs take tiles from a list by falling number, forwards and backwards
// in turn.
// Bound by the chain from a page's scores over its softmax to its outputs, 7 us a page with two tiles taking turns.  2,048 tokens, 32 heads
// of 64: 577 us with multiply-adds, 240 so, at the same error (1.32e-7 and 1.33e-7 of the norm; peaked scores 3.16e-7 and 2.70e-7, 200
// tokens behind 1,600 1.67e-7 and 1.63e-7).
constexpr int kTcRows = 128, kTcD = 64, kTcStages = 2, kTcThreads = 384;
constexpr int kTcTmaWarp = 8, kTcMmaWarp0 = 9, kTcMmaWarp1 = 10, kTcFlagWarp = 11;
constexpr int kTcRegsIssuers = 40, kTcRegsSoftmax = 232;   // 128 x 40 + 256 x 232 = 64,512 = 384 x 168, the launch's registers
constexpr int kTcPart = kPageTokens * kTcD;                // elements of one part of a page's keys or values
constexpr float kTcValueScale = 16777216.f;                // 2^24
constexpr float kTcMostScoreFactor = 0x1p60f, kTcMostValue = 0x1p72f;   // (see above)

__device__ int g_f32_tc_status = 0;

struct TcF32Args {
    PrefillF32Args f;
    __nv_bfloat16* parts;   // [2: keys, values][slot][kv head][3][64][64]; slot = sequence * table_stride + page of the sequence
    int* flags;             // [0]: raised, [1 ..]: per (sequence, page, kv head) of the split
    int n_seqs, n_tiles, n_split;
};

struct TcF32Smem {
    alignas(1024) __nv_bfloat16 q[2][3][kTcRows * kTcD];
    alignas(1024) __nv_bfloat16 k[kTcStages][3][kTcPart];
    alignas(1024) __nv_bfloat16 v[kTcStages][3][kTcPart];
    alignas(8) uint64_t k_full[kTcStages];
    uint64_t k_empty[kTcStages], v_full[kTcStages], v_empty[kTcStages];
    uint64_t q_full[2], s_full[2], p_full[2], pv_done[2];
    uint32_t tmem_base;
    int abort_flag;
    float rest[2][32][kTcRows];   // what additions into the outputs' last 32 dimensions have rounded off
};

// a number as the sum of three bfloat16 numbers
__device__ __forceinline__ void split3(float x, float& a, float& b, float& c) {
    a = __bfloat162float(__float2bfloat16_rn(x));
    const float r = x - a;
    b = __bfloat162float(__float2bfloat16_rn(r));
    c = r - b;
}
__device__ __forceinline__ uint32_t two_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// eight numbers into three 16-byte pieces of their parts
__device__ __forceinline__ void split8(const float (&x)[8], uint4 (&piece)[3]) {
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a0, b0, c0, a1, b1, c1;
        split3(x[2 * i], a0, b0, c0);
        split3(x[2 * i + 1], a1, b1, c1);
        w[0][i] = two_bf16(a0, a1); w[1][i] = two_bf16(b0, b1); w[2][i] = two_bf16(c0, c1);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) piece[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// A CTA per (page of a sequence, kv head): keys [64][D] and values [D][64] into their parts; what lies beyond the sequence's end is 0.
__global__ void __launch_bounds__(128)
split_pages_kernel(const TcF32Args a) {
    const int page = blockIdx.x, g = blockIdx.y, seq = blockIdx.z, G = a.f.n_kv_heads, W = a.f.table_stride;
    const size_t slot = (size_t)seq * W + page;
    pdl_launch_dependents();
    pdl_wait();
    if (page == 0 && g == 0 && seq == 0 && threadIdx.x == 0) a.flags[0] = 0;
    const int valid = a.f.kv_lens[seq] - page * kPageTokens;
    bool bad = false;
    if (valid > 0) {
        const size_t src = ((size_t)a.f.page_table[slot] * G + g) * kTcPart;
        const size_t dst = (slot * G + g) * 3 * kTcPart, values = (size_t)a.n_seqs * W * G * 3 * kTcPart;
#pragma unroll
        for (int i = 0; i < kTcPart / 8 / 128; ++i) {
            const int c = (i * 128 + threadIdx.x) * 8, row = c / 64, col = c % 64;
            float k[8], v[8];
            uint4 piece[3];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                *reinterpret_cast<float4*>(k + 4 * h) = *reinterpret_cast<const float4*>(a.f.k_pool + src + c + 4 * h);
                *reinterpret_cast<float4*>(v + 4 * h) = *reinterpret_cast<const float4*>(a.f.v_pool + src + c + 4 * h);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                k[e] = row < valid ? k[e] : 0.f;
                v[e] = col + e < valid ? v[e] : 0.f;
                bad |= !(fabsf(k[e]) < kTcMostScoreFactor) || !(fabsf(v[e]) < kTcMostValue);
                v[e] *= kTcValueScale;
            }
            split8(k, piece);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(a.parts + dst + p * kTcPart + c) = piece[p];
            split8(v, piece);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(a.parts + values + dst + p * kTcPart + c) = piece[p];
        }
    }
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0) a.flags[1 + slot * G + g] = any;
}

__device__ __forceinline__ void tc_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, int accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// sums of two times sixteen neighbouring columns of this thread's row
__device__ __forceinline__ void tmem_sum16(uint32_t first, uint32_t second, float (&v)[16]) {
    uint32_t a[16], b[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]), "=&r"(a[8]), "=&r"(a[9]),
          "=&r"(a[10]), "=&r"(a[11]), "=&r"(a[12]), "=&r"(a[13]), "=&r"(a[14]), "=&r"(a[15]), "=&r"(b[0]), "=&r"(b[1]), "=&r"(b[2]), "=&r"(b[3]),
          "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]), "=&r"(b[8]), "=&r"(b[9]), "=&r"(b[10]), "=&r"(b[11]), "=&r"(b[12]), "=&r"(b[13]),
          "=&r"(b[14]), "=&r"(b[15])
        : "r"(first), "r"(second) : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(a[i]) + __uint_as_float(b[i]);
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

__global__ void __launch_bounds__(kTcThreads, 1)
attention_prefill_f32_tc_kernel(const __grid_constant__ CUtensorMap map_parts, const TcF32Args a) {
    // Tensor memory, 512 columns: tile t has its scores in 256 t .. + 127 (64 for each half of the dimensions), overwritten by the
    // three parts of its probabilities (bfloat16 pairs, 96) once its threads hold them, and a page's outputs in + 128 .. + 255 (64 for
    // each half of the keys).
    extern __shared__ __align__(1024) uint8_t tc_raw[];
    TcF32Smem& sm = *reinterpret_cast<TcF32Smem*>(((uintptr_t)tc_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the six products, as (part of the first operand, part of the second): smallest first
    constexpr int kFirst[6] = {0, 1, 2, 0, 1, 0}, kSecond[6] = {2, 1, 0, 1, 0, 0};

    if (threadIdx.x == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            mbar_init(&sm.k_full[s], 1); mbar_init(&sm.k_empty[s], 2); mbar_init(&sm.v_full[s], 1); mbar_init(&sm.v_empty[s], 2);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&sm.q_full[t], 4); mbar_init(&sm.s_full[t], 1); mbar_init(&sm.p_full[t], 4); mbar_init(&sm.pv_done[t], 1);
        }
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_parts) : "memory");
    }
    if (warp == kTcMmaWarp0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem_base;
    volatile int* abort_flag = &sm.abort_flag;
    pdl_launch_dependents();
    pdl_wait();

    const int G = a.f.n_kv_heads, group = a.f.n_heads / G, n_pairs = a.f.n_heads / 2;
    const int total = a.n_tiles * n_pairs * a.n_seqs;
    auto run_units = [&](auto role) {
        constexpr int ROLE = decltype(role)::value;   // 1: softmax warps, 0: the others
        int units_done = 0, base = 0;                 // phases of q_full; blocks of earlier units (phases of everything else)
        for (int round = 0;; ++round) {
            const int unit = round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
            if (round * (int)gridDim.x >= total || *abort_flag) break;
            if (unit >= total) continue;
            const int tile = a.n_tiles - 1 - unit / (n_pairs * a.n_seqs), in_tile = unit % (n_pairs * a.n_seqs);
            const int seq = in_tile / n_pairs, head0 = in_tile % n_pairs * 2;
            const int tok0 = a.f.cu_seqlens[seq], q_len = a.f.cu_seqlens[seq + 1] - tok0, q0 = tile * kTcRows;
            if (q0 >= q_len) continue;
            const int kv_len = a.f.kv_lens[seq], p_first = kv_len - q_len + q0, rows = min(kTcRows, q_len - q0);
            const int nb = (p_first + rows - 1) / kPageTokens + 1;

            if (ROLE == 0 && warp == kTcTmaWarp && lane == 0) {
                const int row_k = ((seq * a.f.table_stride) * G + head0 / group) * 3 * 64, row_page = G * 3 * 64;
                const int row_v = row_k + a.n_seqs * a.f.table_stride * G * 3 * 64;
                for (int j = 0; j < nb; ++j) {
                    const int n = base + j, s = n % kTcStages;
                    bool ok = n < kTcStages || mbar_wait(&sm.k_empty[s], ((n / kTcStages) - 1) & 1, abort_flag);
                    if (ok) {
                        mbar_expect_tx(&sm.k_full[s], 3 * kTcPart * 2);
                        for (int p = 0; p < 3; ++p) tma_load_2d(sm.k[s][p], &map_parts, 0, row_k + j * row_page + p * 64, &sm.k_full[s]);
                        ok = n < kTcStages || mbar_wait(&sm.v_empty[s], ((n / kTcStages) - 1) & 1, abort_flag);
                    }
                    if (!ok) { *abort_flag = 1; atomicCAS(&g_f32_tc_status, 0, (1 << 8) | s); break; }
                    mbar_expect_tx(&sm.v_full[s], 3 * kTcPart * 2);
                    for (int p = 0; p < 3; ++p) tma_load_2d(sm.v[s][p], &map_parts, 0, row_v + j * row_page + p * 64, &sm.v_full[s]);
                }
            } else if (ROLE == 0 && (warp == kTcMmaWarp0 || warp == kTcMmaWarp1) && lane == 0) {
                const int t = warp - kTcMmaWarp0;
                constexpr uint32_t idesc = umma_idesc_bf16(kTcRows, 64);
                bool ok = mbar_wait(&sm.q_full[t], units_done & 1, abort_flag);
                if (!ok) { *abort_flag = 1; atomicCAS(&g_f32_tc_status, 0, 2 << 8); }
                auto scores = [&](int j) {
                    const int n = base + j, s = n % kTcStages;
                    if (!mbar_wait(&sm.k_full[s], (n / kTcStages) & 1, abort_flag)) {
                        *abort_flag = 1; atomicCAS(&g_f32_tc_status, 0, (3 << 8) | s); ok = false;
                        return;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int half = 0; half < 2; ++half)
#pragma unroll
                        for (int i = 0; i < 6; ++i) {
                            const uint64_t qd = umma_desc(sm.q[t][kFirst[i]]) + 4 * half, kd = umma_desc(sm.k[s][kSecond[i]]) + 4 * half;
#pragma unroll
                            for (int kk = 0; kk < 2; ++kk) umma_bf16(tmem + 256 * t + 64 * half, qd + 2 * kk, kd + 2 * kk, idesc, (i | kk) != 0);
                        }
                    umma_commit(&sm.s_full[t]);
                    umma_commit(&sm.k_empty[s]);
                };
                if (ok) scores(0);
                for (int j = 0; j < nb && ok; ++j) {
                    const int n = base + j, s = n % kTcStages;
                    if (!mbar_wait(&sm.p_full[t], n & 1, abort_flag) || !mbar_wait(&sm.v_full[s], (n / kTcStages) & 1, abort_flag)) {
                        *abort_flag = 1; atomicCAS(&g_f32_tc_status, 0, (5 << 8) | t); ok = false; break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int half = 0; half < 2; ++half)
#pragma unroll
                        for (int i = 0; i < 6; ++i) {
                            const uint64_t vd = umma_desc(sm.v[s][kSecond[i]]) + 4 * half;
#pragma unroll
                            for (int kk = 0; kk < 2; ++kk)
                                tc_mma_a_tmem(tmem + 256 * t + 128 + 64 * half, tmem + 256 * t + 32 * kFirst[i] + 16 * half + 8 * kk, vd + 2 * kk,
                                              idesc, (i | kk) != 0);
                        }
                    umma_commit(&sm.pv_done[t]);
                    umma_commit(&sm.v_empty[s]);
                    if (j + 1 < nb) scores(j + 1);   // (behind the product that reads the probabilities in their place)
                }
            } else if (ROLE == 1) {
                const int t = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
                const uint32_t mine = tmem + 256 * t + ((uint32_t)(quarter * 32) << 16);
                const int pos = p_first + min(r, rows - 1);           // rows past the end repeat the last one and are not stored
                // ---- this row of Q, in parts, into the swizzled layout the products read (the unit before has formed its last scores)
                bool bad = false;
                const float* qrow = a.f.q + (size_t)(tok0 + q0 + min(r, rows - 1)) * a.f.q_row_stride + (size_t)(head0 + t) * kTcD;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float x[8];
                    uint4 piece[3];
                    *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(qrow + 8 * c);
                    *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(qrow + 8 * c + 4);
#pragma unroll
                    for (int e = 0; e < 8; ++e) bad |= !(fabsf(x[e]) < kTcMostScoreFactor);
                    split8(x, piece);
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(sm.q[t][p]) + r * 128 + ((c ^ (r & 7)) << 4)) = piece[p];
                }
                if (bad) atomicOr(a.flags, 1);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_arrive(&sm.q_full[t]);
                float m = -INFINITY, l = 0.f, l_rest = 0.f;     // l_rest: what the additions into l have rounded off
                // o: the row's outputs; what its additions round off: the first 32 dimensions' in registers, the others' in shared memory
                float o[kTcD], rest[32];
                float* kept = &sm.rest[t][0][r];
#pragma unroll
                for (int d = 0; d < kTcD; ++d) o[d] = 0.f;
#pragma unroll
                for (int d = 0; d < 32; ++d) rest[d] = kept[d * kTcRows] = 0.f;
                auto add_page = [&](float corr) {   // (o += page) corr
#pragma unroll
                    for (int c = 0; c < kTcD; c += 16) {
                        float v[16];
                        tmem_sum16(mine + 128 + c, mine + 192 + c, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float add = v[i] + (c < 32 ? rest[(c + i) & 31] : kept[((c + i) & 31) * kTcRows]), sum = o[c + i] + add;
                            const float lost = (add - (sum - o[c + i])) * corr;
                            if (c < 32) rest[(c + i) & 31] = lost;
                            else kept[((c + i) & 31) * kTcRows] = lost;
                            o[c + i] = sum * corr;
                        }
                    }
                };
                auto wait = [&](uint64_t* bar, int phase, int where) {
                    bool ok = mbar_wait(bar, phase, abort_flag);
                    if (!ok && lane == 0) { *abort_flag = 1; atomicCAS(&g_f32_tc_status, 0, (where << 8) | warp); }
                    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    return ok;
                };
                bool ok = true;
                for (int j = 0; j < nb; ++j) {
                    ok = wait(&sm.s_full[t], (base + j) & 1, 6);
                    if (!ok) break;
                    float s[2][32];
#pragma unroll
                    for (int c = 0; c < 64; c += 16) {
                        float v[16];
                        tmem_sum16(mine + c, mine + 64 + c, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) s[c >> 5][(c & 31) + i] = v[i];
                    }
                    const int key0 = j * kPageTokens;
                    if (key0 + kPageTokens - 1 > p_first) {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
#pragma unroll
                            for (int i = 0; i < 32; ++i) s[c][i] = key0 + 32 * c + i <= pos ? s[c][i] : -INFINITY;
                    }
                    float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) top[i & 3] = fmaxf(top[i & 3], s[c][i]);
                    // (the first page holds position 0, which every row sees: the maximum is finite from there on; 1 / sqrt(64) is exact)
                    const float m_new = fmaxf(m, 0.125f * fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])));
                    const float corr = expf(m - m_new);
                    m = m_new;
                    if (j > 0) {
                        ok = wait(&sm.pv_done[t], (base + j - 1) & 1, 7);
                        if (!ok) break;
                        add_page(corr);
                    }
                    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {       // 16 keys: eight columns of each part
                        uint32_t part[3][8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int at = 16 * (c & 1) + 2 * i;
                            const float p0 = expf(fmaf(0.125f, s[c >> 1][at], -m)), p1 = expf(fmaf(0.125f, s[c >> 1][at + 1], -m));
                            sum[i & 3] += p0 + p1;
                            float a0, b0, c0, a1, b1, c1;
                            split3(p0, a0, b0, c0);
                            split3(p1, a1, b1, c1);
                            part[0][i] = two_bf16(a0, a1); part[1][i] = two_bf16(b0, b1); part[2][i] = two_bf16(c0, c1);
                        }
#pragma unroll
                        for (int p = 0; p < 3; ++p) tmem_st8(mine + 32 * p + 8 * c, part[p]);
                    }
                    {
                        const float before = l * corr, add = ((sum[0] + sum[1]) + (sum[2] + sum[3])) + l_rest * corr;
                        l = before + add;
                        l_rest = add - (l - before);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc_arrive(&sm.p_full[t]);
                }
                if (ok) ok = wait(&sm.pv_done[t], (base + nb - 1) & 1, 8);
                if (ok) {
                    add_page(1.f);
                    if (r < rows) {
                        float* dst = a.f.out + ((size_t)(tok0 + q0 + r) * a.f.n_heads + head0 + t) * kTcD;
#pragma unroll
                        for (int d = 0; d < kTcD; d += 4) {
                            float4 v;
                            v.x = o[d] / l * (1.f / kTcValueScale); v.y = o[d + 1] / l * (1.f / kTcValueScale);
                            v.z = o[d + 2] / l * (1.f / kTcValueScale); v.w = o[d + 3] / l * (1.f / kTcValueScale);
                            *reinterpret_cast<float4*>(dst + d) = v;
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            ++units_done;
            base += nb;
        }
    };
    if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcRegsSoftmax));
        run_units(std::integral_constant<int, 1>{});
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsIssuers));
        if (warp == kTcFlagWarp && blockIdx.x == 0) {
            int bad = 0;
            for (int i = lane; i < a.n_split; i += 32) bad |= a.flags[1 + i];
            if (bad) atomicOr(a.flags, 1);
        }
        run_units(std::integral_constant<int, 0>{});
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kTcMmaWarp0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sm.tmem_base), "r"(512) : "memory");
    }
}

static int launch_prefill_f32_tc(const PrefillF32Args& f, int n_seqs, int max_q_len, void* scratch, cudaStream_t stream) {
    TcF32Args a = {};
    a.f = f;
    a.n_seqs = n_seqs;
    a.n_tiles = (max_q_len + kTcRows - 1) / kTcRows;
    a.n_split = n_seqs * f.table_stride * f.n_kv_heads;
    a.parts = (__nv_bfloat16*)scratch;
    const long long rows = 2ll * a.n_split * 3 * 64;
    a.flags = (int*)((uint8_t*)scratch + (size_t)rows * 64 * 2);
    if (rows >= (1ll << 31) || (long long)a.n_tiles * (f.n_heads / 2) * n_seqs >= (1ll << 30)) return kErrUnsupportedSize;
    CUtensorMap map;
    if (!make_map(&map, scratch, (int)rows, 64, 64, 64)) return kErrUnsupportedSize;
    const size_t smem = sizeof(TcF32Smem) + 1024;
    if (cudaFuncSetAttribute(attention_prefill_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return (int)cudaGetLastError();
    int st = launch_pdl(split_pages_kernel, dim3(f.table_stride, f.n_kv_heads, n_seqs), dim3(128), 0, stream, a);
    if (st != 0) return st;
    const int units = a.n_tiles * (f.n_heads / 2) * n_seqs, sms = device_sm_count();
    st = launch_pdl(attention_prefill_f32_tc_kernel, dim3(units < sms ? units : sms), dim3(kTcThreads), smem, stream, map, a);
    if (st != 0) return st;
    PrefillF32Args again = f;
    again.only_if = a.flags;
    return launch_prefill_f32<kTcD, 4>(again, n_seqs, max_q_len, 0, 1, nullptr, stream);
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

// Bytes of scratch that b200_attention_prefill_f32_tc needs.
extern "C" long long b200_attention_prefill_f32_tc_scratch(int n_seqs, int table_stride, int n_kv_heads) {
    const long long pages = (long long)n_seqs * table_stride * n_kv_heads;
    return pages * 2 * 3 * b200::kTcPart * 2 + (pages + 1) * 4;
}

extern "C" int b200_attention_prefill_f32_tc_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, b200::g_f32_tc_status, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(b200::g_f32_tc_status, &zero, sizeof(int));
    return v;
}

// The same as b200_attention_prefill_f32 without window or terms, head_dim 64 and an even number of query heads to a kv head, on the
// tensor cores (other operands: kErrUnsupportedSize).  scratch: 128-aligned, b200_attention_prefill_f32_tc_scratch bytes.
extern "C" int b200_attention_prefill_f32_tc(const void* q, int q_row_stride, void* out, const int* cu_seqlens, const int* kv_lens,
                                             const int* page_table, int table_stride, const void* k_pool, const void* v_pool,
                                             int n_seqs, int max_q_len, int n_heads, int n_kv_heads, int head_dim, void* scratch,
                                             long long scratch_bytes, cudaStream_t stream) {
    using namespace b200;
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0 || table_stride <= 0) return kErrBadArgument;
    if (head_dim != kTcD || (n_heads / n_kv_heads) % 2 != 0 || n_kv_heads > 65535 || n_seqs > 65535) return kErrUnsupportedSize;
    if (q_row_stride % 4 != 0 || (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15)) return kErrUnsupportedSize;
    if (scratch == nullptr || ((uintptr_t)scratch & 127) || scratch_bytes < b200_attention_prefill_f32_tc_scratch(n_seqs, table_stride, n_kv_heads))
        return kErrBadArgument;
    if ((long long)max_q_len * n_heads > 0x7fffff00ll) return kErrUnsupportedSize;
    PrefillF32Args a = {};
    a.q = (const float*)q; a.out = (float*)out; a.cu_seqlens = cu_seqlens; a.kv_lens = kv_lens; a.page_table = page_table;
    a.k_pool = (const float*)k_pool; a.v_pool = (const float*)v_pool;
    a.q_row_stride = q_row_stride; a.table_stride = table_stride; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads;
    return launch_prefill_f32_tc(a, n_seqs, max_q_len, scratch, stream);
}
