// Causal grouped-query attention over the paged cache, for any head size, any
// number of heads and groups, any mix of query lengths, both precisions.
//
// It stands where gpt-fast expands K/V to all heads and calls SDPA over the
// whole cache with a boolean mask (model.py:209-211): query head h reads
// key/value head h / (H/G); the key at position j is visible to the query at
// position p iff j <= p (and p - j < window when a window is set); scores are
// scaled by `scale`; softmax is 32-bit.  Options that other mixers use: `chunk` (a query
// sees only keys of its own block of `chunk` positions, blocks counted from
// position 0 of the sequence), `sink` (one number per query head whose
// exponential joins the softmax denominator without a value), a value head
// size `dv` of its own, values that are the leading part of the key rows, and a
// bias on the scaled score that depends on head and distance n = p - j only:
// `bias` (a table [bias_len][H], row min(n, bias_len - 1), added) and `slopes`
// (one number per head, slopes[h] * n taken off).  `softcap` > 0 squashes the (scaled, biased)
// score to cap * tanh(score / cap).  `keep_first`: the sequence's first keep_first positions stay
// visible to every later query whatever the window.  `maps` = 2: a head has two queries and a key
// row two keys side by side, each pair a softmax of its own over the same values; the head's output
// is o = o_1 - lambda o_2, divided by its root mean square over dv (diff_eps inside the root) and
// multiplied by out_scale.
//
// One block per (token, query head); prompts in 32-bit share keys and values between rows (attention_prompt_kernel, the same bits).  Keys are visited in chunks of 128 that
// start at multiples of 128 of the ABSOLUTE position, with an online softmax
// between chunks, so a query's result is the same bits whether its token came
// in a long prompt, alone, or in any batch.  It waits for memory, one key row per thread and then one value
// row after the other, so key rows are read four numbers at a time and the value rows' places are worked out once per
// chunk, which leaves eight rows' loads in flight.  This is the kernel of the 32-bit
// path and the fallback of the bfloat16 path; the fast bfloat16 kernels live
// in files of their own.
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

constexpr int CHUNK = 128;      // keys per step = threads per block
constexpr int MAX_DPT = 4;      // head_dim <= CHUNK * MAX_DPT

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u); v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
}

template <typename T>
__global__ void __launch_bounds__(CHUNK)
attention_generic_kernel(const T* __restrict__ q, T* __restrict__ out, GfbPagedKV kv, GfbBatch b,
                         int H, int G, int d, int dv, int v_row, float scale, int window, int chunk,
                         const float* __restrict__ sink, const float* __restrict__ bias, int bias_len,
                         const float* __restrict__ slopes, float softcap, int keep_first, int maps, float lambda,
                         float diff_eps, float out_scale, int* status) {
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;              // [d]
    float* ps = smem + d;          // [CHUNK]
    __shared__ float scratch[32];
    __shared__ __align__(16) long long v_at[CHUNK];   // where each key's value row starts in the pool; negative: no such key
    gfb_pdl_launch();
    gfb_pdl_wait();

    int t = blockIdx.x, h = blockIdx.y;
    int g = h / (H / G);
    int s = b.tok_seq[t];
    int slot = b.slots[s];
    int pos = b.lengths[slot] + (t - b.cu_seqlens[s]);
    const int dkr = d * maps;                    // numbers in a cached key row
    const bool wide = d % 4 == 0 && (reinterpret_cast<uintptr_t>(kv.k_pool) & (4 * sizeof(T) - 1)) == 0;      // key rows of whole 4-number units

    int lo = 0;
    if (window > 0 && pos - window + 1 > 0) lo = pos - window + 1;
    if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
    const int* pt = kv.page_table + (size_t)slot * kv.max_pages;
    const size_t head_off = (size_t)g * kv.page_size * dkr, v_head_off = (size_t)g * kv.page_size * v_row;
    const size_t page_stride = (size_t)G * kv.page_size * dkr, v_page_stride = (size_t)G * kv.page_size * v_row;
    const int kept = lo > 0 ? min(keep_first, lo) : 0;       // positions [0, kept) are seen besides [lo, pos]
    float first[MAX_DPT];                                    // the first map's finished output, while the second runs
#pragma unroll
    for (int i = 0; i < MAX_DPT; i++) first[i] = 0.f;

  for (int map = 0; map < maps; map++) {
    __syncthreads();               // every thread is done with the previous map's qs
    const T* qrow = q + (((size_t)t * H + h) * maps + map) * d;
    for (int i = threadIdx.x; i < d; i += CHUNK) qs[i] = gfb_to_f32(qrow[i]) * scale;
    float m_run = -INFINITY, l_run = 0.f;
    float acc[MAX_DPT];
#pragma unroll
    for (int i = 0; i < MAX_DPT; i++) acc[i] = 0.f;

    for (int c0 = kept > 0 ? 0 : (lo / CHUNK) * CHUNK; c0 <= pos; c0 += CHUNK) {
        if (c0 >= kept && c0 + CHUNK <= lo) continue;          // a block of keys between the kept ones and the window
        __syncthreads();           // qs ready (first pass); ps / v_at free (later passes)
        int j = c0 + threadIdx.x;
        bool live = (j >= lo || j < kept) && j <= pos;
        int page = -1;
        if (live) {
            int pi = j / kv.page_size;
            page = pi < kv.max_pages ? pt[pi] : -1;
            if (page < 0 || page >= kv.n_pages) {
                gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi);
                live = false;
                page = -1;
            }
        }
        v_at[threadIdx.x] = live ? (long long)page * (long long)v_page_stride + (long long)v_head_off + (long long)(j % kv.page_size) * v_row : -1;
        float sc = -INFINITY;
        if (live) {
            const T* krow = (const T*)kv.k_pool + (size_t)page * page_stride + head_off
                            + (size_t)(j % kv.page_size) * dkr + (size_t)map * d;
            float dot = 0.f;
            if (wide) {
                // four numbers per load, eight loads in flight; the sum stays in ascending order
#pragma unroll 8
                for (int i = 0; i < d; i += 4) {
                    float k4[4];
                    load4(krow + i, k4);
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + i);
                    dot = fmaf(q4.x, k4[0], dot); dot = fmaf(q4.y, k4[1], dot); dot = fmaf(q4.z, k4[2], dot); dot = fmaf(q4.w, k4[3], dot);
                }
            } else {
                for (int i = 0; i < d; i++) dot = fmaf(qs[i], gfb_to_f32(krow[i]), dot);
            }
            sc = dot;
            if (bias != nullptr) sc += bias[(size_t)min(pos - j, bias_len - 1) * H + h];
            if (slopes != nullptr) sc -= slopes[h] * (float)(pos - j);
            if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        }
        float m_new = fmaxf(m_run, gfb_block_max(sc, scratch));
        float p = live ? expf(sc - m_new) : 0.f;
        ps[threadIdx.x] = p;
        float l_chunk = gfb_block_sum(p, scratch);     // also orders the ps / v_at stores
        float corr = (m_run == -INFINITY) ? 0.f : expf(m_run - m_new);
        l_run = l_run * corr + l_chunk;
        m_run = m_new;
        int nkeys = min(CHUNK, pos - c0 + 1);
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) {
            int dim = threadIdx.x + r * CHUNK;
            if (dim < dv) {
                float a = acc[r] * corr;
                const T* v_base = (const T*)kv.v_pool + dim;
#pragma unroll 8
                for (int jj = 0; jj < nkeys; jj++) {
                    const long long at = v_at[jj];
                    if (at >= 0) a = fmaf(ps[jj], gfb_to_f32(v_base[at]), a);
                }
                acc[r] = a;
            }
        }
    }
    if (sink != nullptr) {
        // one more term in the denominator, exp(sink_h), with no value behind it
        const float sk = sink[h];
        const float m_fin = fmaxf(m_run, sk);
        const float corr = (m_run == -INFINITY) ? 0.f : expf(m_run - m_fin);
        l_run = l_run * corr + expf(sk - m_fin);
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) acc[r] *= corr;
    }
    float inv = l_run > 0.f ? 1.f / l_run : 0.f;
    if (maps == 1) {
        T* orow = out + ((size_t)t * H + h) * dv;
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) {
            int dim = threadIdx.x + r * CHUNK;
            if (dim < dv) orow[dim] = gfb_from_f32<T>(acc[r] * inv);
        }
    } else if (map == 0) {
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) first[r] = acc[r] * inv;
    } else {
        // the difference of the two maps, normed over the head and scaled
        float ss = 0.f;
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) {
            first[r] -= lambda * (acc[r] * inv);
            if (threadIdx.x + r * CHUNK < dv) ss += first[r] * first[r];
        }
        __syncthreads();
        ss = gfb_block_sum(ss, scratch);
        const float f = out_scale / sqrtf(ss / (float)dv + diff_eps);
        T* orow = out + ((size_t)t * H + h) * dv;
#pragma unroll
        for (int r = 0; r < MAX_DPT; r++) {
            int dim = threadIdx.x + r * CHUNK;
            if (dim < dv) orow[dim] = gfb_from_f32<T>(first[r] * f);
        }
    }
  }
}

// ---- prompts in 32-bit ------------------------------------------------------------------------------
// The same arithmetic in the same order, bit for bit, for ROWS (token, head of a group) rows of one sequence per block: a block per row reads every
// key and value from L2 for itself, row by row of a key per thread.  Here a chunk's 128 keys, and
// then its values, come into shared memory once for the ROWS rows, of which each half of the block takes half.  A thread is a key while scores
// are made and a value column while weights meet values; rows read their queries and weights by broadcast.  Keys that not every row of
// the block sees are left out of a row's sums by a bit, not by a zero, so that a number there that is not finite does no harm.
// 61 and 137 tokens of 24 heads of 128: 70 us with a block per row, 34 so (65 with a thread per key and all sixteen rows of a bit test each).
constexpr int ROWS = 16, MINE = ROWS / 2, PROMPT_DIM = 128, PROMPT_THREADS = 2 * CHUNK;

struct Prompt {
    int d, dv, v_row, window, chunk, bias_len, n_x;
    float scale, softcap;
    const float *sink, *bias, *slopes;
};

__device__ __forceinline__ void row16(float* smem, const float* gmem, bool live) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(gmem), "r"(live ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(PROMPT_THREADS, 2)
attention_prompt_kernel(const float* __restrict__ q, float* __restrict__ out, GfbPagedKV kv, GfbBatch b, int H, int G, const Prompt o, int* status) {
    extern __shared__ __align__(16) float smem[];
    const int pitch = max(o.d, o.dv) + 4, rep = H / G, g = blockIdx.y, tid = threadIdx.x & (CHUNK - 1), half = threadIdx.x / CHUNK;
    const int lane = tid & 31, warp = tid >> 5;       // (within this half)
    float* tile = smem;                               // [CHUNK][pitch]: keys, then values
    float* qs = tile + CHUNK * pitch;                 // [ROWS][d]
    float* ps = qs + ROWS * o.d;                      // [CHUNK][ROWS]
    float* part = ps + CHUNK * ROWS;                  // [ROWS][4]: the warps' maxima
    float* part2 = part + ROWS * 4;                   // ... and their sums
    __shared__ int pos_of[ROWS], lo_of[ROWS], head_of[ROWS];
    __shared__ unsigned char seen[CHUNK][2];          // which of a half's rows see the key
    gfb_pdl_launch();
    gfb_pdl_wait();
    int seq = -1, row0 = 0;
    {
        int left = o.n_x - 1 - (int)blockIdx.x;       // the latest rows first: they see the most keys
        for (int i = 0; i < b.n_seqs; i++) {
            const int nt = ((b.cu_seqlens[i + 1] - b.cu_seqlens[i]) * rep + ROWS - 1) / ROWS;
            if (left < nt) { seq = i; row0 = left * ROWS; break; }
            left -= nt;
        }
    }
    if (seq < 0) return;
    const int t0 = b.cu_seqlens[seq], rows = min(ROWS, (b.cu_seqlens[seq + 1] - t0) * rep - row0), slot = b.slots[seq], start = b.lengths[slot];
    const int* pt = kv.page_table + (size_t)slot * kv.max_pages;
    if (threadIdx.x < ROWS) {
        const int r = threadIdx.x, pos = start + (row0 + r) / rep;
        int lo = (o.window > 0 && pos - o.window + 1 > 0) ? pos - o.window + 1 : 0;
        if (o.chunk > 0) lo = max(lo, (pos / o.chunk) * o.chunk);
        pos_of[r] = r < rows ? pos : -1;              // (no key)
        lo_of[r] = lo;
        head_of[r] = g * rep + (row0 + r) % rep;
    }
    auto q_row = [&](int r) { return (size_t)(t0 + (row0 + r) / rep) * H + g * rep + (row0 + r) % rep; };      // of q and out
    for (int e = threadIdx.x; e < ROWS * o.d; e += PROMPT_THREADS) {
        const int r = e / o.d, i = e - r * o.d;
        qs[e] = r < rows ? q[q_row(r) * o.d + i] * o.scale : 0.f;
    }
    __syncthreads();
    const int r0 = half * MINE;                       // this half's first row
    float m_run[MINE], l_run[MINE], acc[MINE];
#pragma unroll
    for (int r = 0; r < MINE; r++) { m_run[r] = -INFINITY; l_run[r] = acc[r] = 0.f; }
    const int last = pos_of[rows - 1], lowest = lo_of[0], all_from = lo_of[rows - 1], all_to = pos_of[0];      // every row sees keys all_from .. all_to
    const size_t k_head = (size_t)g * kv.page_size * o.d, v_head = (size_t)g * kv.page_size * o.v_row;
    const size_t k_page = (size_t)G * kv.page_size * o.d, v_page = (size_t)G * kv.page_size * o.v_row;
    for (int c0 = lowest / CHUNK * CHUNK; c0 <= last; c0 += CHUNK) {
        const int j = c0 + tid;
        int page = -1, in_page = 0;
        if (j >= lowest && j <= last) {
            const int pi = j / kv.page_size;
            in_page = j - pi * kv.page_size;
            page = pi < kv.max_pages ? pt[pi] : -1;
            if (page < 0 || page >= kv.n_pages) { gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi); page = -1; }
        }
        const int n_keys = min(CHUNK, last - c0 + 1);
        // rows of the tile by whole warps, sixteen keys each, from the places that their keys' threads hold
        auto fetch = [&](const float* pool, size_t at, int n) {
            const int first = 16 * half, many = min(16, n_keys - warp * 32 - first);
#pragma unroll 4
            for (int k = 0; k < many; k++) {
                const size_t from = __shfl_sync(0xffffffffu, (unsigned long long)at, first + k);
                const bool there = __shfl_sync(0xffffffffu, page, first + k) >= 0;
                if (lane * 4 < n) row16(tile + (warp * 32 + first + k) * pitch + lane * 4, pool + from + lane * 4, there);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        };
        fetch((const float*)kv.k_pool, max(page, 0) * k_page + k_head + (size_t)in_page * o.d, o.d);
        __syncthreads();
        uint32_t bits = 0;
        float sc[MINE];
#pragma unroll
        for (int r = 0; r < MINE; r++) sc[r] = 0.f;
        if (page >= 0) {
            const float *krow = tile + tid * pitch, *qr = qs + r0 * o.d;
#pragma unroll 4
            for (int i = 0; i < o.d; i += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(krow + i);
#pragma unroll
                for (int r = 0; r < MINE; r++) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qr + r * o.d + i);
                    sc[r] = fmaf(q4.x, k4.x, sc[r]); sc[r] = fmaf(q4.y, k4.y, sc[r]); sc[r] = fmaf(q4.z, k4.z, sc[r]); sc[r] = fmaf(q4.w, k4.w, sc[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < MINE; r++) {
            const int pos = pos_of[r0 + r];
            if (page >= 0 && j <= pos && j >= lo_of[r0 + r]) {
                bits |= 1u << r;
                if (o.bias != nullptr) sc[r] += o.bias[(size_t)min(pos - j, o.bias_len - 1) * H + head_of[r0 + r]];
                if (o.slopes != nullptr) sc[r] -= o.slopes[head_of[r0 + r]] * (float)(pos - j);
                if (o.softcap > 0.f) sc[r] = o.softcap * tanhf(sc[r] / o.softcap);
            } else {
                sc[r] = -INFINITY;
            }
            const float mx = gfb_warp_max(sc[r]);
            if (lane == 0) part[(r0 + r) * 4 + warp] = mx;
        }
        seen[tid][half] = (unsigned char)bits;
        __syncthreads();                              // every thread is done with its key, too
        fetch((const float*)kv.v_pool, max(page, 0) * v_page + v_head + (size_t)in_page * o.v_row, o.dv);
        float corr[MINE];
#pragma unroll
        for (int r = 0; r < MINE; r++) {
            const float4 p4 = *reinterpret_cast<const float4*>(part + (r0 + r) * 4);
            const float m_new = fmaxf(m_run[r], fmaxf(fmaxf(p4.x, p4.y), fmaxf(p4.z, p4.w)));
            sc[r] = bits >> r & 1 ? expf(sc[r] - m_new) : 0.f;
            corr[r] = (m_run[r] == -INFINITY) ? 0.f : expf(m_run[r] - m_new);
            m_run[r] = m_new;
            const float sum = gfb_warp_sum(sc[r]);
            if (lane == 0) part2[(r0 + r) * 4 + warp] = sum;
        }
#pragma unroll
        for (int r = 0; r < MINE; r += 4) *reinterpret_cast<float4*>(ps + tid * ROWS + r0 + r) = make_float4(sc[r], sc[r + 1], sc[r + 2], sc[r + 3]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < MINE; r++) {
            const float4 p4 = *reinterpret_cast<const float4*>(part2 + (r0 + r) * 4);
            l_run[r] = l_run[r] * corr[r] + ((p4.x + p4.z) + (p4.y + p4.w));       // (the order of gfb_block_sum)
            acc[r] *= corr[r];
        }
        if (tid < o.dv) {
            auto some = [&](int from, int to) {       // keys that not every row sees
                for (int jj = from; jj < to; jj++) {
                    const float v = tile[jj * pitch + tid];
                    const uint32_t who = seen[jj][half];
#pragma unroll
                    for (int r = 0; r < MINE; r++)
                        if (who >> r & 1) acc[r] = fmaf(ps[jj * ROWS + r0 + r], v, acc[r]);
                }
            };
            const int a = min(max(all_from - c0, 0), n_keys), z = max(a, min(n_keys, all_to - c0 + 1));
            some(0, a);
#pragma unroll 4
            for (int jj = a; jj < z; jj++) {          // (a key without a page: a weight of zero and a value of zeros)
                const float v = tile[jj * pitch + tid];
#pragma unroll
                for (int r = 0; r < MINE; r += 4) {
                    const float4 p4 = *reinterpret_cast<const float4*>(ps + jj * ROWS + r0 + r);
                    acc[r] = fmaf(p4.x, v, acc[r]); acc[r + 1] = fmaf(p4.y, v, acc[r + 1]);
                    acc[r + 2] = fmaf(p4.z, v, acc[r + 2]); acc[r + 3] = fmaf(p4.w, v, acc[r + 3]);
                }
            }
            some(z, n_keys);
        }
        __syncthreads();                              // the tile, weights and bits are free
    }
#pragma unroll
    for (int r = 0; r < MINE; r++) {
        if (r0 + r >= rows) break;
        if (o.sink != nullptr) {
            const float sk = o.sink[head_of[r0 + r]];
            const float m_fin = fmaxf(m_run[r], sk);
            const float c = (m_run[r] == -INFINITY) ? 0.f : expf(m_run[r] - m_fin);
            l_run[r] = l_run[r] * c + expf(sk - m_fin);
            acc[r] *= c;
        }
        const float inv = l_run[r] > 0.f ? 1.f / l_run[r] : 0.f;
        if (tid < o.dv) out[q_row(r0 + r) * o.dv + tid] = acc[r] * inv;
    }
}

GFB_API int gfb_attention_generic(const void* q, void* out, int dt,
                                  void* k_pool, void* v_pool, const int* page_table, int max_pages, int page_size,
                                  int n_pages,
                                  const int* cu_seqlens, const int* tok_seq, const int* slots, const int* lengths,
                                  int n_seqs, int n_tokens, int share, int H, int G, int d, int dv, float scale, int window,
                                  int chunk, const float* sink, int values_in_keys, const float* bias, int bias_len,
                                  const float* slopes, float softcap, int keep_first, int maps, float lambda, float diff_eps,
                                  float out_scale, int* status, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (maps != 1 && maps != 2) return gfb_fail("gfb_attention_generic: %d score maps per head (1 or 2)", maps);
    if (keep_first < 0) return gfb_fail("gfb_attention_generic: %d kept first positions", keep_first);
    if (keep_first > 0 && chunk > 0) return gfb_fail("gfb_attention_generic: kept first positions go with a window, not with a block mask");
    if (maps == 2 && (values_in_keys || sink != nullptr)) return gfb_fail("gfb_attention_generic: two maps take values of their own and no sink");
    if (dv <= 0) dv = d;
    if (dv > CHUNK * MAX_DPT) return gfb_fail("gfb_attention_generic: value head size %d exceeds %d", dv, CHUNK * MAX_DPT);
    if (G <= 0 || H % G) return gfb_fail("gfb_attention_generic: %d heads do not divide into %d groups", H, G);
    if (H > 65535) return gfb_fail("gfb_attention_generic: %d heads exceed the grid limit", H);
    if (bias != nullptr && bias_len < 1) return gfb_fail("gfb_attention_generic: a distance table of %d rows", bias_len);
    // values_in_keys: a value is the first dv dimensions of its key row (a latent shared by keys and values), so
    // the value pool is the key pool read with the keys' row stride
    if (values_in_keys && dv > d) return gfb_fail("gfb_attention_generic: values of %d dimensions inside keys of %d", dv, d);
    const int v_row = values_in_keys ? d : dv;
    GfbPagedKV kv{k_pool, values_in_keys ? k_pool : v_pool, page_table, max_pages, page_size, n_pages};
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    dim3 grid(n_tokens, H);
    size_t smem = (size_t)(d + CHUNK) * sizeof(float);
    cudaError_t e;
    // share: where the kernel can, rows of 32-bit numbers share their keys and values.  (A head's pages of whole 16-byte rows; kept first positions
    // and pairs of maps stay with the general kernel.)
    if (dt == GFB_F32 && share && maps == 1 && keep_first == 0 && d % 4 == 0 && dv % 4 == 0 && d <= PROMPT_DIM && dv <= PROMPT_DIM &&
        (((uintptr_t)k_pool | (uintptr_t)kv.v_pool) & 15) == 0) {
        const long n_x = ((long)n_tokens * (H / G) + ROWS - 1) / ROWS + n_seqs;          // an upper bound of the tiles; surplus blocks find no work
        if (n_x > 2147483647L) return gfb_fail("gfb_attention_generic: %ld tiles", n_x);
        const size_t bytes = ((size_t)CHUNK * ((d > dv ? d : dv) + 4) + ROWS * d + CHUNK * ROWS + 8 * ROWS) * 4;
        static size_t configured = 0;
        if (bytes > configured) {
            e = cudaFuncSetAttribute(attention_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e != cudaSuccess) return gfb_fail("gfb_attention_generic: %zu bytes of shared memory refused: %s", bytes, cudaGetErrorString(e));
            configured = bytes;
        }
        const Prompt o{d, dv, v_row, window, chunk, bias_len, (int)n_x, scale, softcap, sink, bias, slopes};
        e = gfb_launch(attention_prompt_kernel, dim3((unsigned)n_x, G), dim3(PROMPT_THREADS), bytes, stream, (const float*)q, (float*)out, kv, b, H, G, o, status);
        return gfb_check(e, "gfb_attention_generic (prompt)");
    }
    if (dt == GFB_BF16)
        e = gfb_launch(attention_generic_kernel<__nv_bfloat16>, grid, dim3(CHUNK), smem, stream,
                       (const __nv_bfloat16*)q, (__nv_bfloat16*)out, kv, b, H, G, d, dv, v_row, scale, window, chunk, sink, bias, bias_len, slopes, softcap, keep_first, maps, lambda, diff_eps, out_scale, status);
    else if (dt == GFB_F32)
        e = gfb_launch(attention_generic_kernel<float>, grid, dim3(CHUNK), smem, stream,
                       (const float*)q, (float*)out, kv, b, H, G, d, dv, v_row, scale, window, chunk, sink, bias, bias_len, slopes, softcap, keep_first, maps, lambda, diff_eps, out_scale, status);
    else
        return gfb_fail("gfb_attention_generic: unknown type %d", dt);
    return gfb_check(e, "gfb_attention_generic");
}
