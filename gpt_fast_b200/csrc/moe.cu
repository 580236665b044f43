// Mixture of experts: a router that picks `top` of E small gated feed-forwards per token, and the experts.
//
// gfb_moe_router        router logits and choice in one launch: a block per token, or per eight tokens of a prompt
// gfb_moe_route         from 32-bit router logits: s = sigmoid(z); the `top` experts with the largest s + correction
//                       (lowest index on ties); weights s / (sum of the chosen s + 1e-20) * scale.  Or (mode ROUTE_SOFTMAX_TOP)
//                       the `top` largest logits themselves, weighted by the softmax over just those, times scale.  Or (mode
//                       ROUTE_SOFTMAX) s = softmax over all E logits, chosen by s + correction, weighted by s * scale.  With
//                       `groups` > 1 only experts of the `keep` groups (of equal size, neighbours) whose largest choice
//                       scores are largest can be chosen (`group_terms` = 2: the groups whose two largest choice scores have the
//                       largest sum).  Mode ROUTE_SIGMOID_PLAIN: weights s * scale, not divided by their sum.
//                       `shared` = 1: every token also runs expert number E with weight 1
// gfb_moe_glu           act[pair, f] = g * sigmoid(alpha g) * (u + shift),  g = min(gate_f . h, limit),
//                       u = clamp(up_f . h, -limit, limit), for every (token, chosen expert) pair
//                       or, for experts of two products (kind RELU2), act[pair, f] = max(up_f . h, 0)^2
// gfb_moe_down          x[t] (+)= sum over the token's chosen experts of weight * (W_down act[pair]); 32-bit sum into the stream
//
// The gate and up rows of an expert alternate in one matrix w13 [E, 2F, D] (RELU2: the up matrix [E, F, D] alone), the down
// matrix is w2 [E, D, F].  A shared expert of the experts' own size is one more matrix behind theirs.
// A pair is p = t * top + r (r: rank of the expert among the token's choices).
//
// Two forms of the expert products.  Few tokens (a decode step): a warp per output number streams the weight row once,
// 16 bytes per lane and load, the token's input staged in shared memory.  Many tokens (a prompt): the pairs are sorted by
// expert (gfb_moe_plan: each expert's rows padded to whole tiles) and the products run tile by tile, each tile with its
// expert's weights, the rows' results brought back to pair order.  The tiles run on the tensor cores (bfloat16: the
// grouped product of the tcgen05 library between gfb_moe_gather_rows and gfb_moe_combine_rows, tiles of 16 to 256 rows) or on
// CUDA cores (32-bit, and shapes the tensor-core tiles do not take: moe_tiles_simt_kernel, tiles of 64 rows).  In every
// form a number is one sum over k in 32-bit in an order that does not depend on the other rows, so a token's result does
// not depend on what else is in the batch.
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

__device__ __forceinline__ float ldw(const void* p, int dt, size_t i) {
    return dt == GFB_BF16 ? __bfloat162float(((const __nv_bfloat16*)p)[i]) : ((const float*)p)[i];
}
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// ------------------------------------------------------------------------------------ router ----
constexpr int MAX_EPL = 16;           // experts per lane: E <= 512
constexpr int ROUTE_WARPS = 4;
enum { ROUTE_SIGMOID = 0, ROUTE_SOFTMAX_TOP = 1, ROUTE_SOFTMAX = 2, ROUTE_SIGMOID_PLAIN = 3 };
constexpr int MAX_GROUPS = 32;        // a lane keeps a group's score

struct RouteArgs {
    int E, top;
    float scale;
    int mode, groups, keep, group_terms, shared;
};

// one token's choice by one warp: `logits` are the token's E router logits.  EPL experts per lane (E <= 32 EPL): every step of the choice
// walks over a lane's experts, so the usual 8 to 32 of them are not walked over as 512.
template <int EPL>
__device__ __forceinline__ void route_token(const float* __restrict__ logits, const void* __restrict__ correction, int c_dt,
                                            const RouteArgs& ra, int* __restrict__ idx, float* __restrict__ weights, int lane) {
    const int E = ra.E, top = ra.top, mode = ra.mode;
    const float scale = ra.scale;
    float s[EPL], c[EPL];
    float z_max = -INFINITY, z_inv = 0.f;
    if (mode == ROUTE_SOFTMAX) {
        for (int e = lane; e < E; e += 32) z_max = fmaxf(z_max, logits[e]);
        z_max = gfb_warp_max(z_max);
        float sum = 0.f;
        for (int e = lane; e < E; e += 32) sum += expf(logits[e] - z_max);
        z_inv = 1.0f / gfb_warp_sum(sum);
    }
#pragma unroll
    for (int i = 0; i < EPL; i++) {
        const int e = lane + 32 * i;
        if (e < E) {
            s[i] = mode == ROUTE_SOFTMAX_TOP ? logits[e] : mode == ROUTE_SOFTMAX ? expf(logits[e] - z_max) * z_inv : sigmoid_f(logits[e]);
            c[i] = s[i] + (correction != nullptr ? ldw(correction, c_dt, e) : 0.f);
        } else {
            s[i] = 0.f;
            c[i] = -INFINITY;
        }
    }
    if (ra.groups > 1) {
        // lane g keeps the score of group g, its largest choice score or the sum of its two largest; the `keep` best groups stay
        // (the lowest index on ties)
        const int per = E / ra.groups;
        float score = -INFINITY;
        for (int g = 0; g < ra.groups; g++) {
            float m = -INFINITY;
#pragma unroll
            for (int i = 0; i < EPL; i++)
                if ((lane + 32 * i) / per == g) m = fmaxf(m, c[i]);            // (experts beyond E are -inf)
            const float top1 = gfb_warp_max(m);
            if (ra.group_terms > 1 && per > 1) {
                // the second largest: the first holder of the largest (by lane) looks at its other experts, every other lane at all
                const int holder = __ffs(__ballot_sync(0xffffffffu, m == top1)) - 1;
                float second = -INFINITY;
                bool skip = lane == holder;
#pragma unroll
                for (int i = 0; i < EPL; i++)
                    if ((lane + 32 * i) / per == g) {
                        if (skip && c[i] == top1) skip = false;
                        else second = fmaxf(second, c[i]);
                    }
                m = top1 + gfb_warp_max(second);
            } else {
                m = top1;
            }
            if (lane == g) score = m;
        }
        unsigned kept = 0u;
        for (int r = 0; r < ra.keep; r++) {
            float best = (lane < ra.groups && !(kept >> lane & 1u)) ? score : -INFINITY;
            int best_g = (lane < ra.groups && !(kept >> lane & 1u)) ? lane : 0x7fffffff;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int og = __shfl_xor_sync(0xffffffffu, best_g, o);
                if (ob > best || (ob == best && og < best_g)) { best = ob; best_g = og; }
            }
            if (best_g < 32) kept |= 1u << best_g;
        }
#pragma unroll
        for (int i = 0; i < EPL; i++) {
            const int e = lane + 32 * i;
            if (e < E && !(kept >> (e / per) & 1u)) c[i] = -INFINITY;
        }
    }
    float sum = 0.f, mine = 0.f;       // lane r keeps the r-th chosen score
    float first = 0.f;                 // the largest chosen logit (softmax over the chosen ones)
    int mine_e = 0;
    for (int r = 0; r < top; r++) {
        float best = -INFINITY, best_s = 0.f;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < EPL; i++)
            if (c[i] > best) { best = c[i]; best_e = lane + 32 * i; best_s = s[i]; }     // ascending e per lane: the lowest index wins a tie
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o), os = __shfl_xor_sync(0xffffffffu, best_s, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; best_s = os; }
        }
#pragma unroll
        for (int i = 0; i < EPL; i++)
            if (lane + 32 * i == best_e) c[i] = -INFINITY;
        if (mode == ROUTE_SOFTMAX_TOP) {
            if (r == 0) first = best_s;
            best_s = expf(best_s - first);
        }
        sum += best_s;
        if (lane == r) { mine = best_s; mine_e = best_e; }
    }
    if (lane < top) {
        idx[lane] = mine_e;
        weights[lane] = mode == ROUTE_SOFTMAX || mode == ROUTE_SIGMOID_PLAIN ? mine * scale : mode == ROUTE_SOFTMAX_TOP ? mine / sum * scale : mine / (sum + 1e-20f) * scale;
    }
    if (ra.shared && lane == 0) {
        idx[top] = E;
        weights[top] = 1.f;
    }
}

static int check_route(const RouteArgs& ra, const char* what) {
    if (ra.E < 1 || ra.E > 32 * MAX_EPL) return gfb_fail("%s: %d experts (1 to %d)", what, ra.E, 32 * MAX_EPL);
    if (ra.top < 1 || ra.top > 32 || ra.top > ra.E) return gfb_fail("%s: %d of %d experts per token (1 to 32)", what, ra.top, ra.E);
    if (ra.groups < 1 || ra.groups > MAX_GROUPS || ra.E % ra.groups || ra.keep < 1 || ra.keep > ra.groups || ra.top > ra.keep * (ra.E / ra.groups))
        return gfb_fail("%s: %d experts from %d of %d groups of %d experts in all", what, ra.top, ra.keep, ra.groups, ra.E);
    if (ra.group_terms < 1 || ra.group_terms > 2) return gfb_fail("%s: a group's score from %d choice scores (1 or 2)", what, ra.group_terms);
    return 0;
}

template <int EPL>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
moe_route_kernel(const float* __restrict__ logits, int ld, const void* __restrict__ correction, int c_dt, RouteArgs ra,
                 int* __restrict__ idx, float* __restrict__ weights, int T) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * ROUTE_WARPS + (threadIdx.x >> 5);
    if (t >= T) return;
    const size_t at = (size_t)t * (ra.top + ra.shared);
    route_token<EPL>(logits + (size_t)t * ld, correction, c_dt, ra, idx + at, weights + at, lane);
}

// idx int32 and weights float32 [T, top + shared]
GFB_API int gfb_moe_route(const float* logits, int ld, const void* correction, int c_dt, int E, int top, float scale, int* idx,
                          float* weights, int T, int mode, int groups, int keep, int group_terms, int shared, cudaStream_t stream) {
    if (T <= 0) return 0;
    const RouteArgs ra{E, top, scale, mode, groups, keep, group_terms, shared ? 1 : 0};
    if (check_route(ra, "gfb_moe_route")) return 1;
    cudaError_t e;
#define GO(EPL) e = gfb_launch(moe_route_kernel<EPL>, dim3((T + ROUTE_WARPS - 1) / ROUTE_WARPS), dim3(32 * ROUTE_WARPS), 0, stream, logits, ld, \
                               correction, c_dt, ra, idx, weights, T)
    if (E <= 32) GO(1);
    else if (E <= 128) GO(4);
    else GO(MAX_EPL);
#undef GO
    return gfb_check(e, "gfb_moe_route");
}

// ------------------------------------------------------------------------------------ few tokens ----
// dot of a weight row with a staged 32-bit vector: lanes take 16 bytes of the row at a time where the row allows it
template <typename T> struct Vec;
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };
template <> struct Vec<float> { static constexpr int N = 4; };

template <typename T>
__device__ __forceinline__ float row_dot(const T* __restrict__ row, const float* __restrict__ v, int n, int lane, bool wide) {
    float acc = 0.f;
    if (wide) {
        constexpr int N = Vec<T>::N;
        for (int c = lane * N; c < n; c += 32 * N) {
            const uint4 raw = *reinterpret_cast<const uint4*>(row + c);
            const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int i = 0; i < N; i++) acc = fmaf(gfb_to_f32(e[i]), v[c + i], acc);
        }
    } else {
        for (int c = lane; c < n; c += 32) acc = fmaf(gfb_to_f32(row[c]), v[c], acc);
    }
    return gfb_warp_sum(acc);
}

// row_dot (its sums in the same order) of two rows of whole aligned 16-byte pieces
template <typename T>
__device__ __forceinline__ void two_rows_dot(const T* __restrict__ row0, const T* __restrict__ row1, const float* __restrict__ v, int n, int lane,
                                             float (&out)[2]) {
    constexpr int N = Vec<T>::N;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll 4
    for (int c = lane * N; c < n; c += 32 * N) {
        const uint4 r0 = *reinterpret_cast<const uint4*>(row0 + c), r1 = *reinterpret_cast<const uint4*>(row1 + c);
#pragma unroll
        for (int i = 0; i < N; i++) {
            a0 = fmaf(gfb_to_f32(reinterpret_cast<const T*>(&r0)[i]), v[c + i], a0);
            a1 = fmaf(gfb_to_f32(reinterpret_cast<const T*>(&r1)[i]), v[c + i], a1);
        }
    }
    out[0] = gfb_warp_sum(a0);
    out[1] = gfb_warp_sum(a1);
}

template <typename T>
__device__ __forceinline__ bool rows_wide(const T* base, int n) {
    return n % Vec<T>::N == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0;
}

// A decode step's router in one launch: a block per token computes the E logits (a warp per two expert rows, the token's input staged in
// shared memory in 32-bit) and its first warp chooses.  What bounds it is latency: the rows are weights, so they are asked into L2 before the
// wait for the kernel ahead, and eight 16-byte loads of a lane are in flight at once.  8 tokens of 2,048 for 16 experts, alone and
// with cold caches: one load at a time 11.7 us, 11.3 so.
constexpr int ROUTER_WARPS = 8;

template <typename T, int EPL>
__global__ void __launch_bounds__(32 * ROUTER_WARPS)
moe_router_kernel(const T* __restrict__ h, const T* __restrict__ router, const void* __restrict__ correction, int c_dt, RouteArgs ra,
                  int* __restrict__ idx, float* __restrict__ weights, int D, int n_extra, float* __restrict__ extra) {
    const int E = ra.E;
    extern __shared__ __align__(16) float rs[];        // the input [D], then the logits [E + n_extra]
    float* z = rs + D;
    gfb_pdl_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x, rows = E + n_extra;
    for (int e = warp; e < rows; e += ROUTER_WARPS)
        for (int c = lane * (128 / (int)sizeof(T)); c < D; c += 32 * (128 / (int)sizeof(T)))
            asm volatile("prefetch.global.L2 [%0];" ::"l"(router + (size_t)e * D + c));
    gfb_pdl_wait();
    for (int i = threadIdx.x; i < D; i += blockDim.x) rs[i] = gfb_to_f32(h[(size_t)t * D + i]);
    __syncthreads();
    const bool wide = rows_wide(router, D);
    for (int e = warp; e < rows; e += 2 * ROUTER_WARPS) {
        const int n = e + ROUTER_WARPS < rows ? 2 : 1;
        float d[2];
        if (wide) {
            two_rows_dot(router + (size_t)e * D, router + (size_t)(e + (n - 1) * ROUTER_WARPS) * D, rs, D, lane, d);
        } else {
            d[0] = row_dot(router + (size_t)e * D, rs, D, lane, false);
            if (n == 2) d[1] = row_dot(router + (size_t)(e + ROUTER_WARPS) * D, rs, D, lane, false);
        }
        if (lane == 0)
            for (int k = 0; k < n; k++) {
                const int ee = e + k * ROUTER_WARPS;
                z[ee] = d[k];
                if (ee >= E) extra[(size_t)t * n_extra + (ee - E)] = d[k];     // rows behind the experts': their logits are handed out as they are
            }
    }
    __syncthreads();
    const size_t at = (size_t)t * (ra.top + ra.shared);
    if (warp == 0) route_token<EPL>(z, correction, c_dt, ra, idx + at, weights + at, lane);
}

// Prompts: a block takes ROUTER_TOKENS tokens, whose inputs sit in shared memory as they are, and a warp takes two of the router's rows at a
// time against all of them (sums in row_dot's order, so a token's logits are the same bits as alone); then a warp chooses for each token.
// What bounds it is the conversions and FMAs of a warp's row pair: 2,048 tokens of 2,048 for 16 experts 16.9 us
// (the product on the tensor cores, zero-padded to 128 columns, and the choice behind it took 19 + 11.1 us and a launch between them).
constexpr int ROUTER_TOKENS = 8;

template <typename T, int EPL>
__global__ void __launch_bounds__(32 * ROUTER_WARPS)
moe_router_tokens_kernel(const T* __restrict__ h, const T* __restrict__ router, const void* __restrict__ correction, int c_dt, RouteArgs ra,
                         int* __restrict__ idx, float* __restrict__ weights, int n_tokens, int D, int n_extra, float* __restrict__ extra) {
    constexpr int N = Vec<T>::N;
    const int E = ra.E, rows = E + n_extra;
    extern __shared__ __align__(16) unsigned char rt_raw[];      // the inputs [ROUTER_TOKENS][D], then the logits [ROUTER_TOKENS][rows]
    T* hs = reinterpret_cast<T*>(rt_raw);
    float* z = reinterpret_cast<float*>(rt_raw + (size_t)ROUTER_TOKENS * D * sizeof(T));
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * ROUTER_TOKENS, nt = min(ROUTER_TOKENS, n_tokens - t0);
#pragma unroll 4
    for (int i = threadIdx.x * N; i < ROUTER_TOKENS * D; i += blockDim.x * N)         // (rows are side by side and whole 16-byte pieces)
        *reinterpret_cast<uint4*>(hs + i) = i < nt * D ? *reinterpret_cast<const uint4*>(h + (size_t)t0 * D + i) : make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (int e = warp; e < rows; e += 2 * ROUTER_WARPS) {
        const bool two = e + ROUTER_WARPS < rows;
        const T* row[2] = {router + (size_t)e * D, router + (size_t)(two ? e + ROUTER_WARPS : e) * D};
        float acc[2][ROUTER_TOKENS];
#pragma unroll
        for (int t = 0; t < ROUTER_TOKENS; t++) acc[0][t] = acc[1][t] = 0.f;
#pragma unroll 2
        for (int c = lane * N; c < D; c += 32 * N) {
            const uint4 r0 = *reinterpret_cast<const uint4*>(row[0] + c), r1 = *reinterpret_cast<const uint4*>(row[1] + c);
            float w[2][N];
#pragma unroll
            for (int k = 0; k < N; k++) { w[0][k] = gfb_to_f32(reinterpret_cast<const T*>(&r0)[k]); w[1][k] = gfb_to_f32(reinterpret_cast<const T*>(&r1)[k]); }
#pragma unroll
            for (int t = 0; t < ROUTER_TOKENS; t++) {
                const uint4 hv = *reinterpret_cast<const uint4*>(hs + (size_t)t * D + c);
#pragma unroll
                for (int k = 0; k < N; k++) {
                    const float v = gfb_to_f32(reinterpret_cast<const T*>(&hv)[k]);
                    acc[0][t] = fmaf(w[0][k], v, acc[0][t]);
                    acc[1][t] = fmaf(w[1][k], v, acc[1][t]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (k == 1 && !two) break;
            const int ee = e + k * ROUTER_WARPS;
#pragma unroll
            for (int t = 0; t < ROUTER_TOKENS; t++) {
                const float d = gfb_warp_sum(acc[k][t]);
                if (lane == 0) {
                    z[t * rows + ee] = d;
                    if (ee >= E && t < nt) extra[(size_t)(t0 + t) * n_extra + (ee - E)] = d;
                }
            }
        }
    }
    __syncthreads();
    for (int t = warp; t < nt; t += ROUTER_WARPS) {
        const size_t at = (size_t)(t0 + t) * (ra.top + ra.shared);
        route_token<EPL>(z + t * rows, correction, c_dt, ra, idx + at, weights + at, lane);
    }
}

// h [T, D] and router [>= E + n_extra, D] of type dt (further rows are padding).  Up to 64 tokens: a block per token; beyond, rows of whole
// 16-byte pieces whose eight inputs fit shared memory: a block per eight tokens; other rows are refused.
// The logits of the n_extra rows behind the experts' go to extra float32 [T, n_extra].
GFB_API int gfb_moe_router(const void* h, const void* router, int dt, const void* correction, int c_dt, int E, int top, float scale,
                           int* idx, float* weights, int T, int D, int mode, int groups, int keep, int group_terms, int shared, int n_extra, float* extra,
                             cudaStream_t stream) {
    if (T <= 0) return 0;
    const RouteArgs ra{E, top, scale, mode, groups, keep, group_terms, shared ? 1 : 0};
    if (check_route(ra, "gfb_moe_router")) return 1;
    if (n_extra < 0 || (n_extra > 0 && extra == nullptr)) return gfb_fail("gfb_moe_router: %d further rows without a place for their logits", n_extra);
    const bool few = T <= 64;
    const size_t smem = few ? (size_t)(D + E + n_extra) * sizeof(float)
                            : ROUTER_TOKENS * ((size_t)D * (dt == GFB_BF16 ? 2 : 4) + (size_t)(E + n_extra) * sizeof(float));
    if (smem > (few ? 48 : 200) * 1024) return gfb_fail("gfb_moe_router: %zu bytes of shared memory", smem);
    const int per = dt == GFB_BF16 ? 8 : 4;
    if (!few && (D % per || (((uintptr_t)h | (uintptr_t)router) & 15))) return gfb_fail("gfb_moe_router: rows of %d numbers are not whole 16-byte pieces", D);
    cudaError_t e = cudaSuccess;
#define GO(T_, EPL)                                                                                                                          \
    do {                                                                                                                                     \
        if (few) {                                                                                                                           \
            e = gfb_launch(moe_router_kernel<T_, EPL>, dim3((unsigned)T), dim3(32 * ROUTER_WARPS), smem, stream, (const T_*)h, (const T_*)router, \
                           correction, c_dt, ra, idx, weights, D, n_extra, extra);                                                           \
        } else {                                                                                                                             \
            if (smem > 48 * 1024) e = cudaFuncSetAttribute(moe_router_tokens_kernel<T_, EPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (e == cudaSuccess)                                                                                                            \
                e = gfb_launch(moe_router_tokens_kernel<T_, EPL>, dim3((unsigned)((T + ROUTER_TOKENS - 1) / ROUTER_TOKENS)), dim3(32 * ROUTER_WARPS), \
                               smem, stream, (const T_*)h, (const T_*)router, correction, c_dt, ra, idx, weights, T, D, n_extra, extra);      \
        }                                                                                                                                    \
    } while (0)
#define PICK(T_) do { if (E <= 32) GO(T_, 1); else if (E <= 128) GO(T_, 4); else GO(T_, MAX_EPL); } while (0)
    if (dt == GFB_BF16) PICK(__nv_bfloat16);
    else if (dt == GFB_F32) PICK(float);
    else return gfb_fail("gfb_moe_router: unknown type %d", dt);
#undef PICK
#undef GO
    return gfb_check(e, "gfb_moe_router");
}

constexpr int GEMV_WARPS = 8;
constexpr int GLU_PER_WARP = 2;       // hidden units per warp: 4 weight rows in flight

enum { KIND_GLU = 0, KIND_RELU2 = 1 };
__device__ __forceinline__ float relu2_f(float z) { const float p = fmaxf(z, 0.f); return p * p; }

template <typename T, int KIND>
__global__ void __launch_bounds__(32 * GEMV_WARPS)
moe_glu_gemv_kernel(const T* __restrict__ h, const int* __restrict__ idx, const T* __restrict__ w13, T* __restrict__ act, int top,
                    int E, int F, int D, float limit, float alpha, float shift) {
    extern __shared__ __align__(16) float hs[];
    gfb_pdl_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pair = blockIdx.y, t = pair / top;
    gfb_pdl_wait();
    const int e = idx[pair];
    for (int i = threadIdx.x; i < D; i += blockDim.x) hs[i] = gfb_to_f32(h[(size_t)t * D + i]);
    __syncthreads();
    if (e < 0 || e >= E) return;
    const T* w = w13 + (size_t)e * (KIND == KIND_RELU2 ? 1 : 2) * F * D;
    const bool wide = rows_wide(w, D);
    const int f0 = (blockIdx.x * GEMV_WARPS + warp) * GLU_PER_WARP;
#pragma unroll
    for (int r = 0; r < GLU_PER_WARP; r++) {
        const int f = f0 + r;
        if (f >= F) break;
        if constexpr (KIND == KIND_RELU2) {
            const float u = row_dot(w + (size_t)f * D, hs, D, lane, wide);
            if (lane == 0) act[(size_t)pair * F + f] = gfb_from_f32<T>(relu2_f(u));
        } else {
            float g = row_dot(w + (size_t)(2 * f) * D, hs, D, lane, wide);
            float u = row_dot(w + (size_t)(2 * f + 1) * D, hs, D, lane, wide);
            if (limit > 0.f) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
            if (lane == 0) act[(size_t)pair * F + f] = gfb_from_f32<T>(g * sigmoid_f(alpha * g) * (u + shift));
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(32 * GEMV_WARPS)
moe_down_gemv_kernel(const T* __restrict__ act, const int* __restrict__ idx, const float* __restrict__ weights, const T* __restrict__ w2,
                     float* __restrict__ x, int top, int E, int F, int D, int store) {
    extern __shared__ __align__(16) float as[];        // [top][F]
    gfb_pdl_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.y;
    gfb_pdl_wait();
    for (int i = threadIdx.x; i < top * F; i += blockDim.x) as[i] = gfb_to_f32(act[(size_t)t * top * F + i]);
    __syncthreads();
    const int n = blockIdx.x * GEMV_WARPS + warp;
    if (n >= D) return;
    const bool wide = rows_wide(w2, F) && ((size_t)D * F) % Vec<T>::N == 0;
    float acc = 0.f;
    for (int r = 0; r < top; r++) {
        const int e = idx[(size_t)t * top + r];
        if (e < 0 || e >= E) continue;
        acc = fmaf(weights[(size_t)t * top + r], row_dot(w2 + ((size_t)e * D + n) * F, as + (size_t)r * F, F, lane, wide), acc);
    }
    if (lane == 0) x[(size_t)t * D + n] = store ? acc : x[(size_t)t * D + n] + acc;
}

template <typename K>
static int allow_smem(K kernel, size_t smem, const char* what) {
    if (smem > 200 * 1024) return gfb_fail("%s: %zu bytes of shared memory", what, smem);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return gfb_fail("%s: %s", what, cudaGetErrorString(e));
    }
    return 0;
}

// ------------------------------------------------------------------------------------ many tokens ----
// The plan: rows of the sorted order.  Expert e's pairs take rows start[e] .. start[e] + count[e] - 1, start[e] a
// multiple of the tile height BM; row_pair[row] is the pair of a row (-1: padding), tile_expert[tile] the expert whose
// weights a tile of that many rows uses (-1: the tile is beyond the last expert's rows), *tiles_used (if asked for) the number
// of tiles with an expert, which come first.  One block builds it; the order of an
// expert's rows among themselves is whatever the atomics give, and no result depends on it.
constexpr int PLAN_THREADS = 1024;

__global__ void __launch_bounds__(PLAN_THREADS)
moe_plan_kernel(const int* __restrict__ idx, int n_pairs, int E, int tile_rows, int* __restrict__ row_pair, int* __restrict__ pair_row,
                int* __restrict__ tile_expert, int max_tiles, int* __restrict__ tiles_used) {
    extern __shared__ int sh[];          // count[E], start[E], fill[E]
    int* count = sh;
    int* start = sh + E;
    int* fill = sh + 2 * E;
    gfb_pdl_launch();
    gfb_pdl_wait();
    for (int e = threadIdx.x; e < E; e += blockDim.x) { count[e] = 0; fill[e] = 0; }
    for (int i = threadIdx.x; i < max_tiles * tile_rows; i += blockDim.x) row_pair[i] = -1;
    for (int i = threadIdx.x; i < max_tiles; i += blockDim.x) tile_expert[i] = -1;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = idx[p];
        if (e >= 0 && e < E) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0;
        for (int e = 0; e < E; e++) {
            start[e] = at;
            const int tiles = (count[e] + tile_rows - 1) / tile_rows;
            for (int i = 0; i < tiles; i++) tile_expert[at / tile_rows + i] = e;
            at += tiles * tile_rows;
        }
        if (tiles_used != nullptr) *tiles_used = at / tile_rows;       // the tiles with rows come first
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = idx[p];
        if (e >= 0 && e < E) {
            const int row = start[e] + atomicAdd(&fill[e], 1);
            row_pair[row] = p;
            pair_row[p] = row;
        } else {
            pair_row[p] = -1;
        }
    }
}

GFB_API int gfb_moe_plan(const int* idx, int n_pairs, int E, int tile_rows, int* row_pair, int* pair_row, int* tile_expert, int max_tiles,
                         int* tiles_used, cudaStream_t stream) {
    if (n_pairs <= 0) return 0;
    const long busy = n_pairs < E ? n_pairs : E;             // experts that can have rows at all
    if (tile_rows < 1 || (long)max_tiles < ((long)n_pairs + busy * (tile_rows - 1)) / tile_rows)
        return gfb_fail("gfb_moe_plan: %d tiles of %d rows cannot hold %d pairs of %d experts", max_tiles, tile_rows, n_pairs, E);
    const size_t smem = (size_t)3 * E * sizeof(int);
    cudaError_t e = gfb_launch(moe_plan_kernel, dim3(1), dim3(PLAN_THREADS), smem, stream, idx, n_pairs, E, tile_rows, row_pair, pair_row,
                               tile_expert, max_tiles, tiles_used);
    return gfb_check(e, "gfb_moe_plan");
}

// Tiles on CUDA cores (the 32-bit path, and bfloat16 shapes the tensor-core tiles do not take): 64 x 64 outputs per block,
// each one thread's ascending sum over k.  RELU2: as GLU with W = the up matrix, act[row, n] = max(., 0)^2.  GLU: A = h rows gathered by pair / top, W = w13 of the tile's expert, the
// output act[row, n / 2] from the gate (even n) and up (odd n) columns.  DOWN: A = act rows (sorted order), W = w2 of
// the tile's expert, the output y[pair, n] in 32-bit, pair order.
constexpr int BM = 64, BN = 64, BK = 16;

enum { TILES_DOWN = 0, TILES_GLU = 1, TILES_RELU2 = 2 };

template <typename T, int WHAT>
__global__ void __launch_bounds__(256)
moe_tiles_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, void* __restrict__ C, const int* __restrict__ row_pair,
                      const int* __restrict__ tile_expert, int top, int N, int K, float limit, float alpha, float shift) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ int src_row[BM];
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int e = tile_expert[blockIdx.y];
    if (e < 0) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    if (threadIdx.x < BM) {
        const int p = row_pair[m0 + threadIdx.x];
        src_row[threadIdx.x] = p < 0 ? -1 : (WHAT != TILES_DOWN ? p / top : m0 + (int)threadIdx.x);
    }
    __syncthreads();
    const T* We = W + (size_t)e * N * K;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int el = threadIdx.x + i * 256;
            const int r = el >> 4, k = el & 15;
            const int gk = k0 + k, gn = n0 + r, sr = src_row[r];
            As[k][r] = (sr >= 0 && gk < K) ? gfb_to_f32(A[(size_t)sr * K + gk]) : 0.f;
            Ws[k][r] = (gn < N && gk < K) ? gfb_to_f32(We[(size_t)gn * K + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = ty * 4 + i;
        const int p = row_pair[m0 + r];
        if (p < 0) continue;
        if (WHAT == TILES_RELU2) {
            T* out = (T*)C + (size_t)(m0 + r) * N;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = n0 + tx * 4 + j;
                if (n < N) out[n] = gfb_from_f32<T>(relu2_f(acc[i][j]));
            }
        } else if (WHAT == TILES_GLU) {
            T* out = (T*)C + (size_t)(m0 + r) * (N >> 1);
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int n = n0 + tx * 4 + j;
                if (n + 1 < N) {
                    float g = acc[i][j], u = acc[i][j + 1];
                    if (limit > 0.f) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
                    out[n >> 1] = gfb_from_f32<T>(g * sigmoid_f(alpha * g) * (u + shift));
                }
            }
        } else {
            float* out = (float*)C + (size_t)p * N;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = n0 + tx * 4 + j;
                if (n < N) out[n] = acc[i][j];
            }
        }
    }
}

// x[t] += sum_r weights[t, r] * y[t * top + r] in ascending r (store: x[t] = that sum)
__global__ void moe_combine_kernel(const float* __restrict__ y, const float* __restrict__ weights, float* __restrict__ x, int top,
                                   int D, long n, int store) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long t = i / D;
    const int c = (int)(i - t * D);
    float acc = 0.f;
    for (int r = 0; r < top; r++) acc = fmaf(weights[t * top + r], y[((size_t)t * top + r) * D + c], acc);
    x[i] = store ? acc : x[i] + acc;
}

// ------------------------------------------------------------------------------------ around the tensor-core tiles ----
// The tensor cores' tiles read their rows where TMA finds them: side by side in the sorted order.  hs[row] = h[row_pair[row] / top]
// (zeros for padding rows), 16 bytes per thread and step, GATHER_ROWS rows' pieces in flight together.  10,240 rows of
// 2,048: a row per block 15.3 us, so 11.1.
constexpr int GATHER_ROWS = 4;

__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const uint4* __restrict__ h, const int* __restrict__ row_pair, uint4* __restrict__ hs, int top, int vec_per_row, int rows) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int row0 = blockIdx.x * GATHER_ROWS;
    int p[GATHER_ROWS];
#pragma unroll
    for (int k = 0; k < GATHER_ROWS; k++) p[k] = row0 + k < rows ? row_pair[row0 + k] : -1;
    for (int i = threadIdx.x; i < vec_per_row; i += blockDim.x) {
        uint4 v[GATHER_ROWS];
#pragma unroll
        for (int k = 0; k < GATHER_ROWS; k++) v[k] = p[k] >= 0 ? h[(size_t)(p[k] / top) * vec_per_row + i] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < GATHER_ROWS; k++)
            if (row0 + k < rows) hs[(size_t)(row0 + k) * vec_per_row + i] = v[k];
    }
}

// h [T, D] bfloat16 with D % 8 == 0 -> hs [rows, D] in the plan's sorted order
GFB_API int gfb_moe_gather_rows(const void* h, const int* row_pair, void* hs, int rows, int top, int D, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (D % 8 || ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(hs)) & 15))
        return gfb_fail("gfb_moe_gather_rows: rows of %d bfloat16 numbers are not whole 16-byte pieces", D);
    cudaError_t e = gfb_launch(moe_gather_rows_kernel, dim3((unsigned)((rows + GATHER_ROWS - 1) / GATHER_ROWS)), dim3(256), 0, stream, (const uint4*)h,
                               row_pair, (uint4*)hs, top, D / 8, rows);
    return gfb_check(e, "gfb_moe_gather_rows");
}

// The plan and the gathered rows of a step of few pairs in one launch: a block per tile (and quarter of its columns) counts the pairs by
// expert for itself, finds its tile's expert in the scan of the counts, lists that expert's pairs in their order and copies their rows.  What
// bounds a decode step here is the chain of launches: 24 pairs of 17 experts, rows of 2,048, took 5.5 + 3.5 us as two, 4.9 us so.
constexpr int PLAN_FEW_PAIRS = 1024, PLAN_FEW_EXPERTS = 1024, PLAN_FEW_ROWS = 64;

__global__ void __launch_bounds__(256)
moe_plan_gather_kernel(const int* __restrict__ idx, int n_pairs, int E, int tile_rows, const uint4* __restrict__ h, uint4* __restrict__ hs, int top,
                       int vec_per_row, int* __restrict__ row_pair, int* __restrict__ pair_row, int* __restrict__ tile_expert,
                       int* __restrict__ tiles_used) {
    __shared__ int experts[PLAN_FEW_PAIRS], count[PLAN_FEW_EXPERTS], mine[PLAN_FEW_ROWS], my_expert, my_first, total;
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, tile = blockIdx.x;
    const bool writer = blockIdx.y == 0;             // one of a tile's blocks writes the plan
    for (int e = tid; e < E; e += blockDim.x) count[e] = 0;
    if (tid < tile_rows) mine[tid] = -1;
    if (tid == 0) my_expert = -1;
    __syncthreads();
    for (int p = tid; p < n_pairs; p += blockDim.x) {
        const int e = idx[p];
        const bool valid = e >= 0 && e < E;
        experts[p] = valid ? e : -1;
        if (valid) atomicAdd(&count[e], 1);
        else if (writer && tile == 0) pair_row[p] = -1;
    }
    __syncthreads();
    if (tid < 32) {
        int at = 0;                                  // tiles of the experts so far
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane, tiles = e < E ? (count[e] + tile_rows - 1) / tile_rows : 0;
            int sum = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            const int first = at + sum - tiles;
            if (tile >= first && tile < first + tiles) { my_expert = e; my_first = (tile - first) * tile_rows; }
            at += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) total = at;
        __syncwarp();
        const int e = my_expert;
        if (e >= 0) {
            int rank = -my_first;
            for (int p0 = 0; p0 < n_pairs; p0 += 32) {
                const int p = p0 + lane;
                const bool in = p < n_pairs && experts[p] == e;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                const int r = rank + __popc(m & ((1u << lane) - 1u));
                if (in && r >= 0 && r < tile_rows) {
                    mine[r] = p;
                    if (writer) pair_row[p] = tile * tile_rows + r;
                }
                rank += __popc(m);
            }
        }
    }
    __syncthreads();
    if (writer) {
        if (tid == 0) {
            tile_expert[tile] = my_expert;
            if (tile == 0) *tiles_used = total;
        }
        if (tid < tile_rows) row_pair[tile * tile_rows + tid] = mine[tid];
    }
    if (my_expert < 0) return;
    const int per = (vec_per_row + gridDim.y - 1) / gridDim.y, v0 = blockIdx.y * per, n = min(per, vec_per_row - v0);
    for (int i = tid; i < tile_rows * n; i += blockDim.x) {
        const int r = i / n, c = v0 + i - r * n, p = mine[r];
        hs[(size_t)(tile * tile_rows + r) * vec_per_row + c] = p < 0 ? make_uint4(0u, 0u, 0u, 0u) : h[(size_t)(p / top) * vec_per_row + c];
    }
}

// gfb_moe_plan and gfb_moe_gather_rows in one launch: at most 1,024 pairs and experts, tiles of at most 64 rows; tiles without rows are not
// written in hs
GFB_API int gfb_moe_plan_gather(const int* idx, int n_pairs, int E, int tile_rows, const void* h, void* hs, int top, int D, int* row_pair,
                                int* pair_row, int* tile_expert, int max_tiles, int* tiles_used, cudaStream_t stream) {
    if (n_pairs <= 0) return 0;
    const long busy = n_pairs < E ? n_pairs : E;
    if (tile_rows < 1 || tile_rows > PLAN_FEW_ROWS || n_pairs > PLAN_FEW_PAIRS || E > PLAN_FEW_EXPERTS)
        return gfb_fail("gfb_moe_plan_gather: %d pairs of %d experts in tiles of %d rows", n_pairs, E, tile_rows);
    if ((long)max_tiles < ((long)n_pairs + busy * (tile_rows - 1)) / tile_rows)
        return gfb_fail("gfb_moe_plan_gather: %d tiles of %d rows cannot hold %d pairs of %d experts", max_tiles, tile_rows, n_pairs, E);
    if (D < 8 || D % 8 || ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(hs)) & 15))
        return gfb_fail("gfb_moe_plan_gather: rows of %d bfloat16 numbers are not whole 16-byte pieces", D);
    const int vec = D / 8, cuts = vec >= 256 ? 4 : 1;
    cudaError_t e = gfb_launch(moe_plan_gather_kernel, dim3(max_tiles, cuts), dim3(256), 0, stream, idx, n_pairs, E, tile_rows, (const uint4*)h,
                               (uint4*)hs, top, vec, row_pair, pair_row, tile_expert, tiles_used);
    return gfb_check(e, "gfb_moe_plan_gather");
}

// x[t] += sum_r weights[t, r] * y[pair_row[t * top + r]] in ascending r (store: x[t] = that sum); y in the plan's sorted order, D % 4 == 0
__global__ void __launch_bounds__(256)
moe_combine_rows_kernel(const float4* __restrict__ y, const int* __restrict__ pair_row, const float* __restrict__ weights,
                        float4* __restrict__ x, int top, int vec_per_row, long n, int store) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long t = i / vec_per_row;
    const int c = (int)(i - t * vec_per_row);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < top; r++) {
        const int row = pair_row[t * top + r];
        if (row < 0) continue;
        const float w = weights[t * top + r];
        const float4 v = y[(size_t)row * vec_per_row + c];
        acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
    }
    float4 o = store ? make_float4(0.f, 0.f, 0.f, 0.f) : x[i];
    o.x += acc.x; o.y += acc.y; o.z += acc.z; o.w += acc.w;
    x[i] = o;
}

GFB_API int gfb_moe_combine_rows(const float* y, const int* pair_row, const float* weights, float* x, int T, int top, int D,
                                 int store, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (D % 4 || ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(x)) & 15))
        return gfb_fail("gfb_moe_combine_rows: rows of %d floats are not whole 16-byte pieces", D);
    const long n = (long)T * (D / 4);
    cudaError_t e = gfb_launch(moe_combine_rows_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, (const float4*)y, pair_row,
                               weights, (float4*)x, top, D / 4, n, store);
    return gfb_check(e, "gfb_moe_combine_rows");
}

// h [T, D], w13 [E, 2F, D], act [rows, F] of type dt.  tiles = 0: the few-token form, act in pair order (rows = T * top);
// otherwise act in the plan's sorted order (rows = max_tiles * 64) and row_pair, tile_expert from gfb_moe_plan with tiles of 64 rows.
// kind 1 (RELU2): w13 is the up matrix [E, F, D] and the constants of the gate are not used.
GFB_API int gfb_moe_glu(const void* h, const int* idx, const void* w13, void* act, int dt, int kind, int T, int top, int E, int F, int D,
                        float limit, float alpha, float shift, const int* row_pair, const int* tile_expert, int max_tiles,
                        cudaStream_t stream) {
    if (T <= 0) return 0;
    typedef __nv_bfloat16 bf16;
    cudaError_t e;
    if (max_tiles > 0) {
        const int N = kind == KIND_RELU2 ? F : 2 * F;
        dim3 grid((N + BN - 1) / BN, max_tiles);
        if (max_tiles > 65535) return gfb_fail("gfb_moe_glu: %d tiles exceed the grid limit", max_tiles);
#define GO(T, W) e = gfb_launch(moe_tiles_simt_kernel<T, W>, grid, dim3(256), 0, stream, (const T*)h, (const T*)w13, act, row_pair, \
                                tile_expert, top, N, D, limit, alpha, shift)
        if (dt == GFB_BF16 && kind == KIND_RELU2) GO(bf16, TILES_RELU2);
        else if (dt == GFB_BF16) GO(bf16, TILES_GLU);
        else if (dt == GFB_F32 && kind == KIND_RELU2) GO(float, TILES_RELU2);
        else if (dt == GFB_F32) GO(float, TILES_GLU);
#undef GO
        else return gfb_fail("gfb_moe_glu: unknown type %d", dt);
        return gfb_check(e, "gfb_moe_glu (tiles)");
    }
    const long pairs = (long)T * top;
    if (pairs > 65535) return gfb_fail("gfb_moe_glu: %ld pairs exceed the grid limit of the few-token form", pairs);
    const size_t smem = (size_t)D * sizeof(float);
    dim3 grid((F + GEMV_WARPS * GLU_PER_WARP - 1) / (GEMV_WARPS * GLU_PER_WARP), (unsigned)pairs);
#define GO(T, K)                                                                                                                   \
    do {                                                                                                                          \
        if (allow_smem(moe_glu_gemv_kernel<T, K>, smem, "gfb_moe_glu")) return 1;                                                 \
        e = gfb_launch(moe_glu_gemv_kernel<T, K>, grid, dim3(32 * GEMV_WARPS), smem, stream, (const T*)h, idx, (const T*)w13, (T*)act, \
                       top, E, F, D, limit, alpha, shift);                                                                        \
    } while (0)
    if (dt == GFB_BF16 && kind == KIND_RELU2) GO(bf16, KIND_RELU2);
    else if (dt == GFB_BF16) GO(bf16, KIND_GLU);
    else if (dt == GFB_F32 && kind == KIND_RELU2) GO(float, KIND_RELU2);
    else if (dt == GFB_F32) GO(float, KIND_GLU);
#undef GO
    else return gfb_fail("gfb_moe_glu: unknown type %d", dt);
    return gfb_check(e, "gfb_moe_glu");
}

// act as gfb_moe_glu left it; w2 [E, D, F]; x float32 [T, D] += the weighted sum of the chosen experts' outputs.
// With tiles: y float32 [T * top, D] is scratch for the experts' outputs in pair order.  store: x = the sum instead of +=.
GFB_API int gfb_moe_down(const void* act, const int* idx, const float* weights, const void* w2, float* x, int dt, int T, int top,
                         int E, int F, int D, const int* row_pair, const int* tile_expert, int max_tiles, float* y,
                         int store, cudaStream_t stream) {
    if (T <= 0) return 0;
    typedef __nv_bfloat16 bf16;
    cudaError_t e;
    if (max_tiles > 0) {
        dim3 grid((D + BN - 1) / BN, max_tiles);
        if (dt == GFB_BF16)
            e = gfb_launch(moe_tiles_simt_kernel<bf16, TILES_DOWN>, grid, dim3(256), 0, stream, (const bf16*)act, (const bf16*)w2, (void*)y,
                           row_pair, tile_expert, top, D, F, 0.f, 0.f, 0.f);
        else if (dt == GFB_F32)
            e = gfb_launch(moe_tiles_simt_kernel<float, TILES_DOWN>, grid, dim3(256), 0, stream, (const float*)act, (const float*)w2, (void*)y,
                           row_pair, tile_expert, top, D, F, 0.f, 0.f, 0.f);
        else return gfb_fail("gfb_moe_down: unknown type %d", dt);
        if (gfb_check(e, "gfb_moe_down (tiles)")) return 1;
        const long n = (long)T * D;
        e = gfb_launch(moe_combine_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, (const float*)y, weights, x, top, D, n, store);
        return gfb_check(e, "gfb_moe_down (combine)");
    }
    if (T > 65535) return gfb_fail("gfb_moe_down: %d tokens exceed the grid limit of the few-token form", T);
    const size_t smem = (size_t)top * F * sizeof(float);
    dim3 grid((D + GEMV_WARPS - 1) / GEMV_WARPS, T);
    if (dt == GFB_BF16) {
        if (allow_smem(moe_down_gemv_kernel<bf16>, smem, "gfb_moe_down")) return 1;
        e = gfb_launch(moe_down_gemv_kernel<bf16>, grid, dim3(32 * GEMV_WARPS), smem, stream, (const bf16*)act, idx, weights, (const bf16*)w2,
                       x, top, E, F, D, store);
    } else if (dt == GFB_F32) {
        if (allow_smem(moe_down_gemv_kernel<float>, smem, "gfb_moe_down")) return 1;
        e = gfb_launch(moe_down_gemv_kernel<float>, grid, dim3(32 * GEMV_WARPS), smem, stream, (const float*)act, idx, weights,
                       (const float*)w2, x, top, E, F, D, store);
    } else return gfb_fail("gfb_moe_down: unknown type %d", dt);
    return gfb_check(e, "gfb_moe_down");
}
