// The selective state space over prompts, in chunks of PC = 64 tokens (gfb_ssd_scan walks token by token):
//
//     dt_t = softplus(dt_raw_t + dt_bias_h);  S_t = 2^(a_t) S_(t-1) + dt_t B_t x_t^T,  a_t = -exp(A_log_h) log2(e) dt_t;  y_t = S_t^T C_t + D_h x_t
//
// With L_i the sum of a over the chunk's tokens up to i and S_0 the state ahead of the chunk,
//
//     y_i = 2^(L_i) S_0^T C_i + sum_(j<=i) (C_i . B_j) 2^(L_i - L_j) dt_j x_j + D_h x_i,     S_0' = 2^(L_end) S_0 + sum_j 2^(L_end - L_j) dt_j B_j x_j^T
//
// Three launches:
//   ssd_scores_kernel   a block per (chunk, group, 16 tokens): C_i . B_j, which all heads of a group share, and C transposed
//   ssd_state_kernel    a block per (sequence, head, 32 columns) walks over the chunks with its part of S in registers and leaves the S_0s
//   ssd_out_kernel      a block per (chunk, head, 64 columns): one product with K = state rows + 64
//
// Everything is 32-bit FMAs; the sums L and their differences are 64-bit (64 numbers per chunk and head), so that a decay between two tokens
// is as exact as its exponent, however much has decayed before them.  Long sums run in pieces of 32 terms that are then added, as the
// token-by-token kernel's lanes do, which keeps their rounding where it was.
//
// What bounds it: the token-by-token kernel is a chain of dependent instructions per token (sequences of 77, 788 and 1,500 tokens,
// 64 heads of 128 x 64: 1,135 us).  Here 2.4 GFMA and the S_0s' way through L2: 274 us,
// of which ssd_state_kernel 156, ssd_out_kernel 121, ssd_scores_kernel 8.  Against 64-bit sums (700 tokens of 4 heads, outputs): 2.0e-7 where
// the decays are close to one (token by token 6.2e-7), 1.3e-7 where they are fast (0.9e-7 to 1.1e-7).
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

namespace {

constexpr int PC = 64;
constexpr int THREADS = 256;
constexpr int VC = 32;                    // columns per block of ssd_state_kernel
constexpr double LOG2E = 1.4426950408889634;

__device__ __forceinline__ float ldw(const void* p, int dt, size_t i) {
    return dt == GFB_BF16 ? __bfloat162float(((const __nv_bfloat16*)p)[i]) : ((const float*)p)[i];
}
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// 16 bytes from global to shared memory, or zeros
__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool live) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(gmem), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct ChunkWork { int seq, t0, n; };

// chunks are numbered through the batch, sequence after sequence
__device__ __forceinline__ bool chunk_work(const GfbBatch& b, int w, ChunkWork& c) {
    int left = w;
    for (int i = 0; i < b.n_seqs; i++) {
        const int q0 = b.cu_seqlens[i], qlen = b.cu_seqlens[i + 1] - q0;
        const int nc = (qlen + PC - 1) / PC;
        if (left < nc) {
            c.seq = i;
            c.t0 = q0 + left * PC;
            c.n = min(PC, qlen - left * PC);
            return true;
        }
        left -= nc;
    }
    return false;
}

// A chunk's scratch, in floats: per group the scores, transposed ([j][i]), and C transposed ([N][PC]); per head S_0 [N][P]
struct Sizes {
    int H, P, N, G;
    __host__ __device__ size_t scores(int g) const { return (size_t)g * (PC * PC + N * PC); }
    __host__ __device__ size_t c_t(int g) const { return scores(g) + PC * PC; }
    __host__ __device__ size_t s0(int h) const { return scores(G) + (size_t)h * N * P; }
    __host__ __device__ size_t all() const { return s0(H); }
};

// dt [PC] and L [PC] of a chunk by one warp (every lane two neighbouring tokens; tokens beyond the chunk have dt = 0)
template <typename TD>
__device__ __forceinline__ void chunk_decays(const TD* __restrict__ dt_raw, int ld_dt, int col, int t0, int n, float bias, double rate, int lane,
                                             float* dt, double* L) {
    float d[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int j = 2 * lane + k;
        d[k] = j < n ? softplus_f(gfb_to_f32(dt_raw[(size_t)(t0 + j) * ld_dt + col]) + bias) : 0.f;
        dt[j] = d[k];
    }
    const double a0 = -rate * (double)d[0], a1 = a0 - rate * (double)d[1];
    double run = a1;                                 // sum up to and with this lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
    }
    const double before = run - a1;
    L[2 * lane] = before + a0;
    L[2 * lane + 1] = run;
}

template <int N>
__global__ void __launch_bounds__(THREADS)
ssd_scores_kernel(const float* __restrict__ x, int ldx, int b_off, int c_off, float* __restrict__ scratch, GfbBatch b, int first_chunk, Sizes z) {
    extern __shared__ __align__(16) float sm[];
    float(*Bs)[N + 4] = reinterpret_cast<float(*)[N + 4]>(sm);                  // [PC]
    float(*Cs)[N + 4] = reinterpret_cast<float(*)[N + 4]>(sm + PC * (N + 4));   // [16]
    gfb_pdl_launch();
    gfb_pdl_wait();
    ChunkWork c;
    if (!chunk_work(b, first_chunk + blockIdx.x, c)) return;
    const int g = blockIdx.y, i0 = blockIdx.z * 16, tid = threadIdx.x;
    float* mine = scratch + (size_t)blockIdx.x * z.all();
    for (int e = tid; e < (PC + 16) * (N / 4); e += THREADS) {
        const int r = e / (N / 4), p = (e - r * (N / 4)) * 4;
        const int j = r < PC ? r : i0 + r - PC;
        const bool live = j < c.n;
        const float* row = x + (size_t)(c.t0 + (live ? j : 0)) * ldx;
        if (r < PC) copy16(&Bs[r][p], row + b_off + g * N + p, live);
        else copy16(&Cs[r - PC][p], row + c_off + g * N + p, live);
    }
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    const int i = tid & 15, jg = tid >> 4;
    float4 acc[4];                                   // four sums per score, of every fourth term
#pragma unroll
    for (int r = 0; r < 4; r++) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < N; k += 4) {
        const float4 cv = ld4(&Cs[i][k]);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float4 bv = ld4(&Bs[jg + 16 * r][k]);
            acc[r].x = fmaf(cv.x, bv.x, acc[r].x); acc[r].y = fmaf(cv.y, bv.y, acc[r].y);
            acc[r].z = fmaf(cv.z, bv.z, acc[r].z); acc[r].w = fmaf(cv.w, bv.w, acc[r].w);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++) mine[z.scores(g) + (size_t)(jg + 16 * r) * PC + i0 + i] = (acc[r].x + acc[r].y) + (acc[r].z + acc[r].w);
    for (int k = jg; k < N; k += 16) mine[z.c_t(g) + (size_t)k * PC + i0 + i] = Cs[i][k];
}

// A thread has 4 state rows x 4 columns of S in registers, a warp 32 x 16; two stages of B and x, so that the next chunk's copies run under
// the current one's products.
template <int N>
struct StateSmem {
    float B[2][PC][N];
    float X[2][PC][VC];
    float w[2][PC];
    float dt[PC];
    double L[PC];
    float decay[2];
};

template <typename TD, int N>
__global__ void __launch_bounds__(N * VC / 16)
ssd_state_kernel(const float* __restrict__ x, int ldx, int b_off, const TD* __restrict__ dt_raw, int ld_dt, int dt_off, const void* __restrict__ dt_bias,
                 const void* __restrict__ a_log, int w_dt, float* __restrict__ scratch, float* __restrict__ state, size_t state_ld, GfbBatch b,
                 int first_chunk, int n_chunks, Sizes z) {
    constexpr int NT = N * VC / 16;                  // threads
    extern __shared__ __align__(16) unsigned char raw[];
    StateSmem<N>& sm = *reinterpret_cast<StateSmem<N>*>(raw);
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int s = blockIdx.x, h = blockIdx.y, p0 = blockIdx.z * VC, g = h / (z.H / z.G);
    int seq0 = 0;
    for (int i = 0; i < s; i++) seq0 += (b.cu_seqlens[i + 1] - b.cu_seqlens[i] + PC - 1) / PC;
    const int q0 = b.cu_seqlens[s], qlen = b.cu_seqlens[s + 1] - q0;
    const int lo = max(seq0, first_chunk), hi = min(seq0 + (qlen + PC - 1) / PC, first_chunk + n_chunks);
    if (lo >= hi) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a warp: 8 groups of four rows x 4 groups of four columns
    const int n0 = (warp >> 1) * 32 + (lane >> 2) * 4, c0 = (warp & 1) * 16 + (lane & 3) * 4;
    const float bias = ldw(dt_bias, w_dt, h);
    const double rate = (double)expf(ldw(a_log, w_dt, h)) * LOG2E;
    float* Sg = state + (size_t)b.slots[s] * state_ld + (size_t)h * N * z.P + p0;
    float S[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) S[i][j] = Sg[(size_t)(n0 + i) * z.P + c0 + j];
    auto fetch = [&](int st, int w) {
        const int t0 = q0 + (w - seq0) * PC, n = min(PC, qlen - (w - seq0) * PC);
        for (int e = tid; e < PC * (N / 4); e += NT) {
            const int j = e / (N / 4), p = (e - j * (N / 4)) * 4;
            copy16(&sm.B[st][j][p], x + (size_t)(t0 + min(j, n - 1)) * ldx + b_off + g * N + p, j < n);
        }
        for (int e = tid; e < PC * (VC / 4); e += NT) {
            const int j = e / (VC / 4), p = (e - j * (VC / 4)) * 4;
            copy16(&sm.X[st][j][p], x + (size_t)(t0 + min(j, n - 1)) * ldx + (size_t)h * z.P + p0 + p, j < n);
        }
        copy_commit();
        if (warp == 0) {
            chunk_decays(dt_raw, ld_dt, dt_off + h, t0, n, bias, rate, lane, sm.dt, sm.L);
            __syncwarp();
            const double end = sm.L[PC - 1];
#pragma unroll
            for (int k = 0; k < 2; k++) sm.w[st][2 * lane + k] = sm.dt[2 * lane + k] * exp2f((float)(end - sm.L[2 * lane + k]));
            if (lane == 0) sm.decay[st] = exp2f((float)end);
            __syncwarp();
        }
    };
    fetch(0, lo);
    int st = 0;
    for (int w = lo; w < hi; w++, st ^= 1) {
        float* S0 = scratch + (size_t)(w - first_chunk) * z.all() + z.s0(h) + p0;
#pragma unroll
        for (int i = 0; i < 4; i++) *reinterpret_cast<float4*>(S0 + (size_t)(n0 + i) * z.P + c0) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
        copy_wait<0>();
        __syncthreads();                             // this chunk's inputs have landed; everybody is done with the other stage
        if (w + 1 < hi) fetch(st ^ 1, w + 1);
        const float d = sm.decay[st];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) S[i][j] *= d;
#pragma unroll 8
        for (int t = 0; t < PC; t++) {
            const float4 bv = ld4(&sm.B[st][t][n0]);
            float4 xv = ld4(&sm.X[st][t][c0]);
            const float wt = sm.w[st][t];
            xv.x *= wt; xv.y *= wt; xv.z *= wt; xv.w *= wt;
            const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                S[i][0] = fmaf(br[i], xv.x, S[i][0]); S[i][1] = fmaf(br[i], xv.y, S[i][1]);
                S[i][2] = fmaf(br[i], xv.z, S[i][2]); S[i][3] = fmaf(br[i], xv.w, S[i][3]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) Sg[(size_t)(n0 + i) * z.P + c0 + j] = S[i][j];
}

// Tokens x columns, 64 x 64 per block: four warps of 32 x 32, a lane has 8 x 4 sums in two groups of four rows.  First C S_0 (both k-major, 32
// state rows per stage, two stages), then the rows' decays, then the scores against the chunk's x.
constexpr int OUT_THREADS = 128, OK = 32;
struct OutSmem {
    float X[2][OK][PC], Z[2][OK][64];
    float dt[PC];
    double L[PC];
};

template <typename TD>
__global__ void __launch_bounds__(OUT_THREADS)
ssd_out_kernel(const float* __restrict__ x, int ldx, const TD* __restrict__ dt_raw, int ld_dt, int dt_off, const void* __restrict__ dt_bias,
               const void* __restrict__ a_log, const void* __restrict__ skip, int w_dt, const float* __restrict__ scratch, float* __restrict__ out,
               GfbBatch b, int first_chunk, Sizes z) {
    __shared__ __align__(16) OutSmem sm;
    gfb_pdl_launch();
    gfb_pdl_wait();
    ChunkWork c;
    if (!chunk_work(b, first_chunk + blockIdx.x, c)) return;
    const int h = blockIdx.y, v0 = blockIdx.z * 64, g = h / (z.H / z.G), N = z.N;
    const float* mine = scratch + (size_t)blockIdx.x * z.all();
    const float *CT = mine + z.c_t(g), *S0 = mine + z.s0(h) + v0, *scores = mine + z.scores(g);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = (warp & 1) * 32 + (lane >> 3) * 4, c0 = (warp >> 1) * 32 + (lane & 7) * 4;
    const float* xg = x + (size_t)h * z.P + v0;
    // stages: N / 32 of state rows, then two of the chunk's tokens (their scores are made below, behind the decays)
    auto fetch = [&](int st, int k0) {
#pragma unroll
        for (int e = tid; e < OK * 16; e += OUT_THREADS) {
            const int k = e >> 4, p = (e & 15) * 4;
            if (k0 < N) {
                copy16(&sm.X[st][k][p], CT + (size_t)(k0 + k) * PC + p, true);
                copy16(&sm.Z[st][k][p], S0 + (size_t)(k0 + k) * z.P + p, true);
            } else {
                const int j = k0 - N + k;
                copy16(&sm.X[st][k][p], scores + (size_t)j * PC + p, true);
                copy16(&sm.Z[st][k][p], xg + (size_t)(c.t0 + min(j, c.n - 1)) * ldx + p, j < c.n);
            }
        }
        copy_commit();
    };
    fetch(0, 0);
    if (warp == 0)
        chunk_decays(dt_raw, ld_dt, dt_off + h, c.t0, c.n, ldw(dt_bias, w_dt, h), (double)expf(ldw(a_log, w_dt, h)) * LOG2E, lane, sm.dt, sm.L);
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    int st = 0;
    for (int k0 = 0; k0 < N + PC; k0 += OK, st ^= 1) {
        copy_wait<0>();
        __syncthreads();
        if (k0 + OK < N + PC) fetch(st ^ 1, k0 + OK);
        if (k0 >= N) {
            // scores of tokens j = k0 - N .. + 31 become (C_i . B_j) 2^(L_i - L_j) dt_j, zero ahead of the diagonal
            for (int e = tid; e < OK * PC; e += OUT_THREADS) {
                const int k = e >> 6, i = e & 63, j = k0 - N + k;
                sm.X[st][k][i] = i >= j ? sm.X[st][k][i] * (exp2f((float)(sm.L[i] - sm.L[j])) * sm.dt[j]) : 0.f;
            }
            if (k0 == N) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float d = exp2f((float)sm.L[r0 + (i & 3) + 16 * (i >> 2)]);
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] *= d;
                }
            }
            __syncthreads();
        }
        float part[8][4];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) part[i][j] = 0.f;
#pragma unroll 8
        for (int k = 0; k < OK; k++) {
            const float4 a = ld4(&sm.X[st][k][r0]), a2 = ld4(&sm.X[st][k][r0 + 16]), v = ld4(&sm.Z[st][k][c0]);
            const float av[8] = {a.x, a.y, a.z, a.w, a2.x, a2.y, a2.z, a2.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                part[i][0] = fmaf(av[i], v.x, part[i][0]); part[i][1] = fmaf(av[i], v.y, part[i][1]);
                part[i][2] = fmaf(av[i], v.z, part[i][2]); part[i][3] = fmaf(av[i], v.w, part[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] += part[i][j];
    }
    const float dskip = skip != nullptr ? ldw(skip, w_dt, h) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = r0 + (i & 3) + 16 * (i >> 2);
        if (row >= c.n) continue;
        const float4 xv = ld4(xg + (size_t)(c.t0 + row) * ldx + c0);
        *reinterpret_cast<float4*>(out + ((size_t)(c.t0 + row) * z.H + h) * z.P + v0 + c0) =
            make_float4(fmaf(dskip, xv.x, acc[i][0]), fmaf(dskip, xv.y, acc[i][1]), fmaf(dskip, xv.z, acc[i][2]), fmaf(dskip, xv.w, acc[i][3]));
    }
}

// chunks that are in flight together: their scratch stays below 256 MB (2,048 tokens of 64 heads of 128 x 64 take 70), or is one chunk's
long chunks_at_once(int n_tokens, int n_seqs, const Sizes& z) {
    const long all = (long)n_tokens / PC + n_seqs;               // an upper bound; surplus blocks find no work
    const long most = (256L << 20) / (long)(z.all() * sizeof(float));
    return all < most ? all : (most > 0 ? most : 1);
}

}  // namespace

// Floats of scratch of gfb_ssd_chunks.
GFB_API long gfb_ssd_chunks_scratch_floats(int n_tokens, int n_seqs, int H, int P, int N, int G) {
    const Sizes z{H, P, N, G};
    return chunks_at_once(n_tokens, n_seqs, z) * (long)z.all();
}

// As gfb_ssd_scan (whose arguments these are), for states of 64 or 128 rows and a multiple of 64 columns; x with 16-byte aligned rows,
// B and C, out and scratch 16-byte aligned.
GFB_API int gfb_ssd_chunks(const float* x, int ldx, int b_off, int c_off, const void* dt_raw, int dt_dt, int ld_dt, int dt_off, const void* dt_bias,
                           const void* a_log, const void* skip, int w_dt, float* state, long state_ld, float* out, float* scratch,
                           const int* cu_seqlens, const int* tok_seq, const int* slots, const int* lengths, int n_seqs, int n_tokens, int H, int P,
                           int N, int G, cudaStream_t stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (G <= 0 || H % G) return gfb_fail("gfb_ssd_chunks: %d heads do not divide into %d groups", H, G);
    if ((N != 64 && N != 128) || P < 64 || P % 64) return gfb_fail("gfb_ssd_chunks: states of %d x %d", N, P);
    if (H > 65535 || G > 65535 || P / VC > 65535) return gfb_fail("gfb_ssd_chunks: %d heads of %d columns exceed the grid limit", H, P);
    if (ldx % 4 || b_off % 4 || c_off % 4 || (((uintptr_t)x | (uintptr_t)out | (uintptr_t)scratch) & 15))
        return gfb_fail("gfb_ssd_chunks: rows, B and C, output and scratch must be 16-byte aligned");
    const Sizes z{H, P, N, G};
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    typedef __nv_bfloat16 bf16;
    const size_t score_smem = (size_t)(PC + 16) * (N + 4) * sizeof(float);
    cudaError_t e = cudaSuccess;
#define ALLOW(K, bytes) if (e == cudaSuccess) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))
    if (N == 128) {
        ALLOW(ssd_scores_kernel<128>, score_smem);
        if (dt_dt == GFB_BF16) { ALLOW((ssd_state_kernel<bf16, 128>), sizeof(StateSmem<128>)); }
        else { ALLOW((ssd_state_kernel<float, 128>), sizeof(StateSmem<128>)); }
    } else {
        if (dt_dt == GFB_BF16) { ALLOW((ssd_state_kernel<bf16, 64>), sizeof(StateSmem<64>)); }
        else { ALLOW((ssd_state_kernel<float, 64>), sizeof(StateSmem<64>)); }
    }
#undef ALLOW
    if (e != cudaSuccess) return gfb_fail("gfb_ssd_chunks: %s", cudaGetErrorString(e));
    if (dt_dt != GFB_BF16 && dt_dt != GFB_F32) return gfb_fail("gfb_ssd_chunks: unknown type %d", dt_dt);
    const long all = (long)n_tokens / PC + n_seqs, step = chunks_at_once(n_tokens, n_seqs, z);
    for (long first = 0; first < all; first += step) {
        const int n = (int)(all - first < step ? all - first : step);
        const dim3 sgrid(n_seqs, H, P / VC), ogrid(n, H, P / 64);
        e = N == 128 ? gfb_launch(ssd_scores_kernel<128>, dim3(n, G, PC / 16), dim3(THREADS), score_smem, stream, x, ldx, b_off, c_off, scratch, b, (int)first, z)
                     : gfb_launch(ssd_scores_kernel<64>, dim3(n, G, PC / 16), dim3(THREADS), score_smem, stream, x, ldx, b_off, c_off, scratch, b, (int)first, z);
#define STATE(TD, N_)                                                                                                                                    \
    if (e == cudaSuccess)                                                                                                                                \
        e = gfb_launch(ssd_state_kernel<TD, N_>, sgrid, dim3(N_ * VC / 16), sizeof(StateSmem<N_>), stream, x, ldx, b_off, (const TD*)dt_raw, ld_dt, dt_off,    \
                       dt_bias, a_log, w_dt, scratch, state, (size_t)state_ld, b, (int)first, n, z)
#define OUT(TD)                                                                                                                                          \
    if (e == cudaSuccess)                                                                                                                                \
        e = gfb_launch(ssd_out_kernel<TD>, ogrid, dim3(OUT_THREADS), 0, stream, x, ldx, (const TD*)dt_raw, ld_dt, dt_off, dt_bias, a_log, skip, w_dt,     \
                       (const float*)scratch, out, b, (int)first, z)
        if (dt_dt == GFB_BF16) {
            if (N == 128) { STATE(bf16, 128); } else { STATE(bf16, 64); }
            OUT(bf16);
        } else {
            if (N == 128) { STATE(float, 128); } else { STATE(float, 64); }
            OUT(float);
        }
#undef STATE
#undef OUT
        if (gfb_check(e, "gfb_ssd_chunks")) return 1;
    }
    return 0;
}
