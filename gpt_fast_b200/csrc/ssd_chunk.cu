// The selective state space over prompts, in chunks of PC = 64 tokens (gfb_ssd_scan walks token by token):
//
//     dt_t = softplus(dt_raw_t + dt_bias_h);  S_t = 2^(a_t) S_(t-1) + dt_t B_t x_t^T,  a_t = -exp(A_log_h) log2(e) dt_t;  y_t = S_t^T C_t + D_h x_t
//
// With L_i the sum of a over the chunk's tokens up to i and S_0 the state ahead of the chunk,
//
//     y_i = 2^(L_i) S_0^T C_i + sum_(j<=i) (C_i . B_j) 2^(L_i - L_j) dt_j x_j + D_h x_i,     S_0' = 2^(L_end) S_0 + sum_j 2^(L_end - L_j) dt_j B_j x_j^T
//
// Four launches:
//   ssd_scores_kernel   a block per (chunk, group, 16 tokens): C_i . B_j, which all heads of a group share, C transposed, and the heads' factors
//   ssd_add_kernel      a block per (chunk, head, 64 rows, 64 columns): what the chunk adds to the state
//   ssd_state_kernel    four numbers of a (sequence, head)'s state per thread walk over the chunks and leave the S_0s
//   ssd_out_kernel      a block per (chunk, head, 64 columns): one product with K = state rows + 64
//
// Everything is 32-bit FMAs; the sums L and their differences are 64-bit (64 numbers per chunk and head), so that a decay between two tokens
// is as exact as its exponent, however much has decayed before them.  Long sums run in pieces of 32 terms that are then added, as the
// token-by-token kernel's lanes do, which keeps their rounding where it was.
//
// What bounds it: the token-by-token kernel is a chain of dependent instructions per token (sequences of 77, 788 and 1,500 tokens,
// 64 heads of 128 x 64: 1,135 us).  Here 2.4 GFMA and the S_0s' way through L2: about 230 us (alone and with cold caches ssd_scores_kernel 18,
// ssd_add_kernel 77, ssd_state_kernel 69, ssd_out_kernel 123).  With the state in a block's registers, walking over a sequence's chunks as it
// added them up, the longest sequence's 24 chunks took 6.5 us each on less than a block per SM: 274 us.  Against 64-bit sums (700 tokens of
// 4 heads, outputs): 1.7e-7 where the decays are close to one (token by token 6.2e-7), 0.7e-7 to 0.9e-7 where they are fast (0.9e-7 to
// 1.1e-7), 0.8e-7 to 1.1e-7 with steps of 0.001 to 0.1 and A of 1 to 16 (1.1e-7 to 1.4e-7).
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

namespace {

constexpr int PC = 64;
constexpr int THREADS = 256;
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

// A chunk's scratch, in floats: per group the scores, transposed ([j][i]), and C transposed ([N][PC]); per head the tokens' factors
// 2^(L_end - L_j) dt_j, the chunk's decay behind them, and S_0 [N][P]
constexpr int WD = PC + 4;
struct Sizes {
    int H, P, N, G;
    __host__ __device__ size_t scores(int g) const { return (size_t)g * (PC * PC + N * PC); }
    __host__ __device__ size_t c_t(int g) const { return scores(g) + PC * PC; }
    __host__ __device__ size_t w(int h) const { return scores(G) + (size_t)h * WD; }
    __host__ __device__ size_t s0(int h) const { return w(H) + (size_t)h * N * P; }
    __host__ __device__ size_t all() const { return s0(H); }
};

// The exponent of a token's decay.  2^-4096 is zero against any 32-bit number, so a decay that forgets everything is that: an infinite one
// (A_log above 88) would leave its sums, and the differences of them, without a value.  (Not a number stays that.)
__device__ __forceinline__ double decay_exponent(double rate, float dt) {
    const double a = -rate * (double)dt;
    return a < -4096.0 ? -4096.0 : a;
}

// dt [PC] and L [PC] of a chunk by one warp (every lane two neighbouring tokens; tokens beyond the chunk have dt = 0 and decay by nothing)
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
    const double a0 = 2 * lane < n ? decay_exponent(rate, d[0]) : 0.0;
    double run = a0 + (2 * lane + 1 < n ? decay_exponent(rate, d[1]) : 0.0);        // sum up to and with this lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
    }
    const double before = __shfl_up_sync(0xffffffffu, run, 1);      // (not run minus this lane's: the second token is not the first one's affair)
    L[2 * lane] = (lane > 0 ? before : 0.0) + a0;
    L[2 * lane + 1] = run;
}

template <typename TD, int N>
__global__ void __launch_bounds__(THREADS)
ssd_scores_kernel(const float* __restrict__ x, int ldx, int b_off, int c_off, const TD* __restrict__ dt_raw, int ld_dt, int dt_off,
                  const void* __restrict__ dt_bias, const void* __restrict__ a_log, int w_dt, float* __restrict__ scratch, GfbBatch b, int first_chunk,
                  Sizes z) {
    extern __shared__ __align__(16) float sm[];
    __shared__ double sL[THREADS / 32][PC];
    __shared__ float sDt[THREADS / 32][PC];
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
    // meanwhile the factors of the group's heads, a warp per head, dealt to the chunk's four blocks
    const int lane = tid & 31, warp = tid >> 5, per_group = z.H / z.G;
    for (int k = blockIdx.z * (THREADS / 32) + warp; k < per_group; k += PC / 16 * (THREADS / 32)) {
        const int h = g * per_group + k;
        chunk_decays(dt_raw, ld_dt, dt_off + h, c.t0, c.n, ldw(dt_bias, w_dt, h), (double)expf(ldw(a_log, w_dt, h)) * LOG2E, lane, sDt[warp], sL[warp]);
        __syncwarp();
        const double end = sL[warp][PC - 1];
        float* w = mine + z.w(h);
#pragma unroll
        for (int q = 0; q < 2; q++) w[lane + 32 * q] = sDt[warp][lane + 32 * q] * exp2f((float)(end - sL[warp][lane + 32 * q]));
        if (lane == 0) w[PC] = exp2f((float)end);
        __syncwarp();
    }
    copy_wait<0>();
    __syncthreads();
    const int i = tid & 15, jg = tid >> 4;
    // The scores are sums of N terms that every later step multiplies, so they are made in 64 bits and rounded once: with 32-bit sums of 32
    // terms the outputs were a fifth to two fifths further from 64 bits than token by token where decays are fast.
    double acc[4][2];
#pragma unroll
    for (int r = 0; r < 4; r++) acc[r][0] = acc[r][1] = 0.0;
#pragma unroll 2
    for (int k = 0; k < N; k += 4) {
        const float4 cv = ld4(&Cs[i][k]);
        const double c0 = cv.x, c1 = cv.y, c2 = cv.z, c3 = cv.w;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float4 bv = ld4(&Bs[jg + 16 * r][k]);
            acc[r][0] = fma(c0, (double)bv.x, acc[r][0]); acc[r][1] = fma(c1, (double)bv.y, acc[r][1]);
            acc[r][0] = fma(c2, (double)bv.z, acc[r][0]); acc[r][1] = fma(c3, (double)bv.w, acc[r][1]);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++) mine[z.scores(g) + (size_t)(jg + 16 * r) * PC + i0 + i] = (float)(acc[r][0] + acc[r][1]);
    for (int k = jg; k < N; k += 16) mine[z.c_t(g) + (size_t)k * PC + i0 + i] = Cs[i][k];
}

// What a chunk adds to the state, all chunks side by side: dS = sum_j B_j (w_j x_j)^T into S_0's place, 64 rows x 64 columns per block, four warps of
// 32 x 32, a lane 8 x 4 sums in two groups of four rows; 32 tokens per stage, two stages.
constexpr int ADD_THREADS = 128, HC = PC / 2;

__global__ void __launch_bounds__(ADD_THREADS)
ssd_add_kernel(const float* __restrict__ x, int ldx, int b_off, float* __restrict__ scratch, GfbBatch b, int first_chunk, Sizes z) {
    __shared__ __align__(16) float B[2][HC][64], X[2][HC][64], w[PC];
    gfb_pdl_launch();
    gfb_pdl_wait();
    ChunkWork c;
    if (!chunk_work(b, first_chunk + blockIdx.x, c)) return;
    const int h = blockIdx.y, g = h / (z.H / z.G), n0 = (int)blockIdx.z % (z.N / 64) * 64, p0 = (int)blockIdx.z / (z.N / 64) * 64;
    float* mine = scratch + (size_t)blockIdx.x * z.all();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = (warp & 1) * 32 + (lane >> 3) * 4, c0 = (warp >> 1) * 32 + (lane & 7) * 4;
    const float *bx = x + b_off + g * z.N + n0, *xx = x + (size_t)h * z.P + p0;
    auto fetch = [&](int st, int j0) {
#pragma unroll
        for (int i = 0; i < HC * 16 / ADD_THREADS; i++) {
            const int e = tid + ADD_THREADS * i, k = e >> 4, p = (e & 15) * 4, j = j0 + k;
            const size_t row = (size_t)(c.t0 + (j < c.n ? j : 0)) * ldx;
            copy16(&B[st][k][p], bx + row + p, j < c.n);
            copy16(&X[st][k][p], xx + row + p, j < c.n);
        }
        copy_commit();
    };
    fetch(0, 0);
    if (tid < PC) w[tid] = mine[z.w(h) + tid];
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
#pragma unroll
    for (int st = 0; st < 2; st++) {
        if (st == 0) { fetch(1, HC); copy_wait<1>(); } else copy_wait<0>();
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < HC; k++) {
            const float4 a = ld4(&B[st][k][r0]), a2 = ld4(&B[st][k][r0 + 16]);
            float4 v = ld4(&X[st][k][c0]);
            const float wk = w[st * HC + k];
            v.x *= wk; v.y *= wk; v.z *= wk; v.w *= wk;
            const float av[8] = {a.x, a.y, a.z, a.w, a2.x, a2.y, a2.z, a2.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                acc[i][0] = fmaf(av[i], v.x, acc[i][0]); acc[i][1] = fmaf(av[i], v.y, acc[i][1]);
                acc[i][2] = fmaf(av[i], v.z, acc[i][2]); acc[i][3] = fmaf(av[i], v.w, acc[i][3]);
            }
        }
    }
    float* S0 = mine + z.s0(h) + p0 + c0;
#pragma unroll
    for (int i = 0; i < 8; i++)
        *reinterpret_cast<float4*>(S0 + (size_t)(n0 + r0 + (i & 3) + 16 * (i >> 2)) * z.P) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// The walk over a sequence's chunks, four numbers of the state per thread: S_0 of a chunk takes the place of what the chunk adds, S <- decay S + dS.
// Bound by that traffic; AHEAD chunks' loads are in flight together (sequences of 77, 788 and 1,500 tokens, 64 heads of 128 x 64: four 66 us, eight 55).
constexpr int AHEAD = 8;

__global__ void __launch_bounds__(THREADS)
ssd_state_kernel(float* scratch, float* __restrict__ state, size_t state_ld, GfbBatch b, int first_chunk, int n_chunks, Sizes z) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int s = blockIdx.x, h = blockIdx.y, at = (blockIdx.z * THREADS + threadIdx.x) * 4;
    int seq0 = 0;
    for (int i = 0; i < s; i++) seq0 += (b.cu_seqlens[i + 1] - b.cu_seqlens[i] + PC - 1) / PC;
    const int lo = max(seq0, first_chunk), hi = min(seq0 + (b.cu_seqlens[s + 1] - b.cu_seqlens[s] + PC - 1) / PC, first_chunk + n_chunks);
    if (lo >= hi || at >= z.N * z.P) return;
    float* Sg = state + (size_t)b.slots[s] * state_ld + (size_t)h * z.N * z.P + at;      // (of any alignment)
    float4 S = make_float4(Sg[0], Sg[1], Sg[2], Sg[3]);
    for (int w0 = lo; w0 < hi; w0 += AHEAD) {
        float4 add[AHEAD];
        float d[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const float* m = scratch + (size_t)(min(w0 + i, hi - 1) - first_chunk) * z.all();
            add[i] = ld4(m + z.s0(h) + at);
            d[i] = m[z.w(h) + PC];
        }
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            if (w0 + i >= hi) break;
            *reinterpret_cast<float4*>(scratch + (size_t)(w0 + i - first_chunk) * z.all() + z.s0(h) + at) = S;
            S = make_float4(fmaf(S.x, d[i], add[i].x), fmaf(S.y, d[i], add[i].y), fmaf(S.z, d[i], add[i].z), fmaf(S.w, d[i], add[i].w));
        }
    }
    Sg[0] = S.x; Sg[1] = S.y; Sg[2] = S.z; Sg[3] = S.w;
}

// Tokens x columns, 64 x 64 per block: four warps of 32 x 32, a lane has 8 x 4 sums in two groups of four rows.  First C S_0 (both k-major, 32
// state rows per stage, two stages), then the rows' decays, then the scores against the chunk's x.
constexpr int OUT_THREADS = 128, OK = 32;
struct OutSmem {
    float X[2][OK][PC], Z[2][OK][64];
    float dt[PC];
    double L[PC];
};

// One output number ahead of the skip, over the tokens up to its own only; sums in ssd_out_kernel's order.
__device__ __noinline__ float out_number(const float* CT, const float* S0, const float* scores, const float* x, int ldx, const double* L, const float* dt,
                                         int row, int N, int P) {
    float acc = 0.f;
    for (int k0 = 0; k0 < N; k0 += OK) {
        float part = 0.f;
        for (int k = k0; k < k0 + OK; k++) part = fmaf(CT[(size_t)k * PC + row], S0[(size_t)k * P], part);
        acc += part;
    }
    acc = __fmul_rn(acc, exp2f((float)L[row]));             // (not an FMA with the first sum below)
    for (int j0 = 0; j0 <= row; j0 += OK) {
        float part = 0.f;
        for (int j = j0; j < j0 + OK && j <= row; j++)
            part = fmaf(scores[(size_t)j * PC + row] * (exp2f((float)(L[row] - L[j])) * dt[j]), x[(size_t)j * ldx], part);
        acc += part;
    }
    return acc;
}

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
    // The zeros ahead of the diagonal meet later tokens' x above: one that is not finite makes NaN of them.  Such a block (and one whose own
    // numbers are not finite) works its numbers out once more, each from the tokens up to its own.
    bool odd = false;
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) odd |= r0 + (i & 3) + 16 * (i >> 2) < c.n && !(fabsf(acc[i][j]) <= 3.4028235e38f);
    if (__syncthreads_or(odd)) {
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int row = r0 + (i & 3) + 16 * (i >> 2);
                if (row < c.n) acc[i][j] = out_number(CT, S0 + c0 + j, scores, xg + (size_t)c.t0 * ldx + c0 + j, ldx, sm.L, sm.dt, row, N, z.P);
            }
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
    if (H > 65535 || G > 65535 || P / 8 > 65535) return gfb_fail("gfb_ssd_chunks: %d heads of %d columns exceed the grid limit", H, P);
    if (ldx % 4 || b_off % 4 || c_off % 4 || (((uintptr_t)x | (uintptr_t)out | (uintptr_t)scratch) & 15))
        return gfb_fail("gfb_ssd_chunks: rows, B and C, output and scratch must be 16-byte aligned");
    const Sizes z{H, P, N, G};
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    typedef __nv_bfloat16 bf16;
    const size_t score_smem = (size_t)(PC + 16) * (N + 4) * sizeof(float);
    cudaError_t e = cudaSuccess;
#define ALLOW(K, bytes) if (e == cudaSuccess) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))
    if (N == 128) {
        if (dt_dt == GFB_BF16) { ALLOW((ssd_scores_kernel<bf16, 128>), score_smem); }
        else { ALLOW((ssd_scores_kernel<float, 128>), score_smem); }
    }
#undef ALLOW
    if (e != cudaSuccess) return gfb_fail("gfb_ssd_chunks: %s", cudaGetErrorString(e));
    if (dt_dt != GFB_BF16 && dt_dt != GFB_F32) return gfb_fail("gfb_ssd_chunks: unknown type %d", dt_dt);
    const long all = (long)n_tokens / PC + n_seqs, step = chunks_at_once(n_tokens, n_seqs, z);
    for (long first = 0; first < all; first += step) {
        const int n = (int)(all - first < step ? all - first : step);
        const dim3 ogrid(n, H, P / 64);
#define SCORES(TD, N_)                                                                                                                                   \
    e = gfb_launch(ssd_scores_kernel<TD, N_>, dim3(n, G, PC / 16), dim3(THREADS), score_smem, stream, x, ldx, b_off, c_off, (const TD*)dt_raw, ld_dt, dt_off, \
                   dt_bias, a_log, w_dt, scratch, b, (int)first, z)
#define OUT(TD)                                                                                                                                          \
    if (e == cudaSuccess)                                                                                                                                \
        e = gfb_launch(ssd_out_kernel<TD>, ogrid, dim3(OUT_THREADS), 0, stream, x, ldx, (const TD*)dt_raw, ld_dt, dt_off, dt_bias, a_log, skip, w_dt,     \
                       (const float*)scratch, out, b, (int)first, z)
        if (N == 128) { if (dt_dt == GFB_BF16) SCORES(bf16, 128); else SCORES(float, 128); }
        else { if (dt_dt == GFB_BF16) SCORES(bf16, 64); else SCORES(float, 64); }
        if (e == cudaSuccess) e = gfb_launch(ssd_add_kernel, dim3(n, H, N / 64 * (P / 64)), dim3(ADD_THREADS), 0, stream, x, ldx, b_off, scratch, b, (int)first, z);
        if (e == cudaSuccess)
            e = gfb_launch(ssd_state_kernel, dim3(n_seqs, H, (N * P / 4 + THREADS - 1) / THREADS), dim3(THREADS), 0, stream, scratch, state, (size_t)state_ld, b,
                           (int)first, n, z);
        if (dt_dt == GFB_BF16) { OUT(bf16); } else { OUT(float); }
#undef SCORES
#undef OUT
        if (gfb_check(e, "gfb_ssd_chunks")) return 1;
    }
    return 0;
}
