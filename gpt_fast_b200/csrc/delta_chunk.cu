// The gated delta rule over prompts, in chunks of PC = 64 tokens (gfb_delta_rule walks token by token):
//
//     S <- diag(g_t) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t          per head, S [d][dv]
//
// with q and k unit vectors (q also times q_scale), beta = sigmoid(.), g = exp(-exp(A_log) softplus(a + dt_bias)) per key channel, or per
// head.  With G_i the sum of log2 g over the chunk's tokens up to i and S_0 the state ahead of the chunk, unrolling the recurrence gives
//
//     (I + diag(beta) A) U = diag(beta) (V - Kt S_0),   A_ij = sum_c k_ic k_jc 2^(G_ic - G_jc) for j < i,   Kt_i = k_i 2^(G_i)
//     o_i = Qt_i S_0 + sum_(j<=i) B_ij u_j,             B_ij = sum_c q_ic k_jc 2^(G_ic - G_jc),             Qt_i = q_i 2^(G_i)
//     S_0' = diag(2^(G_end)) S_0 + Kh^T U,              Kh_j = k_j 2^(G_end - G_j)
//
// (the WY form of the products of (I - beta k k^T) diag(g)).  So with T = (I + diag(beta) A)^-1, W = T diag(beta) Kt and Y = T diag(beta) V,
// which depend on no state, only U = Y - W S_0 and S_0' remain to be done chunk after chunk.  Three launches:
//
//   delta_chunk_kernel   a block per (chunk, head), all side by side: norms, decays, A, B, T, W, Y, Kh, Qt
//   delta_scan_kernel    a block per (sequence, head, 16 value columns) walks over the chunks: two small products per chunk
//   delta_out_kernel     a block per (chunk, head, 64 value columns): o = [Qt | B] [S_0 ; U], one product with K = d + 64
//
// Everything is 32-bit FMAs.  No power with a positive exponent is taken, whatever the decays: G runs within sub-chunks of 16 tokens; a
// pair of tokens in two sub-chunks factors through the decay between the later one's start and the earlier one's end, and a pair
// within one takes 2^(L_i - L_j) channel by channel, L summed in 64 bits and kept as two 32-bit numbers, so that a decay between two tokens
// is as exact as its exponent.  Long sums run in pieces of 16 or 32 terms that are then added, as the token-by-token kernel's lanes
// do, which keeps their rounding where it was.  T is made from the inverses of its four 16 x 16 diagonal blocks.
//
// What bounds it: the token-by-token kernel took 0.48 us per token whatever the hardware's width (a chain of dependent instructions;
// 2,048 tokens of 16 heads of 128 x 128: 980 us).  Here the chain is one step per 64 tokens: 313 us, of which delta_chunk_kernel 150 (shared
// memory and the latency of its staging loads; with single FMAs instead of pairs 23 more, with the pairs of a sub-chunk as a square 13),
// delta_scan_kernel 120 (shared memory, 76 %), delta_out_kernel 43.  Against 64-bit sums (700 tokens of 4 heads, outputs): 2.0e-7 where
// the decays are close to one (token by token 3.4e-7), 1.4e-7 to 1.6e-7 where they are fast (1.5e-7 to 1.7e-7), 1.8e-7 with steps of 0.001
// to 0.1 and A of 1 to 16 (2.2e-7 to 3.7e-7).  Keys that are alike make T far from the identity: at a correlation of 0.9 and beta near one
// 1.8e-7 to 4.1e-7 (1.6e-7 to 3.8e-7), of 0.99 up to 7.0e-7 (3.9e-7).
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

namespace {

constexpr int PC = 64;           // tokens per chunk
constexpr int SUB = 16;          // tokens per sub-chunk
constexpr int THREADS = 256;
constexpr int DT = 32, DTP = DT + 4;      // key channels per pass of delta_chunk_kernel
constexpr int AP = PC + 4;                // row length of a 64 x 64 matrix in shared memory
constexpr int VC = 16;                    // value columns per block of delta_scan_kernel
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ldw(const void* p, int dt, size_t i) {
    return dt == GFB_BF16 ? __bfloat162float(((const __nv_bfloat16*)p)[i]) : ((const float*)p)[i];
}
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// two 32-bit numbers per instruction (sm_100), each rounded as by the single form
typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { f32x2 r; const f32x2 m = pack2(-1.f, -1.f); asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(m), "l"(a)); return r; }
__device__ __forceinline__ float half_sum(f32x2 v) { float a, b; unpack2(v, a, b); return a + b; }
// 2^x for x <= 0 (results below 2^-126 become zero)
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ f32x2 ex22(f32x2 v) { float a, b; unpack2(v, a, b); return pack2(ex2(a), ex2(b)); }
__device__ __forceinline__ ulonglong2 ldp(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }      // four numbers as two pairs
__device__ __forceinline__ void copy16(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
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

// What delta_chunk_kernel leaves per (chunk, head), in floats behind one another
struct Sizes {
    int d, dv;
    __host__ __device__ size_t w() const { return 0; }                                        // W [PC][d]
    __host__ __device__ size_t kh() const { return (size_t)PC * d; }                          // Kh [PC][d]
    __host__ __device__ size_t qb() const { return (size_t)2 * PC * d; }                      // [Qt | B] transposed: [d + PC][PC]
    __host__ __device__ size_t su() const { return qb() + (size_t)(d + PC) * PC; }            // [S_0 ; Y, then U]: [d + PC][dv]
    __host__ __device__ size_t decay() const { return su() + (size_t)(d + PC) * dv; }         // 2^(G_end) [d]
    __host__ __device__ size_t all() const { return decay() + d; }
};

struct ChunkSmem {
    union {
        struct { float q[PC][DTP], k[PC][DTP], L[PC][DTP], Lo[PC][DTP], qt[PC][DTP], kt[PC][DTP], kh[PC][DTP]; };
        struct { float N[PC][AP], T[PC][AP], R[PC][AP]; };     // diag(beta) A, its inverse, right-hand sides
    };
    float P[3][SUB][SUB + 1];
    double sums[16][THREADS];     // of A and B so far, a thread's own: six far pairs of B, of A, two near ones of B, of A
    double tot[8][DT];            // decay sums of half sub-chunks
    float M[4][DT];               // decay of a whole sub-chunk, and of all behind it
    float qn[PC], kn[PC], beta[PC];
};

template <typename TB>
__global__ void __launch_bounds__(THREADS, 2)
delta_chunk_kernel(const float* __restrict__ qkv, int ldq, int q_off, int k_off, int v_off, const TB* __restrict__ beta_raw, int ld_b, int beta_off,
                   const float* __restrict__ a_raw, int ld_a, int a_off, const void* __restrict__ dt_bias, const void* __restrict__ a_log, int w_dt,
                   float* __restrict__ scratch, GfbBatch b, int first_chunk, int H, int KH, int d, int dv, float q_scale, float unit_eps, int head_decay) {
    extern __shared__ __align__(16) unsigned char raw[];
    ChunkSmem& sm = *reinterpret_cast<ChunkSmem*>(raw);
    gfb_pdl_launch();
    gfb_pdl_wait();
    ChunkWork c;
    if (!chunk_work(b, first_chunk + blockIdx.x, c)) return;
    const Sizes z{d, dv};
    const int h = blockIdx.y, kvh = h / (H / KH);
    float* mine = scratch + ((size_t)blockIdx.x * H + h) * z.all();
    float *W = mine + z.w(), *Kh = mine + z.kh(), *QB = mine + z.qb(), *SU = mine + z.su(), *dec = mine + z.decay();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
    const float* qg = qkv + q_off + (size_t)kvh * d;
    const float* kg = qkv + k_off + (size_t)kvh * d;
    // the factors that make q and k unit vectors: a warp per token
    for (int j = warp; j < PC; j += THREADS / 32) {
        float sq = 0.f, sk = 0.f;
        if (j < c.n)
            for (int i = lane; i < d; i += 32) {
                const float x = qg[(size_t)(c.t0 + j) * ldq + i], y = kg[(size_t)(c.t0 + j) * ldq + i];
                sq = fmaf(x, x, sq);
                sk = fmaf(y, y, sk);
            }
        sq = gfb_warp_sum(sq);
        sk = gfb_warp_sum(sk);
        if (lane == 0) {
            sm.qn[j] = (1.0f / sqrtf(sq + unit_eps)) * q_scale;
            sm.kn[j] = 1.0f / sqrtf(sk + unit_eps);
        }
    }
    if (tid < PC) sm.beta[tid] = tid < c.n ? 1.0f / (1.0f + expf(-gfb_to_f32(beta_raw[(size_t)(c.t0 + tid) * ld_b + beta_off + h]))) : 0.f;
    __syncthreads();
    const float rate = expf(ldw(a_log, w_dt, h)) * LOG2E;
    // Thread (ty, tx) owns tokens ty + 16 r (one per sub-chunk) against tokens tx + 16 c: B in [0], A in [1]
    // (far: sub-chunks (1,0), (2,1), (2,0), (3,2), (3,1), (3,0)).
    // The sums that make T and B are what the outputs' error hangs on, most of all where keys are alike and T is far from the identity: a pass
    // sums 16 even and 16 odd channels in 32 bits, and the passes add up in 64 (strongly alike keys, beta near one: chains of 64 terms
    // left the outputs 1.0e-6 from 64 bits, token by token 3.9e-7).
    f32x2 diag = 0ull;
    // Pairs within a sub-chunk: row u has u earlier tokens and row 15 - u has 15 - u, so that the two together fill 15 of 16 lanes, and the last
    // lane takes the later row's own pair.  128 threads are a sub-chunk, which leaves two sub-chunks to a thread where a square has four; the
    // first eight tokens' own pairs, whose decay is one, are taken by eight threads each.
    const int u = ty & 7, fi = (tid >> 7) * SUB + (tx < u ? u : 15 - u), fj = (tid >> 7) * SUB + (tx < u ? tx : tx - u);
    const int di = (tid >> 6) * SUB + ((tid >> 3) & 7);
    const int dd = tid & 31, oct = tid >> 5;        // staging: a channel, eight tokens
#pragma unroll 1
    for (int d0 = 0; d0 < d; d0 += DT) {
        const int ch = d0 + dd;
        float gi[8], qi[8], ki[8];
        const float bias = head_decay ? ldw(dt_bias, w_dt, h) : ldw(dt_bias, w_dt, (size_t)h * d + ch);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int j = oct * 8 + i;
            const bool live = j < c.n;
            const size_t t = (size_t)(c.t0 + (live ? j : 0));
            gi[i] = a_raw[t * ld_a + a_off + (head_decay ? (size_t)h : (size_t)h * d + ch)];
            qi[i] = live ? qg[t * ldq + ch] * sm.qn[j] : 0.f;
            ki[i] = live ? kg[t * ldq + ch] * sm.kn[j] : 0.f;
        }
        double sum = 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            // 2^-4096 is zero against any 32-bit number, so a decay that forgets everything is that: an infinite one (A_log above 88, an
            // infinite input) would leave the sums, and the differences of them, without a value.  (Not a number stays that.)
            const float g = oct * 8 + i < c.n ? -rate * softplus_f(gi[i] + bias) : 0.f;
            gi[i] = g < -4096.f ? -4096.f : g;
            sum += (double)gi[i];
        }
        __syncthreads();                            // the previous pass is done with everything below
        sm.tot[oct][dd] = sum;
        __syncthreads();
        {
            const int sub = oct >> 1;
            const double before = (oct & 1) ? sm.tot[oct - 1][dd] : 0.0, whole = sm.tot[oct & ~1][dd] + sm.tot[oct | 1][dd];
            double ahead = 0.0, behind = 0.0;        // the sub-chunks before and behind this one
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const double w = sm.tot[2 * m][dd] + sm.tot[2 * m + 1][dd];
                if (m < sub) ahead += w;
                if (m > sub) behind += w;
            }
            if (!(oct & 1)) sm.M[sub][dd] = ex2((float)whole);
            const float pa = ex2((float)ahead), pb = ex2((float)behind);
            double run = before;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int j = oct * 8 + i;
                run += (double)gi[i];
                const float L = (float)run, e = ex2(L);
                // the decays behind the token within its sub-chunk: never above zero, also where rounding made the two sums cross
                const float rest = (float)(whole - run);
                const float kh = ki[i] * ex2(rest > 0.f ? 0.f : rest);
                sm.q[j][dd] = qi[i];
                sm.k[j][dd] = ki[i];
                sm.L[j][dd] = L;
                sm.Lo[j][dd] = (float)(run - (double)L);
                sm.qt[j][dd] = qi[i] * e;
                sm.kt[j][dd] = ki[i] * e;
                sm.kh[j][dd] = kh;
                Kh[(size_t)j * d + ch] = kh * pb;
                W[(size_t)j * d + ch] = sm.beta[j] * (ki[i] * e * pa);       // the right-hand side that becomes W
                gi[i] = qi[i] * e * pa;
            }
            if (oct == 0) dec[ch] = ex2((float)(whole + behind));
            float4* out = reinterpret_cast<float4*>(QB + (size_t)ch * PC + oct * 8);
            out[0] = make_float4(gi[0], gi[1], gi[2], gi[3]);
            out[1] = make_float4(gi[4], gi[5], gi[6], gi[7]);
        }
        __syncthreads();
        f32x2 far[2][6] = {{0ull, 0ull, 0ull, 0ull, 0ull, 0ull}, {0ull, 0ull, 0ull, 0ull, 0ull, 0ull}}, near[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll 1
        for (int x = 0; x < DT; x += 4) {
            {
                const ulonglong2 M1 = ldp(&sm.M[1][x]), M2 = ldp(&sm.M[2][x]);
                const ulonglong2 h0 = ldp(&sm.kh[tx][x]), h1 = ldp(&sm.kh[tx + 16][x]), h2 = ldp(&sm.kh[tx + 32][x]);
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const float(*rows)[DTP] = m == 0 ? sm.qt : sm.kt;
                    const ulonglong2 r1 = ldp(&rows[ty + 16][x]), r2 = ldp(&rows[ty + 32][x]), r3 = ldp(&rows[ty + 48][x]);
                    const f32x2 a2x = mul2(r2.x, M1.x), a2y = mul2(r2.y, M1.y), a3x = mul2(r3.x, M2.x), a3y = mul2(r3.y, M2.y);
                    const f32x2 b3x = mul2(a3x, M1.x), b3y = mul2(a3y, M1.y);
                    fma2(far[m][0], r1.x, h0.x); fma2(far[m][0], r1.y, h0.y);
                    fma2(far[m][1], r2.x, h1.x); fma2(far[m][1], r2.y, h1.y);
                    fma2(far[m][2], a2x, h0.x); fma2(far[m][2], a2y, h0.y);
                    fma2(far[m][3], r3.x, h2.x); fma2(far[m][3], r3.y, h2.y);
                    fma2(far[m][4], a3x, h1.x); fma2(far[m][4], a3y, h1.y);
                    fma2(far[m][5], b3x, h0.x); fma2(far[m][5], b3y, h0.y);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int i = fi + 32 * r, j = fj + 32 * r;
                const ulonglong2 li = ldp(&sm.L[i][x]), lj = ldp(&sm.L[j][x]);
                const ulonglong2 ri = ldp(&sm.Lo[i][x]), rj = ldp(&sm.Lo[j][x]);
                const ulonglong2 k2 = ldp(&sm.k[j][x]);
                const f32x2 ex = mul2(k2.x, ex22(add2(sub2(li.x, lj.x), sub2(ri.x, rj.x))));
                const f32x2 ey = mul2(k2.y, ex22(add2(sub2(li.y, lj.y), sub2(ri.y, rj.y))));
                const ulonglong2 q2 = ldp(&sm.q[i][x]), c2 = ldp(&sm.k[i][x]);
                fma2(near[0][r], q2.x, ex); fma2(near[0][r], q2.y, ey);
                fma2(near[1][r], c2.x, ex); fma2(near[1][r], c2.y, ey);
            }
        }
#pragma unroll
        for (int f = 0; f < 16; f++) {
            float even, odd;
            unpack2(f < 12 ? far[f / 6][f % 6] : near[(f - 12) / 2][f % 2], even, odd);
            const double both = (double)even + (double)odd;
            sm.sums[f][tid] = d0 == 0 ? both : sm.sums[f][tid] + both;
        }
        {
            const ulonglong2 q2 = ldp(&sm.q[di][(tid & 7) * 4]), k2 = ldp(&sm.k[di][(tid & 7) * 4]);
            fma2(diag, q2.x, k2.x); fma2(diag, q2.y, k2.y);
        }
    }
    __syncthreads();                                 // the matrices take the place of q, k, L
    // B transposed (zeros above the diagonal) and diag(beta) A; T is kept transposed too, so that four rows of it are one load
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int i = ty + 16 * r;
        const float be = sm.beta[i];
#pragma unroll
        for (int cc = 0; cc < 4; cc++) {
            const int j = tx + 16 * cc;
            const int f = cc < r ? (r == 1 ? 0 : r == 2 ? 2 - cc : 5 - cc) : 0;
            sm.T[j][i] = 0.f;
            if (cc == r && tx <= ty) continue;       // below
            sm.R[j][i] = cc < r ? (float)sm.sums[f][tid] : 0.f;
            if (cc < r) sm.N[i][j] = be * (float)sm.sums[6 + f][tid];
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i = fi + 32 * r, j = fj + 32 * r;
        sm.R[j][i] = (float)sm.sums[12 + r][tid];
        if (j < i) sm.N[i][j] = sm.beta[i] * (float)sm.sums[14 + r][tid];
    }
    float own = half_sum(diag);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) own += __shfl_xor_sync(0xffffffffu, own, o);
    if ((tid & 7) == 0) sm.R[di][di] = own;
    __syncthreads();
    for (int e = tid; e < PC * 16; e += THREADS) {
        const int j = e >> 4, i = (e & 15) * 4;
        *reinterpret_cast<float4*>(QB + (size_t)(d + j) * PC + i) = ld4(&sm.R[j][i]);
    }
    // the inverses of the diagonal blocks of I + N: a thread per column, forward substitution
    if (tid < PC) {
        const int o = (tid >> 4) * SUB, col = tid & 15;
        float x[SUB];
#pragma unroll
        for (int i = 0; i < SUB; i++) {
            float v = i == col ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < i; j++) v = fmaf(-sm.N[o + i][o + j], x[j], v);
            x[i] = v;                                // zero above the diagonal by itself
            sm.T[o + col][o + i] = v;
        }
    }
    // blocks below the diagonal, one diagonal of blocks after the other: T_rc = -T_rr sum_(c <= m < r) N_rm T_mc
    for (int off = 1; off < 4; off++) {
        __syncthreads();
        for (int k = 0; k < 4 - off; k++) {          // thread (ty, tx): one number of each block
            const int r = k + off;
            float v = 0.f;
            for (int m = k * SUB; m < r * SUB; m++) v = fmaf(sm.N[r * SUB + ty][m], sm.T[k * SUB + tx][m], v);
            sm.P[k][ty][tx] = v;
        }
        __syncthreads();
        for (int k = 0; k < 4 - off; k++) {
            const int r = k + off;
            float v = 0.f;
#pragma unroll
            for (int m = 0; m < SUB; m++)
                if (m <= ty) v = fmaf(sm.T[r * SUB + m][r * SUB + ty], sm.P[k][m][tx], v);       // (a later row need not be finite)
            sm.T[k * SUB + tx][r * SUB + ty] = -v;
        }
    }
    // W = T (diag(beta) Kt) in place, Y = T (diag(beta) V): 64 columns at a time
    const int tiles = (d + dv) / 64;
    for (int tile = 0; tile < tiles; tile++) {
        const bool of_w = tile * 64 < d;
        const int c0 = of_w ? tile * 64 : tile * 64 - d;
        __syncthreads();
        for (int e = tid; e < PC * 16; e += THREADS) {
            const int j = e >> 4, cc = (e & 15) * 4;
            float4 v;
            if (of_w) {
                v = ld4(W + (size_t)j * d + c0 + cc);
            } else {
                v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < c.n) {
                    const float be = sm.beta[j];
                    const float* p = qkv + (size_t)(c.t0 + j) * ldq + v_off + (size_t)h * dv + c0 + cc;
                    v = make_float4(be * p[0], be * p[1], be * p[2], be * p[3]);
                }
            }
            *reinterpret_cast<float4*>(&sm.R[j][cc]) = v;
        }
        __syncthreads();
        // rows 4 ty .. + 3 (their sub-chunk and those before it), columns 4 tx .. + 3
        float acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int cc = 0; cc < 4; cc++) acc[r][cc] = 0.f;
        for (int J = 0; J <= ty >> 2; J++) {
            f32x2 part[4][2] = {{0ull, 0ull}, {0ull, 0ull}, {0ull, 0ull}, {0ull, 0ull}};
            const int before = J < ty >> 2 ? SUB : 4 * (ty & 3);      // tokens ahead of all four rows, then their own, of which a row
#pragma unroll 4                                                      // takes those up to itself (a later one need not be finite)
            for (int jj = 0; jj < before; jj++) {
                const ulonglong2 v = ldp(&sm.R[16 * J + jj][4 * tx]);
                const float4 t4 = ld4(&sm.T[16 * J + jj][4 * ty]);
                const f32x2 t0 = pack2(t4.x, t4.x), t1 = pack2(t4.y, t4.y), t2 = pack2(t4.z, t4.z), t3 = pack2(t4.w, t4.w);
                fma2(part[0][0], t0, v.x); fma2(part[0][1], t0, v.y);
                fma2(part[1][0], t1, v.x); fma2(part[1][1], t1, v.y);
                fma2(part[2][0], t2, v.x); fma2(part[2][1], t2, v.y);
                fma2(part[3][0], t3, v.x); fma2(part[3][1], t3, v.y);
            }
            if (J == ty >> 2) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const ulonglong2 v = ldp(&sm.R[4 * ty + q][4 * tx]);
                    const float4 t4 = ld4(&sm.T[4 * ty + q][4 * ty]);
                    const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
                    for (int r = q; r < 4; r++) {
                        const f32x2 tr = pack2(t[r], t[r]);
                        fma2(part[r][0], tr, v.x); fma2(part[r][1], tr, v.y);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                float a, e, i, o;
                unpack2(part[r][0], a, e);
                unpack2(part[r][1], i, o);
                acc[r][0] += a; acc[r][1] += e; acc[r][2] += i; acc[r][3] += o;
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int i = 4 * ty + r;
            float* dst = of_w ? W + (size_t)i * d + c0 + 4 * tx : SU + (size_t)(d + i) * dv + c0 + 4 * tx;
            *reinterpret_cast<float4*>(dst) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
    }
}

// A block has S [d][16] of one (sequence, head) in shared memory, transposed, and two stages of W, Kh, Y and the decays: the next
// chunk's copies run under the current one's products.  U = Y - W S: lane (rg, kq) of a warp takes rows rg + 16 i and every fourth group
// of four k, so that the 16-byte loads of eight neighbouring lanes fall into 32 banks (rows of W are padded to d + 16 numbers); the four
// lanes' sums meet by shuffles, each lane ending with one row.  Kh^T U likewise over the chunk's tokens.
template <int D>
struct ScanSmem {
    float W[2][PC][D + 16];
    float K[2][PC][D + 8];
    float U[2][PC][VC + 4];
    float dec[2][D];
    float S[VC][D + 4];
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
delta_scan_kernel(float* __restrict__ scratch, float* __restrict__ state, size_t state_ld, GfbBatch b, int first_chunk, int n_chunks, int H, int dv) {
    extern __shared__ __align__(16) unsigned char raw[];
    ScanSmem<D>& sm = *reinterpret_cast<ScanSmem<D>*>(raw);
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int s = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * VC;
    const Sizes z{D, dv};
    int lo = 0;
    for (int i = 0; i < s; i++) lo += (b.cu_seqlens[i + 1] - b.cu_seqlens[i] + PC - 1) / PC;
    int hi = lo + (b.cu_seqlens[s + 1] - b.cu_seqlens[s] + PC - 1) / PC;
    lo = max(lo, first_chunk);
    hi = min(hi, first_chunk + n_chunks);
    if (lo >= hi) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* Sg = state + (size_t)b.slots[s] * state_ld + (size_t)h * D * dv + v0;
    for (int e = tid; e < D * VC; e += THREADS) {
        const int k = e / VC, v = e - k * VC;
        sm.S[v][k] = Sg[(size_t)k * dv + v];
    }
    auto fetch = [&](int st, int w) {
        const float* m = scratch + ((size_t)(w - first_chunk) * H + h) * z.all();
        constexpr int PIECES = D / 4;
        for (int e = tid; e < PC * PIECES; e += THREADS) {
            const int j = e / PIECES, c = (e - j * PIECES) * 4;
            copy16(&sm.W[st][j][c], m + z.w() + (size_t)j * D + c);
            copy16(&sm.K[st][j][c], m + z.kh() + (size_t)j * D + c);
        }
        {
            const int j = tid >> 2, c = (tid & 3) * 4;
            copy16(&sm.U[st][j][c], m + z.su() + (size_t)(D + j) * dv + v0 + c);
        }
        if (tid < D / 4) copy16(&sm.dec[st][tid * 4], m + z.decay() + tid * 4);
        copy_commit();
    };
    fetch(0, lo);
    int st = 0;
    const int q4 = lane & 3, rg8 = lane >> 2;
    for (int w = lo; w < hi; w++, st ^= 1) {
        float* SU = scratch + ((size_t)(w - first_chunk) * H + h) * z.all() + z.su() + v0;
        copy_wait<0>();
        __syncthreads();                             // this chunk's inputs have landed; everybody is done with the other stage and S is new
        if (w + 1 < hi) fetch(st ^ 1, w + 1);
        // the state ahead of the chunk, for the outputs
        for (int e = tid; e < D * 4; e += THREADS) {
            const int k = e >> 2, c = (e & 3) * 4;
            *reinterpret_cast<float4*>(SU + (size_t)k * dv + c) = make_float4(sm.S[c][k], sm.S[c + 1][k], sm.S[c + 2][k], sm.S[c + 3][k]);
        }
        {
            const int rg = rg8 + 8 * (warp & 1), cg = (warp >> 1) * 4;     // rows rg + 16 i, columns cg .. + 3
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
#pragma unroll 2
            for (int k0 = 0; k0 < D; k0 += 16) {
                float4 a[4], x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] = ld4(&sm.W[st][rg + 16 * i][k0 + 4 * q4]);
#pragma unroll
                for (int j = 0; j < 4; j++) x[j] = ld4(&sm.S[cg + j][k0 + 4 * q4]);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        acc[i][j] = fmaf(a[i].x, x[j].x, fmaf(a[i].y, x[j].y, fmaf(a[i].z, x[j].z, fmaf(a[i].w, x[j].w, acc[i][j]))));
            }
            // lanes q4 ^ 2 swap halves of the rows, lanes q4 ^ 1 halves of what is left: lane q4 ends with row i = q4
            float two[2][4], one[4];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float give = (q4 & 2) ? acc[i][j] : acc[i + 2][j], keep = (q4 & 2) ? acc[i + 2][j] : acc[i][j];
                    two[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
                }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float give = (q4 & 1) ? two[0][j] : two[1][j], keep = (q4 & 1) ? two[1][j] : two[0][j];
                one[j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
            }
            const int row = rg + 16 * q4;
            float4 u = ld4(&sm.U[st][row][cg]);
            u = make_float4(u.x - one[0], u.y - one[1], u.z - one[2], u.w - one[3]);
            *reinterpret_cast<float4*>(&sm.U[st][row][cg]) = u;              // this thread's own four numbers
            *reinterpret_cast<float4*>(SU + (size_t)(D + row) * dv + cg) = u;
        }
        __syncthreads();
        {
            // key channels kk .. + 3 and D / 2 + kk .. + 3, columns cg .. + 3, tokens q4, q4 + 4, ...
            constexpr int KG = D / 8;                // groups of key channels: 16 or 8
            const int g = rg8 + 8 * (KG == 16 ? (warp & 1) : 0), kk = 4 * g;
            const int cg = (KG == 16 ? warp >> 1 : warp & 3) * 4;
            if (KG == 16 || warp < 4) {
                float acc[8][4];
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
#pragma unroll 4
                for (int t = q4; t < PC; t += 4) {
                    const float4 a = ld4(&sm.K[st][t][kk]), a2 = ld4(&sm.K[st][t][D / 2 + kk]), u = ld4(&sm.U[st][t][cg]);
                    const float kv[8] = {a.x, a.y, a.z, a.w, a2.x, a2.y, a2.z, a2.w};
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        acc[i][0] = fmaf(kv[i], u.x, acc[i][0]); acc[i][1] = fmaf(kv[i], u.y, acc[i][1]);
                        acc[i][2] = fmaf(kv[i], u.z, acc[i][2]); acc[i][3] = fmaf(kv[i], u.w, acc[i][3]);
                    }
                }
                float four[4][4], two[2][4];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float give = (q4 & 2) ? acc[i][j] : acc[i + 4][j], keep = (q4 & 2) ? acc[i + 4][j] : acc[i][j];
                        four[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
                    }
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float give = (q4 & 1) ? four[i][j] : four[i + 2][j], keep = (q4 & 1) ? four[i + 2][j] : four[i][j];
                        two[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
                    }
                const int k = (q4 & 2 ? D / 2 : 0) + kk + (q4 & 1 ? 2 : 0);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float e = sm.dec[st][k + i];
#pragma unroll
                    for (int j = 0; j < 4; j++) sm.S[cg + j][k + i] = fmaf(e, sm.S[cg + j][k + i], two[i][j]);
                }
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < D * VC; e += THREADS) {
        const int k = e / VC, v = e - k * VC;
        Sg[(size_t)k * dv + v] = sm.S[v][k];
    }
}

// o [64][64 columns] = X^T Z, X = [Qt | B]^T [K][64], Z = [S_0 ; U] [K][dv]: both k-major, 32 k per stage, two stages.  Four warps of 32 x
// 32, a lane has 8 x 4 sums in two groups of four rows.
constexpr int OUT_THREADS = 128, OK = 32;

// One number of it over the tokens up to its own only; sums in delta_out_kernel's order.
__device__ __noinline__ float out_number(const float* X, const float* Z, int row, int d, int dv) {
    float acc = 0.f;
    for (int k0 = 0; k0 <= d + row; k0 += OK) {
        float part = 0.f;
        for (int k = k0; k < k0 + OK && k <= d + row; k++) part = fmaf(X[(size_t)k * PC + row], Z[(size_t)k * dv], part);
        acc += part;
    }
    return acc;
}

__global__ void __launch_bounds__(OUT_THREADS)
delta_out_kernel(const float* __restrict__ scratch, float* __restrict__ out, GfbBatch b, int first_chunk, int H, int d, int dv) {
    __shared__ __align__(16) float X[2][OK][PC], Z[2][OK][64];
    gfb_pdl_launch();
    gfb_pdl_wait();
    ChunkWork c;
    if (!chunk_work(b, first_chunk + blockIdx.x, c)) return;
    const Sizes z{d, dv};
    const int h = blockIdx.y, v0 = blockIdx.z * 64, K = d + PC;
    const float* m = scratch + ((size_t)blockIdx.x * H + h) * z.all();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = (warp & 1) * 32 + (lane >> 3) * 4, c0 = (warp >> 1) * 32 + (lane & 7) * 4;
    auto fetch = [&](int st, int k0) {
#pragma unroll
        for (int e = tid; e < OK * 16; e += OUT_THREADS) {
            const int k = e >> 4, p = (e & 15) * 4;
            copy16(&X[st][k][p], m + z.qb() + (size_t)(k0 + k) * PC + p);
            copy16(&Z[st][k][p], m + z.su() + (size_t)(k0 + k) * dv + v0 + p);
        }
        copy_commit();
    };
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    fetch(0, 0);
    int st = 0;
    for (int k0 = 0; k0 < K; k0 += OK, st ^= 1) {
        copy_wait<0>();
        __syncthreads();
        if (k0 + OK < K) fetch(st ^ 1, k0 + OK);
        float part[8][4];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) part[i][j] = 0.f;
#pragma unroll 8
        for (int k = 0; k < OK; k++) {
            const float4 a = ld4(&X[st][k][r0]), a2 = ld4(&X[st][k][r0 + 16]), v = ld4(&Z[st][k][c0]);
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
    // The zeros of B meet later tokens' u above: one that is not finite makes NaN of them.  Such a block (and one whose own numbers are not
    // finite) works its numbers out once more, each from the tokens up to its own.
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
                if (row < c.n) acc[i][j] = out_number(m + z.qb(), m + z.su() + v0 + c0 + j, row, d, dv);
            }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = r0 + (i & 3) + 16 * (i >> 2);
        if (row < c.n)
            *reinterpret_cast<float4*>(out + ((size_t)(c.t0 + row) * H + h) * dv + v0 + c0) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// chunks that are in flight together: their scratch stays below 256 MB (2,048 tokens of 16 heads of 128 x 128 take 110), or is one
// chunk's
long chunks_at_once(int n_tokens, int n_seqs, int H, int d, int dv) {
    const long all = (long)n_tokens / PC + n_seqs;               // an upper bound; surplus blocks find no work
    const long each = (long)(Sizes{d, dv}.all() * sizeof(float)) * H;
    const long most = (256L << 20) / each;
    return all < most ? all : (most > 0 ? most : 1);
}

}  // namespace

// Floats of scratch of gfb_delta_chunks.
GFB_API long gfb_delta_chunks_scratch_floats(int n_tokens, int n_seqs, int H, int d, int dv) {
    return chunks_at_once(n_tokens, n_seqs, H, d, dv) * H * (long)Sizes{d, dv}.all();
}

// As gfb_delta_rule (whose arguments these are), for key heads of 64 or 128 and value heads of a multiple of 64; qkv and a_raw are only
// read.  state with state_ld and every sequence's part of it need no alignment; out and scratch 16 bytes.
GFB_API int gfb_delta_chunks(const float* qkv, int ldq, int q_off, int k_off, int v_off, const void* beta_raw, int b_dt, int ld_b, int beta_off,
                             const float* a_raw, int ld_a, int a_off, const void* dt_bias, const void* a_log, int w_dt, float* state,
                             long state_ld, float* out, float* scratch, const int* cu_seqlens, const int* tok_seq, const int* slots,
                             const int* lengths, int n_seqs, int n_tokens, int H, int KH, int d, int dv, float q_scale, float unit_eps,
                             int head_decay, cudaStream_t stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (KH <= 0 || H % KH) return gfb_fail("gfb_delta_chunks: %d heads do not divide into %d query/key heads", H, KH);
    if ((d != 64 && d != 128) || dv < 64 || dv % 64) return gfb_fail("gfb_delta_chunks: heads of %d x %d", d, dv);
    if (H > 65535 || dv / VC > 65535) return gfb_fail("gfb_delta_chunks: %d heads of %d columns exceed the grid limit", H, dv);
    if (((uintptr_t)out | (uintptr_t)scratch) & 15) return gfb_fail("gfb_delta_chunks: output and scratch must be 16-byte aligned");
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    const long all = (long)n_tokens / PC + n_seqs, step = chunks_at_once(n_tokens, n_seqs, H, d, dv);
    typedef __nv_bfloat16 bf16;
    cudaError_t e = cudaFuncSetAttribute(b_dt == GFB_BF16 ? (const void*)delta_chunk_kernel<bf16> : (const void*)delta_chunk_kernel<float>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkSmem));
    if (e == cudaSuccess)
        e = d == 128 ? cudaFuncSetAttribute(delta_scan_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanSmem<128>))
                     : cudaFuncSetAttribute(delta_scan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanSmem<64>));
    if (e != cudaSuccess) return gfb_fail("gfb_delta_chunks: %s", cudaGetErrorString(e));
    for (long first = 0; first < all; first += step) {
        const int n = (int)(all - first < step ? all - first : step);
#define CHUNKS(TB)                                                                                                                           \
    e = gfb_launch(delta_chunk_kernel<TB>, dim3(n, H), dim3(THREADS), sizeof(ChunkSmem), stream, qkv, ldq, q_off, k_off, v_off, (const TB*)beta_raw, \
                   ld_b, beta_off, a_raw, ld_a, a_off, dt_bias, a_log, w_dt, scratch, b, (int)first, H, KH, d, dv, q_scale, unit_eps, head_decay)
        if (b_dt == GFB_BF16) CHUNKS(bf16);
        else if (b_dt == GFB_F32) CHUNKS(float);
        else return gfb_fail("gfb_delta_chunks: unknown type %d", b_dt);
#undef CHUNKS
        const dim3 grid(n_seqs, H, dv / VC);
        if (e == cudaSuccess && d == 128)
            e = gfb_launch(delta_scan_kernel<128>, grid, dim3(THREADS), sizeof(ScanSmem<128>), stream, scratch, state, (size_t)state_ld, b, (int)first, n, H, dv);
        else if (e == cudaSuccess)
            e = gfb_launch(delta_scan_kernel<64>, grid, dim3(THREADS), sizeof(ScanSmem<64>), stream, scratch, state, (size_t)state_ld, b, (int)first, n, H, dv);
        if (e == cudaSuccess)
            e = gfb_launch(delta_out_kernel, dim3(n, H, dv / 64), dim3(OUT_THREADS), 0, stream, (const float*)scratch, out, b, (int)first, H, d, dv);
        if (gfb_check(e, "gfb_delta_chunks")) return 1;
    }
    return 0;
}
