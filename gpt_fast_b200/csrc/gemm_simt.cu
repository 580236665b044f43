// C[M,N] = A[M,K] * W[N,K]^T on CUDA cores, any M, N, K, both precisions.
//
// This is the 32-bit product for short sums and for rows that are no multiple of
// 16 bytes (gemm_split.cu has the others), and the fallback of the bfloat16
// path for shapes the tensor-core kernel refuses (such rows too).
// It stands where gpt-fast calls nn.Linear (model.py:195, :215,
// :227, :145).  Each output element is a sum over slices of SLICE numbers of k:
// a slice is one thread's sum in ascending order, and the slices are added in
// ascending order, whatever M, the tile's size and its position are: a row's
// result does not depend on which other rows are in the batch.
//
// The FMA pipe bounds it from about 20 rows on (73 TFLOP/s at 1,930 MHz), the weight stream below.  A thread keeps 8 x 8 sums, so a
// warp issues 4 16-byte shared-memory loads per 64 FMAs, and the next 16 k of both operands travel to registers under the
// products of the current ones.  The slices are what fills the chip: a 32-bit layer of a short prompt has fewer tiles than two per SM
// (198 rows, 3,072 columns: 192 of 64 x 64), so a tile's slices then go to blocks of their own, which leave 32-bit partial
// sums, and a second kernel adds them; with tiles enough a block walks over all slices itself.  Both give the same bits.
// Measured against one sum per thread over all of K in 64 x 64 tiles of 4 x 4 sums: 198 rows of 3,072 numbers times 16,384 columns 1,137 -> 541 us
// (37 TFLOP/s), of 8,192 numbers times 3,072 columns 1,012 -> 297, of 3,072 times 5,120 496 -> 181; 500 rows of 3,072 times 5,120: 343 us, 46 TFLOP/s.
//
// Epilogues: STORE (C = acc, cast), ADD (C is 32-bit, C += acc: the residual
// sum), SWIGLU (W's rows alternate gate, up; C[M, N/2] = silu(gate) * up), and
// the unary activations GELU (exact, with erf), GELU_TANH and SILU (C = f(acc)).
#include "common.cuh"

GFB_DEFINE_LAST_ERROR()

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_GELU = 4, EPI_GELU_TANH = 5, EPI_SILU = 6, EPI_RELU2 = 7 };   // 3: the tensor-core kernel's partial sums

template <int EPI>
__device__ __forceinline__ float unary(float z) {
    if (EPI == EPI_GELU) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
    if (EPI == EPI_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
    if (EPI == EPI_SILU) return z / (1.0f + expf(-z));
    if (EPI == EPI_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
    return z;
}

constexpr int BK = 16, THREADS = 128;
constexpr int SLICE = 512;                        // numbers of k per slice: a fixed part of the order of summation

// four neighbouring numbers of a row
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}

// two 32-bit numbers per instruction (sm_100), each rounded as by the single form
typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }

// numbers k .. k + 3 of row r of an operand with `rows` rows; zeros beyond its ends.  WIDE: rows of whole 4-number units, aligned
template <typename T, bool WIDE>
__device__ __forceinline__ float4 fetch4(const T* __restrict__ p, int r, int rows, int k, int k_end, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r >= rows || k >= k_end) return v;
    const T* q = p + (size_t)r * K + k;
    if (WIDE) return load4(q);                    // (k_end is a multiple of four then)
    v.x = gfb_to_f32(q[0]);
    if (k + 1 < k_end) v.y = gfb_to_f32(q[1]);
    if (k + 2 < k_end) v.z = gfb_to_f32(q[2]);
    if (k + 3 < k_end) v.w = gfb_to_f32(q[3]);
    return v;
}

template <typename TC, int EPI>
__device__ __forceinline__ void finish(TC* __restrict__ C, int m, int n, int N, float v, float next) {
    if (EPI == EPI_SWIGLU) {                      // an even column (gate) with the one behind it (up); N is even
        if ((n & 1) == 0) C[(size_t)m * (N >> 1) + (n >> 1)] = gfb_from_f32<TC>(v / (1.f + expf(-v)) * next);
    } else if (EPI == EPI_ADD) {
        C[(size_t)m * N + n] = gfb_from_f32<TC>(gfb_to_f32(C[(size_t)m * N + n]) + v);
    } else {
        C[(size_t)m * N + n] = gfb_from_f32<TC>(unary<EPI>(v));
    }
}

// Four warps in WM x WN; a warp takes 32 x 64 of the tile (TM = 8: its lanes in 4 x 8, a lane's 8 x 8 sums lie in two groups of four rows, 16
// apart, and two of four columns, 32 apart, so that every 16-byte load of shared memory is one pass), or 8 x 32 (TM = 2: lanes in
// 4 x 8, 2 x 4 sums, for a few rows that only wait for the weights).  SPLIT: blockIdx.z takes one slice and leaves its sums in
// partial [slices][M][N]; else the running total of the slices before the last stands in partial [M][N] (a second set of sums in registers
// cost a third of the rate: 2,048 rows of 3,072 times 5,120 columns 2,043 us, 1,570 us so).
template <typename TA, typename TW, typename TC, int EPI, int WM, int WN, int TM, bool WIDE, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 3)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M, int N, int K, float* __restrict__ partial) {
    static_assert(WM * WN * 32 == THREADS && (TM == 8 || TM == 2), "four warps");
    constexpr int TN = TM == 8 ? 8 : 4, BM = WM * 4 * TM, BN = WN * 8 * TN;
    constexpr int LA = (BM * BK / 4 + THREADS - 1) / THREADS, LW = (BN * BK / 4 + THREADS - 1) / THREADS;   // 4-number loads per thread and step
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Ws[2][BK][BN + 4];
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int am = (warp % WM) * 4 * TM + (lane >> 3) * (TM == 8 ? 4 : 2), wn = (warp / WM) * 8 * TN + (lane & 7) * 4;   // first row and column in the tile
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int k_begin = SPLIT ? (int)blockIdx.z * SLICE : 0, k_last = SPLIT ? min(K, k_begin + SLICE) : K;
    const int lr = tid >> 2, lk = (tid & 3) * 4;                    // the row (of every 32) and the four k this thread loads
    f32x2 sum[TM][TN / 2];                        // neighbouring columns share an FMA instruction
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) sum[i][j] = 0ull;

    float4 ra[LA], rw[LW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; i++) ra[i] = lr + 32 * i < BM ? fetch4<TA, WIDE>(A, m0 + lr + 32 * i, M, k0 + lk, k_last, K) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LW; i++) rw[i] = lr + 32 * i < BN ? fetch4<TW, WIDE>(W, n0 + lr + 32 * i, N, k0 + lk, k_last, K) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto stage = [&](int s) {
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int r = lr + 32 * i;
            if (r < BM) { As[s][lk][r] = ra[i].x; As[s][lk + 1][r] = ra[i].y; As[s][lk + 2][r] = ra[i].z; As[s][lk + 3][r] = ra[i].w; }
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int r = lr + 32 * i;
            if (r < BN) { Ws[s][lk][r] = rw[i].x; Ws[s][lk + 1][r] = rw[i].y; Ws[s][lk + 2][r] = rw[i].z; Ws[s][lk + 3][r] = rw[i].w; }
        }
    };
    fetch(k_begin);
    stage(0);
    __syncthreads();
    int s = 0;
    for (int k0 = k_begin; k0 < k_last; k0 += BK, s ^= 1) {
        const bool more = k0 + BK < k_last;
        if (more) fetch(k0 + BK);
#pragma unroll 8
        for (int k = 0; k < BK; k++) {
            float a[TM];
            f32x2 w[TN / 2];
            if (TM == 8) {
                const float4 a0 = *reinterpret_cast<const float4*>(&As[s][k][am]), a1 = *reinterpret_cast<const float4*>(&As[s][k][am + 16]);
                a[0] = a0.x; a[1] = a0.y; a[2 % TM] = a0.z; a[3 % TM] = a0.w; a[4 % TM] = a1.x; a[5 % TM] = a1.y; a[6 % TM] = a1.z; a[7 % TM] = a1.w;
            } else {
                const float2 a0 = *reinterpret_cast<const float2*>(&As[s][k][am]);
                a[0] = a0.x; a[1] = a0.y;
            }
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[s][k][wn + 8 * j]);
                w[j / 2] = v.x; w[j / 2 + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const f32x2 both = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) fma2(sum[i][j], both, w[j]);
            }
        }
        if (!SPLIT && (k0 + BK) % SLICE == 0 && more) {             // a slice ends: into the running total (the first one as it is)
            const bool first = k0 < SLICE;
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const int m = m0 + am + (i & 3) + 16 * (i >> 2);
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    const int n = n0 + wn + (j & 3) + 32 * (j >> 2);
                    float v[2];
                    unpack2(sum[i][j / 2], v[0], v[1]);
                    if (m < M && n < N) {
                        float* t = partial + (size_t)m * N + n;
                        *t = first ? v[j & 1] : *t + v[j & 1];
                    }
                }
#pragma unroll
                for (int j = 0; j < TN / 2; j++) sum[i][j] = 0ull;
            }
        }
        if (more) stage(s ^ 1);
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + am + (i & 3) + 16 * (i >> 2);
        if (m >= M) continue;
        float acc[TN];
#pragma unroll
        for (int j = 0; j < TN; j += 2) unpack2(sum[i][j / 2], acc[j], acc[j + 1]);
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + wn + (j & 3) + 32 * (j >> 2);
            if (n >= N) continue;
            if (SPLIT) {
                partial[((size_t)blockIdx.z * M + m) * N + n] = acc[j];
            } else if (K > SLICE) {
                const float* t = partial + (size_t)m * N;
                const int other = EPI == EPI_SWIGLU ? (n ^ 1) : n;
                finish<TC, EPI>(C, m, n, N, t[n] + acc[j], t[other] + acc[j ^ 1]);
            } else {
                finish<TC, EPI>(C, m, n, N, acc[j], acc[j ^ 1]);
            }
        }
    }
}

// the slices of every sum, in ascending order, and the epilogue; a thread per pair of columns
template <typename TC, int EPI>
__global__ void __launch_bounds__(256)
gemm_simt_sum_kernel(const float* __restrict__ partial, TC* __restrict__ C, int M, int N, int slices) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int half = (N + 1) / 2;
    const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (e >= (size_t)M * half) return;
    const int m = (int)(e / half), n = (int)(e - (size_t)m * half) * 2;
    const float* p = partial + (size_t)m * N + n;
    const bool two = n + 1 < N;
    float v0 = p[0], v1 = two ? p[1] : 0.f;
    for (int s = 1; s < slices; s++) {
        const float* q = p + (size_t)s * M * N;
        v0 += q[0];
        if (two) v1 += q[1];
    }
    finish<TC, EPI>(C, m, n, N, v0, v1);
    if (two) finish<TC, EPI>(C, m, n + 1, N, v1, 0.f);
}

// Rows of a tile: 64 x 128, or 32 x 256 where that leaves at least an eighth fewer rows of empty work, or 16 x 64.
static int tile_rows(int M) {
    if (M <= 16) return 16;
    const int by64 = (M + 63) / 64 * 64, by32 = (M + 31) / 32 * 32;
    return by32 * 8 <= by64 * 7 ? 32 : 64;
}
static int tile_cols(int bm) { return bm == 16 ? 64 : bm == 32 ? 256 : 128; }

static int slices_of(int K) { return (K + SLICE - 1) / SLICE; }

// Slices go to blocks of their own while the tiles alone are fewer than six for each of 148 SMs (a block of 128 threads, several of
// which share an SM): beyond that the last round's idle SMs cost less than the partial sums' way through memory.  198 rows times 16,384
// columns (448 tiles, K = 3,072): 717 us in slices of 1,024 with two blocks per SM, 541 in slices of 512 with three.
static bool split(int M, int N, int K) {
    const int bm = tile_rows(M), bn = tile_cols(bm);
    const long tiles = (long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return slices_of(K) > 1 && slices_of(K) <= 65535 && tiles < 6 * 148;
}

// The rows of A that one launch takes.  Partial sums stay below 256 MB (or are one row tile's), as the chunked recurrences' scratch does:
// a product that needs more is done in portions of rows behind one another, in the same scratch.  28 slices of 1,728 x 4,096 would be
// 793 MB beside a result of 28.
constexpr long SCRATCH_BYTES = 256L << 20;
struct Portion { int rows; bool apart; };         // apart: slices in blocks of their own
static Portion portion(int M, int N, int K) {
    const int bm = tile_rows(M), slices = slices_of(K);
    if (slices == 1) return {M, false};
    bool apart = split(M, N, K);
    long most = SCRATCH_BYTES / 4 / N / (apart ? slices : 1) / bm * bm;
    if (apart && most < bm) {
        apart = false;
        most = SCRATCH_BYTES / 4 / N / bm * bm;
    }
    if (most < bm) most = bm;
    return {M < most ? M : (int)most, apart};
}

// Floats of scratch of a product (0: none).
GFB_API long gfb_gemm_simt_scratch_floats(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= SLICE) return 0;
    const Portion p = portion(M, N, K);
    return (long)(p.apart ? slices_of(K) : 1) * p.rows * N;
}

template <typename TA, typename TW, typename TC, int EPI>
static int run(const TA* A, const TW* W, TC* C, int M, int N, int K, bool apart, float* partial, cudaStream_t stream) {
    const int bm = tile_rows(M), bn = tile_cols(bm);
    const dim3 grid((N + bn - 1) / bn, (M + bm - 1) / bm, apart ? slices_of(K) : 1);
    const bool wide = K % 4 == 0 && ((uintptr_t)A & (4 * sizeof(TA) - 1)) == 0 && ((uintptr_t)W & (4 * sizeof(TW) - 1)) == 0;
    cudaError_t e;
#define GO(WM_, WN_, TM_, WIDE_) \
    e = apart ? gfb_launch(gemm_simt_kernel<TA, TW, float, EPI_STORE, WM_, WN_, TM_, WIDE_, true>, grid, dim3(THREADS), 0, stream, A, W, (float*)nullptr, M, N, K, partial) \
              : gfb_launch(gemm_simt_kernel<TA, TW, TC, EPI, WM_, WN_, TM_, WIDE_, false>, grid, dim3(THREADS), 0, stream, A, W, C, M, N, K, partial)
    if (bm == 16) { if (wide) GO(2, 2, 2, true); else GO(2, 2, 2, false); }
    else if (bm == 32) { if (wide) GO(1, 4, 8, true); else GO(1, 4, 8, false); }
    else { if (wide) GO(2, 2, 8, true); else GO(2, 2, 8, false); }
#undef GO
    if (gfb_check(e, "gfb_gemm_simt")) return 1;
    if (!apart) return 0;
    const size_t pairs = (size_t)M * ((N + 1) / 2);
    e = gfb_launch(gemm_simt_sum_kernel<TC, EPI>, dim3((unsigned)((pairs + 255) / 256)), dim3(256), 0, stream, (const float*)partial, C, M, N, slices_of(K));
    return gfb_check(e, "gfb_gemm_simt (sum)");
}

template <typename TA, typename TW, typename TC, int EPI>
static int portions(const void* A, const void* W, void* C, int M, int N, int K, float* partial, cudaStream_t stream) {
    if ((M + tile_rows(M) - 1) / tile_rows(M) > 65535) return gfb_fail("gfb_gemm_simt: M = %d is too large", M);
    const Portion p = portion(M, N, K);
    const size_t out_cols = EPI == EPI_SWIGLU ? N / 2 : N;
    for (int m = 0; m < M; m += p.rows)
        if (run<TA, TW, TC, EPI>((const TA*)A + (size_t)m * K, (const TW*)W, (TC*)C + m * out_cols, M - m < p.rows ? M - m : p.rows, N, K, p.apart, partial, stream))
            return 1;
    return 0;
}

template <typename TA, typename TW, typename TC>
static int launch(const void* A, const void* W, void* C, int M, int N, int K, int epi, float* partial, cudaStream_t stream) {
    if (epi == EPI_STORE) return portions<TA, TW, TC, EPI_STORE>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_ADD) return portions<TA, TW, TC, EPI_ADD>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_SWIGLU) return portions<TA, TW, TC, EPI_SWIGLU>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_GELU) return portions<TA, TW, TC, EPI_GELU>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_GELU_TANH) return portions<TA, TW, TC, EPI_GELU_TANH>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_SILU) return portions<TA, TW, TC, EPI_SILU>(A, W, C, M, N, K, partial, stream);
    if (epi == EPI_RELU2) return portions<TA, TW, TC, EPI_RELU2>(A, W, C, M, N, K, partial, stream);
    return gfb_fail("gfb_gemm_simt: unknown epilogue %d", epi);
}

// in_dt: type of A and W; out_dt: type of C (ADD needs 32-bit C).  partial: room for gfb_gemm_simt_scratch_floats numbers where
// that is not 0.
GFB_API int gfb_gemm_simt(const void* A, const void* W, void* C, int in_dt, int out_dt, int M, int N, int K,
                          int epi, float* partial, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return gfb_fail("gfb_gemm_simt: K = %d", K);
    if (epi == EPI_ADD && out_dt != GFB_F32) return gfb_fail("gfb_gemm_simt: the residual sum is kept in 32-bit");
    if (epi == EPI_SWIGLU && (N & 1)) return gfb_fail("gfb_gemm_simt: SwiGLU needs an even number of rows, got %d", N);
    if (partial == nullptr && gfb_gemm_simt_scratch_floats(M, N, K) > 0) return gfb_fail("gfb_gemm_simt: K = %d needs room for its slices", K);
    typedef __nv_bfloat16 bf16;
    if (in_dt == GFB_F32 && out_dt == GFB_F32) return launch<float, float, float>(A, W, C, M, N, K, epi, partial, stream);
    if (in_dt == GFB_BF16 && out_dt == GFB_BF16) return launch<bf16, bf16, bf16>(A, W, C, M, N, K, epi, partial, stream);
    if (in_dt == GFB_BF16 && out_dt == GFB_F32) return launch<bf16, bf16, float>(A, W, C, M, N, K, epi, partial, stream);
    return gfb_fail("gfb_gemm_simt: unsupported types in %d out %d", in_dt, out_dt);
}
