// C[M,N] = A[M,K] * W[N,K]^T of 32-bit numbers on the tensor cores, each number as the sum of three bfloat16.
//
// a = a1 + a2 + a3 without a remainder from 2^-110 on (8 bits each; a1 truncated, so that the largest numbers stay finite), likewise w, and
//     a w = a1 w1 + (a1 w2 + a2 w1) + (a1 w3 + a2 w2 + a3 w1) + terms below 2^-22 of it and of either sign:
// six bfloat16 products with exact 16-bit results.  What is left to lose is the order and the rounding of the sum, which the tensor cores cut
// off instead of rounding.  So an accumulator in tensor memory holds 32 numbers of k at most, its small terms first, and a thread
// adds the accumulators up in registers, rounding each sum: 2 sums cut off and one rounded per 32 numbers, where the CUDA cores' chain
// rounds 32 times.  Against 64 bits, numbers of unit scale: 0.9e-7 (K = 512) to 2.1e-7 (14,336), on CUDA cores 4.1e-7; sums that are
// little more than their largest product 5.5e-8, there 2.8e-8, since the one sum that counts is cut off here and rounded there.
//
// us here | on CUDA cores, captured, K = 3,072: 198 rows times 16,384 columns 107 | 525, times 5,120 42 | 179; one row times 16,384 84 | 103, times
// 128,256 481 | 700; 2,048 rows times 5,120 360 | 1,417; 198 rows of 8,192 numbers times 3,072 57 | 288.  At 198 rows the tensor pipe is busy for 69 % of
// the time (12 multiplications of 128 x 208 x 16 read 10 KB each per stage, beside the copies and the planes); at few rows the way from weight to sum bounds it.
//
// An element's order of summation depends on N and K alone: accumulators of 32 k in ascending order, in `splits_of(N, K)`
// portions of K whose sums are added in ascending order by a kernel of their own.  A row's bits do not depend on the other rows.
//
// Roles in a block of 320 threads: warp 0 = TMA producer, warp 1 = tensor memory and MMA issue (one lane each), warps 2 to 9 split the
// weights (32-bit tile in shared memory -> three bfloat16 planes) and then add the accumulator of the stage before.  The 128 weight
// rows of a tile are the rows of the MMA, up to 256 tokens its columns.  The activations come in three planes that `split_rows_kernel`
// wrote, since every block reads them; a weight is read, and split, once per 256 tokens.
//
// A sum that is not finite (an infinite or NaN operand: its pieces cannot hold it; an overflow on the way), or so small that the operands' pieces
// may have missed bits that count, is worked out once more from the 32-bit numbers, by a warp, before the epilogue: eight columns that read a row of A
// once, given up where all are NaN.  That is for the odd row.  Where every sum needs it, 198 rows of 3,072 numbers times 16,384 columns
// take 1.4 ms with NaNs throughout and 10.2 ms with an infinity in every row (column by column 23.1), 16 rows of 1,024 times 4,096 0.1 and 0.2 ms.
// Every wait is bounded by time, as in the bfloat16 product.
//
// Epilogues as in gemm_simt.cu, which keeps the products this kernel does not take (rows that are no multiple of 16 bytes, bfloat16).
#include "common.cuh"

#include <cuda.h>

GFB_DEFINE_LAST_ERROR()

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_GELU = 4, EPI_GELU_TANH = 5, EPI_SILU = 6, EPI_RELU2 = 7 };

namespace {

constexpr int BM = 128;              // weight rows per tile
constexpr int BK = 32;               // k per stage and per accumulator
constexpr int THREADS = 320, SPLITTERS = 8;
constexpr int W_STAGE = BM * BK * 4, W_PLANE = BM * BK * 2, X_ROW = BK * 2;
constexpr int MAX_RING = 8;
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

// Stages of the 32-bit weights, of the activations' planes and of the weights' planes (each with an accumulator of its own), by 16-column
// groups per warp (tiles of up to 32 * CH tokens).  A stage of few tokens is over sooner than its way from plane to sum, so more are under way.
template <int CH> struct Ring {
    static constexpr int W = CH == 8 ? 4 : CH == 4 ? 4 : CH == 2 ? 5 : 6, X = CH == 8 ? 2 : 3, P = CH == 8 ? 2 : CH == 4 ? 3 : 4;
    static constexpr int COLS = CH == 4 ? 512 : P * 32 * CH;                        // of tensor memory: a power of two
};

struct Barriers {
    unsigned long long w_full[MAX_RING], w_empty[MAX_RING], x_full[MAX_RING], x_empty[MAX_RING];
    unsigned long long planes[4];    // the weights' planes of a stage are written
    unsigned long long done[4];      // a stage's accumulator is complete, its planes are free
    unsigned long long taken[4];     // an accumulator has been added up
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int which) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 128; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > WAIT_LIMIT_NS) {
            *abort_flag = 1;
            gfb_report(status, GFB_ERR_WAIT_TIMEOUT, which, (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)));
            return false;
        }
        __nanosleep(64);
    }
}
// The same for a whole warp: one answer for all its lanes.  Where a wait runs out lanes can differ (one sees the abort flag, another its barrier), and
// a warp that parted there would never meet again at the aligned instructions behind it.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int which) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, which));
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}

// Shared-memory matrix descriptor of a K-major tile of 64-byte rows with 64-byte swizzle: groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                        // layout: 64-byte swizzle
    return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// the eight warps that split and add, all or none
__device__ __forceinline__ bool splitters_all(bool flag) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"((uint32_t)flag) : "memory");
    return all != 0;
}

// Two numbers into three pairs of bfloat16 (the first number in the low half).  Each remainder is exact; one that is not finite stays
// so in the sum.
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    p1 = __byte_perm(ua, ub, 0x7632);                                            // the upper halves: truncated
    const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(ra, rb);
    p2 = *reinterpret_cast<const uint32_t*>(&h2);
    const __nv_bfloat162 h3 = __floats2bfloat162_rn(ra - __uint_as_float(p2 << 16), rb - __uint_as_float(p2 & 0xffff0000u));
    p3 = *reinterpret_cast<const uint32_t*>(&h3);
}

template <int EPI>
__device__ __forceinline__ float unary(float z) {
    if (EPI == EPI_GELU) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
    if (EPI == EPI_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
    if (EPI == EPI_SILU) return z / (1.0f + expf(-z));
    if (EPI == EPI_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
    return z;
}

// Row m of A times rows n .. n + COLS - 1 of W (the last of them at most N - 1) by a whole warp, in 64 bits, so that only infinities and NaNs of the
// operands, or a sum beyond 32 bits, come out as such.  Column n + u's sum goes to lane u.  The order of a sum is that of its k alone.
constexpr int COLS = 8, LOOK = 512;
__device__ __noinline__ float whole_dots(const float* __restrict__ A, const float* __restrict__ W, int m, int n, int N, int K) {
    const int lane = threadIdx.x & 31;
    const float* a = A + (size_t)m * K;
    double s[COLS];
#pragma unroll
    for (int u = 0; u < COLS; u++) s[u] = 0.0;
    for (int k0 = 0; k0 < K; k0 += LOOK) {
        const int end = min(K, k0 + LOOK);
#pragma unroll 4
        for (int k = k0 + lane; k < end; k += 32) {
            const double x = a[k];
#pragma unroll
            for (int u = 0; u < COLS; u++) s[u] = fma(x, (double)W[(size_t)min(n + u, N - 1) * K + k], s[u]);
        }
        bool over = true;                        // NaNs stay what they are
#pragma unroll
        for (int u = 0; u < COLS; u++) over = over && __any_sync(0xffffffffu, isnan(s[u]));
        if (over) break;
    }
    float mine = 0.f;
#pragma unroll
    for (int u = 0; u < COLS; u++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
        if (lane == u) mine = (float)s[u];
    }
    return mine;
}

// Where pieces miss a number.  bfloat16 ends at 2^-133 (and as normal numbers at 2^-126), so a number below 2^-110 loses its last bits, at most
// 2^-126 of it however the tensor cores take subnormal pieces.  A row of A without a number of 2^-96 has all its sums worked out from the 32-bit
// numbers (`least` infinite), a row of zeros none (zero).  In any other row its own numbers lose less than 2^-30 of the largest, and the weights' losses, K 2^-126 times that
// largest at most, are below 2^-26 of every sum from K 2^-100 times the largest (and 2^-100 K) on; smaller sums are worked out as well.
constexpr float SMALL_ROW = 0x1p-96f, SMALL_SUM = 0x1p-100f;

// Whether a sum of a row may have to be worked out once more: not finite, or smaller than the row's `least` (as bits: not in [least, infinity)).
__device__ __forceinline__ bool doubtful(float v, uint32_t least) { return (__float_as_uint(v) & 0x7fffffffu) - least >= 0x7f800000u - least; }

// Four neighbouring sums of row m, from column n on: the doubtful ones are worked out once more (a whole warp comes here).  A sum of zero is
// left in any row but a small one: its weights are zeros, or none of them is a number of bfloat16 (2^-133).
__device__ __noinline__ float4 mended(float4 sums, const float* __restrict__ A, const float* __restrict__ W, uint32_t least, int m, int n, int N, int K) {
    float v[4] = {sums.x, sums.y, sums.z, sums.w};
    const int lane = threadIdx.x & 31;
    uint32_t bad = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (n + u < N && doubtful(v[u], least) && (v[u] != 0.f || least == 0x7f800000u)) bad |= 1u << u;
    }
    uint32_t lanes = __ballot_sync(0xffffffffu, bad != 0);
    while (lanes) {                              // two lanes' columns at a time, where they are neighbours in a row
        const int l = __ffs(lanes) - 1;
        const int mm = __shfl_sync(0xffffffffu, m, l), nn = __shfl_sync(0xffffffffu, n, l);
        const bool pair = l < 31 && __shfl_sync(0xffffffffu, m, (l + 1) & 31) == mm && __shfl_sync(0xffffffffu, n, (l + 1) & 31) == nn + 4;
        const float s = whole_dots(A, W, mm, nn, N, K);
        const int from = lane == l ? 0 : 4;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float x = __shfl_sync(0xffffffffu, s, from + u);
            if ((lane == l || (pair && lane == l + 1)) && (bad >> u & 1)) v[u] = x;
        }
        lanes &= ~((pair ? 3u : 1u) << l);
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// four neighbouring sums through the epilogue; n is a multiple of four
template <int EPI>
__device__ __forceinline__ void finish4(float* __restrict__ C, int m, int n, int N, const float (&v)[4]) {
    if (n >= N) return;
    if (EPI == EPI_SWIGLU) {                      // gate, up, gate, up; N is even
        float* c = C + (size_t)m * (N >> 1) + (n >> 1);
        c[0] = v[0] / (1.f + expf(-v[0])) * v[1];
        if (n + 2 < N) c[1] = v[2] / (1.f + expf(-v[2])) * v[3];
        return;
    }
    float* c = C + (size_t)m * N + n;
    if ((N & 3) == 0 && ((uintptr_t)C & 15) == 0) {
        float4 o = EPI == EPI_ADD ? *reinterpret_cast<const float4*>(c) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (EPI == EPI_ADD) { o.x += v[0]; o.y += v[1]; o.z += v[2]; o.w += v[3]; }
        else o = make_float4(unary<EPI>(v[0]), unary<EPI>(v[1]), unary<EPI>(v[2]), unary<EPI>(v[3]));
        *reinterpret_cast<float4*>(c) = o;
        return;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (n + u < N) c[u] = EPI == EPI_ADD ? c[u] + v[u] : unary<EPI>(v[u]);
}

// planes[p][m][k]: piece p of A[m][k], zeros from K to Kp.  A block takes a row, eight numbers per thread and step, and says from which size
// on (by its bits) the row's sums are to be had from pieces (see below).
constexpr int ROW_THREADS = 1024;            // at most

__global__ void __launch_bounds__(ROW_THREADS)
split_rows_kernel(const float* __restrict__ A, __nv_bfloat16* __restrict__ planes, uint32_t* __restrict__ least, int M, int K, int Kp, int wide) {
    __shared__ uint32_t warps[ROW_THREADS / 32];
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int m = blockIdx.x;
    uint32_t largest = 0;                                            // by its bits: infinities and NaNs are the largest
    for (int k = threadIdx.x * 8; k < Kp; k += blockDim.x * 8) {
        const float* a = A + (size_t)m * K + k;
        float v[8];
        if (wide && k + 8 <= K) {
            const float4 lo = *reinterpret_cast<const float4*>(a), hi = *reinterpret_cast<const float4*>(a + 4);
            v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = k + i < K ? a[i] : 0.f;
        }
        uint32_t p[3][4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            split2(v[2 * i], v[2 * i + 1], p[0][i], p[1][i], p[2][i]);
            largest = max(largest, max(__float_as_uint(v[2 * i]) & 0x7fffffffu, __float_as_uint(v[2 * i + 1]) & 0x7fffffffu));
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
            *reinterpret_cast<uint4*>(planes + (size_t)q * M * Kp + (size_t)m * Kp + k) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
    largest = __reduce_max_sync(0xffffffffu, largest);
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = largest;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    largest = __reduce_max_sync(0xffffffffu, threadIdx.x < blockDim.x / 32 ? warps[threadIdx.x] : 0u);
    const float top = __uint_as_float(largest);
    if (threadIdx.x == 0) least[m] = largest == 0 ? 0u : __float_as_uint(top < SMALL_ROW ? INFINITY : (float)K * SMALL_SUM * fmaxf(top, 1.f));
}

// A tile of 128 weight rows (blockIdx.y) by bn tokens (blockIdx.x; bn a multiple of 16, at most 32 * CH) over one portion of K (blockIdx.z).
// PARTIAL: the sums go to C [splits][M][N] as they are.
template <int CH, int EPI, bool PARTIAL>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* __restrict__ A,
                  const float* __restrict__ W, const uint32_t* __restrict__ least, float* __restrict__ C, int M, int N, int K, int bn, int stages_per_split,
                  int* status) {
    constexpr int NW = Ring<CH>::W, NX = Ring<CH>::X, NP = Ring<CH>::P, LAG = NW - NX;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t ws = base, ps = ws + NW * W_STAGE, xs = ps + NP * 3 * W_PLANE;
    const int x_plane = bn * X_ROW;
    Barriers* bars = reinterpret_cast<Barriers*>(aligned + NW * W_STAGE + NP * 3 * W_PLANE + NX * 3 * (32 * CH * X_ROW));
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * bn, n0 = blockIdx.y * BM;
    const int first = blockIdx.z * stages_per_split, n_stages = min(stages_per_split, (K + BK - 1) / BK - first);

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_x)) : "memory");
        for (int s = 0; s < NW; s++) {
            mbar_init(smem_u32(&bars->w_full[s]), 1);
            mbar_init(smem_u32(&bars->w_empty[s]), SPLITTERS);
        }
        for (int s = 0; s < NX; s++) {
            mbar_init(smem_u32(&bars->x_full[s]), 1);
            mbar_init(smem_u32(&bars->x_empty[s]), 1);
        }
        for (int b = 0; b < NP; b++) {
            mbar_init(smem_u32(&bars->planes[b]), SPLITTERS);
            mbar_init(smem_u32(&bars->done[b]), 1);
            mbar_init(smem_u32(&bars->taken[b]), SPLITTERS);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"((uint32_t)Ring<CH>::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    gfb_pdl_launch();
    gfb_pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            // The weights run ahead of the activations by the difference of the rings' lengths: a stage of weights is free once it is
            // split, one of activations once it is multiplied.
            for (int i = 0; i < n_stages + LAG; i++) {
                if (i < n_stages) {
                    const int s = i % NW;
                    if (!mbar_wait(smem_u32(&bars->w_empty[s]), (uint32_t)(i / NW & 1) ^ 1u, abort_flag, status, 1)) break;
                    mbar_expect_tx(smem_u32(&bars->w_full[s]), W_STAGE);
                    tma_load_2d(ws + s * W_STAGE, &map_w, (first + i) * BK, n0, smem_u32(&bars->w_full[s]));
                }
                const int j = i - LAG;
                if (j >= 0) {
                    const int s = j % NX;
                    if (!mbar_wait(smem_u32(&bars->x_empty[s]), (uint32_t)(j / NX & 1) ^ 1u, abort_flag, status, 2)) break;
                    mbar_expect_tx(smem_u32(&bars->x_full[s]), 3 * x_plane);
                    tma_load_3d(xs + s * 3 * x_plane, &map_x, (first + j) * BK, m0, 0, smem_u32(&bars->x_full[s]));
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            for (int i = 0; i < n_stages; i++) {
                const int s = i % NX, b = i % NP;
                if (!mbar_wait(smem_u32(&bars->taken[b]), (uint32_t)(i / NP & 1) ^ 1u, abort_flag, status, 3)) break;
                if (!mbar_wait(smem_u32(&bars->x_full[s]), (uint32_t)(i / NX & 1), abort_flag, status, 4)) break;
                if (!mbar_wait(smem_u32(&bars->planes[b]), (uint32_t)(i / NP & 1), abort_flag, status, 5)) break;
                tc_fence_after();
                const uint32_t acc = tmem + (uint32_t)(b * 32 * CH);
                const uint64_t dw = umma_smem_desc(ps + b * 3 * W_PLANE), dx = umma_smem_desc(xs + s * 3 * x_plane);
                constexpr int WP[6] = {2, 1, 0, 1, 0, 0}, XP[6] = {0, 1, 2, 0, 1, 0};       // the smallest terms first
#pragma unroll
                for (int t = 0; t < 6; t++)
#pragma unroll
                    for (int k = 0; k < BK / 16; k++)
                        umma_bf16(acc, dw + (WP[t] * W_PLANE >> 4) + 2 * k, dx + (uint64_t)(XP[t] * x_plane >> 4) + 2 * k, idesc, (t | k) != 0);
                umma_commit(smem_u32(&bars->x_empty[s]));
                umma_commit(smem_u32(&bars->done[b]));
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2, w8 = warp - 2;
        const int groups = bn >> 4, low = (groups + 1) >> 1;
        const int g0 = half ? low : 0, mine = half ? groups - low : low;           // this warp's groups of 16 columns
        const int n_tok = min(bn, M - m0);
        const uint32_t lowest = !PARTIAL && w8 + SPLITTERS * lane < n_tok ? least[m0 + w8 + SPLITTERS * lane] : 0u;     // of the warp's tokens below, one per lane
        float sum[CH][16];
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int j = 0; j < 16; j++) sum[c][j] = 0.f;
        bool ok = true;
        for (int i = 0; i < n_stages + NP - 1 && ok; i++) {
            if (i < n_stages) {                  // (the planes are free: stage i - NP has been added up below)
                const int s = i % NW, b = i % NP;
                ok = mbar_wait_warp(smem_u32(&bars->w_full[s]), (uint32_t)(i / NW & 1), abort_flag, status, 6);
                if (!ok) break;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = w8 * 16 + h * 8 + (lane >> 2), g = lane & 3;     // a row's eight numbers from 8 g on
                    const uint8_t* src = aligned + s * W_STAGE + r * 128;
                    const float4 lo = *reinterpret_cast<const float4*>(src + (((2 * g) ^ (r & 7)) << 4));
                    const float4 hi = *reinterpret_cast<const float4*>(src + (((2 * g + 1) ^ (r & 7)) << 4));
                    uint32_t p[3][4];
                    split2(lo.x, lo.y, p[0][0], p[1][0], p[2][0]);
                    split2(lo.z, lo.w, p[0][1], p[1][1], p[2][1]);
                    split2(hi.x, hi.y, p[0][2], p[1][2], p[2][2]);
                    split2(hi.z, hi.w, p[0][3], p[1][3], p[2][3]);
                    uint8_t* dst = aligned + NW * W_STAGE + b * 3 * W_PLANE + r * X_ROW + ((g ^ (r >> 1 & 3)) << 4);
#pragma unroll
                    for (int t = 0; t < 3; t++) *reinterpret_cast<uint4*>(dst + t * W_PLANE) = make_uint4(p[t][0], p[t][1], p[t][2], p[t][3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(smem_u32(&bars->w_empty[s]));
                    mbar_arrive(smem_u32(&bars->planes[b]));
                }
            }
            if (const int d = i - (NP - 1); d >= 0) {
                const int b = d % NP;
                ok = mbar_wait_warp(smem_u32(&bars->done[b]), (uint32_t)(d / NP & 1), abort_flag, status, 7);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 32 * CH + g0 * 16);
#pragma unroll
                for (int c = 0; c < CH; c++)
                    if (c < mine) {
                        uint32_t raw[16];
                        tmem_ld16(taddr + c * 16, raw);
#pragma unroll
                        for (int j = 0; j < 16; j++) sum[c][j] += __uint_as_float(raw[j]);
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->taken[b]));
            }
        }
        // The tile goes through shared memory (every copy has landed and been read), so that a warp writes a token's 128 rows side by side.
        if (splitters_all(ok)) {
            float* tile = reinterpret_cast<float*>(aligned);                        // [tokens][128 rows]
#pragma unroll
            for (int c = 0; c < CH; c++)
                if (c < mine)
#pragma unroll
                    for (int j = 0; j < 16; j++) tile[((g0 + c) * 16 + j) * BM + q * 32 + lane] = sum[c][j];
            asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
            const int n = n0 + 4 * lane;
#pragma unroll 2
            for (int j = w8; j < n_tok; j += SPLITTERS) {
                float4 t = *reinterpret_cast<const float4*>(tile + j * BM + 4 * lane);
                if (!PARTIAL) {
                    const uint32_t low = __shfl_sync(0xffffffffu, lowest, j / SPLITTERS);
                    if (__any_sync(0xffffffffu, doubtful(t.x, low) || doubtful(t.y, low) || doubtful(t.z, low) || doubtful(t.w, low)))
                        t = mended(t, A, W, low, m0 + j, n, N, K);
                }
                const float v[4] = {t.x, t.y, t.z, t.w};
                if (PARTIAL) finish4<EPI_STORE>(C + (size_t)blockIdx.z * M * N, m0 + j, n, N, v);
                else finish4<EPI>(C, m0 + j, n, N, v);
            }
        }
    }

    if (*abort_flag) {                           // copies that were issued may still be landing
        unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Ring<CH>::COLS) : "memory");
    }
}

// the portions of every sum, in ascending order, and the epilogue; a thread per four columns
template <int EPI>
__global__ void __launch_bounds__(256, 5)        // (the rare call may spill; the sums want many blocks under way)
split_sum_kernel(const float* __restrict__ partial, const float* __restrict__ A, const float* __restrict__ W, const uint32_t* __restrict__ least,
                 float* __restrict__ C, int M, int N, int K, int splits) {
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int units = (N + 3) / 4;
    const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
    const bool in = e < (size_t)M * units;
    const int m = in ? (int)(e / units) : 0, n = in ? (int)(e - (size_t)m * units) * 4 : N;      // (n = N: nothing to do, but the warp stays whole)
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (in) {
        const float* p = partial + (size_t)m * N + n;
        const bool wide = (N & 3) == 0;                             // (partial is 16-byte aligned)
        for (int s = 0; s < splits; s++, p += (size_t)M * N) {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
            if (wide) {
                const float4 x = *reinterpret_cast<const float4*>(p);
                t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (n + u < N) t[u] = p[u];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = s == 0 ? t[u] : v[u] + t[u];
        }
    }
    const uint32_t low = least[m];
    if (__any_sync(0xffffffffu, in && (doubtful(v[0], low) || doubtful(v[1], low) || doubtful(v[2], low) || doubtful(v[3], low)))) {
        const float4 t = mended(make_float4(v[0], v[1], v[2], v[3]), A, W, low, m, n, N, K);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    finish4<EPI>(C, m, n, N, v);
}

// ---- host side ----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

int encoded(CUresult r, const char* what) {
    return r == CUDA_SUCCESS ? 0 : gfb_fail("gfb_gemm_split: cuTensorMapEncodeTiled failed with %d (%s)", (int)r, what);
}

int make_maps(CUtensorMap* mw, CUtensorMap* mx, const float* W, const void* planes, int M, int N, int K, int Kp, int bn) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return gfb_fail("gfb_gemm_split: the driver does not export cuTensorMapEncodeTiled");
    const cuuint32_t ones[3] = {1, 1, 1};
    const cuuint64_t wd[2] = {(cuuint64_t)K, (cuuint64_t)N}, wstr[1] = {(cuuint64_t)K * 4};
    const cuuint32_t wb[2] = {BK, BM};
    if (encoded(enc(mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), wd, wstr, wb, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE), "weights")) return 1;
    const cuuint64_t xd[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3}, xstr[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)M * Kp * 2};
    const cuuint32_t xb[3] = {BK, (cuuint32_t)bn, 3};
    return encoded(enc(mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(planes), xd, xstr, xb, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE), "activations");
}

// Portions of K, each summed by blocks of its own, so that one tile of tokens fills the chip: a cost model in stages of 32 k, six of which go
// into a block's start and end, with the partial sums' way through memory.  By N and K alone, since it is part of the order of summation.
int stages_per_split(int N, int K) {
    const long tiles = (N + BM - 1) / BM;
    const int all = (K + BK - 1) / BK;
    int best = all;
    double best_cost = 0;
    // Few tiles of long rows take more portions.  us for one row | on CUDA cores: 8,192 numbers times 256 columns 13.1 | 15.4 (16 portions: 16.7), 14,336 times
    // 256 15.3 | 22.6 (24.8), times 2 14.8 | 13.9 (24.7), 28,672 times 2 20.9 | 14.8 (43.9), times 512 27.8 | 39.1 (44.4).
    const long few = K / (256 * (tiles > 2 ? tiles / 2 : 1));
    const int most = few > 64 ? 64 : few < 16 ? 16 : (int)few;
    for (int s = 1; s <= most && s <= all; s++) {
        const int per = (all + s - 1) / s, real = (all + per - 1) / per;
        if (real != s) continue;
        const double cost = (double)((tiles * s + 147) / 148) * (per + 6) + (s > 1 ? 4 + s * (N / 3000.0) : 0);
        if (s == 1 || cost < best_cost) { best = per; best_cost = cost; }
    }
    return best;
}
int splits_of(int N, int K) {
    const int per = stages_per_split(N, K);
    return ((K + BK - 1) / BK + per - 1) / per;
}

long aligned(long bytes) { return (bytes + 255) / 256 * 256; }

// The rows of A that one launch takes: its planes and partial sums stay below 256 MB (or are one tile's).
constexpr long SCRATCH_BYTES = 256L << 20;
long row_bytes(int N, int K) {
    const int splits = splits_of(N, K);
    return 4 + 6L * ((K + 7) / 8 * 8) + (splits > 1 ? 4L * splits * N : 0);
}
int portion(int M, int N, int K) {
    long most = (SCRATCH_BYTES - 512) / row_bytes(N, K) / 256 * 256;
    if (most < 256) most = 256;
    return M < most ? M : (int)most;
}

template <int CH> size_t smem_bytes() {
    return 1024 + (size_t)Ring<CH>::W * W_STAGE + Ring<CH>::P * 3 * W_PLANE + (size_t)Ring<CH>::X * 3 * (32 * CH * X_ROW) + sizeof(Barriers);
}

template <int CH, int EPI, bool PARTIAL>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const float* A, const float* W, const uint32_t* least, float* C, int M, int N, int K, int bn, int* status, cudaStream_t stream) {
    static_assert(Ring<CH>::W * W_STAGE + Ring<CH>::P * 3 * W_PLANE + Ring<CH>::X * 3 * 32 * CH * X_ROW >= 32 * CH * BM * 4, "the tile of sums fits the rings");
    static_assert(Ring<CH>::X <= Ring<CH>::W && Ring<CH>::W <= MAX_RING, "rings");
    auto kern = gemm_split_kernel<CH, EPI, PARTIAL>;
    const size_t smem = smem_bytes<CH>();
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return gfb_fail("gfb_gemm_split: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    const dim3 grid((M + bn - 1) / bn, (N + BM - 1) / BM, PARTIAL ? splits_of(N, K) : 1);
    const int per = PARTIAL ? stages_per_split(N, K) : (K + BK - 1) / BK;
    return gfb_check(gfb_launch(kern, grid, dim3(THREADS), smem, stream, mw, mx, A, W, least, C, M, N, K, bn, per, status), "gfb_gemm_split");
}

template <int EPI, bool PARTIAL>
int launch_by_width(const CUtensorMap& mw, const CUtensorMap& mx, const float* A, const float* W, const uint32_t* least, float* C, int M, int N, int K, int bn, int* status,
                    cudaStream_t stream) {
    if (bn <= 32) return launch<1, EPI, PARTIAL>(mw, mx, A, W, least, C, M, N, K, bn, status, stream);
    if (bn <= 64) return launch<2, EPI, PARTIAL>(mw, mx, A, W, least, C, M, N, K, bn, status, stream);
    if (bn <= 128) return launch<4, EPI, PARTIAL>(mw, mx, A, W, least, C, M, N, K, bn, status, stream);
    return launch<8, EPI, PARTIAL>(mw, mx, A, W, least, C, M, N, K, bn, status, stream);
}

template <int EPI>
int run(const float* A, const float* W, float* C, int M, int N, int K, uint8_t* scratch, int* status, cudaStream_t stream) {
    const int Kp = (K + 7) / 8 * 8, splits = splits_of(N, K);
    __nv_bfloat16* planes = reinterpret_cast<__nv_bfloat16*>(scratch);
    uint32_t* least = reinterpret_cast<uint32_t*>(scratch + aligned(6L * M * Kp));
    float* partial = reinterpret_cast<float*>(scratch + aligned(6L * M * Kp) + aligned(4L * M));
    const int steps = (Kp / 8 + ROW_THREADS - 1) / ROW_THREADS, row_threads = ((Kp / 8 + steps - 1) / steps + 31) / 32 * 32;
    if (gfb_check(gfb_launch(split_rows_kernel, dim3((unsigned)M), dim3((unsigned)row_threads), 0, stream, A, planes, least, M, K, Kp, (int)(((uintptr_t)A & 15) == 0)),
                  "gfb_gemm_split (rows)")) return 1;
    const int tiles = (M + 255) / 256, bn = ((M + tiles - 1) / tiles + 15) / 16 * 16;
    CUtensorMap mw, mx;
    if (make_maps(&mw, &mx, W, planes, M, N, K, Kp, bn)) return 1;
    if (splits == 1) return launch_by_width<EPI, false>(mw, mx, A, W, least, C, M, N, K, bn, status, stream);
    if (launch_by_width<EPI_STORE, true>(mw, mx, A, W, least, partial, M, N, K, bn, status, stream)) return 1;
    const size_t sums = (size_t)M * ((N + 3) / 4);
    return gfb_check(gfb_launch(split_sum_kernel<EPI>, dim3((unsigned)((sums + 255) / 256)), dim3(256), 0, stream, (const float*)partial, A, W, (const uint32_t*)least, C, M, N, K,
                                splits), "gfb_gemm_split (sum)");
}

template <int EPI>
int portions(const float* A, const float* W, float* C, int M, int N, int K, uint8_t* scratch, int* status, cudaStream_t stream) {
    const int rows = portion(M, N, K);
    const size_t out_cols = EPI == EPI_SWIGLU ? N / 2 : N;
    for (int m = 0; m < M; m += rows)
        if (run<EPI>(A + (size_t)m * K, W, C + m * out_cols, M - m < rows ? M - m : rows, N, K, scratch, status, stream)) return 1;
    return 0;
}

}  // namespace

// Bytes of scratch of a product.
GFB_API long gfb_gemm_split_scratch_bytes(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const long rows = portion(M, N, K);
    return aligned(6L * rows * ((K + 7) / 8 * 8)) + aligned(4L * rows) + (splits_of(N, K) > 1 ? 4L * splits_of(N, K) * rows * N : 0);
}

// A, W, C 32-bit; W 16-byte aligned with rows of whole 16-byte units; scratch: gfb_gemm_split_scratch_bytes, 256-byte aligned.
GFB_API int gfb_gemm_split(const float* A, const float* W, float* C, int M, int N, int K, int epi, void* scratch, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4) return gfb_fail("gfb_gemm_split: K = %d must be a positive multiple of 4 (16-byte rows for TMA)", K);
    if ((uintptr_t)W & 15) return gfb_fail("gfb_gemm_split: the weights must be 16-byte aligned");
    if ((uintptr_t)scratch & 255 || scratch == nullptr) return gfb_fail("gfb_gemm_split: needs 256-byte aligned scratch");
    if (epi == EPI_SWIGLU && (N & 1)) return gfb_fail("gfb_gemm_split: SwiGLU needs an even number of rows, got %d", N);
    if ((N + BM - 1) / BM > 65535) return gfb_fail("gfb_gemm_split: N = %d is too large", N);
    uint8_t* s = static_cast<uint8_t*>(scratch);
    if (epi == EPI_STORE) return portions<EPI_STORE>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_ADD) return portions<EPI_ADD>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_SWIGLU) return portions<EPI_SWIGLU>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_GELU) return portions<EPI_GELU>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_GELU_TANH) return portions<EPI_GELU_TANH>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_SILU) return portions<EPI_SILU>(A, W, C, M, N, K, s, status, stream);
    if (epi == EPI_RELU2) return portions<EPI_RELU2>(A, W, C, M, N, K, s, status, stream);
    return gfb_fail("gfb_gemm_split: unknown epilogue %d", epi);
}
