// Prefill attention on the 5th-generation tensor cores (tcgen05), head_dim 128 or 64, bfloat16.
//
// Causal attention of a run of new tokens over the paged cache (gpt-fast: the
// SDPA call of model.py:209-211).  A block owns one key/value head and a tile of
// TQ = 128 / (heads per group) consecutive query tokens of one sequence (rounded down: 42 tokens
// and 126 rows for 3 heads per group); its rows are the (token, head of the group) pairs, one per
// tensor-memory lane.
// Keys and values are visited 128 at a time (two pages of 64):
//
//   S = Q K^T        tcgen05.mma, A = Q and B = K from shared memory (TMA, 128B swizzle),
//                    S (32-bit) in tensor memory, two buffers
//   softmax          4 warps, one row per thread: tcgen05.ld of S, running maximum and sum
//                    in 32-bit registers, P rounded to bfloat16 and stored back into
//                    tensor memory (tcgen05.st); the reference maximum follows the true one
//                    lazily (steps of 2^8), and only then O is rescaled in tensor memory
//   O += P V         tcgen05.mma with A = P from tensor memory and B = V from shared
//                    memory as an MN-major operand (V lies [key][dim] in the cache)
//
// The MMA warp issues S of the next 128 keys before it waits for P of the current
// ones, so the tensor cores work while the softmax warps do.  Warp 0 is the TMA
// producer (Q once through a 3-D map over [token, head, dim] that lays the rows out
// as (token, head of group); K and V pages through 2-D maps over the pools), warp 1
// allocates tensor memory and issues the MMAs, warps 2..5 are the softmax and
// epilogue warps.  Every wait is bounded by wall-clock time (see gemm_tc.cu).
#include "common.cuh"

#include <cuda.h>
#include <cuda_fp16.h>

GFB_DEFINE_LAST_ERROR()

namespace {

constexpr int D = 128;                    // head_dim
constexpr int PAGE = 64;
constexpr int ROWS = 128;                 // query rows per block
constexpr int KEYS = 128;                 // keys per iteration (two pages)
constexpr int HALF_BYTES = 128 * 128;     // 128 rows x 64 elements x 2 bytes: one swizzled half tile
constexpr int TILE_BYTES = 2 * HALF_BYTES;
constexpr int KV_STAGES = 2;
static_assert(KV_STAGES == 2, "the one-tile kernel frees K/V stage s by the barriers of score buffer s");
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

// tensor-memory columns
constexpr uint32_t COL_S = 0;             // two score buffers of 128 columns
constexpr uint32_t COL_O = 256;           // output accumulator, 128 columns
constexpr uint32_t COL_P = 384;           // two probability buffers of 64 columns (bfloat16 pairs)

struct Bars {
    unsigned long long q_full, q_empty, o_free;
    unsigned long long k_full[KV_STAGES];     // (a K stage is free again when the scores of its block are done: s_full,
    unsigned long long v_full[KV_STAGES];     //  a V stage when its P V is: pv_done; a commit per barrier costs MMA issue time)
    unsigned long long s_full[2], s_empty[2];
    // P of the even / odd key blocks is written: one barrier would count two blocks together, since the scores of the next block are
    // issued ahead of the wait for P of this one and the quarters of the rows do not wait for one another
    unsigned long long p_ready[2];
    unsigned long long pv_done[2];            // P V of the even / odd key blocks has landed
    unsigned long long o_full;                // the item's last P V has landed (one phase per item)
    unsigned long long xch[4];                // per quarter of the rows: both warps of a row have written their half's maximum
    unsigned long long fin[4];                // the same for their sums at the end of an item
    unsigned long long tbl_free, tbl_full;    // the distance table in shared memory: all eight softmax warps have left the previous item's / written this item's
    uint32_t tmem_base;
    int abort_flag;
    float mx_half[2][2][ROWS];                // [key block parity][half][row]
    float l_half[2][2][ROWS];                 // [item parity][half][row]
};

// The first TMA copy through a tensor map fetches the 128-byte map; asking for it at once hides that behind the
// block's set-up.
__device__ __forceinline__ void prefetch_map(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
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
            gfb_report(status, GFB_ERR_WAIT_TIMEOUT, 100 + which, (int)(blockIdx.x + gridDim.x * blockIdx.y));
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
// K-major operand tile with 128-byte swizzle (rows of 128 bytes, 8-row groups 1024 bytes apart)
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// MN-major operand tile with 128-byte swizzle: rows are K (keys), 64 MN elements (dims) per 128-byte
// row; 8-row groups 1024 bytes apart (stride offset), the next 64 dims one half tile further (leading offset)
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t saddr, uint32_t half_bytes = HALF_BYTES) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(half_bytes >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N, int b_mn_major) { return idesc_bf16(M, N, b_mn_major) & ~((1u << 7) | (1u << 10)); }
__device__ __forceinline__ void umma_ss(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
// The same load without the wait, and the wait as a separate step that names the registers, so that the compiler
// keeps every use of them behind it: several loads can then be in flight before one wait.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait32(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
          "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
          "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
        :: "memory");
}
// a whole row of 128 scores: four loads in flight, then the wait
__device__ __forceinline__ void tmem_ld_row128(uint32_t taddr, float (*v)[32]) {
    uint32_t r[4][32];
#pragma unroll
    for (int c = 0; c < 4; c++) tmem_ld32_issue(taddr + c * 32, r[c]);
#pragma unroll
    for (int c = 0; c < 4; c++) tmem_ld_wait32(r[c]);
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
        for (int i = 0; i < 32; i++) v[c][i] = __uint_as_float(r[c][i]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr),
          "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
          "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
          "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
          "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
          "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
          "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
          "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
          "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// one column: a number per lane
__device__ __forceinline__ void tmem_st1(uint32_t taddr, float v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(__float_as_uint(v)) : "memory");
}
__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r) :: "memory");
    return __uint_as_float(r);
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two 32-bit lanes per instruction (sm_100): r = a * b + c and r = a + b on pairs; the maximum of three
__device__ __forceinline__ void fma2(float a0, float a1, float b, float c, float& r0, float& r1) {
    unsigned long long pa, pb, pc, pr;
    asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a0), "f"(a1));
    asm("mov.b64 %0, {%1, %1};" : "=l"(pb) : "f"(b));
    asm("mov.b64 %0, {%1, %1};" : "=l"(pc) : "f"(c));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(pr) : "l"(pa), "l"(pb), "l"(pc));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(pr));
}
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1) {
    unsigned long long pa, pb;
    asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a0), "f"(a1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b0), "f"(b1));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(pa) : "l"(pa), "l"(pb));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(pa));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack2_half(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// A bias on the score that depends on the head and on the distance n = query position - key position only, in units of
// the raw score (the bias divided by the score scale), so that it joins the score before scale and exponential.
//   table   null, or four copies [4][H][len] of a per-head array in which ascending entries belong to ascending keys:
//           entry u holds the bias at distance top - u; the first entries (distances beyond the last one the table tells
//           apart) all hold the far value, the entries beyond `top` (keys behind the query, masked anyway) are padding.
//           Copy s is the array moved down by s entries, so the 16-byte loads of a thread, whose first entry can have
//           any index, are aligned in the copy s = index mod 4.
//   slopes  null, or [H]: slopes[h] * n is taken off.
//   s_len, s_stride  (the one-tile kernel) not 0: the softmax warps copy the item's heads into shared memory, s_len entries
//           per head s_stride apart, entry k for distance k - TABLE_AHEAD, and read their biases there: read from global
//           memory, four copies of every head of a group outgrow the L1 cache and every block waits for L2.
struct DistanceBias {
    const float* table;
    int len, top;
    const float* slopes;
    int s_len, s_stride;
};
constexpr int TABLE_AHEAD = 256;         // entries for keys behind the query (masked): a tile's last block reaches up to 254 keys past a row
constexpr int TABLE_BEYOND = 256;        // entries past the window: a tile's first block starts up to 127 keys before its first row's window, rows are up to 127 apart

// v[c][i] belongs to key key0 + 32 c + i.
template <int NC>
__device__ __forceinline__ void add_distance_bias(float (&v)[NC][32], const DistanceBias& db, int H, int head, int row_pos, int key0) {
    if (db.table != nullptr) {
        // A block whose keys all lie beyond the table's reach starts below entry 0: the first NC * 32 entries hold the
        // far value, so the clamp reads the right numbers.  The upper clamp only moves loads of masked keys.
        const int u0 = min(max(db.top - row_pos + key0, 0), db.len - NC * 32 - 4);
        const int s = u0 & 3;
        const float4* src = reinterpret_cast<const float4*>(db.table + ((size_t)s * H + head) * db.len + (u0 - s));
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 t = __ldg(src + c * 8 + (i >> 2));
                v[c][i] += t.x; v[c][i + 1] += t.y; v[c][i + 2] += t.z; v[c][i + 3] += t.w;
            }
    }
    if (db.slopes != nullptr) {
        const float sl = __ldg(db.slopes + head);
        const float at0 = sl * (float)(key0 - row_pos);            // exact: distances are far below 2^24
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int i = 0; i < 32; i++) v[c][i] += fmaf(sl, (float)(c * 32 + i), at0);
    }
}

// The first key the query at `pos` sees: the window's edge, or the start of its block of `chunk` positions
// (blocks counted from position 0), whichever is later.
__device__ __forceinline__ int first_key(int pos, int window, int chunk) {
    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
    return lo;
}

// One (sequence, tile of TQ query tokens, key/value head) unit of work.
struct TileWork {
    int seq, tq0, g;
    int t_first, nq, slot, pos0, last_pos, first_lo, last_lo, blk0, n_iter, last_page;
};
// Work item w of the grid's list (long tiles first: the tile index runs backwards); false: an empty item.
__device__ __forceinline__ bool tile_work(const GfbBatch& b, int w, int n_x, int G, int TQ, int window, int chunk, TileWork& t) {
    const int xi = w / G;
    t.g = w - xi * G;
    t.seq = -1;
    int left = n_x - 1 - xi;
    for (int i = 0; i < b.n_seqs; i++) {
        const int qlen = b.cu_seqlens[i + 1] - b.cu_seqlens[i];
        const int nt = (qlen + TQ - 1) / TQ;
        if (left < nt) { t.seq = i; t.tq0 = left * TQ; break; }
        left -= nt;
    }
    if (t.seq < 0) return false;
    t.t_first = b.cu_seqlens[t.seq];
    const int qlen = b.cu_seqlens[t.seq + 1] - t.t_first;
    t.nq = min(TQ, qlen - t.tq0);
    t.slot = b.slots[t.seq];
    t.pos0 = b.lengths[t.slot] + t.tq0;
    t.last_pos = t.pos0 + t.nq - 1;
    t.first_lo = first_key(t.pos0, window, chunk);
    t.last_lo = first_key(t.last_pos, window, chunk);
    t.blk0 = t.first_lo / KEYS;
    t.n_iter = t.last_pos / KEYS + 1 - t.blk0;                   // key blocks [blk0, blk0 + n_iter)
    t.last_page = t.last_pos / PAGE;
    return true;
}

// The items are sorted by weight (long tiles first), so the blocks take them in a snake: pass 0 hands items
// 0 .. P-1 to blocks 0 .. P-1, pass 1 hands items P .. 2P-1 to blocks P-1 .. 0, and so on: the block with the
// heaviest item of one pass gets the lightest of the next.  (Past the end of the list the index only grows.)
__device__ __forceinline__ int snake_item(int pass, int block, int P) {
    return pass * P + ((pass & 1) ? P - 1 - block : block);
}

// Persistent: every block walks over its share of the n_work items (`snake_item`).  Barriers, tensor memory and the
// pipeline state are set up once; the counters of K/V stages and score buffers run on across items, so the first
// loads and the first S = Q K^T of the next item are under way while the softmax warps still write the
// previous item's output.  Two more barriers order the reuse of Q in shared memory (q_empty: the item's last
// S has read it) and of O in tensor memory (o_free: the softmax warps have read the finished output).
template <int DH>
__global__ void __launch_bounds__(320, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                       const int* __restrict__ page_table, int max_pages, int n_pages_pool,
                       GfbBatch b, int H, int G, float scale_log2e, int window, int chunk, const float* __restrict__ sink,
                       DistanceBias db, int n_x, int* status, float cap_raw, float* __restrict__ lse_out) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_q); prefetch_map(&map_k); prefetch_map(&map_v); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t qs = base;                                            // [2 halves][128 rows][128 B]
    const uint32_t ks = base + TILE_BYTES;                               // KV_STAGES x same, rows = keys
    const uint32_t vs = ks + KV_STAGES * TILE_BYTES;
    Bars* bars = reinterpret_cast<Bars*>(aligned + (size_t)(1 + 2 * KV_STAGES) * TILE_BYTES);
    float* bias_s = reinterpret_cast<float*>(aligned + (size_t)(1 + 2 * KV_STAGES) * TILE_BYTES + ((sizeof(Bars) + 15) & ~(size_t)15));
    volatile int* abort_flag = &bars->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rep = H / G;
    const int TQ = ROWS / rep;
    const int n_work = n_x * G;
    constexpr int NH = DH / 64;                                          // swizzled half tiles (64 dims) per operand tile

    // Rows beyond TQ * rep (heads per group that do not divide 128: 126 rows for 3, 125 for 5, ...) are never
    // written by the Q copy; they are zeroed once so that their scores are finite.  Nothing of them is stored.
    for (int i = threadIdx.x; i < (ROWS - TQ * rep) * 8 * NH; i += blockDim.x) {
        const int row = TQ * rep + i / (8 * NH), chunk = i % (8 * NH);  // NH halves x 8 chunks of 16 bytes per row
        *reinterpret_cast<uint4*>(aligned + (chunk >> 3) * HALF_BYTES + row * 128 + (chunk & 7) * 16) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bars->q_full), 1);
        mbar_init(smem_u32(&bars->q_empty), 1);
        mbar_init(smem_u32(&bars->o_free), 8);
        for (int s = 0; s < KV_STAGES; s++) {
            mbar_init(smem_u32(&bars->k_full[s]), 1);
            mbar_init(smem_u32(&bars->v_full[s]), 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&bars->s_full[s]), 1);
            mbar_init(smem_u32(&bars->s_empty[s]), 8);
            mbar_init(smem_u32(&bars->p_ready[s]), 8);
        }
        for (int s = 0; s < 4; s++) {
            mbar_init(smem_u32(&bars->xch[s]), 2);
            mbar_init(smem_u32(&bars->fin[s]), 2);
        }
        for (int s = 0; s < 2; s++) mbar_init(smem_u32(&bars->pv_done[s]), 1);
        mbar_init(smem_u32(&bars->o_full), 1);
        mbar_init(smem_u32(&bars->tbl_free), 8);
        mbar_init(smem_u32(&bars->tbl_full), 8);
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
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
            uint32_t jj = 0, it = 0;                                     // key blocks and items so far
            bool ok = true;
            for (int pass = 0, w; (w = snake_item(pass, (int)blockIdx.x, (int)gridDim.x)) < n_work && ok; pass++) {
                TileWork t;
                if (!tile_work(b, w, n_x, G, TQ, window, chunk, t)) continue;
                const int* pt = page_table + (size_t)t.slot * max_pages;
                if (it > 0) ok = mbar_wait(smem_u32(&bars->q_empty), (it - 1u) & 1u, abort_flag, status, 11);
                if (!ok) break;
                // Q: rows ordered (token, head of group); a 3-D box {64 dims, rep heads, TQ tokens} per half
                mbar_expect_tx(smem_u32(&bars->q_full), (uint32_t)(NH * 128 * rep * TQ));
                tma_load_3d(qs, &map_q, 0, t.g * rep, t.t_first + t.tq0, smem_u32(&bars->q_full));
                if (NH == 2) tma_load_3d(qs + HALF_BYTES, &map_q, 64, t.g * rep, t.t_first + t.tq0, smem_u32(&bars->q_full));
                it++;
                for (int j = 0; j < t.n_iter; j++, jj++) {
                    const int s = jj % KV_STAGES;
                    const uint32_t ph = (jj / KV_STAGES) & 1u;
                    int pg[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        int pi = (t.blk0 + j) * 2 + h;
                        if (pi > t.last_page) pi = t.last_page;         // no such page: any finite data, masked later
                        int page = pt[pi];
                        if (page < 0 || page >= n_pages_pool) { gfb_report(status, GFB_ERR_PAGE_TABLE, t.slot, pi); page = 0; }
                        pg[h] = page;
                    }
                    if (!mbar_wait(smem_u32(&bars->s_full[s]), ph ^ 1u, abort_flag, status, 1)) { ok = false; break; }   // the scores of block jj - 2 are done
                    mbar_expect_tx(smem_u32(&bars->k_full[s]), NH * HALF_BYTES);
#pragma unroll
                    for (int h = 0; h < 2; h++) {                       // page h -> rows 64h .. 64h+63 of both halves
                        const int row = (pg[h] * G + t.g) * PAGE;
                        tma_load_2d(ks + s * TILE_BYTES + h * (PAGE * 128), &map_k, 0, row, smem_u32(&bars->k_full[s]));
                        if (NH == 2) tma_load_2d(ks + s * TILE_BYTES + HALF_BYTES + h * (PAGE * 128), &map_k, 64, row, smem_u32(&bars->k_full[s]));
                    }
                    if (!mbar_wait(smem_u32(&bars->pv_done[s]), ph ^ 1u, abort_flag, status, 2)) { ok = false; break; }   // P V of block jj - 2 is done
                    mbar_expect_tx(smem_u32(&bars->v_full[s]), NH * HALF_BYTES);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int row = (pg[h] * G + t.g) * PAGE;
                        tma_load_2d(vs + s * TILE_BYTES + h * (PAGE * 128), &map_v, 0, row, smem_u32(&bars->v_full[s]));
                        if (NH == 2) tma_load_2d(vs + s * TILE_BYTES + HALF_BYTES + h * (PAGE * 128), &map_v, 64, row, smem_u32(&bars->v_full[s]));
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = idesc_bf16(ROWS, KEYS, 0);
            constexpr uint32_t idesc_o = idesc_bf16(ROWS, DH, 1);
            uint32_t jj = 0, it = 0;
            bool ok = true;
            auto issue_s = [&](uint32_t u, bool last_of_item) -> bool {   // S of key block number u (running count)
                const int s = u % KV_STAGES, sb = u & 1u;
                if (!mbar_wait(smem_u32(&bars->k_full[s]), (u / KV_STAGES) & 1u, abort_flag, status, 3)) return false;
                if (!mbar_wait(smem_u32(&bars->s_empty[sb]), ((u >> 1) & 1u) ^ 1u, abort_flag, status, 4)) return false;
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < DH / 16; k++) {
                    const uint32_t off = (k >> 2) * HALF_BYTES;
                    umma_ss(tmem + COL_S + sb * 128, desc_kmajor(qs + off) + 2 * (k & 3),
                            desc_kmajor(ks + s * TILE_BYTES + off) + 2 * (k & 3), idesc_s, k != 0);
                }
                umma_commit(smem_u32(&bars->s_full[sb]));
                if (last_of_item) umma_commit(smem_u32(&bars->q_empty));   // Q may be overwritten once these have run
                return true;
            };
            for (int pass = 0, w; (w = snake_item(pass, (int)blockIdx.x, (int)gridDim.x)) < n_work && ok; pass++) {
                TileWork t;
                if (!tile_work(b, w, n_x, G, TQ, window, chunk, t)) continue;
                ok = mbar_wait(smem_u32(&bars->q_full), it & 1u, abort_flag, status, 5);
                ok = ok && issue_s(jj, t.n_iter == 1);
                for (int j = 0; j < t.n_iter && ok; j++, jj++) {
                    if (j + 1 < t.n_iter) ok = issue_s(jj + 1, j + 2 == t.n_iter);
                    if (!ok) break;
                    const int s = jj % KV_STAGES;
                    ok = mbar_wait(smem_u32(&bars->v_full[s]), (jj / KV_STAGES) & 1u, abort_flag, status, 6);
                    ok = ok && mbar_wait(smem_u32(&bars->p_ready[jj & 1u]), (jj >> 1) & 1u, abort_flag, status, 7);
                    // the first P V of an item overwrites O: the previous item's output must have been read
                    if (ok && j == 0 && it > 0) ok = mbar_wait(smem_u32(&bars->o_free), (it - 1u) & 1u, abort_flag, status, 12);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)                       // 16 keys per MMA: 8 columns of P, 2 KB of V
                        umma_ts(tmem + COL_O, tmem + COL_P + (jj & 1u) * 64 + kk * 8,
                                desc_mnmajor(vs + s * TILE_BYTES + kk * 2048), idesc_o, (j | kk) != 0);
                    umma_commit(smem_u32(&bars->pv_done[s]));
                    if (j + 1 == t.n_iter) umma_commit(smem_u32(&bars->o_full));
                }
                it++;
            }
        }
    } else {
        // Eight softmax warps: warps 2..5 take the first 64 keys of every block, warps 6..9 the second 64.  Warp q of
        // either half holds rows 32 q .. 32 q + 31, one row per thread, so a row is shared by two warps on the same SM
        // sub-partition: while one waits for a result the other issues.  They agree on the row's maximum through
        // shared memory once per block and add their sums at the end of an item.
        const int half = warp >= 6 ? 1 : 0;
        const int q = warp & 3;
        const int r = q * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        const int tq = r / rep;
        uint32_t jj = 0, it = 0;                                       // key blocks and items so far
        bool ok = true;
        for (int pass = 0, w; (w = snake_item(pass, (int)blockIdx.x, (int)gridDim.x)) < n_work && ok; pass++) {
            TileWork t;
            if (!tile_work(b, w, n_x, G, TQ, window, chunk, t)) continue;
            const bool row_ok = tq < t.nq;
            const int row_pos = t.pos0 + tq;
            const int row_lo = first_key(row_pos, window, chunk);
            if (db.s_stride > 0) {
                // the table of this item's heads: wait until no warp reads the previous item's, write a share, wait for all shares
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->tbl_free));
                ok = mbar_wait_warp(smem_u32(&bars->tbl_free), it & 1u, abort_flag, status, 15);
                if (!ok) break;
                for (int k = (warp - 2) * 32 + lane; k < rep * db.s_len; k += 256) {
                    const int hl = k / db.s_len, kk = k - hl * db.s_len;
                    const int u = min(max(db.top - (kk - TABLE_AHEAD), 0), db.len - 1);
                    bias_s[hl * db.s_stride + kk] = __ldg(db.table + (size_t)(t.g * rep + hl) * db.len + u);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->tbl_full));
                ok = mbar_wait_warp(smem_u32(&bars->tbl_full), it & 1u, abort_flag, status, 16);
                if (!ok) break;
            }
            float m_run = -INFINITY, l_run = 0.f;                        // l_run: this warp's half of the row's sum
            for (int j = 0; j < t.n_iter && ok; j++, jj++) {
                const uint32_t sb = jj & 1u;
                const int key0 = (t.blk0 + j) * KEYS + half * 64;        // this warp's first key
                ok = mbar_wait_warp(smem_u32(&bars->s_full[sb]), (jj >> 1) & 1u, abort_flag, status, 8);
                if (!ok) break;
                tc_fence_after();
                // a block needs no mask when the tile's first row sees its last key and its last row (whose window or chunk
                // starts latest) sees its first key
                const bool need_mask = key0 + 63 > t.pos0 || key0 < t.last_lo || t.nq < TQ;
                // this warp's half of the row into registers
                uint32_t raw[2][32];
                tmem_ld32_issue(lane_base + COL_S + sb * 128 + half * 64, raw[0]);
                tmem_ld32_issue(lane_base + COL_S + sb * 128 + half * 64 + 32, raw[1]);
                tmem_ld_wait32(raw[0]);
                tmem_ld_wait32(raw[1]);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->s_empty[sb]));    // one arrival per warp
                float v[2][32];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int i = 0; i < 32; i++) v[c][i] = __uint_as_float(raw[c][i]);
                if (db.s_stride > 0) {
                    // ascending keys are descending distances; the strides keep the lanes of a warp on different banks
                    const float* e = bias_s + (r - tq * rep) * db.s_stride + TABLE_AHEAD + (row_pos - key0);
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int i = 0; i < 32; i++) v[c][i] += e[-(c * 32 + i)];
                    if (db.slopes != nullptr) {
                        DistanceBias only_slopes = db;
                        only_slopes.table = nullptr;
                        add_distance_bias<2>(v, only_slopes, H, t.g * rep + (r - tq * rep), row_pos, key0);
                    }
                } else if (db.table != nullptr || db.slopes != nullptr)
                    add_distance_bias<2>(v, db, H, t.g * rep + (r - tq * rep), row_pos, key0);
                if (cap_raw > 0.f) {
                    // a soft cap on the scaled score, in units of the raw score: cap tanh(s / cap), tanh(x) = 1 - 2 / (e^2x + 1)
                    const float two_over = 2.8853900817779268f / cap_raw;    // 2 log2(e) / cap
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int i = 0; i < 32; i++) {
                            const float e = fast_exp2(v[c][i] * two_over);
                            v[c][i] = cap_raw - __fdividef(2.f * cap_raw, e + 1.f);
                        }
                }
                if (need_mask) {                                             // only blocks on the diagonal or at the window's edge
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int i = 0; i < 32; i++) {
                            const int kj = key0 + c * 32 + i;
                            if (!(row_ok && kj <= row_pos && kj >= row_lo)) v[c][i] = -INFINITY;
                        }
                }
                float mx4[4];                                                // four chains
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float* x = &v[c >> 1][(c & 1) * 16];
                    mx4[c] = fmaxf(x[0], x[1]);
#pragma unroll
                    for (int i = 2; i < 16; i += 2) mx4[c] = max3(mx4[c], x[i], x[i + 1]);
                }
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // the other half's maximum (buffers by block parity: a warp cannot be two blocks ahead of its partner)
                bars->mx_half[sb][half][r] = mx;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->xch[q]));
                ok = mbar_wait_warp(smem_u32(&bars->xch[q]), jj & 1u, abort_flag, status, 13);
                if (!ok) break;
                mx = fmaxf(mx, bars->mx_half[sb][half ^ 1][r]);
                // The running maximum only has to keep the exponentials in range, so it follows the true maximum
                // lazily: it moves (and O is rescaled) only when the true maximum has grown by more than 2^8 in
                // the exponent; until then probabilities may reach 256, which bfloat16 and the 32-bit sums hold.
                // Sum and output use the same reference, so the quotient at the end is exact either way.
                float m_new = m_run;
                if (mx > m_run && (m_run == -INFINITY || (mx - m_run) * scale_log2e > 8.f)) m_new = mx;
                const float corr = (m_run == -INFINITY || m_new == m_run) ? 1.f : fast_exp2((m_run - m_new) * scale_log2e);   // a row without keys so far has O = 0, l = 0
                const float mneg = (m_new == -INFINITY) ? 0.f : -m_new * scale_log2e;
                // probabilities (2^-inf = 0 for masked scores), rounded to bfloat16 into tensor memory
                float rs2[2] = {0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t pk[16];
                    float rs_odd = 0.f;                                      // rs2[c] and rs_odd: one packed sum
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float t0, t1;
                        fma2(v[c][i], v[c][i + 1], scale_log2e, mneg, t0, t1);
                        const float p0 = fast_exp2(t0), p1 = fast_exp2(t1);
                        add2(rs2[c], rs_odd, p0, p1);
                        pk[i >> 1] = pack2(p0, p1);
                    }
                    rs2[c] += rs_odd;
                    tmem_st16(lane_base + COL_P + sb * 64 + half * 32 + c * 16, pk);
                }
                const float rs = rs2[0] + rs2[1];
                // O of the earlier blocks follows the new maximum, each warp its 64 columns, after the previous P V has
                // landed.  Rarely, so most phases of that barrier are never looked at; the parity wait is valid all the
                // same: the phase before the awaited one (P V of block jj - 3) is over, since the scores of this block
                // were issued behind the P V of block jj - 2, and the phase after it (block jj + 1) cannot have begun,
                // since that P V is issued behind this block's, which waits for this warp's arrival below.
                if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                    ok = mbar_wait_warp(smem_u32(&bars->pv_done[(jj - 1u) & 1u]), ((jj - 1u) >> 1) & 1u, abort_flag, status, 9);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < NH; c++) {
                        float o[32];
                        tmem_ld32(lane_base + COL_O + half * (DH / 2) + c * 32, o);
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] *= corr;
                        tmem_st32(lane_base + COL_O + half * (DH / 2) + c * 32, o);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->p_ready[sb]));
                l_run = l_run * corr + rs;
                m_run = m_new;
            }
            // All P V of the item have landed: a barrier of its own with one phase per item.  (A parity wait on pv_done
            // is only valid while that barrier can be neither a phase behind nor a phase ahead of the awaited one; at the
            // end of an item, with the waits of the earlier blocks left out, it could be either.)
            if (ok) ok = mbar_wait_warp(smem_u32(&bars->o_full), it & 1u, abort_flag, status, 10);
            if (!ok) break;
            tc_fence_after();
            // the row's sum: both halves are under the same reference
            bars->l_half[it & 1u][half][r] = l_run;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->fin[q]));
            ok = mbar_wait_warp(smem_u32(&bars->fin[q]), it & 1u, abort_flag, status, 14);
            if (!ok) break;
            l_run += bars->l_half[it & 1u][half ^ 1][r];
            it++;
            const int head = t.g * rep + (r - tq * rep);
            // a sink: one more term of the sum under the row's reference maximum, with no value behind it
            if (sink != nullptr && m_run != -INFINITY) l_run += fast_exp2(sink[head] * 1.4426950408889634f - m_run * scale_log2e);
            const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
            // the row's log-sum-exp in units of log2, for a caller that merges further keys into the row afterwards
            if (lse_out != nullptr && row_ok && half == 0)
                lse_out[(size_t)(t.t_first + t.tq0 + tq) * H + head] = l_run > 0.f ? fmaf(m_run, scale_log2e, log2f(l_run)) : -INFINITY;
            __nv_bfloat16* dst = out + ((size_t)(t.t_first + t.tq0 + tq) * H + head) * DH + half * (DH / 2);   // each warp stores its half of the columns
#pragma unroll 1
            for (int c = 0; c < NH; c++) {
                float v[32];
                tmem_ld32(lane_base + COL_O + half * (DH / 2) + c * 32, v);   // warp-collective: also for idle rows
                if (row_ok) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 pk;
                        pk.x = pack2(v[i] * inv, v[i + 1] * inv); pk.y = pack2(v[i + 2] * inv, v[i + 3] * inv);
                        pk.z = pack2(v[i + 4] * inv, v[i + 5] * inv); pk.w = pack2(v[i + 6] * inv, v[i + 7] * inv);
                        *reinterpret_cast<uint4*>(dst + c * 32 + i) = pk;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->o_free));         // O may be overwritten by the next item
        }
    }

    if (*abort_flag) {
        unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- two query tiles per block ------------------------------------------------------------------
// The same algorithm with TWO tiles of 128 rows (2 TQ consecutive tokens) in one block, each with its own
// four softmax warps, sharing every K/V page that is loaded.  The tensor pipe alternates between the
// tiles: while the warps of one tile work through their exponentials, it computes P V of the other tile
// and that tile's next scores.  Tensor memory: S of tile x in columns 128 x .. 128 x + 127, O of tile x in
// 256 + 128 x ...; P (bfloat16) overwrites the first 64 columns of its own S once the scores are in
// registers, and the next S of that tile is issued behind the P V that reads it (the pipe runs in order).
struct Bars2 {
    unsigned long long q_full;
    unsigned long long k_full[KV_STAGES], k_empty[KV_STAGES];
    unsigned long long v_full[KV_STAGES], v_empty[KV_STAGES];
    unsigned long long s_full[2];
    unsigned long long p_ready[2];
    unsigned long long pv_done[2];
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(320, 1)
attn_prefill_tc2_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                        const int* __restrict__ page_table, int max_pages, int n_pages_pool,
                        GfbBatch b, int H, int G, float scale_log2e, int window, int chunk, const float* __restrict__ sink,
                        DistanceBias db, int* status) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_q); prefetch_map(&map_k); prefetch_map(&map_v); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t qs = base;                                            // 2 tiles x [2 halves][128 rows][128 B]
    const uint32_t ks = base + 2 * TILE_BYTES;
    const uint32_t vs = ks + KV_STAGES * TILE_BYTES;
    Bars2* bars = reinterpret_cast<Bars2*>(aligned + (size_t)(2 + 2 * KV_STAGES) * TILE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rep = H / G;
    const int TQ = ROWS / rep;
    for (int i = threadIdx.x; i < 2 * (ROWS - TQ * rep) * 16; i += blockDim.x) {      // both tiles' idle rows, as in the one-tile kernel
        const int x = i / ((ROWS - TQ * rep) * 16), k = i - x * (ROWS - TQ * rep) * 16;
        const int row = TQ * rep + (k >> 4), chunk = k & 15;
        *reinterpret_cast<uint4*>(aligned + x * TILE_BYTES + (chunk >> 3) * HALF_BYTES + row * 128 + (chunk & 7) * 16) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    int seq = -1, tq0 = 0;
    {
        int left = (int)gridDim.x - 1 - (int)blockIdx.x;                 // long tiles first
        for (int i = 0; i < b.n_seqs; i++) {
            int qlen = b.cu_seqlens[i + 1] - b.cu_seqlens[i];
            int nt = (qlen + 2 * TQ - 1) / (2 * TQ);
            if (left < nt) { seq = i; tq0 = left * 2 * TQ; break; }
            left -= nt;
        }
    }
    if (seq < 0) return;
    const int g = blockIdx.y;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bars->q_full), 1);
        for (int s = 0; s < KV_STAGES; s++) {
            mbar_init(smem_u32(&bars->k_full[s]), 1);
            mbar_init(smem_u32(&bars->k_empty[s]), 1);
            mbar_init(smem_u32(&bars->v_full[s]), 1);
            mbar_init(smem_u32(&bars->v_empty[s]), 1);
        }
        for (int x = 0; x < 2; x++) {
            mbar_init(smem_u32(&bars->s_full[x]), 1);
            mbar_init(smem_u32(&bars->p_ready[x]), 4);
            mbar_init(smem_u32(&bars->pv_done[x]), 1);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    gfb_pdl_launch();
    gfb_pdl_wait();

    const int t_first = b.cu_seqlens[seq];
    const int qlen = b.cu_seqlens[seq + 1] - t_first;
    const int slot = b.slots[seq];
    const int len0 = b.lengths[slot];
    // per tile: tokens [tq0 + x TQ, +nq), positions from pos0, key blocks [lo_blk, hi_blk)
    int nq[2], pos0[2], lo_blk[2], hi_blk[2];
#pragma unroll
    for (int x = 0; x < 2; x++) {
        nq[x] = min(TQ, qlen - (tq0 + x * TQ));
        pos0[x] = len0 + tq0 + x * TQ;
        if (nq[x] > 0) {
            const int first_lo = first_key(pos0[x], window, chunk);
            lo_blk[x] = first_lo / KEYS;
            hi_blk[x] = (pos0[x] + nq[x] - 1) / KEYS + 1;
        } else {
            lo_blk[x] = 0;
            hi_blk[x] = 0;
        }
    }
    const int blk0 = nq[1] > 0 ? min(lo_blk[0], lo_blk[1]) : lo_blk[0];
    const int blk1 = max(hi_blk[0], hi_blk[1]);
    const int n_iter = blk1 - blk0;
    const int last_page = (len0 + min(qlen, tq0 + 2 * TQ) - 1) / PAGE;
    const int* pt = page_table + (size_t)slot * max_pages;
    auto active = [&](int x, int j) { return blk0 + j >= lo_blk[x] && blk0 + j < hi_blk[x]; };

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(smem_u32(&bars->q_full), (uint32_t)(2 * 2 * 128 * rep * TQ));
#pragma unroll
            for (int x = 0; x < 2; x++) {                                // rows beyond the batch are filled with zeros
                tma_load_3d(qs + x * TILE_BYTES, &map_q, 0, g * rep, t_first + tq0 + x * TQ, smem_u32(&bars->q_full));
                tma_load_3d(qs + x * TILE_BYTES + HALF_BYTES, &map_q, 64, g * rep, t_first + tq0 + x * TQ, smem_u32(&bars->q_full));
            }
            for (int j = 0; j < n_iter; j++) {
                const int s = j % KV_STAGES;
                const uint32_t ph = (uint32_t)(j / KV_STAGES) & 1u;
                int pg[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    int pi = (blk0 + j) * 2 + h;
                    if (pi > last_page) pi = last_page;
                    int page = pt[pi];
                    if (page < 0 || page >= n_pages_pool) { gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi); page = 0; }
                    pg[h] = page;
                }
                if (!mbar_wait(smem_u32(&bars->k_empty[s]), ph ^ 1u, abort_flag, status, 1)) break;
                mbar_expect_tx(smem_u32(&bars->k_full[s]), TILE_BYTES);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = (pg[h] * G + g) * PAGE;
                    tma_load_2d(ks + s * TILE_BYTES + h * (PAGE * 128), &map_k, 0, row, smem_u32(&bars->k_full[s]));
                    tma_load_2d(ks + s * TILE_BYTES + HALF_BYTES + h * (PAGE * 128), &map_k, 64, row, smem_u32(&bars->k_full[s]));
                }
                if (!mbar_wait(smem_u32(&bars->v_empty[s]), ph ^ 1u, abort_flag, status, 2)) break;
                mbar_expect_tx(smem_u32(&bars->v_full[s]), TILE_BYTES);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = (pg[h] * G + g) * PAGE;
                    tma_load_2d(vs + s * TILE_BYTES + h * (PAGE * 128), &map_v, 0, row, smem_u32(&bars->v_full[s]));
                    tma_load_2d(vs + s * TILE_BYTES + HALF_BYTES + h * (PAGE * 128), &map_v, 64, row, smem_u32(&bars->v_full[s]));
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = idesc_bf16(ROWS, KEYS, 0);
            constexpr uint32_t idesc_o = idesc_bf16(ROWS, D, 1);
            uint32_t n_pv[2] = {0, 0};                                   // P V products issued per tile
            bool ok = mbar_wait(smem_u32(&bars->q_full), 0, abort_flag, status, 5);
            auto issue_s = [&](int x, int j) {                           // K stage of block j is known to be loaded
                const int s = j % KV_STAGES;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t off = (k >> 2) * HALF_BYTES;
                    umma_ss(tmem + 128 * x, desc_kmajor(qs + x * TILE_BYTES + off) + 2 * (k & 3),
                            desc_kmajor(ks + s * TILE_BYTES + off) + 2 * (k & 3), idesc_s, k != 0);
                }
                umma_commit(smem_u32(&bars->s_full[x]));
            };
            auto k_ready = [&](int j) {
                return mbar_wait(smem_u32(&bars->k_full[j % KV_STAGES]), (uint32_t)(j / KV_STAGES) & 1u, abort_flag, status, 3);
            };
            if (ok && n_iter > 0) {
                ok = k_ready(0);
                if (ok) {
                    tc_fence_after();
                    if (active(0, 0)) issue_s(0, 0);
                    if (active(1, 0)) issue_s(1, 0);
                    umma_commit(smem_u32(&bars->k_empty[0]));
                }
            }
            for (int j = 0; j < n_iter && ok; j++) {
                const int s = j % KV_STAGES;
                bool k_next = false;                                     // whether K of block j + 1 has been waited for
                ok = mbar_wait(smem_u32(&bars->v_full[s]), (uint32_t)(j / KV_STAGES) & 1u, abort_flag, status, 6);
#pragma unroll
                for (int x = 0; x < 2 && ok; x++) {
                    if (active(x, j)) {
                        ok = mbar_wait(smem_u32(&bars->p_ready[x]), n_pv[x] & 1u, abort_flag, status, 7);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)                   // 16 keys per MMA: 8 columns of P, 2 KB of V
                            umma_ts(tmem + 256 + 128 * x, tmem + 128 * x + kk * 8,
                                    desc_mnmajor(vs + s * TILE_BYTES + kk * 2048), idesc_o, (n_pv[x] | (uint32_t)kk) != 0);
                        umma_commit(smem_u32(&bars->pv_done[x]));
                        n_pv[x]++;
                    }
                    if (j + 1 < n_iter && active(x, j + 1)) {            // the tile's next scores, behind its P V
                        if (!k_next) { ok = k_ready(j + 1); k_next = true; if (!ok) break; tc_fence_after(); }
                        issue_s(x, j + 1);
                    }
                }
                if (!ok) break;
                umma_commit(smem_u32(&bars->v_empty[s]));
                if (j + 1 < n_iter) {
                    if (!k_next) { ok = k_ready(j + 1); if (!ok) break; }
                    umma_commit(smem_u32(&bars->k_empty[(j + 1) % KV_STAGES]));
                }
            }
        }
    } else {
        const int x = (warp - 2) >> 2;                                   // warps 2..5: tile 0, warps 6..9: tile 1
        const int q = warp & 3;
        const int r = q * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t col_s = 128 * x, col_o = 256 + 128 * x;
        const int tq = r / rep;
        const bool row_ok = tq < nq[x];
        const int row_pos = pos0[x] + tq;
        const int row_lo = first_key(row_pos, window, chunk);
        const int last_lo = first_key(pos0[x] + max(nq[x], 1) - 1, window, chunk);
        float m_run = -INFINITY, l_run = 0.f;
        uint32_t n_done = 0;                                             // blocks of this tile finished
        bool ok = true;
        for (int j = 0; j < n_iter && ok; j++) {
            if (!active(x, j)) continue;
            const int key0 = (blk0 + j) * KEYS;
            ok = mbar_wait_warp(smem_u32(&bars->s_full[x]), n_done & 1u, abort_flag, status, 8);
            if (!ok) break;
            tc_fence_after();
            const bool need_mask = key0 + KEYS - 1 > pos0[x] || key0 < last_lo || nq[x] < TQ;
            float v[4][32];
            tmem_ld_row128(lane_base + col_s, v);
            if (db.table != nullptr || db.slopes != nullptr)
                add_distance_bias<4>(v, db, H, g * rep + (r - tq * rep), row_pos, key0);
            if (need_mask) {
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const int kj = key0 + c * 32 + i;
                        if (!(row_ok && kj <= row_pos && kj >= row_lo)) v[c][i] = -INFINITY;
                    }
            }
            float mx4[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                mx4[c] = fmaxf(v[c][0], v[c][1]);
#pragma unroll
                for (int i = 2; i < 32; i += 2) mx4[c] = max3(mx4[c], v[c][i], v[c][i + 1]);
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            float m_new = m_run;                                         // lazy reference maximum, as in the one-tile kernel
            if (mx > m_run && (m_run == -INFINITY || (mx - m_run) * scale_log2e > 8.f)) m_new = mx;
            const float corr = (m_run == -INFINITY || m_new == m_run) ? 1.f : fast_exp2((m_run - m_new) * scale_log2e);   // a row without keys so far has O = 0, l = 0
            const float mneg = (m_new == -INFINITY) ? 0.f : -m_new * scale_log2e;
            // P over the first half of this tile's own scores: all of this row's scores are in registers by now,
            // and a thread only ever touches its own row (lane) of tensor memory
            float rs4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t pk[16];
                float rs_odd = 0.f;                                      // rs4[c] and rs_odd: one packed sum
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float t0, t1;
                    fma2(v[c][i], v[c][i + 1], scale_log2e, mneg, t0, t1);
                    const float p0 = fast_exp2(t0), p1 = fast_exp2(t1);
                    add2(rs4[c], rs_odd, p0, p1);
                    pk[i >> 1] = pack2(p0, p1);
                }
                rs4[c] += rs_odd;
                tmem_st16(lane_base + col_s + c * 16, pk);
            }
            // O follows the reference maximum, rarely (S of this block was issued behind the tile's previous P V, so
            // that phase is over and the wait only orders the accesses)
            if (n_done > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                ok = mbar_wait_warp(smem_u32(&bars->pv_done[x]), (n_done - 1u) & 1u, abort_flag, status, 9);
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < 4; c++) {
                    float o[32];
                    tmem_ld32(lane_base + col_o + c * 32, o);
#pragma unroll
                    for (int i = 0; i < 32; i++) o[i] *= corr;
                    tmem_st32(lane_base + col_o + c * 32, o);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->p_ready[x]));
            l_run = l_run * corr + (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
            m_run = m_new;
            n_done++;
        }
        if (ok && n_done > 0) ok = mbar_wait_warp(smem_u32(&bars->pv_done[x]), (n_done - 1u) & 1u, abort_flag, status, 10);
        if (ok && n_done > 0) {
            tc_fence_after();
            const int head = g * rep + (r - tq * rep);
            if (sink != nullptr && m_run != -INFINITY) l_run += fast_exp2(sink[head] * 1.4426950408889634f - m_run * scale_log2e);
            const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
            __nv_bfloat16* dst = out + ((size_t)(t_first + tq0 + x * TQ + tq) * H + head) * D;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                float v[32];
                tmem_ld32(lane_base + col_o + c * 32, v);
                if (row_ok) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 pk;
                        pk.x = pack2(v[i] * inv, v[i + 1] * inv); pk.y = pack2(v[i + 2] * inv, v[i + 3] * inv);
                        pk.z = pack2(v[i + 4] * inv, v[i + 5] * inv); pk.w = pack2(v[i + 6] * inv, v[i + 7] * inv);
                        *reinterpret_cast<uint4*>(dst + c * 32 + i) = pk;
                    }
                }
            }
        }
    }

    if (*abort_flag) {
        unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- prompts against a shared latent ---------------------------------------------------------------
// All heads read the same cached rows (gfb_latent_attention states the arithmetic): keys are whole rows of R + 64 numbers (R = 128, 256,
// 384 or 512), values their first R.  A tile is 128 (token, head) pairs of one sequence.  A 32-bit accumulator of 128 x 512 would take
// all of an SM's tensor memory, so an item is a tile AND one half of the value columns: two blocks score the same keys, each
// adds its own half of P V.  That is 1.5 times the products of one pass, on a pipe that the scores alone (36 MMAs of 128 x 64 per page) keep
// busy while four softmax warps, a row per thread, work on the page before.
//
// A page's rows lie in shared memory as swizzled pieces of [64 keys][64 dims]: the block's own value half (also the B operand of P V,
// MN-major) and the rest (the other half and the rotated part), each with two stages of its own, so that a page's rest is free again when
// its scores are done and its own half when its P V is.  What makes room for both (144 KB) is Q: the 256 numbers of the own half stand in
// tensor memory as the A operand (128 columns), only the rest (80 KB) in shared memory.
//   tensor memory: O 0..255, two score buffers of 64 columns (P overwrites the first 32 of its own) 256..383, Q's half 384..511
//
// Measured (16 heads, R = 512, one prompt): 4,096 tokens 492 us, 590 TFLOP/s of scores and weighted sums, where the
// mma.sync kernel (gfb_latent_attention, which decode steps and other sizes keep) took 1,723 us, 169 TFLOP/s.
constexpr int LK = 64;                          // keys per iteration: one page
constexpr int PIECE_BYTES = LK * 128;           // [64 keys][64 dims]
constexpr int QPIECE_BYTES = ROWS * 128;        // [128 rows][64 dims]
constexpr uint32_t LCOL_S = 256, LCOL_Q = 384;
constexpr int LAT_THREADS = 192;

struct LatBars {
    unsigned long long q_full, qt_full;           // Q's rest in shared memory (TMA), Q's own half in tensor memory (four softmax warps)
    unsigned long long rest_full[2], own_full[2];
    unsigned long long rest_done[2];              // the scores' first part has read the rest of page j (a commit)
    unsigned long long s_full[2], pv_done[2];     // scores of page j are there; P V of page j is done (which also frees the own half's stage)
    // all four warps' P of page j, a barrier per score buffer: the scores of page j + 1 are issued ahead of the wait for P of page j, so a
    // warp may arrive for page j + 1 while another has not arrived for page j, and one barrier would count the two together.  An arrival for
    // page j + 2 needs that page's scores, which are issued behind the wait for page j.
    unsigned long long p_ready[2], o_full;
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(LAT_THREADS, 1)
latent_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __nv_bfloat16* __restrict__ q,
                         __nv_bfloat16* __restrict__ out, const int* __restrict__ page_table, int max_pages, int n_pages_pool, GfbBatch b, int H,
                         int R, float scale_log2e, int window, const float* __restrict__ sink, int n_x, int* status) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_q); prefetch_map(&map_k); }
    const int hc = R / 128, rc = hc + 1;          // pieces of the own half and of the rest
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t qs = base, rs = qs + rc * QPIECE_BYTES, os = rs + 2 * rc * PIECE_BYTES;
    LatBars* bars = reinterpret_cast<LatBars*>(aligned + rc * QPIECE_BYTES + 2 * (rc + hc) * PIECE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int Dk = R + 64;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bars->q_full), 1);
        mbar_init(smem_u32(&bars->qt_full), 4);
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&bars->rest_full[s]), 1);
            mbar_init(smem_u32(&bars->own_full[s]), 1);
            mbar_init(smem_u32(&bars->rest_done[s]), 1);
            mbar_init(smem_u32(&bars->s_full[s]), 1);
            mbar_init(smem_u32(&bars->pv_done[s]), 1);
            mbar_init(smem_u32(&bars->p_ready[s]), 4);
        }
        mbar_init(smem_u32(&bars->o_full), 1);
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    gfb_pdl_launch();
    gfb_pdl_wait();

    // the item: a tile of rows (the latest rows of the last sequence first: they see the most keys) and a half of the value columns
    const int half = blockIdx.x & 1;
    int seq = -1, m0 = 0;
    {
        int left = n_x - 1 - (int)(blockIdx.x >> 1);
        for (int i = 0; i < b.n_seqs; i++) {
            const int nt = ((b.cu_seqlens[i + 1] - b.cu_seqlens[i]) * H + ROWS - 1) / ROWS;
            if (left < nt) { seq = i; m0 = left * ROWS; break; }
            left -= nt;
        }
    }
    if (seq >= 0) {
        const int t0 = b.cu_seqlens[seq], rows_here = min(ROWS, (b.cu_seqlens[seq + 1] - t0) * H - m0);
        const int slot = b.slots[seq], start = b.lengths[slot];
        const int first_pos = start + m0 / H, last_pos = start + (m0 + rows_here - 1) / H;
        const int blk0 = window > 0 ? max(0, first_pos - window + 1) / LK : 0, n_iter = last_pos / LK + 1 - blk0;
        const int own0 = half * hc * 64;              // the own half's first number in a row
        const size_t row0 = (size_t)t0 * H + m0;      // the tile's first row of q and out

        if (warp == 0) {
            if (lane == 0) {
                // the rest of a row: the other half's pieces, then the rotated part
                mbar_expect_tx(smem_u32(&bars->q_full), (uint32_t)rc * QPIECE_BYTES);
                for (int c = 0; c < rc; c++)
                    tma_load_2d(qs + c * QPIECE_BYTES, &map_q, c < hc ? (1 - half) * hc * 64 + c * 64 : R, (int)row0, smem_u32(&bars->q_full));
                const int* pt = page_table + (size_t)slot * max_pages;
                for (int j = 0; j < n_iter; j++) {
                    const int s = j & 1;
                    const uint32_t ph = (uint32_t)(j >> 1) & 1u;
                    const int pi = blk0 + j;
                    int page = pi < max_pages ? pt[pi] : -1;
                    if (page < 0 || page >= n_pages_pool) { gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi); page = 0; }
                    if (!mbar_wait(smem_u32(&bars->rest_done[s]), ph ^ 1u, abort_flag, status, 21)) break;
                    mbar_expect_tx(smem_u32(&bars->rest_full[s]), (uint32_t)rc * PIECE_BYTES);
                    for (int c = 0; c < rc; c++)
                        tma_load_2d(rs + (s * rc + c) * PIECE_BYTES, &map_k, c < hc ? (1 - half) * hc * 64 + c * 64 : R, page * LK, smem_u32(&bars->rest_full[s]));
                    if (!mbar_wait(smem_u32(&bars->pv_done[s]), ph ^ 1u, abort_flag, status, 22)) break;
                    mbar_expect_tx(smem_u32(&bars->own_full[s]), (uint32_t)hc * PIECE_BYTES);
                    for (int c = 0; c < hc; c++)
                        tma_load_2d(os + (s * hc + c) * PIECE_BYTES, &map_k, own0 + c * 64, page * LK, smem_u32(&bars->own_full[s]));
                }
            }
        } else if (warp == 1) {
            if (lane == 0) {
                const uint32_t idesc_s = idesc_bf16(ROWS, LK, 0), idesc_o = idesc_bf16(ROWS, hc * 64, 1);
                auto issue_s = [&](int j) -> bool {
                    const int s = j & 1;
                    const uint32_t ph = (uint32_t)(j >> 1) & 1u, d = tmem + LCOL_S + s * LK;
                    if (!mbar_wait(smem_u32(&bars->rest_full[s]), ph, abort_flag, status, 23)) return false;
                    tc_fence_after();
                    for (int c = 0; c < rc; c++) {
                        const uint64_t da = desc_kmajor(qs + c * QPIECE_BYTES), db = desc_kmajor(rs + (s * rc + c) * PIECE_BYTES);
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ss(d, da + 2 * k, db + 2 * k, idesc_s, (c | k) != 0);
                    }
                    umma_commit(smem_u32(&bars->rest_done[s]));
                    if (!mbar_wait(smem_u32(&bars->own_full[s]), ph, abort_flag, status, 24)) return false;
                    tc_fence_after();
                    for (int c = 0; c < hc; c++) {
                        const uint64_t db = desc_kmajor(os + (s * hc + c) * PIECE_BYTES);
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ts(d, tmem + LCOL_Q + c * 32 + k * 8, db + 2 * k, idesc_s, 1);
                    }
                    umma_commit(smem_u32(&bars->s_full[s]));
                    return true;
                };
                bool ok = mbar_wait(smem_u32(&bars->q_full), 0, abort_flag, status, 25);
                ok = ok && mbar_wait(smem_u32(&bars->qt_full), 0, abort_flag, status, 26);
                tc_fence_after();
                ok = ok && issue_s(0);
                for (int j = 0; j < n_iter && ok; j++) {
                    // the next page's scores go ahead of this page's P V (their buffer's last P was read by the P V before, in order)
                    if (j + 1 < n_iter) ok = issue_s(j + 1);
                    const int s = j & 1;
                    ok = ok && mbar_wait(smem_u32(&bars->p_ready[s]), (uint32_t)(j >> 1) & 1u, abort_flag, status, 27);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)                       // 16 keys per MMA: 8 columns of P, 2 KB of every piece
                        umma_ts(tmem, tmem + LCOL_S + s * LK + kk * 8, desc_mnmajor(os + s * hc * PIECE_BYTES + kk * 2048, PIECE_BYTES), idesc_o, (j | kk) != 0);
                    umma_commit(smem_u32(&bars->pv_done[s]));
                    if (j + 1 == n_iter) umma_commit(smem_u32(&bars->o_full));
                }
            }
        } else {
            const int quarter = warp & 3;
            const int r = quarter * 32 + lane;
            const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
            const bool row_ok = r < rows_here;
            const int row_pos = start + (m0 + r) / H;
            const int row_lo = window > 0 ? max(0, row_pos - window + 1) : 0;
            const int last_lo = window > 0 ? max(0, last_pos - window + 1) : 0;
            // Q's own half into tensor memory: a row per thread, two numbers per column (rows beyond the tile: zeros)
            {
                const uint4* src = reinterpret_cast<const uint4*>(q + (row0 + (row_ok ? r : 0)) * Dk + own0);
                for (int c = 0; c < 2 * hc; c++) {
                    uint32_t v[16];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint4 x = row_ok ? src[c * 4 + i] : make_uint4(0u, 0u, 0u, 0u);
                        v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
                    }
                    tmem_st16(lane_base + LCOL_Q + c * 16, v);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->qt_full));
            }
            float m_run = -INFINITY, l_run = 0.f;
            bool ok = true;
            for (int j = 0; j < n_iter; j++) {
                const int s = j & 1, key0 = (blk0 + j) * LK;
                ok = mbar_wait_warp(smem_u32(&bars->s_full[s]), (uint32_t)(j >> 1) & 1u, abort_flag, status, 28);
                if (!ok) break;
                tc_fence_after();
                uint32_t raw[2][32];
                tmem_ld32_issue(lane_base + LCOL_S + s * LK, raw[0]);
                tmem_ld32_issue(lane_base + LCOL_S + s * LK + 32, raw[1]);
                tmem_ld_wait32(raw[0]);
                tmem_ld_wait32(raw[1]);
                float v[2][32];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int i = 0; i < 32; i++) v[c][i] = __uint_as_float(raw[c][i]);
                // only pages on the diagonal, at the window's edge or of a tile with empty rows
                if (key0 + LK - 1 > first_pos || key0 < last_lo || rows_here < ROWS) {
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int i = 0; i < 32; i++) {
                            const int kj = key0 + c * 32 + i;
                            if (!(row_ok && kj <= row_pos && kj >= row_lo)) v[c][i] = -INFINITY;
                        }
                }
                float mx4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float* x = &v[c >> 1][(c & 1) * 16];
                    mx4[c] = fmaxf(x[0], x[1]);
#pragma unroll
                    for (int i = 2; i < 16; i += 2) mx4[c] = max3(mx4[c], x[i], x[i + 1]);
                }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // The reference is the true maximum, so that a row's largest weight is one, and the sum is that of the rounded weights.  With a
                // reference that lags by up to 2^8, as in the kernels above, rows with few large weights were up to 20 % further from 64 bits than
                // the mma.sync kernel's (1,024 tokens, queries of twice unit size: 0.00209 for 0.00174; so 0.00173).  It costs a tenth of the time.
                const float m_new = fmaxf(m_run, mx);
                const float corr = (m_run == -INFINITY || m_new == m_run) ? 1.f : fast_exp2((m_run - m_new) * scale_log2e);
                const float mneg = (m_new == -INFINITY) ? 0.f : -m_new * scale_log2e;
                float rsum[2] = {0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t pk[16];
                    float odd = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float a0, a1;
                        fma2(v[c][i], v[c][i + 1], scale_log2e, mneg, a0, a1);
                        const float p0 = fast_exp2(a0), p1 = fast_exp2(a1);
                        const uint32_t both = pack2(p0, p1);
                        add2(rsum[c], odd, __uint_as_float(both << 16), __uint_as_float(both & 0xffff0000u));
                        pk[i >> 1] = both;
                    }
                    rsum[c] += odd;
                    tmem_st16(lane_base + LCOL_S + s * LK + c * 16, pk);
                }
                // O follows a new reference, behind the previous P V: the scores of this page were issued behind the P V of page j - 2,
                // and that of page j + 1 waits for this warp, so the barrier's phase is the awaited one or the one before it
                if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                    ok = mbar_wait_warp(smem_u32(&bars->pv_done[(j - 1) & 1]), (uint32_t)((j - 1) >> 1) & 1u, abort_flag, status, 29);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 2 * hc; c++) {
                        float o[32];
                        tmem_ld32(lane_base + c * 32, o);
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] *= corr;
                        tmem_st32(lane_base + c * 32, o);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->p_ready[s]));
                l_run = l_run * corr + (rsum[0] + rsum[1]);
                m_run = m_new;
            }
            if (ok) ok = mbar_wait_warp(smem_u32(&bars->o_full), 0, abort_flag, status, 30);
            if (ok) {
                tc_fence_after();
                if (sink != nullptr && m_run != -INFINITY) l_run += fast_exp2(sink[(m0 + r) % H] * 1.4426950408889634f - m_run * scale_log2e);
                const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
                __nv_bfloat16* dst = out + (row0 + r) * R + own0;
#pragma unroll 1
                for (int c = 0; c < 2 * hc; c++) {
                    float o[32];
                    tmem_ld32(lane_base + c * 32, o);                      // warp-collective: also for idle rows
                    if (row_ok) {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            uint4 pk;
                            pk.x = pack2(o[i] * inv, o[i + 1] * inv); pk.y = pack2(o[i + 2] * inv, o[i + 3] * inv);
                            pk.z = pack2(o[i + 4] * inv, o[i + 5] * inv); pk.w = pack2(o[i + 6] * inv, o[i + 7] * inv);
                            *reinterpret_cast<uint4*>(dst + c * 32 + i) = pk;
                        }
                    }
                }
            }
        }
    }
    if (*abort_flag) {
        unsigned long long w0 = global_ns();
        while (global_ns() - w0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- a product with a weight per head -----------------------------------------------------------------
// out[t, h, n] = sum_k in[t, h, k] W_h[k, n], optionally times a sigmoid gate (gfb_headwise_linear states the arguments): latent attention's
// move of the queries into the latent space and of the attended latent out of it.  A block takes 128 tokens of one head and 128 columns:
// A is the tokens' rows through a map over the whole input (the head is a column offset), B the weight as it lies, [k][n], an MN-major operand
// in two pieces of 64 columns.  Three stages of 64 k (32 KB each), so that two blocks share an SM and one's epilogue runs under the other's
// loads.  The epilogue passes 32-bit rows through shared memory, so that gates and results move as whole lines.
//
// What bounds it is memory (K = 128 or 512: 4,096 tokens of 16 heads read and write 90 MB).  The mma.sync form (64 x 64 tiles without a
// pipeline), us for 4,096 tokens, 16 heads, 128 -> 512 and back: 234 -> 105 (34 us alone for
// 128 -> 512, without the events' cost).
constexpr int HW_STAGES = 3, HW_STAGE_BYTES = 2 * HALF_BYTES, HW_PITCH = 132;
constexpr uint32_t HW_SMEM = 1024 + HW_STAGES * HW_STAGE_BYTES + 128;
static_assert(4 * 32 * HW_PITCH * 4 <= HW_STAGES * HW_STAGE_BYTES, "the epilogue's rows take the ring's place");

struct HwBars {
    unsigned long long full[HW_STAGES], empty[HW_STAGES], done;
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(192)
headwise_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, int in_off, int in_stride,
                   __nv_bfloat16* __restrict__ out, int ld_out, int out_off, int out_stride, const __nv_bfloat16* __restrict__ gate, int ld_gate,
                   int gate_off, int gate_cols, int n_tokens, int K, int N, int* status) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_a); prefetch_map(&map_w); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    HwBars* bars = reinterpret_cast<HwBars*>(aligned + HW_STAGES * HW_STAGE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * ROWS, h = blockIdx.y, n0 = blockIdx.z * 128, nkb = K / 64;
    if (threadIdx.x == 0) {
        for (int s = 0; s < HW_STAGES; s++) { mbar_init(smem_u32(&bars->full[s]), 1); mbar_init(smem_u32(&bars->empty[s]), 1); }
        mbar_init(smem_u32(&bars->done), 1);
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(128u) : "memory");
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
            for (int kb = 0; kb < nkb; kb++) {
                const int s = kb % HW_STAGES;
                if (!mbar_wait(smem_u32(&bars->empty[s]), ((uint32_t)(kb / HW_STAGES) & 1u) ^ 1u, abort_flag, status, 31)) break;
                const uint32_t full = smem_u32(&bars->full[s]), at = base + s * HW_STAGE_BYTES;
                mbar_expect_tx(full, HW_STAGE_BYTES);
                tma_load_2d(at, &map_a, in_off + h * in_stride + kb * 64, t0, full);
                tma_load_2d(at + HALF_BYTES, &map_w, n0, h * K + kb * 64, full);
                tma_load_2d(at + HALF_BYTES + PIECE_BYTES, &map_w, n0 + 64, h * K + kb * 64, full);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_bf16(ROWS, 128, 1);
            bool ok = true;
            for (int kb = 0; kb < nkb && ok; kb++) {
                const int s = kb % HW_STAGES;
                ok = mbar_wait(smem_u32(&bars->full[s]), (uint32_t)(kb / HW_STAGES) & 1u, abort_flag, status, 32);
                if (!ok) break;
                tc_fence_after();
                const uint32_t at = base + s * HW_STAGE_BYTES;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    umma_ss(tmem, desc_kmajor(at) + 2 * k, desc_mnmajor(at + HALF_BYTES + k * 2048, PIECE_BYTES), idesc, (kb | k) != 0);
                umma_commit(smem_u32(&bars->empty[s]));
            }
            if (ok) umma_commit(smem_u32(&bars->done));
        }
    } else {
        const int q = warp & 3;
        float* mine = reinterpret_cast<float*>(aligned) + q * 32 * HW_PITCH;
        if (mbar_wait_warp(smem_u32(&bars->done), 0, abort_flag, status, 33)) {      // every copy has landed and been read
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 128; c += 32) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c, v);
#pragma unroll
                for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(mine + lane * HW_PITCH + c + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
            __syncwarp();
            const int rows = min(32, n_tokens - (t0 + q * 32));
#pragma unroll 4
            for (int r = 0; r < rows; r++) {
                const size_t t = (size_t)(t0 + q * 32 + r);
                float4 v = *reinterpret_cast<const float4*>(mine + r * HW_PITCH + lane * 4);
                if (gate != nullptr) {
                    const __nv_bfloat16* g = gate + t * ld_gate + gate_off + (gate_cols == 1 ? h : h * N + n0 + lane * 4);
                    float z[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) z[i] = 1.0f / (1.0f + expf(-__bfloat162float(g[gate_cols == 1 ? 0 : i])));
                    v.x *= z[0]; v.y *= z[1]; v.z *= z[2]; v.w *= z[3];
                }
                *reinterpret_cast<uint2*>(out + t * ld_out + out_off + (size_t)h * out_stride + n0 + lane * 4) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
            }
        }
    }
    if (*abort_flag) {
        unsigned long long w0 = global_ns();
        while (global_ns() - w0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128u) : "memory");
    }
}

// ---- prompts with their keys and values expanded -------------------------------------------------------
// A prompt whose keys are mostly its own new tokens is better off with every head's keys and values written out once: a (query, key, head)
// then takes 2 (192 + 128) operations where attention on the latent takes 2 (576 + 512), and the expansion, 2 * 512 * 256 per key and head,
// is what the queries' way into the latent space and the outputs' way back cost per token.  latent_expand_kernel makes them,
// latent_heads_kernel attends.
//
// Keys are rounded to bfloat16, as queries are on the other way.  A rounded value where that way rounds the sum of values would cost precision in rows
// that see few keys (1,200 tokens: 0.00274 from 64 bits for 0.00265), so values and weights are float16, each column of values times the power of two
// that takes its largest possible number (v_scale, from the weights; a normed latent is bounded) to 2^14 .. 2^15: a number keeps 11 bits down to 2^-29
// of that.  4,096 tokens of 16 heads, the whole layer: 0.0042 from 64 bits, attention on the latent 0.0046.
//
// Measured there (R = 512): expansion 25 us, attention 123 (700 and 700 TFLOP/s), where the queries' and outputs' products and attention on the latent take
// 34 + 64 and 491.
//
// keys, values [H][n_seqs * cap][128]: key j of sequence i in row i * cap + j, cap a multiple of 128.  A block takes 128 keys of one head, two
// pages of the cache: both products over the latent share the page's tile (A); B is Wuk_h [128][R] as it lies, and Wuv_h [R][128], an
// MN-major operand in two pieces of 64 columns.  Two stages of 64 k (48 KB each), so that two blocks share an SM and one's epilogue runs under
// the other's loads, which bound it: 32 KB of weights per 64 k from L2.  Rows past the sequence's end, or of pages ahead of the
// window, are zeros, so that no weight of zero meets a NaN.
constexpr int LE_STAGES = 2, LE_STAGE_BYTES = 3 * HALF_BYTES;
constexpr uint32_t LE_SMEM = 1024 + LE_STAGES * LE_STAGE_BYTES + 128;
static_assert(4 * 32 * HW_PITCH * 4 <= LE_STAGES * LE_STAGE_BYTES, "the epilogue's rows take the ring's place");

struct LeBars {
    unsigned long long full[LE_STAGES], empty[LE_STAGES], done;
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(192)
latent_expand_kernel(const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_uk, const __grid_constant__ CUtensorMap map_uv,
                     __nv_bfloat16* __restrict__ keys, __half* __restrict__ values, const float* __restrict__ v_scale, const int* __restrict__ page_table,
                     int max_pages, int n_pages_pool, GfbBatch b, int H, int R, int cap, int window, int* status) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_c); prefetch_map(&map_uk); prefetch_map(&map_uv); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    LeBars* bars = reinterpret_cast<LeBars*>(aligned + LE_STAGES * LE_STAGE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = cap / KEYS, tile = blockIdx.x / H, h = blockIdx.x - tile * H, seq = tile / tiles, key0 = (tile - seq * tiles) * KEYS;
    if (threadIdx.x == 0) {
        for (int s = 0; s < LE_STAGES; s++) { mbar_init(smem_u32(&bars->full[s]), 1); mbar_init(smem_u32(&bars->empty[s]), 1); }
        mbar_init(smem_u32(&bars->done), 1);
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int slot = b.slots[seq], start = b.lengths[slot], new_tokens = b.cu_seqlens[seq + 1] - b.cu_seqlens[seq], len = start + new_tokens;
    const int lo = window > 0 ? max(0, start - window + 1) : 0;      // the first key that any new token sees
    const bool idle = new_tokens <= 0 || key0 >= len || key0 + KEYS <= lo;
    if (idle) {
    } else if (warp == 0) {
        if (lane == 0) {
            int page[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {                            // (a page that no token sees: another one, its rows become zeros)
                const int pi = min(max(key0 / PAGE + i, lo / PAGE), (len - 1) / PAGE);
                page[i] = pi < max_pages ? page_table[(size_t)slot * max_pages + pi] : -1;
                if (page[i] < 0 || page[i] >= n_pages_pool) { gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi); page[i] = 0; }
            }
            for (int kb = 0; kb < R / 64; kb++) {
                const int s = kb % LE_STAGES;
                if (!mbar_wait(smem_u32(&bars->empty[s]), ((uint32_t)(kb / LE_STAGES) & 1u) ^ 1u, abort_flag, status, 41)) break;
                const uint32_t full = smem_u32(&bars->full[s]), at = base + s * LE_STAGE_BYTES;
                mbar_expect_tx(full, LE_STAGE_BYTES);
                tma_load_2d(at, &map_c, kb * 64, page[0] * PAGE, full);
                tma_load_2d(at + PIECE_BYTES, &map_c, kb * 64, page[1] * PAGE, full);
                tma_load_2d(at + HALF_BYTES, &map_uk, kb * 64, h * D, full);
                tma_load_2d(at + 2 * HALF_BYTES, &map_uv, 0, h * R + kb * 64, full);
                tma_load_2d(at + 2 * HALF_BYTES + PIECE_BYTES, &map_uv, 64, h * R + kb * 64, full);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc_k = idesc_bf16(ROWS, D, 0), idesc_v = idesc_bf16(ROWS, D, 1);
            bool ok = true;
            for (int kb = 0; kb < R / 64 && ok; kb++) {
                const int s = kb % LE_STAGES;
                ok = mbar_wait(smem_u32(&bars->full[s]), (uint32_t)(kb / LE_STAGES) & 1u, abort_flag, status, 42);
                if (!ok) break;
                tc_fence_after();
                const uint32_t at = base + s * LE_STAGE_BYTES;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    umma_ss(tmem, desc_kmajor(at) + 2 * k, desc_kmajor(at + HALF_BYTES) + 2 * k, idesc_k, (kb | k) != 0);
                    umma_ss(tmem + D, desc_kmajor(at) + 2 * k, desc_mnmajor(at + 2 * HALF_BYTES + k * 2048, PIECE_BYTES), idesc_v, (kb | k) != 0);
                }
                umma_commit(smem_u32(&bars->empty[s]));
            }
            if (ok) umma_commit(smem_u32(&bars->done));
        }
    } else {
        const int q = warp & 3;
        float* mine = reinterpret_cast<float*>(aligned) + q * 32 * HW_PITCH;
        if (mbar_wait_warp(smem_u32(&bars->done), 0, abort_flag, status, 43)) {      // every copy has landed and been read
            tc_fence_after();
            const size_t row0 = ((size_t)h * b.n_seqs + seq) * cap + key0 + q * 32;
#pragma unroll 1
            for (int half = 0; half < 2; half++) {
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    float v[32];
                    tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + half * D + c, v);
#pragma unroll
                    for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(mine + lane * HW_PITCH + c + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
                __syncwarp();
                uint16_t* out = (half ? reinterpret_cast<uint16_t*>(values) : reinterpret_cast<uint16_t*>(keys)) + row0 * D + lane * 4;
                const float4 sc = half ? *reinterpret_cast<const float4*>(v_scale + h * D + lane * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll 4
                for (int r = 0; r < 32; r++) {
                    const float4 v = *reinterpret_cast<const float4*>(mine + r * HW_PITCH + lane * 4);
                    const int key = key0 + q * 32 + r;
                    const bool there = key < len && key >= (lo & ~(PAGE - 1));
                    const uint2 both = half ? make_uint2(pack2_half(v.x * sc.x, v.y * sc.y), pack2_half(v.z * sc.z, v.w * sc.w))
                                            : make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
                    *reinterpret_cast<uint2*>(out + (size_t)r * D) = there ? both : make_uint2(0u, 0u);
                }
                __syncwarp();
            }
        }
    }
    if (*abort_flag) {
        unsigned long long w0 = global_ns();
        while (global_ns() - w0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

// Attention of one head over its expanded keys [128 | the 64 rotated numbers all heads share, in the cache's rows] and values [128], the output
// times a sigmoid gate.  As attn_prefill_tc2_kernel: two tiles of 128 tokens per block share every 128 keys, and the tensor pipe alternates between
// them.  What bounds it is a tile's chain of scores, softmax and P V, so each has eight softmax warps: two threads share a row, 64 keys each, and
// tell each other their maximum (and in the end their sum) through a column of tensor memory that the scores have left (4,096 tokens of
// 16 heads: a thread per row 129 us, two 123; the products of both tiles behind one another 137).  Q of both tiles (96 KB) leaves a ring of eight slots of 16 KB for three pieces of K, [128 keys][64
// dims], and two of V, [64 keys][128 dims], per 128 keys, in the order in which they are freed: V_j, K_(j+1), V_(j+1), ...; a
// piece takes the slot of the eighth piece before it.
// float16 has more bits than bfloat16 and far fewer exponents, so weights are lifted to the top of its range: the reference of the exponentials lags a
// row's maximum by up to 2^LH_LAG and stands for 2^LH_LIFT, so that the largest weight of a row lies between 2^LH_LIFT and 2^15, one 2^29 below
// it keeps ten bits and one 2^35 below it is not lost; and the sum takes the weights as they are rounded for P V.  (Sums of unrounded weights up to 2^8
// lost a flat tail 2^25.5 below a row's peak, and kept it in the denominator: 2.8e-3 of a row at 131,072 keys.)
//   tensor memory: S of tile x in columns 128 x .. 128 x + 127 (P overwrites the first half), O of tile x in 256 + 128 x ..
constexpr int LH_Q_BYTES = 3 * HALF_BYTES, LH_SLOTS = 8;
constexpr float LH_LAG = 3.f, LH_LIFT = 15.f - LH_LAG;
struct LhBars {
    unsigned long long q_full;
    unsigned long long k_full[2], k_empty[2], v_full[2], v_empty[2];   // of even and odd key blocks
    unsigned long long s_full[2], p_ready[2], pv_done[2];              // per tile
    unsigned long long told[2][4];                                     // per tile and quarter of its rows: both halves of the keys have told
    uint32_t tmem_base;
    int abort_flag;
};
constexpr int LH_THREADS = 64 + 2 * 256;
constexpr uint32_t LH_SMEM = 1024 + 2 * LH_Q_BYTES + LH_SLOTS * HALF_BYTES + sizeof(LhBars);
static_assert(LH_SMEM <= 227 * 1024, "shared memory");

__global__ void __launch_bounds__(LH_THREADS, 1)
latent_heads_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_kr, const __grid_constant__ CUtensorMap map_v, int q_off, __nv_bfloat16* __restrict__ out,
                    const float* __restrict__ v_unscale, const __nv_bfloat16* __restrict__ gate, int ld_gate, int gate_off, int gate_per_head, const int* __restrict__ page_table,
                    int max_pages, int n_pages_pool, GfbBatch b, int H, int R, int cap, float scale_log2e, int window, const float* __restrict__ sink,
                    int n_x, int* status) {
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 0) { prefetch_map(&map_q); prefetch_map(&map_qr); prefetch_map(&map_k); prefetch_map(&map_kr); prefetch_map(&map_v); }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t qs = base, ring = base + 2 * LH_Q_BYTES;
    LhBars* bars = reinterpret_cast<LhBars*>(aligned + 2 * LH_Q_BYTES + LH_SLOTS * HALF_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bars->q_full), 1);
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&bars->k_full[s]), 1);
            mbar_init(smem_u32(&bars->k_empty[s]), 1);
            mbar_init(smem_u32(&bars->v_full[s]), 1);
            mbar_init(smem_u32(&bars->v_empty[s]), 1);
            mbar_init(smem_u32(&bars->s_full[s]), 1);
            mbar_init(smem_u32(&bars->p_ready[s]), 8);
            mbar_init(smem_u32(&bars->pv_done[s]), 1);
            for (int k = 0; k < 4; k++) mbar_init(smem_u32(&bars->told[s][k]), 2);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    gfb_pdl_launch();
    gfb_pdl_wait();

    // the item: two tiles of tokens (the latest of the last sequence first: they see the most keys) of one head
    const int xi = (int)blockIdx.x / H, head = (int)blockIdx.x - xi * H;
    int seq = -1, tq0 = 0;
    {
        int left = n_x - 1 - xi;
        for (int i = 0; i < b.n_seqs; i++) {
            const int nt = (b.cu_seqlens[i + 1] - b.cu_seqlens[i] + 2 * ROWS - 1) / (2 * ROWS);
            if (left < nt) { seq = i; tq0 = left * 2 * ROWS; break; }
            left -= nt;
        }
    }
    if (seq >= 0) {
        const int t_first = b.cu_seqlens[seq], qlen = b.cu_seqlens[seq + 1] - t_first, slot = b.slots[seq], len0 = b.lengths[slot];
        if (threadIdx.x == 0 && len0 + qlen > cap) gfb_report(status, GFB_ERR_CACHE_RANGE, t_first + qlen - 1, len0 + qlen - 1);   // more than the host's bound
        // per tile: tokens [tq0 + 128 x, +nq), positions from pos0, key blocks [lo_blk, hi_blk)
        int nq[2], pos0[2], lo_blk[2], hi_blk[2];
#pragma unroll
        for (int x = 0; x < 2; x++) {
            nq[x] = min(ROWS, qlen - (tq0 + x * ROWS));
            pos0[x] = len0 + tq0 + x * ROWS;
            lo_blk[x] = nq[x] > 0 ? first_key(pos0[x], window, 0) / KEYS : 0;
            hi_blk[x] = nq[x] > 0 ? (pos0[x] + nq[x] - 1) / KEYS + 1 : 0;
        }
        const int blk0 = lo_blk[0], n_iter = max(hi_blk[0], hi_blk[1]) - blk0;      // (the second tile's tokens are later ones)
        auto active = [&](int x, int j) { return blk0 + j >= lo_blk[x] && blk0 + j < hi_blk[x]; };

        if (warp == 0) {
            if (lane == 0) {
                mbar_expect_tx(smem_u32(&bars->q_full), 2 * LH_Q_BYTES);
#pragma unroll
                for (int x = 0; x < 2; x++) {                                // rows beyond the batch are filled with zeros
                    const int t = t_first + tq0 + x * ROWS;
                    tma_load_2d(qs + x * LH_Q_BYTES, &map_q, q_off + head * 192, t, smem_u32(&bars->q_full));
                    tma_load_2d(qs + x * LH_Q_BYTES + HALF_BYTES, &map_q, q_off + head * 192 + 64, t, smem_u32(&bars->q_full));
                    tma_load_2d(qs + x * LH_Q_BYTES + 2 * HALF_BYTES, &map_qr, head * 64, t, smem_u32(&bars->q_full));
                }
                const int* pt = page_table + (size_t)slot * max_pages;
                const int row0 = (head * b.n_seqs + seq) * cap, lo_page = first_key(len0, window, 0) / PAGE, last_page = (len0 + qlen - 1) / PAGE;
                auto slot_at = [&](int piece) { return ring + (uint32_t)(piece % LH_SLOTS) * HALF_BYTES; };
                // pieces 5 j .. 5 j + 2 are K of block j, 5 j + 3 and 5 j + 4 its V
                auto load_k = [&](int j) -> bool {
                    const uint32_t full = smem_u32(&bars->k_full[j & 1]), ph = ((uint32_t)(j >> 1) & 1u) ^ 1u;
                    const int row = row0 + (blk0 + j) * KEYS;
                    int page[2];                                         // (asked for ahead of the waits)
#pragma unroll
                    for (int i = 0; i < 2; i++) {                        // (no such page, or one ahead of the window: any other, masked later)
                        const int pi = min(max((blk0 + j) * 2 + i, lo_page), last_page);
                        page[i] = pi < max_pages ? pt[pi] : -1;
                    }
                    if (!mbar_wait(smem_u32(&bars->k_empty[j & 1]), ph, abort_flag, status, 44)) return false;       // K of block j - 2
                    mbar_expect_tx(full, 3 * HALF_BYTES);
                    tma_load_2d(slot_at(5 * j), &map_k, 0, row, full);
                    if (!mbar_wait(smem_u32(&bars->v_empty[j & 1]), ph, abort_flag, status, 45)) return false;       // V of block j - 2
                    tma_load_2d(slot_at(5 * j + 1), &map_k, 64, row, full);
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        if (page[i] < 0 || page[i] >= n_pages_pool) { gfb_report(status, GFB_ERR_PAGE_TABLE, slot, (blk0 + j) * 2 + i); page[i] = 0; }
                        tma_load_2d(slot_at(5 * j + 2) + i * PIECE_BYTES, &map_kr, R, page[i] * PAGE, full);
                    }
                    return true;
                };
                bool ok = load_k(0);
                for (int j = 0; j < n_iter && ok; j++) {
                    const uint32_t full = smem_u32(&bars->v_full[j & 1]);
                    const int row = row0 + (blk0 + j) * KEYS;
                    if (j > 0) ok = mbar_wait(smem_u32(&bars->k_empty[(j - 1) & 1]), (uint32_t)((j - 1) >> 1) & 1u, abort_flag, status, 46);   // K of block j - 1
                    if (!ok) break;
                    mbar_expect_tx(full, 2 * HALF_BYTES);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        tma_load_2d(slot_at(5 * j + 3 + (i >> 1)) + (i & 1) * PIECE_BYTES, &map_v, (i & 1) * 64, row + (i >> 1) * 64, full);
                    if (j + 1 < n_iter) ok = load_k(j + 1);
                }
            }
        } else if (warp == 1) {
            if (lane == 0) {
                constexpr uint32_t idesc_s = idesc_bf16(ROWS, KEYS, 0), idesc_o = idesc_f16(ROWS, D, 1);
                uint32_t n_pv[2] = {0, 0};                                   // P V products issued per tile
                bool ok = mbar_wait(smem_u32(&bars->q_full), 0, abort_flag, status, 47);
                auto slot_at = [&](int piece) { return ring + (uint32_t)(piece % LH_SLOTS) * HALF_BYTES; };
                auto issue_s = [&](int x, int j) {                           // K of block j is known to be loaded
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const uint64_t da = desc_kmajor(qs + x * LH_Q_BYTES + c * HALF_BYTES), db = desc_kmajor(slot_at(5 * j + c));
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_ss(tmem + 128 * x, da + 2 * k, db + 2 * k, idesc_s, (c | k) != 0);
                    }
                    umma_commit(smem_u32(&bars->s_full[x]));
                };
                auto k_ready = [&](int j) { return mbar_wait(smem_u32(&bars->k_full[j & 1]), (uint32_t)(j >> 1) & 1u, abort_flag, status, 48); };
                ok = ok && k_ready(0);
                if (ok) {
                    tc_fence_after();
                    if (active(0, 0)) issue_s(0, 0);
                    if (active(1, 0)) issue_s(1, 0);
                    umma_commit(smem_u32(&bars->k_empty[0]));
                }
                for (int j = 0; j < n_iter && ok; j++) {
                    bool k_next = false;                                     // whether K of block j + 1 has been waited for
                    ok = mbar_wait(smem_u32(&bars->v_full[j & 1]), (uint32_t)(j >> 1) & 1u, abort_flag, status, 49);
#pragma unroll
                    for (int x = 0; x < 2 && ok; x++) {
                        if (active(x, j)) {
                            ok = mbar_wait(smem_u32(&bars->p_ready[x]), n_pv[x] & 1u, abort_flag, status, 50);
                            if (!ok) break;
                            tc_fence_after();
#pragma unroll
                            for (int kk = 0; kk < 8; kk++)                   // 16 keys per MMA: 8 columns of P, 2 KB of either half of the dims
                                umma_ts(tmem + 256 + 128 * x, tmem + 128 * x + kk * 8,
                                        desc_mnmajor(slot_at(5 * j + 3 + (kk >> 2)) + (kk & 3) * 2048, PIECE_BYTES), idesc_o, (n_pv[x] | (uint32_t)kk) != 0);
                            umma_commit(smem_u32(&bars->pv_done[x]));
                            n_pv[x]++;
                        }
                        if (j + 1 < n_iter && active(x, j + 1)) {            // the tile's next scores, behind its P V
                            if (!k_next) { ok = k_ready(j + 1); k_next = true; if (!ok) break; tc_fence_after(); }
                            issue_s(x, j + 1);
                        }
                    }
                    if (!ok) break;
                    umma_commit(smem_u32(&bars->v_empty[j & 1]));
                    if (j + 1 < n_iter) {
                        if (!k_next) { ok = k_ready(j + 1); if (!ok) break; }
                        umma_commit(smem_u32(&bars->k_empty[(j + 1) & 1]));
                    }
                }
            }
        } else {
            const int x = (warp - 2) >> 3, half = (warp - 2) >> 2 & 1;       // warps 2..9: tile 0, 10..17: tile 1; the first four of them keys 0..63
            const int q = warp & 3, r = q * 32 + lane;
            const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
            const uint32_t col_s = 128 * x, col_o = 256 + 128 * x + 64 * half;       // (each half also rescales and writes half of O)
            const uint32_t told = smem_u32(&bars->told[x][q]);
            // the last column of either half of the scores: its own half's thread writes it behind its loads, the other reads it ahead of
            // what comes next there (P of the second half in columns 32 .. 63, the next scores)
            const uint32_t col_mine = lane_base + col_s + 63 + 64 * half, col_other = lane_base + col_s + 63 + 64 * (half ^ 1);
            uint32_t n_told = 0;
            auto exchange = [&](float mine, float& other) -> bool {
                tmem_st1(col_mine, mine);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(told);
                if (!mbar_wait(told, n_told & 1u, abort_flag, status, 54)) return false;
                n_told++;
                tc_fence_after();
                other = tmem_ld1(col_other);
                return true;
            };
            const bool row_ok = r < nq[x];
            const int row_pos = pos0[x] + r, row_lo = first_key(row_pos, window, 0), last_lo = first_key(pos0[x] + max(nq[x], 1) - 1, window, 0);
            float m_run = -INFINITY, l_run = 0.f;
            uint32_t n_done = 0;                                             // blocks of this tile finished
            bool ok = true;
            for (int j = 0; j < n_iter && ok; j++) {
                if (!active(x, j)) continue;
                const int key0 = (blk0 + j) * KEYS + 64 * half;
                ok = mbar_wait_warp(smem_u32(&bars->s_full[x]), n_done & 1u, abort_flag, status, 51);
                if (!ok) break;
                tc_fence_after();
                uint32_t raw[2][32];
                tmem_ld32_issue(lane_base + col_s + 64 * half, raw[0]);
                tmem_ld32_issue(lane_base + col_s + 64 * half + 32, raw[1]);
                tmem_ld_wait32(raw[0]);
                tmem_ld_wait32(raw[1]);
                float v[2][32];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int i = 0; i < 32; i++) v[c][i] = __uint_as_float(raw[c][i]);
                if (key0 + 63 > pos0[x] || key0 < last_lo || nq[x] < ROWS) {
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int i = 0; i < 32; i++) {
                            const int kj = key0 + c * 32 + i;
                            if (!(row_ok && kj <= row_pos && kj >= row_lo)) v[c][i] = -INFINITY;
                        }
                }
                float mx4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float* y = &v[c >> 1][(c & 1) * 16];
                    mx4[c] = fmaxf(y[0], y[1]);
#pragma unroll
                    for (int i = 2; i < 16; i += 2) mx4[c] = max3(mx4[c], y[i], y[i + 1]);
                }
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])), theirs;
                ok = exchange(mx, theirs);
                if (!ok) break;
                mx = fmaxf(mx, theirs);
                float m_new = m_run;
                if (mx > m_run && (m_run == -INFINITY || (mx - m_run) * scale_log2e > LH_LAG)) m_new = mx;
                const float corr = (m_run == -INFINITY || m_new == m_run) ? 1.f : fast_exp2((m_run - m_new) * scale_log2e);
                const float mneg = (m_new == -INFINITY) ? 0.f : LH_LIFT - m_new * scale_log2e;
                float rsum[2] = {0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t pk[16];
                    float odd = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float a0, a1;
                        fma2(v[c][i], v[c][i + 1], scale_log2e, mneg, a0, a1);
                        const __half2 p = __floats2half2_rn(fast_exp2(a0), fast_exp2(a1));
                        const float2 rounded = __half22float2(p);        // what P V takes is what the sum takes
                        add2(rsum[c], odd, rounded.x, rounded.y);
                        pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&p);
                    }
                    rsum[c] += odd;
                    tmem_st16(lane_base + col_s + 32 * half + c * 16, pk);   // (both halves of this row's scores are in registers by now)
                }
                // O follows a new reference, rarely (S of this block was issued behind the tile's previous P V, so that the wait only orders the accesses)
                if (n_done > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                    ok = mbar_wait_warp(smem_u32(&bars->pv_done[x]), (n_done - 1u) & 1u, abort_flag, status, 52);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 2; c++) {
                        float o[32];
                        tmem_ld32(lane_base + col_o + c * 32, o);
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] *= corr;
                        tmem_st32(lane_base + col_o + c * 32, o);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->p_ready[x]));
                l_run = l_run * corr + (rsum[0] + rsum[1]);
                m_run = m_new;
                n_done++;
            }
            if (ok && n_done > 0) ok = mbar_wait_warp(smem_u32(&bars->pv_done[x]), (n_done - 1u) & 1u, abort_flag, status, 53);
            if (ok && n_done > 0) {
                tc_fence_after();
                float theirs;
                ok = exchange(l_run, theirs);                                // (the last P has been read)
                l_run = half ? theirs + l_run : l_run + theirs;
            }
            if (ok && n_done > 0) {
                if (sink != nullptr && m_run != -INFINITY) l_run += fast_exp2(sink[head] * 1.4426950408889634f + (LH_LIFT - m_run * scale_log2e));
                const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
                const size_t t = (size_t)(t_first + tq0 + x * ROWS + (row_ok ? r : 0));
                const int dim0 = 64 * half;
                __nv_bfloat16* dst = out + (t * H + head) * D + dim0;
                const __nv_bfloat16* gt = gate + t * ld_gate + gate_off;
                const float per_head = gate_per_head ? 1.0f / (1.0f + expf(-__bfloat162float(gt[head]))) : 1.f;
#pragma unroll 1
                for (int c = 0; c < 2; c++) {
                    float o[32];
                    tmem_ld32(lane_base + col_o + c * 32, o);
                    if (row_ok) {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            const float* un = v_unscale + head * D + dim0 + c * 32 + i;
                            const float4 u0 = *reinterpret_cast<const float4*>(un), u1 = *reinterpret_cast<const float4*>(un + 4);
                            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
                            float y[8];
#pragma unroll
                            for (int e = 0; e < 8; e++) y[e] = o[i + e] * inv * u[e] * per_head;
                            if (!gate_per_head) {
                                const uint4 g8 = *reinterpret_cast<const uint4*>(gt + head * D + dim0 + c * 32 + i);
                                const uint32_t g4[4] = {g8.x, g8.y, g8.z, g8.w};
#pragma unroll
                                for (int e = 0; e < 4; e++) {
                                    y[2 * e] *= 1.0f / (1.0f + expf(-__uint_as_float(g4[e] << 16)));
                                    y[2 * e + 1] *= 1.0f / (1.0f + expf(-__uint_as_float(g4[e] & 0xffff0000u)));
                                }
                            }
                            *reinterpret_cast<uint4*>(dst + c * 32 + i) = make_uint4(pack2(y[0], y[1]), pack2(y[2], y[3]), pack2(y[4], y[5]), pack2(y[6], y[7]));
                        }
                    }
                }
            }
        }
    }
    if (*abort_flag) {
        unsigned long long w0 = global_ns();
        while (global_ns() - w0 < 50000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

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

}  // namespace

// Causal attention for runs of new tokens on tcgen05; head_dim 128, pages of 64, at most 8 heads per group
// with 128 % (heads per group) == 0.  tiles: query tiles of 128 rows per block, 1 or 2, or 0 to let the
// function choose by the amount of work.  max_blocks: cap of the one-tile kernel's grid (0: one block per SM).
GFB_API int gfb_attn_prefill_tc_masked(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, int tiles, int max_blocks, int* status, cudaStream_t stream);

GFB_API int gfb_attn_prefill_tc(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                int tiles, int max_blocks, int* status, cudaStream_t stream) {
    return gfb_attn_prefill_tc_masked(q, out, k_pool, v_pool, page_table, max_pages, page_size, n_pages, cu_seqlens, tok_seq, slots,
                                      lengths, n_seqs, n_tokens, H, G, d, scale, window, 0, nullptr, tiles, max_blocks, status, stream);
}

// The same with a block mask (chunk > 0: a query sees only the keys of its own block of `chunk` positions, blocks
// counted from position 0) and a sink (float32 [H] or null: exp(sink_h) joins the softmax denominator of head h).
GFB_API int gfb_attn_prefill_tc_biased(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, const float* bias, int bias_len, int bias_top,
                                       const float* slopes, int tiles, int max_blocks, int* status, cudaStream_t stream);

GFB_API int gfb_attn_prefill_tc_masked(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, int tiles, int max_blocks, int* status, cudaStream_t stream) {
    return gfb_attn_prefill_tc_biased(q, out, k_pool, v_pool, page_table, max_pages, page_size, n_pages, cu_seqlens, tok_seq, slots,
                                      lengths, n_seqs, n_tokens, H, G, d, scale, window, chunk, sink, nullptr, 0, 0, nullptr, tiles,
                                      max_blocks, status, stream);
}

// Kept first positions: behind the windowed attention, every query whose window no longer reaches the sequence's start takes
// the first positions it does not see (j < min(keep_first, first key of its window)) into its row: with the row's log-sum-exp
// L (log2 units) from the attention kernel and x_j = log2(e) cap(scale q.k_j),
//     M = max(L, max_j x_j),  w = 2^(L - M),  out <- (w out + sum_j 2^(x_j - M) v_j) / (w + sum_j 2^(x_j - M)).
// One warp per (token, head), a lane holds DH / 32 dimensions of the row; the kept positions are few.
template <int DH>
__global__ void __launch_bounds__(128)
attn_kept_merge_kernel(const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ out, const float* __restrict__ lse,
                       const __nv_bfloat16* __restrict__ k_pool, const __nv_bfloat16* __restrict__ v_pool,
                       const int* __restrict__ page_table, int max_pages, int n_pages, GfbBatch b, int H, int G, float scale,
                       float softcap, int window, int keep_first, int* status) {
    constexpr int PER = DH / 32;
    gfb_pdl_launch();
    gfb_pdl_wait();
    const int lane = threadIdx.x & 31;
    const long item = (long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (item >= (long)b.n_tokens * H) return;
    const int t = (int)(item / H), h = (int)(item - (long)t * H);
    const int s = b.tok_seq[t];
    const int slot = b.slots[s];
    const int pos = b.lengths[slot] + (t - b.cu_seqlens[s]);
    const int kept = min(keep_first, pos - window + 1);
    if (kept <= 0) return;
    const int g = h / (H / G);
    const size_t at = (size_t)item * DH + lane * PER;
    float qv[PER], acc[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) { qv[i] = __bfloat162float(q[at + i]); acc[i] = __bfloat162float(out[at + i]); }
    float m = lse[item], den = 1.f;                              // the row so far, in units of 2^m
    if (m == -INFINITY) {
        den = 0.f;
#pragma unroll
        for (int i = 0; i < PER; i++) acc[i] = 0.f;
    }
    for (int j = 0; j < kept; j++) {
        const int pi = j / PAGE;
        const int page = pi < max_pages ? page_table[(size_t)slot * max_pages + pi] : -1;
        if (page < 0 || page >= n_pages) {
            if (lane == 0) gfb_report(status, GFB_ERR_PAGE_TABLE, slot, pi);
            return;
        }
        const size_t row = (((size_t)page * G + g) * PAGE + (j - pi * PAGE)) * DH + lane * PER;
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < PER; i++) dot = fmaf(qv[i], __bfloat162float(k_pool[row + i]), dot);
        float sc = gfb_warp_sum(dot) * scale;
        if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        const float x = sc * 1.4426950408889634f;
        const float m_new = fmaxf(m, x);
        const float down = m == -INFINITY ? 0.f : exp2f(m - m_new), p = exp2f(x - m_new);
        den = den * down + p;
#pragma unroll
        for (int i = 0; i < PER; i++) acc[i] = acc[i] * down + p * __bfloat162float(v_pool[row + i]);
        m = m_new;
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
    for (int i = 0; i < PER; i++) out[at + i] = __float2bfloat16_rn(acc[i] * inv);
}

// The same with a bias by head and distance in units of the raw score (the bias divided by `scale`): `bias` null or
// float32 [4][H][bias_len], the four moved copies of the per-head array that `DistanceBias` describes, with distance 0 at
// entry bias_top; `slopes` null or float32 [H].
// ... and with a soft cap on the scaled score (softcap > 0: cap tanh(s / cap)) and kept first positions (keep_first > 0, with a
// window: the sequence's first keep_first positions stay visible to every later query).  Both run in the one-tile kernel; the
// kept positions are merged into the rows by a second kernel, for which the first leaves every row's log-sum-exp in `lse`
// (float32 [n_tokens * H], the caller's scratch).
GFB_API int gfb_attn_prefill_tc_capped(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, const float* bias, int bias_len, int bias_top,
                                       const float* slopes, float softcap, int keep_first, float* lse, int tiles, int max_blocks,
                                       int* status, cudaStream_t stream);

GFB_API int gfb_attn_prefill_tc_biased(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, const float* bias, int bias_len, int bias_top,
                                       const float* slopes, int tiles, int max_blocks, int* status, cudaStream_t stream) {
    return gfb_attn_prefill_tc_capped(q, out, k_pool, v_pool, page_table, max_pages, page_size, n_pages, cu_seqlens, tok_seq, slots,
                                      lengths, n_seqs, n_tokens, H, G, d, scale, window, chunk, sink, bias, bias_len, bias_top, slopes,
                                      0.f, 0, nullptr, tiles, max_blocks, status, stream);
}

GFB_API int gfb_attn_prefill_tc_capped(const void* q, void* out, void* k_pool, void* v_pool, const int* page_table, int max_pages,
                                       int page_size, int n_pages, const int* cu_seqlens, const int* tok_seq, const int* slots,
                                       const int* lengths, int n_seqs, int n_tokens, int H, int G, int d, float scale, int window,
                                       int chunk, const float* sink, const float* bias, int bias_len, int bias_top,
                                       const float* slopes, float softcap, int keep_first, float* lse, int tiles, int max_blocks,
                                       int* status, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (softcap < 0.f || keep_first < 0 || ((softcap > 0.f || keep_first > 0) && !(scale > 0.f)))
        return gfb_fail("gfb_attn_prefill_tc: a soft cap of %f, %d kept first positions, a scale of %f", softcap, keep_first, scale);
    if (keep_first > 0 && (window <= 0 || chunk > 0)) keep_first = 0;          // no window: every earlier position is seen anyway
    if (keep_first > 0 && (lse == nullptr || sink != nullptr || bias != nullptr || slopes != nullptr))
        return gfb_fail("gfb_attn_prefill_tc: kept first positions need scratch for the rows' log-sum-exp and go without a sink or a distance bias");
    if (keep_first == 0) lse = nullptr;
    if (softcap > 0.f || keep_first > 0) tiles = 1;
    const float cap_raw = softcap > 0.f ? softcap / scale : 0.f;
    if (bias != nullptr && (bias_len % 4 || bias_len < 128 + 4 + 384 || bias_top < 127 || bias_top + 384 >= bias_len
                            || (reinterpret_cast<uintptr_t>(bias) & 15)))
        return gfb_fail("gfb_attn_prefill_tc: a distance array of %d entries with distance 0 at %d (128 far entries ahead of the table, "
                        "384 behind distance 0, a multiple of 4, 16-byte aligned)", bias_len, bias_top);
    DistanceBias db{bias, bias_len, bias_top, slopes, 0, 0};
    if (page_size != PAGE || (d != 64 && d != 128))
        return gfb_fail("gfb_attn_prefill_tc: built for pages of %d and head_dim 64 or 128, got %d and %d", PAGE, page_size, d);
    if (G <= 0 || H % G) return gfb_fail("gfb_attn_prefill_tc: %d heads over %d groups", H, G);
    const int rep = H / G;
    if (rep > 8) return gfb_fail("gfb_attn_prefill_tc: %d heads per group (at most 8)", rep);
    const int TQ = ROWS / rep;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return gfb_fail("gfb_attn_prefill_tc: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap mq, mk, mv;
    {
        cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)H, (cuuint64_t)n_tokens};
        cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)H * d * 2};
        cuuint32_t box[3] = {64, (cuuint32_t)rep, (cuuint32_t)TQ};
        cuuint32_t es[3] = {1, 1, 1};
        CUresult r = enc(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return gfb_fail("gfb_attn_prefill_tc: tensor map of q refused (%d)", (int)r);
    }
    if ((long long)n_pages * G * PAGE > 2147483647LL)           // TMA coordinates are 32-bit
        return gfb_fail("gfb_attn_prefill_tc: %d pages x %d heads x %d tokens do not fit the 32-bit row coordinate of a tensor map",
                        n_pages, G, PAGE);
    for (int i = 0; i < 2; i++) {
        cuuint64_t dims[2] = {(cuuint64_t)d, (cuuint64_t)n_pages * G * PAGE};
        cuuint64_t strides[1] = {(cuuint64_t)d * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)PAGE};
        cuuint32_t es[2] = {1, 1};
        CUresult r = enc(i ? &mv : &mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, i ? v_pool : k_pool, dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return gfb_fail("gfb_attn_prefill_tc: tensor map of the cache refused (%d)", (int)r);
    }
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    if (tiles < 0 || tiles > 2) return gfb_fail("gfb_attn_prefill_tc: %d query tiles per block (0 = choose, 1 or 2)", tiles);
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
    }
    cudaError_t e;
    const long blocks2 = ((long)(n_tokens + 2 * TQ - 1) / (2 * TQ)) * G;
    if (d == 128 && (tiles == 2 || (tiles == 0 && blocks2 >= 6L * sms))) {
        // enough work for several rounds of blocks of two tiles, which share their K/V loads and keep the tensor
        // pipe busier (measured: from about 7,000 tokens of one sequence on, at 32 heads in 8 groups); with less
        // work the persistent one-tile kernel balances the SMs better
        size_t smem = 1024 + (size_t)(2 + 2 * KV_STAGES) * TILE_BYTES + sizeof(Bars2);
        static size_t configured2 = 0;
        if (smem > configured2) {
            cudaError_t a = cudaFuncSetAttribute(attn_prefill_tc2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (a != cudaSuccess) return gfb_fail("gfb_attn_prefill_tc: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(a));
            configured2 = smem;
        }
        dim3 grid((n_tokens + 2 * TQ - 1) / (2 * TQ) + n_seqs, G);
        e = gfb_launch(attn_prefill_tc2_kernel, grid, dim3(320), smem, stream, mq, mk, mv, (__nv_bfloat16*)out,
                       page_table, max_pages, n_pages, b, H, G, scale * 1.4426950408889634f, window, chunk, sink, db, status);
    } else {
        size_t smem = 1024 + (size_t)(1 + 2 * KV_STAGES) * TILE_BYTES + ((sizeof(Bars) + 15) & ~(size_t)15);
        if (bias != nullptr && window > 0) {
            // the table of a group's heads in shared memory, where it fits beside the tiles: every distance a tile can meet
            // under its window, the stride chosen so that the 32 rows of a warp (tokens x heads of the group) read 32 banks
            const int s_len = TABLE_AHEAD + window + TABLE_BEYOND;
            const int want = 32 % rep == 0 ? (32 / rep) % 32 : 1;
            const int s_stride = s_len + ((want - s_len) % 32 + 32) % 32;
            const size_t bytes = (size_t)rep * s_stride * sizeof(float);
            if (smem + bytes <= 227 * 1024) {
                db.s_len = s_len;
                db.s_stride = s_stride;
                smem += bytes;
            }
        }
        static size_t configured = 0;
        if (smem > configured) {
            cudaError_t a = cudaFuncSetAttribute(attn_prefill_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (a == cudaSuccess) a = cudaFuncSetAttribute(attn_prefill_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (a != cudaSuccess) return gfb_fail("gfb_attn_prefill_tc: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(a));
            configured = smem;
        }
        const int n_x = (n_tokens + TQ - 1) / TQ + n_seqs;           // an upper bound of the tiles; surplus items are empty
        long blocks = (long)n_x * G;
        const long cap = max_blocks > 0 ? max_blocks : sms;           // one block per SM walks over the items
        if (blocks > cap) blocks = cap;
        if (d == 128)
            e = gfb_launch(attn_prefill_tc_kernel<128>, dim3((unsigned)blocks), dim3(320), smem, stream, mq, mk, mv, (__nv_bfloat16*)out,
                           page_table, max_pages, n_pages, b, H, G, scale * 1.4426950408889634f, window, chunk, sink, db, n_x, status, cap_raw, lse);
        else
            e = gfb_launch(attn_prefill_tc_kernel<64>, dim3((unsigned)blocks), dim3(320), smem, stream, mq, mk, mv, (__nv_bfloat16*)out,
                           page_table, max_pages, n_pages, b, H, G, scale * 1.4426950408889634f, window, chunk, sink, db, n_x, status, cap_raw, lse);
    }
    if (gfb_check(e, "gfb_attn_prefill_tc")) return 1;
    if (keep_first > 0) {
        const dim3 grid((unsigned)(((long)n_tokens * H + 3) / 4));
        if (d == 128)
            e = gfb_launch(attn_kept_merge_kernel<128>, grid, dim3(128), 0, stream, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, (const float*)lse,
                           (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, page_table, max_pages, n_pages, b, H, G, scale, softcap,
                           window, keep_first, status);
        else
            e = gfb_launch(attn_kept_merge_kernel<64>, grid, dim3(128), 0, stream, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, (const float*)lse,
                           (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, page_table, max_pages, n_pages, b, H, G, scale, softcap,
                           window, keep_first, status);
        return gfb_check(e, "gfb_attn_prefill_tc (kept first positions)");
    }
    return 0;
}

// Prompts against a shared latent (the arguments are gfb_latent_attention's): q bfloat16 [T, H, R + 64], out bfloat16 [T, H * R], cached rows of
// R + 64 numbers in pages of 64, R = 128, 256, 384 or 512, scale > 0; everything 16-byte aligned.
GFB_API int gfb_latent_prefill_tc(const void* q, void* out, void* k_pool, const int* page_table, int max_pages, int page_size, int n_pages,
                                  const int* cu_seqlens, const int* tok_seq, const int* slots, const int* lengths, int n_seqs, int n_tokens, int H,
                                  int Dk, int R, float scale, int window, const float* sink, int* status, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (page_size != PAGE || R < 128 || R > 512 || R % 128 || Dk != R + 64 || !(scale > 0.f) || H < 1)
        return gfb_fail("gfb_latent_prefill_tc: rows of %d with %d value columns in pages of %d, scale %f", Dk, R, page_size, scale);
    if ((((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool) & 15) != 0) return gfb_fail("gfb_latent_prefill_tc: operands must be 16-byte aligned");
    if ((long long)n_pages * PAGE > 2147483647LL || (long long)n_tokens * H + ROWS > 2147483647LL)
        return gfb_fail("gfb_latent_prefill_tc: %d pages or %d x %d rows do not fit the 32-bit row coordinate of a tensor map", n_pages, n_tokens, H);
    EncodeTiledFn enc = encode_fn();
    if (!enc) return gfb_fail("gfb_latent_prefill_tc: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap mq, mk;
    for (int i = 0; i < 2; i++) {
        cuuint64_t dims[2] = {(cuuint64_t)Dk, i ? (cuuint64_t)n_pages * PAGE : (cuuint64_t)n_tokens * H};
        cuuint64_t strides[1] = {(cuuint64_t)Dk * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)(i ? LK : ROWS)};
        cuuint32_t es[2] = {1, 1};
        CUresult r = enc(i ? &mk : &mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, i ? k_pool : const_cast<void*>(q), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return gfb_fail("gfb_latent_prefill_tc: tensor map refused (%d)", (int)r);
    }
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    const int hc = R / 128;
    const size_t smem = 1024 + (size_t)(hc + 1) * QPIECE_BYTES + 2 * (size_t)(2 * hc + 1) * PIECE_BYTES + sizeof(LatBars);
    cudaError_t e = cudaFuncSetAttribute(latent_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gfb_fail("gfb_latent_prefill_tc: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
    const long n_x = ((long)n_tokens * H + ROWS - 1) / ROWS + n_seqs;          // an upper bound of the tiles; surplus blocks find no work
    if (2 * n_x > 2147483647L) return gfb_fail("gfb_latent_prefill_tc: %ld tiles", n_x);
    e = gfb_launch(latent_prefill_tc_kernel, dim3((unsigned)(2 * n_x)), dim3(LAT_THREADS), smem, stream, mq, mk, (const __nv_bfloat16*)q,
                   (__nv_bfloat16*)out, page_table, max_pages, n_pages, b, H, R, scale * 1.4426950408889634f, window, sink, (int)n_x, status);
    return gfb_check(e, "gfb_latent_prefill_tc");
}

// gfb_headwise_linear (whose arguments these are) on tcgen05: bfloat16, K a multiple of 64, N of 128, input and weight 16-byte aligned with
// ld_in, in_off and in_stride multiples of 8, output 8-byte aligned with ld_out, out_off and out_stride multiples of 4.
GFB_API int gfb_headwise_linear_tc(const void* in, int ld_in, int in_off, int in_stride, const void* w, void* out, int ld_out, int out_off,
                                   int out_stride, const void* gate, int ld_gate, int gate_off, int gate_cols, int n_tokens, int H, int K, int N,
                                   int* status, cudaStream_t stream) {
    if (n_tokens <= 0 || H <= 0 || N <= 0) return 0;
    if (K < 64 || K % 64 || N % 128 || ld_in % 8 || in_off % 8 || in_stride % 8 || ld_out % 4 || out_off % 4 || out_stride % 4 ||
        (((uintptr_t)in | (uintptr_t)w) & 15) || ((uintptr_t)out & 7))
        return gfb_fail("gfb_headwise_linear_tc: %d -> %d per head, rows of %d and %d, or pointers that are not aligned", K, N, ld_in, ld_out);
    if (H > 65535 || N / 128 > 65535 || (long long)H * K > 2147483647LL) return gfb_fail("gfb_headwise_linear_tc: %d heads of %d x %d exceed the grid limit", H, K, N);
    EncodeTiledFn enc = encode_fn();
    if (!enc) return gfb_fail("gfb_headwise_linear_tc: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap ma, mw;
    for (int i = 0; i < 2; i++) {
        cuuint64_t dims[2] = {i ? (cuuint64_t)N : (cuuint64_t)ld_in, i ? (cuuint64_t)H * K : (cuuint64_t)n_tokens};
        cuuint64_t strides[1] = {dims[0] * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)(i ? 64 : ROWS)};
        cuuint32_t es[2] = {1, 1};
        CUresult r = enc(i ? &mw : &ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(i ? w : in), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return gfb_fail("gfb_headwise_linear_tc: tensor map refused (%d)", (int)r);
    }
    cudaError_t e = cudaFuncSetAttribute(headwise_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HW_SMEM);
    if (e != cudaSuccess) return gfb_fail("gfb_headwise_linear_tc: %u bytes of shared memory refused: %s", HW_SMEM, cudaGetErrorString(e));
    e = gfb_launch(headwise_tc_kernel, dim3((n_tokens + ROWS - 1) / ROWS, H, N / 128), dim3(192), HW_SMEM, stream, ma, mw, in_off, in_stride,
                   (__nv_bfloat16*)out, ld_out, out_off, out_stride, (const __nv_bfloat16*)gate, ld_gate, gate_off, gate_cols, n_tokens, K, N, status);
    return gfb_check(e, "gfb_headwise_linear_tc");
}

// Prompts with every head's keys and values expanded (head and value size 128, 64 rotated numbers, rank R a multiple of 64).  proj bfloat16 [T, ld]:
// at q_off H heads of 192 query numbers of which the first 128 are read, at gate_off H gates (gate_per_head) or H * 128; q_rot [T, H, 64]: the
// rotated query parts; wuk [H, 128, R], wuv [H, R, 128]; v_scale float32 [2][H * 128]: powers of two and
// their reciprocals, by which the values stay within float16; keys, values [H, n_seqs * cap, 128]: scratch, cap a multiple of 128 that no sequence's length
// exceeds; out [T, H * 128].  The cache holds the new tokens' rows already.  Everything 16-byte aligned, ld, q_off and gate_off multiples of 8.
GFB_API int gfb_latent_expanded(const void* proj, int ld, int q_off, int gate_off, int gate_per_head, const void* q_rot, const void* wuk, const void* wuv,
                                const float* v_scale, void* keys, void* values, void* out, void* k_pool, const int* page_table, int max_pages, int page_size, int n_pages,
                                const int* cu_seqlens, const int* tok_seq, const int* slots, const int* lengths, int n_seqs, int n_tokens, int H, int R,
                                int cap, float scale, int window, const float* sink, int* status, cudaStream_t stream) {
    if (n_tokens <= 0 || H <= 0) return 0;
    if (page_size != PAGE || R < 64 || R % 64 || cap < KEYS || cap % KEYS || !(scale > 0.f) || ld % 8 || q_off % 8 || gate_off % 8)
        return gfb_fail("gfb_latent_expanded: rank %d, pages of %d, rows of %d, scale %f", R, page_size, ld, scale);
    if (((uintptr_t)proj | (uintptr_t)q_rot | (uintptr_t)wuk | (uintptr_t)wuv | (uintptr_t)v_scale | (uintptr_t)keys | (uintptr_t)values | (uintptr_t)out | (uintptr_t)k_pool) & 15)
        return gfb_fail("gfb_latent_expanded: operands must be 16-byte aligned");
    const long long rows = (long long)n_seqs * cap, n_x = ((long long)n_tokens + 2 * ROWS - 1) / (2 * ROWS) + n_seqs;   // an upper bound of the tiles
    if ((long long)n_pages * PAGE > 2147483647LL || rows * H > 2147483647LL || (long long)H * R > 2147483647LL || n_x * H > 2147483647LL)
        return gfb_fail("gfb_latent_expanded: %d pages, %lld rows of %d heads do not fit the 32-bit row coordinate of a tensor map", n_pages, rows, H);
    EncodeTiledFn enc = encode_fn();
    if (!enc) return gfb_fail("gfb_latent_expanded: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap maps[7];
    const struct { const void* p; long long cols, rows; int box; } what[7] = {
        {k_pool, R + 64, (long long)n_pages * PAGE, PAGE}, {wuk, R, (long long)H * D, D}, {wuv, D, (long long)H * R, 64}, {proj, ld, n_tokens, ROWS},
        {q_rot, (long long)H * 64, n_tokens, ROWS}, {keys, D, rows * H, KEYS}, {values, D, rows * H, 64}};
    for (int i = 0; i < 7; i++) {
        cuuint64_t dims[2] = {(cuuint64_t)what[i].cols, (cuuint64_t)what[i].rows};
        cuuint64_t strides[1] = {dims[0] * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)what[i].box};
        cuuint32_t es[2] = {1, 1};
        CUresult r = enc(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(what[i].p), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return gfb_fail("gfb_latent_expanded: tensor map %d refused (%d)", i, (int)r);
    }
    GfbBatch b{cu_seqlens, tok_seq, slots, lengths, n_seqs, n_tokens};
    cudaError_t e = cudaFuncSetAttribute(latent_expand_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LE_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(latent_heads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LH_SMEM);
    if (e != cudaSuccess) return gfb_fail("gfb_latent_expanded: %u and %u bytes of shared memory refused: %s", LE_SMEM, LH_SMEM, cudaGetErrorString(e));
    e = gfb_launch(latent_expand_kernel, dim3((unsigned)(rows / KEYS * H)), dim3(192), LE_SMEM, stream, maps[0], maps[1], maps[2], (__nv_bfloat16*)keys,
                   (__half*)values, v_scale, page_table, max_pages, n_pages, b, H, R, cap, window, status);
    if (gfb_check(e, "gfb_latent_expanded (keys and values)")) return 1;
    e = gfb_launch(latent_heads_kernel, dim3((unsigned)(n_x * H)), dim3(LH_THREADS), LH_SMEM, stream, maps[3], maps[4], maps[5], maps[0], maps[6], q_off,
                   (__nv_bfloat16*)out, v_scale + (size_t)H * D, (const __nv_bfloat16*)proj, ld, gate_off, gate_per_head, page_table, max_pages, n_pages, b, H, R, cap,
                   scale * 1.4426950408889634f, window, sink, (int)n_x, status);
    return gfb_check(e, "gfb_latent_expanded");
}
