// The float32 matrix product on the 5th-generation tensor cores:
//   out[M,N] = x[M,K] . W[N,K]^T                       (mode 0; mode 3 with xIELU on the sums)
//   out[M,N] = silu(x . Wgate^T) * (x . Wup^T)          (mode 2, W = [gate; up], N rows each; the other gates as in gemm.cu)
// A float32 number is the sum of three bfloat16 numbers (8 + 8 + 8 significant bits, each rounded to nearest, the
// remainders exact), so x . w is the sum of nine exact bfloat16 products; the six largest are taken (the three left out
// are below 2^-26 of |x w|). The second and third piece are kept 2^8 and 2^16 times as large, so that they do not fall under
// bfloat16's range before the number itself does (without, the error of numbers below 2^-110 grew to 2e-3 at 2^-126; now only
// subnormal numbers below 2^-133, whose first piece is 0, meet the other operand's first 8 to 16 bits alone); the
// accumulator then holds 2^16 times the sums of the smallest products, 2^8 times the next ones', and the mma that goes on
// to larger ones scales it down (scale-input-d). What limits the result is then the accumulator of the tensor cores, so it never holds more
// than 64 columns of K: within such a chunk the small products go first and the large ones last (four additions at full
// size), and the chunk's sums are drained from tensor memory and added up in float32 registers, in order. The error
// against float64 (2-norm, relative) is 0.8e-7 at K = 64, 1.1e-7 at 2,560 and 1.3e-7 at 9,728, where one float32 FMA chain over K
// (sgemm) has 1.4e-7, 9.1e-7 and 17.7e-7.
//
// Summation order: K in S groups of whole chunks, a group's chunks in order, then the groups in order. S depends on
// (N, K) alone, and nothing else of the order on the number of rows: a row's result does not depend on the rows beside it.
// A unit of several groups keeps their sum in tensor memory where there is room for it (544 rows, 2,560 outputs of 4,096: 97 us when
// every group was added into the output); else it adds each into the output.
// Where a unit of work holds one group (split) the groups leave as partial sums [S][M][N] for the consumer to add
// up in the same order; where it holds all of them (few units otherwise) it adds group after group into ``out`` itself.
//
// What bounds it: few rows: the weights' bytes from HBM while all SMs have a unit, then the chunks of the units left (about 1,150
// clocks each, whatever their height); many rows: the six products, one sixth of the bfloat16 rate, under the power cap.
// Roles of a block (one per SM, persistent over units), in two forms: tiles of more than 32 rows of x, and FEW:
//   convert (8 warps; FEW 16 in two groups that take chunks in turn): two threads take row r of a stage's weights (up to 128 rows x
//               64 columns, float32, TMA with 128-byte swizzle), 32 columns each, and write its three bfloat16 pieces into tensor
//               memory, where the mma reads its A operand from (96 columns a buffer, 2 to 4 buffers). In shared memory the pieces
//               would cost 48 KB a stage written, and the mma 8 instead of 4 KB read per 128 x 128 x 16 product. One group alone
//               takes 1,250 clocks a chunk with loads, arithmetic and stores one after the other.
//   drain (8 warps, two threads a row, half of the columns each; FEW 4, one thread a row): adds up the accumulators in turn; epilogue.
//   a warp for the TMA of the weights, one for x, two that issue tcgen05.mma: they take chunks in turn, so that the three waits of a
//               chunk (250 to 350 clocks together) run beside the mma of the other one's.
//   x: FEW and at most 4 rows: the warp loads them as float32 and takes them apart itself, two chunks ahead; else TMA of the pieces
//               ([3][M][Kp] bfloat16, made by split_rows before: as the B operand they come ready from shared memory).
// Measured in a graph, dependent launches, weights not in the L2 (2,560 wide layers of 9,728; one converting group, one mma warp,
// descriptors built at each mma and split_rows in front of every product -> this kernel). One row: q/k/v 14.9 -> 13.0 us, output
// projection 12.0 -> 10.2, gated 57.8 -> 50.9, down 20.2 -> 18.6 (the weights' bytes take 9.6, 6.4, 30.5, 15.2), a head of 50,000
// 87 -> 82 (6.2 TB/s). 544 rows: 113 -> 86, 100 -> 63, 362 -> 298, 167 -> 156 (the sums kept in tensor memory took 99 -> 86 and 71 -> 63
// of that). The gated product's tensor pipe is 64 % busy at 544 rows; at one row 13 %, and its SMs 67 % of the time (203 units in two
// waves).
// Infinities, NaN and numbers beyond bfloat16's largest: a piece times a zero piece is NaN where the product is not. A
// thread that finds a sum that is not finite works that one out again by plain FMA from x and W.
#include <cuda.h>

#include "common.cuh"

namespace {

constexpr int BK = 64, ROWS = 128, MAX_NT = 128, MAX_STAGES = 12, MAX_BUFS = 4;
constexpr int A_COLS = 96;
constexpr int DIRECT_ROWS = 4;                    // up to so many rows of x are taken apart by the product itself
constexpr int EX_BYTES = 2 * 32 * 64 * 4, FEW_NT = 32;   // up to FEW_NT rows a tile: the kernel's form for few rows
#ifndef DK_WAIT_CYCLES
#define DK_WAIT_CYCLES 2000000000LL               // about a second: a wait this long has failed
#endif
#ifdef DK_TEST_STALL
// Test build only: with the flag set no weights are requested, so the waits of all other roles run out (after DK_WAIT_CYCLES,
// which such a build makes short): a code in *err, tensor memory given back, the kernel returns.
__device__ int dk_stall_flag;
DK_EXPORT int dk_test_stall(int on) { return (int)cudaMemcpyToSymbol(dk_stall_flag, &on, sizeof(int)); }
#define DK_STALLED (dk_stall_flag != 0)
#else
#define DK_STALLED false
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (clock64() - t0 > DK_WAIT_CYCLES) return false;
    }
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                     smem_u32(dst)),
                 "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(
            smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy)
        : "memory");
}
// K-major operand, 128-byte swizzle, rows 128 bytes apart, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d),
                 "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}
// The same onto the accumulator times 2^-8.
__device__ __forceinline__ void umma_ts_down8(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, 1, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%4, %4, %4, %4}, p, 8; }" ::"r"(d),
        "r"(a_tmem), "l"(b), "r"(idesc), "r"(0)
        : "memory");
}
// One lane of a converged warp. The compiler keeps the operands of an mma issued under it in uniform registers; under
// ``lane == 0`` it moves every one of them there first, 80 clocks an mma instead of 50 (the head's product of one row: 601 us
// instead of 343).
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// What a pair (two float32 in one register pair) has left beside its rounding to bfloat16, times 2^8; exact.
__device__ __forceinline__ void remainder_up8(uint64_t& pair, uint32_t rounded) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(rounded << 16), "r"(rounded & 0xffff0000u));
    asm("sub.rn.f32x2 %0, %0, %1;" : "+l"(pair) : "l"(r));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(pair) : "l"(0x4380000043800000ull));
}
__device__ __forceinline__ uint32_t round_pair(uint64_t pair) {
    uint32_t lo, hi, out;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(pair));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return out;
}
// The three bfloat16 pieces of a and b, packed in pairs (a in the low half): a = hi + mid / 2^8 + lo / 2^16. Two numbers an
// instruction: with one at a time two sequences generating 12 tokens took 71.5 ms instead of 66.2 unscaled; a gated product of one
// row takes 57.2 us (56.0 unscaled).
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    uint64_t pair;
    asm("mov.b64 %0, {%1, %2};" : "=l"(pair) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
    hi = round_pair(pair);
    remainder_up8(pair, hi);
    mid = round_pair(pair);
    remainder_up8(pair, mid);
    lo = round_pair(pair);
}

// x [M][K] float32 -> pieces [3][M][Kp] bfloat16, Kp = K rounded up to 8, zeros behind K. A thread takes 8 columns.
// Bound by its bytes: 10 a number. It stands directly before the product, so it triggers its launch before its own wait.
__global__ void split_rows_kernel(const float* x, bf16* out, int M, int K, int Kp) {
    pdl_launch_dependents();
    pdl_wait();
    const long long per_row = Kp / 8, i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= per_row * M) return;
    const long long row = i / per_row;
    const int k = (int)(i - row * per_row) * 8;
    const float* p = x + row * K + k;
    float v[8];
    if (K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        const float4 b = k + 4 < K ? *reinterpret_cast<const float4*>(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = k + e < K ? p[e] : 0.f;
    }
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) split_pair(v[2 * e], v[2 * e + 1], h[e], m[e], l[e]);
    const size_t plane = (size_t)M * Kp, at = (size_t)row * Kp + k;
    *reinterpret_cast<uint4*>(out + at) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(out + plane + at) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4*>(out + 2 * plane + at) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The gates of gemm.cu's sgemm: 0 SiLU, 1 the tanh form of GELU, 2 the clamped gate with its limit.
__device__ __forceinline__ float gated(float v, float u, float act_pos, float act_neg) {
    if (act_pos > 1.5f) {
        const float g = fminf(v, act_neg), c = fminf(fmaxf(u, -act_neg), act_neg);
        return g / (1.f + expf(-1.702f * g)) * (c + 1.f);
    }
    const float a = act_pos > 0.5f ? 1.5957691216057308f * v * fmaf(0.044715f * v, v, 1.f) : v;
    return v / (1.f + expf(-a)) * u;
}

struct Product {
    const float *x, *W;
    float *out, *parts;          // parts: [S][M][N] where a unit holds one group
    int M, N, K, Kp;
    int tile_n, tiles, nt, row_tiles, groups, group_len, split;   // tile_n: outputs a tile (weight rows; mode 2: half of them)
    int w_stages, x_stages, w_box, bufs, kept;   // w_box: bytes between boxes of weights in shared memory; bufs: pieces of W, accumulators
    // kept: the sums of the groups so far stay in tensor memory, behind the buffers, until the last group
    float act_pos, act_neg;
};

// Plain FMA over one row and the same groups of K: for sums that are not finite.
__device__ __noinline__ float plain_sum(const float* x, const float* w, int K, int k0, int k1, int group) {
    float total = 0.f;
    for (int k = k0; k < k1; k += group) {
        float s = 0.f;
        for (int i = k; i < min(min(k + group, k1), K); i++) {
            s = fmaf(x[i], w[i], s);
            if (s != s) return s;            // nothing makes a number of it again
        }
        total = k == k0 ? s : total + s;
    }
    return total;
}

// FEW (tiles of at most FEW_NT rows): 16 converting warps in two groups that take chunks in turn, and 4 draining ones; else 8 and 8.
template <bool FEW>
struct Warps {
    static constexpr int CONVERT = FEW ? 16 : 8, DRAIN = FEW ? 4 : 8, LOADER = CONVERT + DRAIN, THREADS = (LOADER + 4) * 32;
};

template <int MODE, bool FEW>
__global__ void __launch_bounds__(Warps<FEW>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ Product p, int* err) {
    constexpr int CONVERT = Warps<FEW>::CONVERT, DRAIN = Warps<FEW>::DRAIN, LOADER = Warps<FEW>::LOADER;
    constexpr int HALF_COLS = FEW ? FEW_NT : MAX_NT / 2;      // columns a draining thread adds up: all, or half of them
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int x_piece = p.nt * 128, x_stage = 3 * x_piece;
    const int w_half = (MODE == 2 ? 2 : 1) * p.w_box, w_stage = 2 * w_half;   // rows x 32 floats (mode 2: gate rows, up rows), twice
    uint8_t* smem_w = smem;
    uint8_t* smem_x = smem_w + p.w_stages * w_stage;
    float* exchange = reinterpret_cast<float*>(smem_x + p.x_stages * x_stage);          // mode 2: [2][32][64] up sums
    uint64_t* w_full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(exchange) + EX_BYTES);
    uint64_t *w_empty = w_full + MAX_STAGES, *x_full = w_empty + MAX_STAGES, *x_empty = x_full + MAX_STAGES;
    uint64_t *a_full = x_empty + MAX_STAGES, *a_empty = a_full + MAX_BUFS, *acc_full = a_empty + MAX_BUFS, *acc_empty = acc_full + MAX_BUFS;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + MAX_BUFS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_blocks = (p.K + BK - 1) / BK;
    const int slices = p.split ? p.groups : 1, per = p.split ? p.group_len : k_blocks;
    const int units = p.tiles * slices * p.row_tiles;
    // unit -> (tile, slice, rows of x); rows run fastest, so that the blocks at work at one time share weights
#define UNIT(u)                                                                                              \
    const int rt = (u) % p.row_tiles, ts = (u) / p.row_tiles, slice = ts % slices, n0 = ts / slices * p.tile_n; \
    const int m0 = rt * p.nt, kb0 = slice * per, kb1 = min(k_blocks, kb0 + per);                             \
    (void)m0, (void)n0, (void)kb0, (void)kb1

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; s++) {
            mbar_init(&w_full[s], 1), mbar_init(&w_empty[s], 8);
            mbar_init(&x_full[s], 1), mbar_init(&x_empty[s], 1);
        }
        for (int b = 0; b < MAX_BUFS; b++) {
            mbar_init(&a_full[b], 8), mbar_init(&a_empty[b], 1);
            mbar_init(&acc_full[b], 1), mbar_init(&acc_empty[b], DRAIN);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == LOADER + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, a_base = tmem + p.bufs * p.nt;   // accumulators of nt columns, then the pieces of W

    if (warp == LOADER) {
        if (lane == 0) {  // ------------------------------------ weights (no kernel of a step writes them)
            const uint64_t stream_once = l2_evict_first();
            const uint32_t tx = (MODE == 2 ? 2 : 1) * p.tile_n * 256;
            int s = 0, it = 0;
            uint32_t round = 0;
            bool ok = !DK_STALLED;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                UNIT(u);
                for (int kb = kb0; kb < kb1; kb++, it++, s = s + 1 == p.w_stages ? 0 : s + 1, round ^= (s == 0)) {
                    if (it >= p.w_stages && !mbar_wait(&w_empty[s], round ^ 1)) {
                        atomicExch(err, 11);
                        ok = false;
                        break;
                    }
                    uint8_t* stage = smem_w + s * w_stage;
                    mbar_expect_tx(&w_full[s], tx);
                    for (int h = 0; h < 2; h++) {
                        if (p.row_tiles == 1) {
                            tma_load_2d(stage + h * w_half, &map_w, kb * BK + 32 * h, n0, &w_full[s], stream_once);
                            if (MODE == 2)
                                tma_load_2d(stage + h * w_half + p.w_box, &map_w, kb * BK + 32 * h, p.N + n0, &w_full[s], stream_once);
                        } else {
                            tma_load_2d(stage + h * w_half, &map_w, kb * BK + 32 * h, n0, &w_full[s]);
                            if (MODE == 2)
                                tma_load_2d(stage + h * w_half + p.w_box, &map_w, kb * BK + 32 * h, p.N + n0, &w_full[s]);
                        }
                    }
                }
            }
        }
    } else if (FEW && warp == LOADER + 2 && p.M <= DIRECT_ROWS) {  // ----------- few rows of x: taken apart here
        pdl_wait();
        if (lane == 0) pdl_launch_dependents();
        const bool aligned = (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
        const int row = lane >> 3;
        int s = 0, it = 0;
        uint32_t round = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            UNIT(u);
            float va[2][8], vb[2][8];                         // two chunks at a time, the next two on their way
            auto load = [&](float (&v)[2][8], int kb) {
#pragma unroll
                for (int j = 0; j < 2; j++)                   // a lane takes 8 columns of row lane / 8
#pragma unroll
                    for (int e = 0; e < 8; e += 4) {          // K is a multiple of 4; zeros behind it
                        const int k = (kb + j) * BK + (lane & 7) * 8 + e;
                        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (row < p.M && kb + j < kb1 && k < p.K) {
                            const float* src = p.x + (size_t)row * p.K + k;
                            if (aligned) f = *reinterpret_cast<const float4*>(src);
                            else f = make_float4(src[0], src[1], src[2], src[3]);
                        }
                        v[j][e] = f.x, v[j][e + 1] = f.y, v[j][e + 2] = f.z, v[j][e + 3] = f.w;
                    }
            };
            auto put = [&](const float (&v)[2][8], int kb) {
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (kb + j >= kb1 || !ok) continue;
                    if (it >= p.x_stages) ok = __all_sync(0xffffffffu, mbar_wait(&x_empty[s], round ^ 1));
                    if (!ok) {
                        atomicExch(err, 12);
                        continue;
                    }
                    if (row < p.M) {                          // rows behind M hold anything: their sums are never stored
                        uint32_t h[4], m[4], l[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) split_pair(v[j][2 * e], v[j][2 * e + 1], h[e], m[e], l[e]);
                        uint8_t* to = smem_x + s * x_stage + row * 128 + (((lane & 7) ^ (row & 7)) << 4);
                        *reinterpret_cast<uint4*>(to) = make_uint4(h[0], h[1], h[2], h[3]);
                        *reinterpret_cast<uint4*>(to + x_piece) = make_uint4(m[0], m[1], m[2], m[3]);
                        *reinterpret_cast<uint4*>(to + 2 * x_piece) = make_uint4(l[0], l[1], l[2], l[3]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&x_full[s]);
                    it++;
                    if (++s == p.x_stages) s = 0, round ^= 1;
                }
            };
            load(va, kb0);
            for (int kb = kb0; kb < kb1 && ok; kb += 4) {
                load(vb, kb + 2);
                put(va, kb);
                load(va, kb + 4);
                put(vb, kb + 2);
            }
        }
    } else if (warp == LOADER + 2) {
        if (lane == 0) {  // ------------------------------------ the pieces of x
            pdl_wait();
            pdl_launch_dependents();
            int s = 0, it = 0;
            uint32_t round = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                UNIT(u);
                for (int kb = kb0; kb < kb1; kb++, it++, s = s + 1 == p.x_stages ? 0 : s + 1, round ^= (s == 0)) {
                    if (it >= p.x_stages && !mbar_wait(&x_empty[s], round ^ 1)) {
                        atomicExch(err, 12);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&x_full[s], x_stage);
                    for (int q = 0; q < 3; q++)
                        tma_load_2d(smem_x + s * x_stage + q * x_piece, &map_x, kb * BK, q * p.M + m0, &x_full[s]);
                }
            }
        }
    } else if (warp == LOADER + 1 || warp == LOADER + 3) {
        // ------------------------ mma: two warps take chunks in turn, so that the waits of one run beside the mma of the other
        const int mine = warp == LOADER + 3;
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.nt >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
        int xs = 0, it = 0, b = 0;
        uint32_t xround = 0, phase = 0;
        // a piece further on in shared memory is an addition to the low half of the descriptor (in units of 16 bytes)
        const uint64_t x_desc = umma_desc(smem_u32(smem_x));
        const uint32_t piece = (uint32_t)x_piece >> 4;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            UNIT(u);
            for (int kb = kb0; kb < kb1; kb++, it++, xs = xs + 1 == p.x_stages ? 0 : xs + 1, xround ^= (xs == 0),
                     b = b + 1 == p.bufs ? 0 : b + 1, phase ^= (b == 0)) {
                if ((it & 1) != mine) continue;
                ok = mbar_wait(&x_full[xs], xround) && mbar_wait(&a_full[b], phase) &&
                     (it < p.bufs || mbar_wait(&acc_empty[b], phase ^ 1));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    atomicExch(err, 13);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint32_t d = tmem + b * p.nt, a = a_base + b * A_COLS;
                    const uint64_t xb = x_desc + (uint32_t)(xs * 3) * piece, x_at[3] = {xb, xb + piece, xb + 2 * piece};
                    // (piece of W, piece of x), 0 the largest; the products grow from the first to the last, at 2^16, 2^8 and 1
                    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                    for (int q = 0; q < 6; q++)
#pragma unroll
                        for (int k = 0; k < BK / 16; k++) {
                            const uint32_t ak = a + PA[q] * 32 + k * 8;
                            const uint64_t bk = x_at[PB[q]] + 2 * k;
                            if (k == 0 && q > 0 && PA[q] + PB[q] < PA[q - 1] + PB[q - 1]) umma_ts_down8(d, ak, bk, idesc);
                            else umma_ts(d, ak, bk, idesc, (q | k) != 0);
                        }
                    umma_commit(&x_empty[xs]);
                    umma_commit(&a_empty[b]);
                    umma_commit(&acc_full[b]);
                }
                __syncwarp();
            }
        }
    } else if (warp < CONVERT) {  // -------------------------------------------------- convert
        const int r = threadIdx.x & 127, h = (warp >> 2) & 1, group = warp >> 3;
        const uint32_t to = a_base + h * 16 + ((uint32_t)((warp & 3) * 32) << 16);
        // where row r of a half stage lies; lanes without a row of the tile read the first one's, and their sums are never stored
        const int in_tile = MODE == 2 ? r & 63 : r;
        const int place = in_tile < p.tile_n ? (MODE == 2 ? (r >> 6) * p.w_box : 0) + in_tile * 128 : 0, turn = (place >> 7) & 7;
        const bool idle = (MODE == 2 ? (warp & 1) * 32 : (warp & 3) * 32) >= p.tile_n;     // no lane of the warp has one
        int ws = 0, it = 0, b = 0;
        uint32_t wround = 0, phase = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            UNIT(u);
            for (int kb = kb0; kb < kb1; kb++, it++, ws = ws + 1 == p.w_stages ? 0 : ws + 1, wround ^= (ws == 0),
                     b = b + 1 == p.bufs ? 0 : b + 1, phase ^= (b == 0)) {
                if (FEW && (it & 1) != group) continue;
                ok = mbar_wait(&w_full[ws], wround);
                if (ok && it >= p.bufs) ok = mbar_wait(&a_empty[b], phase ^ 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    atomicExch(err, 14);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!idle) {
                    const uint8_t* row = smem_w + ws * w_stage + h * w_half + place;
                    uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float4 v = *reinterpret_cast<const float4*>(row + ((c ^ turn) << 4));
                        split_pair(v.x, v.y, hi[2 * c], mid[2 * c], lo[2 * c]);
                        split_pair(v.z, v.w, hi[2 * c + 1], mid[2 * c + 1], lo[2 * c + 1]);
                    }
                    tmem_st16(to + b * A_COLS, hi);
                    tmem_st16(to + b * A_COLS + 32, mid);
                    tmem_st16(to + b * A_COLS + 64, lo);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_empty[ws]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[b]);
            }
        }
    } else {  // ---------------------------------------------------------------- drain and epilogue
        const int q = warp & 3, r = q * 32 + lane;
        const int half = FEW ? 0 : (warp - CONVERT) >> 2, split_at = FEW ? p.nt : (p.nt / 2 + 15) / 16 * 16;      // columns [0, split_at), [split_at, nt)
        const int j0 = half * split_at, cols = half ? p.nt - split_at : split_at, pieces = cols / 16;
        float* ex = exchange + half * 32 * 64;
        const bool is_up = MODE == 2 && q >= 2;
        const int local = MODE == 2 ? (r & 63) : r;
        pdl_wait();                       // nothing is stored before the kernels before this one are done
        int b = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            UNIT(u);
            const int n = n0 + local;
            const bool mine = local < p.tile_n && n < p.N;
            float* out = p.split ? p.parts + (size_t)slice * p.M * p.N : p.out;
            unsigned long long bad = 0;          // this thread's columns with a sum that is not finite
            for (int g0 = kb0; g0 < kb1; g0 += p.group_len) {
                float tot[HALF_COLS];
#pragma unroll
                for (int j = 0; j < HALF_COLS; j++) tot[j] = 0.f;
                const int g1 = min(kb1, g0 + p.group_len);
                for (int kb = g0; kb < g1; kb++, b = b + 1 == p.bufs ? 0 : b + 1, phase ^= (b == 0)) {
                    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], phase));
                    if (!ok) {             // go on without waiting: the warps meet at barriers below, and the sums are not valid
                        atomicExch(err, 15);
                        continue;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t acc = tmem + b * p.nt + j0 + ((uint32_t)(q * 32) << 16);
#pragma unroll
                    for (int c = 0; c < HALF_COLS / 16; c++)
                        if (c < pieces) {
                            uint32_t v[16];
                            tmem_ld16(acc + c * 16, v);
#pragma unroll
                            for (int i = 0; i < 16; i++) tot[c * 16 + i] += __uint_as_float(v[i]);
                        }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[b]);
                }
                // ---- the group's sums leave, or join those of the groups before it
                const bool last = g1 == kb1;
                if (MODE != 2 && p.kept) {
                    const uint32_t sums = a_base + p.bufs * A_COLS + j0 + ((uint32_t)(q * 32) << 16);
#pragma unroll
                    for (int c = 0; c < HALF_COLS / 16; c++)
                        if (c < pieces) {
                            uint32_t v[16];
                            if (g0 != kb0) {
                                tmem_ld16(sums + c * 16, v);
#pragma unroll
                                for (int i = 0; i < 16; i++) tot[c * 16 + i] = __uint_as_float(v[i]) + tot[c * 16 + i];
                            }
                            if (!last) {
#pragma unroll
                                for (int i = 0; i < 16; i++) v[i] = __float_as_uint(tot[c * 16 + i]);
                                tmem_st16(sums + c * 16, v);
                            }
                        }
                    if (!last) {
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        continue;
                    }
                }
                if (MODE == 2) {           // one group; gate sums in the warps of lanes 0..63, up sums in the others
#pragma unroll
                    for (int c = 0; c < HALF_COLS; c += 32)
                        if (c < cols) {
                            if (is_up) {
#pragma unroll
                                for (int i = 0; i < 32; i++) ex[i * 64 + local] = tot[c + i];
                            }
                            asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                            if (!is_up) {
#pragma unroll
                                for (int i = 0; i < 32; i++) {
                                    const int m = m0 + j0 + c + i;
                                    const float up = ex[i * 64 + local];
                                    if (mine && c + i < cols && m < p.M) {
                                        if (!(fabsf(tot[c + i]) <= 3.402823466e38f && fabsf(up) <= 3.402823466e38f)) bad |= 1ull << (c + i);
                                        out[(size_t)m * p.N + n] = gated(tot[c + i], up, p.act_pos, p.act_neg);
                                    }
                                }
                            }
                            asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                        }
                } else if (mine) {
                    const bool first = g0 == kb0 || p.kept;
                    const int rows = min(cols, p.M - m0 - j0);
                    float* dst = out + (size_t)(m0 + j0) * p.N + n;
#pragma unroll
                    for (int c = 0; c < HALF_COLS; c += 8)
                        if (c < rows) {
                            if (!first) {
                                float before[8];
#pragma unroll
                                for (int i = 0; i < 8; i++) before[i] = c + i < rows ? dst[(size_t)(c + i) * p.N] : 0.f;
#pragma unroll
                                for (int i = 0; i < 8; i++) tot[c + i] = before[i] + tot[c + i];
                            }
#pragma unroll
                            for (int i = 0; i < 8; i++)
                                if (c + i < rows) {
                                    if (!(fabsf(tot[c + i]) <= 3.402823466e38f)) bad |= 1ull << (c + i);
                                    dst[(size_t)(c + i) * p.N] = MODE == 3 && last ? xielu_f(tot[c + i], p.act_pos, p.act_neg) : tot[c + i];
                                }
                        }
                }
            }
            if (bad != 0 && ok) {          // those outputs again, without the pieces
                const int k0 = kb0 * BK, k1 = min(p.K, kb1 * BK), group = p.group_len * BK;
                for (int m = m0 + j0; m < min(p.M, m0 + j0 + cols); m++) {
                    if (!((bad >> (m - m0 - j0)) & 1)) continue;
                    const float v = plain_sum(p.x + (size_t)m * p.K, p.W + (size_t)n * p.K, p.K, k0, k1, group);
                    float o = v;
                    if (MODE == 2)
                        o = gated(v, plain_sum(p.x + (size_t)m * p.K, p.W + (size_t)(p.N + n) * p.K, p.K, k0, k1, group), p.act_pos, p.act_neg);
                    if (MODE == 3) o = xielu_f(v, p.act_pos, p.act_neg);
                    out[(size_t)m * p.N + n] = o;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == LOADER + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
#undef UNIT
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encoder() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiled)p;
    }
    return fn;
}

// Row-major matrix [rows, cols]: boxes of box_rows x 128 bytes, 128-byte swizzle, zero fill.
int make_map(CUtensorMap* map, CUtensorMapDataType type, int size, const void* base, long long rows, long long cols, int box_rows) {
    EncodeTiled enc = encoder();
    if (!enc) return (int)cudaErrorNotSupported;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * size};
    cuuint32_t box[2] = {(cuuint32_t)(128 / size), (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = enc(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <int MODE, bool FEW>
int launch_as(Product p, const bf16* pieces, int* err, cudaStream_t st) {
    const int x_stage = 3 * p.nt * 128;
    const size_t tail = EX_BYTES + (4 * MAX_STAGES + 4 * MAX_BUFS) * sizeof(uint64_t) + 16;
    const size_t budget = 227 * 1024 - tail - 1024;
    p.w_box = (p.tile_n + 7) / 8 * 1024;                      // 128 bytes a row, boxes at multiples of the swizzle's 1024
    const int w_stage = (MODE == 2 ? 4 : 2) * p.w_box;
    p.bufs = 512 / (p.nt + A_COLS) < MAX_BUFS ? 512 / (p.nt + A_COLS) : MAX_BUFS;
    p.kept = MODE != 2 && !p.split && p.groups > 1 && p.bufs * (p.nt + A_COLS) + p.nt <= 512;
    // a stage of x is free when its mma are done, a stage of W once it is converted (``bufs`` more wait in tensor memory)
    p.x_stages = p.nt > 64 ? 2 : 4;                           // even: see below
    p.w_stages = (int)((budget - (size_t)p.x_stages * x_stage) / w_stage);
    if (p.w_stages > MAX_STAGES) p.w_stages = MAX_STAGES;
    // Warps that take chunks in turn (mma; converting ones, FEW) need an even number of the stages that loads fill, which come in any
    // order: each then belongs to one of them. A warp that met a stage's barrier only every second time could take the phase before
    // for its own. (Buffers that warps fill or empty in order may be three.)
    if (FEW) p.w_stages &= ~1;
    if (p.w_stages < 1 || (FEW && p.bufs % 2 != 0)) return (int)cudaErrorInvalidValue;
    const size_t smem = 1024 + (size_t)p.w_stages * w_stage + (size_t)p.x_stages * x_stage + tail;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<MODE, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    CUtensorMap mx{}, mw;
    int rc = FEW && p.M <= DIRECT_ROWS ? 0 : make_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pieces, 3LL * p.M, p.Kp, p.nt);
    if (rc) return rc;
    rc = make_map(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p.W, MODE == 2 ? 2LL * p.N : p.N, p.K, p.tile_n);
    if (rc) return rc;
    const long long units = (long long)p.tiles * (p.split ? p.groups : 1) * p.row_tiles;
    if (units > (1LL << 30)) return (int)cudaErrorInvalidValue;
    return dk_launch(gemm_f32_tc_kernel<MODE, FEW>, dim3((unsigned)(units < sms ? units : sms)), dim3(Warps<FEW>::THREADS), smem, st, mx, mw, p, err);
}

template <int MODE>
int launch(const Product& p, const bf16* pieces, int* err, cudaStream_t st) {
    return p.nt <= FEW_NT ? launch_as<MODE, true>(p, pieces, err, st) : launch_as<MODE, false>(p, pieces, err, st);
}

}  // namespace

// x [M,K], W [N,K] (mode 2: [2N,K] = gate rows then up rows), out [M,N], all float32; K % 4 == 0, W on a 16-byte boundary.
// pieces: scratch of 3 * M * Kp bfloat16, Kp = K rounded up to a multiple of 8, on a 16-byte boundary (null with at most 4 rows
// in row tiles of at most 32). groups, group_len:
// K's chunks of 64 columns in ``groups`` groups of ``group_len`` (the last may be shorter, none empty; 1 in mode 2).
// parts: null, or [groups][M][N] (mode 0): the groups' sums, left for the consumer to add up. tile_n: outputs a tile, at
// most 128 (mode 2: 64). nt: rows of x a tile, a multiple of 16, at most 128. err: device int, receives a code if a bounded
// wait ran out. act_pos, act_neg: as in dk_sgemm.
DK_EXPORT int dk_gemm_f32_tc(const float* x, const float* W, float* out, void* pieces, int M, int N, int K, int mode, int groups,
                             int group_len, float* parts, int tile_n, int nt, int* err, float act_pos, float act_neg,
                             cudaStream_t st) {
    const int k_blocks = (K + BK - 1) / BK, Kp = (K + 7) / 8 * 8;
    if (M < 1 || N < 1 || K < 4 || K % 4 != 0 || err == nullptr || (pieces == nullptr && !(M <= DIRECT_ROWS && nt <= FEW_NT)) || (mode != 0 && mode != 2 && mode != 3))
        return (int)cudaErrorInvalidValue;
    if (((uintptr_t)W | (uintptr_t)pieces) % 16 != 0 || 3LL * M > (1LL << 30)) return (int)cudaErrorInvalidValue;
    if (groups < 1 || group_len < 1 || (long long)groups * group_len < k_blocks || (long long)(groups - 1) * group_len >= k_blocks ||
        (mode == 2 && groups != 1) || (parts != nullptr && mode != 0) || (parts == nullptr && out == nullptr))
        return (int)cudaErrorInvalidValue;
    if (tile_n < 1 || tile_n > (mode == 2 ? 64 : 128) || nt < 16 || nt > MAX_NT || nt % 16 != 0) return (int)cudaErrorInvalidValue;
    if (M > DIRECT_ROWS || nt > FEW_NT) {
        const long long threads = (long long)M * (Kp / 8);
        const int e = dk_launch(split_rows_kernel, dim3((unsigned)((threads + 127) / 128)), dim3(128), 0, st, x, (bf16*)pieces, M, K, Kp);
        if (e) return e;
    }
    Product p{};
    p.x = x, p.W = W, p.out = out, p.parts = parts, p.M = M, p.N = N, p.K = K, p.Kp = Kp;
    p.tile_n = tile_n, p.tiles = (N + tile_n - 1) / tile_n, p.nt = nt, p.row_tiles = (M + nt - 1) / nt;
    p.groups = groups, p.group_len = group_len, p.split = parts != nullptr;
    p.act_pos = act_pos, p.act_neg = act_neg;
    if (mode == 2) return launch<2>(p, (const bf16*)pieces, err, st);
    if (mode == 3) return launch<3>(p, (const bf16*)pieces, err, st);
    return launch<0>(p, (const bf16*)pieces, err, st);
}
