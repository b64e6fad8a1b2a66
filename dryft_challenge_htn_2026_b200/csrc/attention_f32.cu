// Causal grouped-query attention over the paged cache in float32 on the CUDA cores, for head sizes 64 and 128 and up to 16
// query heads a key/value head. Built per head size with -DHD=64 or -DHD=128; other sizes: attention_generic.cu.
//
// Formula (reference: engine/engine.py:148-164, engine/fused.py:301-343): query head h reads kv head h / (nh / nkv);
// score = q.k * scale; a query at position p sees keys j <= p (and j > p - window when a window is set); softmax; P.V.
//
// Order of the arithmetic, the same in both kernels, so that a row's result does not depend on the rows beside it nor on whether
// it came as part of a prompt or as a single token: a page of 64 keys at a time: scores (one FMA chain over the head), their
// maximum, weights against that maximum, their sum (a fixed tree), P.V (one FMA chain over the page); then the page is merged
// into what the pages before it gave (merge()).
//
//   prompts: a block takes 64 or 32 rows (rows / G queries of one sequence x the G query heads of one kv head) through its pages. Q, K,
//       V in shared memory (K's place takes P afterwards: 98 or 82 KB, two blocks an SM); S = Q.K^T with 4 x 4 (2 x 4) scores a
//       thread, P.V with 4 (2) rows x HD / 16 columns a thread; keys that every row of the tile sees go four at a time, only the few
//       behind them with a test a row. Bound by the chain load - scores - weights - P.V, whose shared-memory reads the two blocks of
//       an SM wait for: 18 us a page of 64 rows, 11.6 of 32, two blocks side by side (tiles of 32, 544 tokens: FMA pipe 37 %, issue
//       slots 54 %, 2.5 of the 4 stalled warps an issue on shared memory). The tiles with the most pages of all heads start first:
//       with the tiles of one head after those of another the last head's longest tiles came last. 32 heads of 128, that and tiles of
//       64 -> now: 100 tokens 31 -> 16 us, 300 70 -> 53, 544 156 -> 110 (124 in tiles of 64), 1,000 397 -> 264, 4,000 3,970 -> 3,640.
//   single tokens: a block a (sequence, kv head, page), the pages merged by a second kernel. 2 sequences of 100 tokens: 203 us with
//       a warp a row, whose keys follow one another at 2 us each -> 7.2 + 2.3 us.
#include "common.cuh"

namespace {

constexpr int THREADS = 256, LDK = HD + 4, LDP = DK_PAGE + 4, MAX_G = 16;
constexpr int CV = HD / 64;                               // float4 columns of P.V a thread

// A page's (maximum mp, sum lp) into the running (m, l): the factors of the old and of the page's values.
__device__ __forceinline__ void merge(float& m, float& l, float mp, float lp, float& a, float& b) {
    const float mn = fmaxf(m, mp);
    a = m == -INFINITY ? 0.f : expf(m - mn);
    b = expf(mp - mn);
    l = __fmaf_rn(l, a, __fmul_rn(lp, b));
    m = mn;
}
__device__ __forceinline__ float merged(float acc, float page, float a, float b) { return __fmaf_rn(acc, a, __fmul_rn(page, b)); }

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One page of one kv head, dense [64][HD], into rows of ld floats.
__device__ __forceinline__ void load_page(float* dst, int ld, const float* store, int page, int nkv, int kvh) {
    const float* src = store + kv_offset(page, nkv, kvh, 0, HD);
    for (int i = threadIdx.x; i < DK_PAGE * HD / 4; i += THREADS) copy16(dst + (i / (HD / 4)) * ld + (i % (HD / 4)) * 4, src + i * 4);
}

// s[i][j] += q[i] . k[tx + 16 j] over the head, one FMA chain each
template <int NI>
__device__ __forceinline__ void scores(float (&s)[NI][4], const float* const (&q)[NI], const float* k, int tx) {
#pragma unroll 4
    for (int d = 0; d < HD; d += 4) {
        float4 a[NI], b[4];
#pragma unroll
        for (int i = 0; i < NI; i++) a[i] = *reinterpret_cast<const float4*>(q[i] + d);
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4*>(k + (tx + 16 * j) * LDK + d);
#pragma unroll
        for (int i = 0; i < NI; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
            }
    }
}

// Scores of a row (a thread has keys tx + 16 j, its 16 neighbours the others) -> weights against the page's maximum; their
// maximum and sum in every lane of the 16.
__device__ __forceinline__ void weights(float (&s)[4], float scale, int key0, int lo, int pos, int tx, float& mp, float& lp) {
    mp = -INFINITY;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int key = key0 + tx + 16 * j;
        s[j] = key >= lo && key <= pos ? __fmul_rn(s[j], scale) : -INFINITY;
        mp = fmaxf(mp, s[j]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, o));
#pragma unroll
    for (int j = 0; j < 4; j++) {
        // -inf: a key out of sight, or one whose score is; in a page of none but those, -inf - mp would be NaN
        s[j] = s[j] == -INFINITY ? 0.f : expf(__fsub_rn(s[j], mp));
    }
    lp = __fadd_rn(__fadd_rn(__fadd_rn(s[0], s[1]), s[2]), s[3]);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) lp = __fadd_rn(lp, __shfl_xor_sync(0xffffffffu, lp, o));
}

template <int ROWS>
__global__ void __launch_bounds__(THREADS, 2)
prompt_kernel(const float* q, float* out, const float* k_store, const float* v_store, const int* tiles, const int* cu_q,
              const int* seq_pos0, const int* page_table, int pt_stride, int nh, int nkv, int window, float scale) {
    constexpr int NI = ROWS / 16;                           // rows a thread
    extern __shared__ __align__(16) float smem[];
    float *q_s = smem, *k_s = q_s + ROWS * HD, *p_s = k_s, *v_s = k_s + DK_PAGE * LDK;
    pdl_wait();
    pdl_launch_dependents();
    // kv heads run fastest: the tiles come with the most keys first, and those of all heads start first
    const int tile = blockIdx.x / nkv, kvh = blockIdx.x - tile * nkv, seq = tiles[2 * tile], q0 = tiles[2 * tile + 1];
    const int G = nh / nkv, flat0 = cu_q[seq] + q0, rows = min(ROWS / G, cu_q[seq + 1] - flat0) * G;
    const int pos0 = seq_pos0[seq] + q0, last = pos0 + rows / G - 1;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int* pt = page_table + (size_t)seq * pt_stride;
    for (int i = threadIdx.x; i < ROWS * (HD / 4); i += THREADS) {
        const int r = i / (HD / 4), c = (i % (HD / 4)) * 4;
        if (r < rows) copy16(q_s + r * HD + c, q + ((size_t)(flat0 + r / G) * nh + kvh * G + r % G) * HD + c);
    }
    const float* qr[NI];
    int pos[NI], lo[NI];
    float m[NI], l[NI], acc[NI][4 * CV];
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const int r = ty * NI + i;
        qr[i] = q_s + min(r, rows - 1) * HD;
        pos[i] = r < rows ? pos0 + r / G : -1;              // a row that is not there sees nothing
        lo[i] = window > 0 ? max(0, pos[i] - window + 1) : 0;
        m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * CV; c++) acc[i][c] = 0.f;
    }
    const int first_page = (window > 0 ? max(0, pos0 - window + 1) : 0) / DK_PAGE, last_page = last / DK_PAGE;
    for (int pg = first_page; pg <= last_page; pg++) {
        const int key0 = pg * DK_PAGE, page = pt[pg];
        load_page(k_s, LDK, k_store, page, nkv, kvh);
        load_page(v_s, HD, v_store, page, nkv, kvh);
        copy_wait();
        __syncthreads();
        float s[NI][4] = {}, a[NI], b[NI];
        scores<NI>(s, qr, k_s, tx);
        __syncthreads();                                    // P goes where K was
#pragma unroll
        for (int i = 0; i < NI; i++) {
            float mp, lp;
            weights(s[i], scale, key0, lo[i], pos[i], tx, mp, lp);
            a[i] = 1.f, b[i] = -1.f;                       // negative: nothing of this page for the row
            if (mp != -INFINITY) merge(m[i], l[i], mp, lp, a[i], b[i]);
            else if (lp != 0.f) l[i] = lp;                  // a NaN among the scores and nothing finite
#pragma unroll
            for (int j = 0; j < 4; j++) p_s[(ty * NI + i) * LDP + tx + 16 * j] = s[i][j];
        }
        __syncthreads();
        float o[NI][4 * CV] = {};
        // the page's first keys, as far as every row sees all of them (fours of them: none where a window cuts the page)
        const int open = window <= 0 || key0 >= last - window + 1 ? min(DK_PAGE, max(0, pos0 - key0 + 1) & ~3) : 0;
#pragma unroll 2
        for (int j = 0; j < open; j += 4) {
            float4 p[NI];
#pragma unroll
            for (int i = 0; i < NI; i++) p[i] = *reinterpret_cast<const float4*>(p_s + (ty * NI + i) * LDP + j);
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int c = 0; c < CV; c++) {
                    const float4 v = *reinterpret_cast<const float4*>(v_s + (j + e) * HD + c * 64 + tx * 4);
#pragma unroll
                    for (int i = 0; i < NI; i++) {
                        const float w = e == 0 ? p[i].x : e == 1 ? p[i].y : e == 2 ? p[i].z : p[i].w;
                        o[i][c * 4] = fmaf(w, v.x, o[i][c * 4]), o[i][c * 4 + 1] = fmaf(w, v.y, o[i][c * 4 + 1]);
                        o[i][c * 4 + 2] = fmaf(w, v.z, o[i][c * 4 + 2]), o[i][c * 4 + 3] = fmaf(w, v.w, o[i][c * 4 + 3]);
                    }
                }
        }
        // a value that a row does not see must not meet its zero weight
        for (int j = open; j < min(DK_PAGE, last - key0 + 1); j++)
#pragma unroll
            for (int i = 0; i < NI; i++)
                if (key0 + j >= lo[i] && key0 + j <= pos[i]) {
                    const float w = p_s[(ty * NI + i) * LDP + j];
#pragma unroll
                    for (int c = 0; c < CV; c++) {
                        const float4 v = *reinterpret_cast<const float4*>(v_s + j * HD + c * 64 + tx * 4);
                        o[i][c * 4] = fmaf(w, v.x, o[i][c * 4]), o[i][c * 4 + 1] = fmaf(w, v.y, o[i][c * 4 + 1]);
                        o[i][c * 4 + 2] = fmaf(w, v.z, o[i][c * 4 + 2]), o[i][c * 4 + 3] = fmaf(w, v.w, o[i][c * 4 + 3]);
                    }
                }
#pragma unroll
        for (int i = 0; i < NI; i++)
            if (b[i] >= 0.f || b[i] != b[i])
#pragma unroll
                for (int c = 0; c < 4 * CV; c++) acc[i][c] = merged(acc[i][c], o[i][c], a[i], b[i]);
        __syncthreads();                                    // the next page goes over this one
    }
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const int r = ty * NI + i;
        if (r >= rows) continue;
        const float inv = 1.f / l[i];
        float* dst = out + ((size_t)(flat0 + r / G) * nh + kvh * G + r % G) * HD + tx * 4;
#pragma unroll
        for (int c = 0; c < CV; c++)
            *reinterpret_cast<float4*>(dst + c * 64) =
                make_float4(acc[i][c * 4] * inv, acc[i][c * 4 + 1] * inv, acc[i][c * 4 + 2] * inv, acc[i][c * 4 + 3] * inv);
    }
}

// Block (page, kv head, sequence): the G query heads' results over one page -> ws_acc [seq][h][pages][HD], ws_ml [..][2].
__global__ void __launch_bounds__(THREADS)
page_kernel(const float* q, const float* k_store, const float* v_store, const int* row_pos, const int* page_table, int pt_stride,
            int nh, int nkv, int window, float scale, float* ws_acc, float* ws_ml) {
    extern __shared__ __align__(16) float smem[];
    float *k_s = smem, *v_s = k_s + DK_PAGE * LDK, *q_s = v_s + DK_PAGE * HD, *p_s = q_s + MAX_G * HD;
    const int pg = blockIdx.x, kvh = blockIdx.y, seq = blockIdx.z, G = nh / nkv, pages = gridDim.x;
    pdl_wait();
    pdl_launch_dependents();
    const int pos = row_pos[seq], key0 = pg * DK_PAGE, lo = window > 0 ? max(0, pos - window + 1) : 0;
    if (pos < 0 || key0 > pos || key0 + DK_PAGE <= lo) return;
    const int page = page_table[(size_t)seq * pt_stride + pg];
    load_page(k_s, LDK, k_store, page, nkv, kvh);
    load_page(v_s, HD, v_store, page, nkv, kvh);
    const size_t head0 = (size_t)seq * nh + kvh * G;
    for (int i = threadIdx.x; i < G * (HD / 4); i += THREADS) copy16(q_s + i * 4, q + head0 * HD + i * 4);
    copy_wait();
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (ty / 2 * 2 < G) {                                   // whole warps: two rows each
        const float* qr[1] = {q_s + min(ty, G - 1) * HD};
        float s[1][4] = {}, mp, lp;
        scores<1>(s, qr, k_s, tx);
        weights(s[0], scale, key0, lo, pos, tx, mp, lp);
#pragma unroll
        for (int j = 0; j < 4; j++) p_s[ty * LDP + tx + 16 * j] = s[0][j];
        if (tx == 0 && ty < G) {
            ws_ml[((head0 + ty) * pages + pg) * 2] = mp;
            ws_ml[((head0 + ty) * pages + pg) * 2 + 1] = lp;
        }
    }
    __syncthreads();
    constexpr int SHARE = THREADS / HD, PER = MAX_G / SHARE;        // rows go round the threads of a column
    const int d = threadIdx.x % HD, g0 = threadIdx.x / HD;
    const int from = max(lo - key0, 0), to = min(pos - key0, DK_PAGE - 1);
    float o[PER] = {};
    for (int j = from; j <= to; j++) {
        const float v = v_s[j * HD + d];
#pragma unroll
        for (int i = 0; i < PER; i++)
            if (g0 + i * SHARE < G) o[i] = fmaf(p_s[(g0 + i * SHARE) * LDP + j], v, o[i]);
    }
#pragma unroll
    for (int i = 0; i < PER; i++)
        if (g0 + i * SHARE < G) ws_acc[((head0 + g0 + i * SHARE) * pages + pg) * HD + d] = o[i];
}

// Block (head, sequence): the pages' results in order.
__global__ void __launch_bounds__(HD)
merge_kernel(const float* ws_acc, const float* ws_ml, float* out, const int* row_pos, int nh, int pages, int window) {
    pdl_launch_dependents();
    pdl_wait();
    const int pos = row_pos[blockIdx.y], d = threadIdx.x;
    const size_t head = (size_t)blockIdx.y * nh + blockIdx.x;
    float m = -INFINITY, l = 0.f, acc = 0.f;
    if (pos >= 0) {
        const int lo = window > 0 ? max(0, pos - window + 1) : 0;
#pragma unroll 8
        for (int pg = lo / DK_PAGE; pg <= pos / DK_PAGE; pg++) {
            const float mp = ws_ml[(head * pages + pg) * 2], lp = ws_ml[(head * pages + pg) * 2 + 1];
            const float page = ws_acc[(head * pages + pg) * HD + d];
            if (mp != -INFINITY) {
                float a, b;
                merge(m, l, mp, lp, a, b);
                acc = merged(acc, page, a, b);
            } else if (lp != 0.f) {
                l = lp;
            }
        }
    }
    out[head * HD + d] = pos >= 0 ? acc * (1.f / l) : 0.f;
}

template <int ROWS>
int launch_prompt(const float* q, float* out, const float* k_store, const float* v_store, const int* tiles, int n_tiles, const int* cu_q,
                  const int* seq_pos0, const int* page_table, int pt_stride, int nh, int nkv, int window, float scale, cudaStream_t st) {
    if ((long long)n_tiles * nkv > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    constexpr size_t smem = (size_t)(ROWS * HD + DK_PAGE * LDK + DK_PAGE * HD) * sizeof(float);
    static_assert(ROWS * LDP <= DK_PAGE * LDK, "P takes K's place");
    cudaError_t e = cudaFuncSetAttribute(prompt_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    return dk_launch(prompt_kernel<ROWS>, dim3((unsigned)(n_tiles * nkv)), dim3(THREADS), smem, st, q, out, k_store, v_store, tiles, cu_q, seq_pos0,
                     page_table, pt_stride, nh, nkv, window, scale);
}

}  // namespace

// q, out [T][nh * HD]; k_store, v_store [pages][nkv][64][HD]; tiles [n][2] = (sequence, first query of a tile of tile_rows / (nh / nkv)
// queries within its portion), tile_rows 64 or 32; cu_q [sequences + 1]; seq_pos0 [sequences]. Every row of q belongs to a sequence's
// portion.
DK_EXPORT int dk_attn_f32_prompt(const float* q, float* out, const float* k_store, const float* v_store, const int* tiles, int n_tiles,
                                 int tile_rows, const int* cu_q, const int* seq_pos0, const int* page_table, int pt_stride, int nh,
                                 int nkv, int window, float scale, cudaStream_t st) {
    if (nkv < 1 || nh % nkv != 0 || nh / nkv > MAX_G || ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_store | (uintptr_t)v_store) % 16 != 0)
        return (int)cudaErrorInvalidValue;
    if (tile_rows == 64)
        return launch_prompt<64>(q, out, k_store, v_store, tiles, n_tiles, cu_q, seq_pos0, page_table, pt_stride, nh, nkv, window, scale, st);
    if (tile_rows == 32)
        return launch_prompt<32>(q, out, k_store, v_store, tiles, n_tiles, cu_q, seq_pos0, page_table, pt_stride, nh, nkv, window, scale, st);
    return (int)cudaErrorInvalidValue;
}

// One token a sequence: q, out [n_seq][nh * HD], row_pos [n_seq] (negative: a padding row, zeros). ws_acc: n_seq * nh * pt_stride *
// HD floats, ws_ml: n_seq * nh * pt_stride * 2.
DK_EXPORT int dk_attn_f32_decode(const float* q, float* out, const float* k_store, const float* v_store, const int* row_pos,
                                 const int* page_table, int pt_stride, int n_seq, int nh, int nkv, int window, float scale,
                                 float* ws_acc, float* ws_ml, cudaStream_t st) {
    if (nkv < 1 || nh % nkv != 0 || nh / nkv > MAX_G || n_seq > 65535 || nkv > 65535 ||
        ((uintptr_t)q | (uintptr_t)k_store | (uintptr_t)v_store) % 16 != 0)
        return (int)cudaErrorInvalidValue;
    constexpr size_t smem = (size_t)(DK_PAGE * LDK + DK_PAGE * HD + MAX_G * HD + MAX_G * LDP) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(page_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int rc = dk_launch(page_kernel, dim3(pt_stride, nkv, n_seq), dim3(THREADS), smem, st, q, k_store, v_store, row_pos,
                             page_table, pt_stride, nh, nkv, window, scale, ws_acc, ws_ml);
    if (rc) return rc;
    return dk_launch(merge_kernel, dim3(nh, n_seq), dim3(HD), 0, st, (const float*)ws_acc, (const float*)ws_ml, out, row_pos, nh,
                     pt_stride, window);
}
