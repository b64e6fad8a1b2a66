// Memory-bound row kernels: embedding gather + RMSNorm, residual add + RMSNorm, SiLU(gate)*up,
// and per-head RMSNorm + rotary position encoding + key/value cache write.
//
// The residual stream `h` is float32 for every model dtype; sums of squares, rsqrt, rotation and
// the residual add are computed in float32. T is the activation/weight dtype (float or bf16).
// Reference formulas (KrishP147/Dryft-Challenge-HTN-2026): engine/engine.py:107-115 (RMSNorm,
// rotate-half RoPE), engine/fused.py:152-172 (add+norm), :175-188 (SiLU*up), :415-475 (q/k norm,
// RoPE, cache write).
#include "common.cuh"

// ---------------------------------------------------------------------------------------------
// h[row] = embed[tok[row]];  a[row] = rmsnorm(h[row]) * w
template <typename T>
__global__ void embed_rmsnorm_kernel(const int* tok, const T* __restrict__ embed,
                                     const float* __restrict__ w, float eps, int H, int V,
                                     float* h, T* a) {
    __shared__ float red[33];
    pdl_launch_dependents();   // before the wait: see pdl_launch_dependents
    pdl_wait();
    const size_t row = blockIdx.x;
    int t = tok[row];
    t = t < 0 ? 0 : (t >= V ? V - 1 : t);  // ids are validated on the host; never read out of bounds
    const T* e = embed + (size_t)t * H;
    float* hr = h + row * H;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float v = to_f(e[i]);
        hr[i] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)H + eps);
    if (w == nullptr) {   // no norm: a, when given, is the row itself in the storage type
        if (a != nullptr)
            for (int i = threadIdx.x; i < H; i += blockDim.x) a[row * H + i] = from_f<T>(hr[i]);
        return;
    }
    T* ar = a + row * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) ar[i] = from_f<T>(hr[i] * rs * w[i]);
}

// h[row] += delta[row] (if delta);  a[out_row] = rmsnorm(h[row]) * w.
// With `rows` the kernel gathers: out_row = blockIdx.x, row = rows[blockIdx.x], and h is not
// written back (used for the final norm at the positions whose logits are wanted).
// ``parts``: n_parts float32 partial sums [n_parts][rows of h][H] (the split-K output of the skinny
// product) that are added up in order and then added to h like delta.
template <typename T>
__global__ void add_rmsnorm_kernel(float* h, const T* delta, const float* parts, int n_parts, size_t part_stride,
                                   const int* rows, const float* __restrict__ w, float eps,
                                   int H, T* a) {
    __shared__ float red[33];
    extern __shared__ float vals[];  // H floats when gathering (h stays untouched)
    pdl_wait();
    pdl_launch_dependents();
    const size_t out_row = blockIdx.x;
    const size_t row = rows ? (size_t)rows[out_row] : out_row;
    float* hr = h + row * H;
    const T* dr = delta ? delta + row * H : nullptr;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float v = hr[i];
        if (dr) v += to_f(dr[i]);
        if (parts) {
            float d = 0.f;
            for (int k = 0; k < n_parts; k++) d += parts[(size_t)k * part_stride + row * H + i];
            v += d;
        }
        if (rows) vals[i] = v; else hr[i] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)H + eps);
    T* ar = a + out_row * H;
    const float* src = rows ? vals : hr;
    for (int i = threadIdx.x; i < H; i += blockDim.x) ar[i] = from_f<T>(src[i] * rs * w[i]);
}

// The same for few rows (decode, and short prefill steps whose products leave partial sums), built
// for latency: one block per row, one or two groups of 4 columns a thread, values kept in registers
// between the two passes, every load of a pass requested before any is used, and what never comes
// from the kernel before this one (norm weight, row index) fetched before the wait for it.
// H % 4 == 0, H <= 8192.
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const bf16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(bf16* p, float4 v) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&lo);
    o.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = o;
}
template <typename T, int QPT>
__global__ void add_rmsnorm_quad_kernel(float* h, const T* delta, const float* parts, int n_parts, size_t part_stride,
                                        const int* rows, const float* __restrict__ w, float eps, int H, T* a) {
    __shared__ float red[33];
    // QPT groups of 4 columns a thread: group q of thread t is columns 4 * (t + q * blockDim.x) ...
    const size_t out_row = blockIdx.x;
    const size_t row = rows ? (size_t)rows[out_row] : out_row;
    float4 w4[QPT];
#pragma unroll
    for (int q = 0; q < QPT; q++) {
        const int c = (threadIdx.x + q * blockDim.x) * 4;
        w4[q] = c < H ? ld4(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_launch_dependents();   // before the wait: see pdl_launch_dependents
    pdl_wait();
    float4 v[QPT];
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < QPT; q++) {
        const int c = (threadIdx.x + q * blockDim.x) * 4;
        v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < H) {
            v[q] = ld4(h + row * H + c);
            if (delta) {
                const float4 d = ld4(delta + row * H + c);
                v[q].x += d.x, v[q].y += d.y, v[q].z += d.z, v[q].w += d.w;
            }
            if (parts) {
                float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
                for (int k = 0; k < n_parts; k++) {
                    const float4 p = ld4(parts + (size_t)k * part_stride + row * H + c);
                    d.x += p.x, d.y += p.y, d.z += p.z, d.w += p.w;
                }
                v[q].x += d.x, v[q].y += d.y, v[q].z += d.z, v[q].w += d.w;
            }
            if (!rows && (delta || parts)) st4(h + row * H + c, v[q]);
        }
        ss += v[q].x * v[q].x + v[q].y * v[q].y + v[q].z * v[q].z + v[q].w * v[q].w;
    }
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)H + eps);
#pragma unroll
    for (int q = 0; q < QPT; q++) {
        const int c = (threadIdx.x + q * blockDim.x) * 4;
        if (c < H)
            st4(a + out_row * H + c, make_float4(v[q].x * rs * w4[q].x, v[q].y * rs * w4[q].y, v[q].z * rs * w4[q].z, v[q].w * rs * w4[q].w));
    }
}

// out[r, c] = silu(gu[r, c]) * gu[r, I + c],  gu rows are [gate | up] of width 2*I
template <typename T>
__global__ void silu_mul_kernel(const T* gu, T* out, size_t n, int I) {
    pdl_wait();
    pdl_launch_dependents();
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    size_t r = idx / I, c = idx % I;
    float g = to_f(gu[r * 2 * I + c]);
    float u = to_f(gu[r * 2 * I + I + c]);
    out[idx] = from_f<T>(g / (1.f + expf(-g)) * u);
}

// ---------------------------------------------------------------------------------------------
// A head's sum of squares is that of its pairs' (d, d + hd/2): a lane's pairs in order, then the lanes by halves (warp_sum).
__device__ __forceinline__ float pair_squares(float first, float second) { return fmaf(first, first, __fmul_rn(second, second)); }

// One warp per (token, head) over nh query heads, nkv key heads and nkv value heads of a fused
// projection row qkv[t] = [q | k | v]. Query and key heads: optional RMSNorm over the head
// (weights qn / kn), optional rotate-half rotation by the angle table at the token's position.
// q goes to q_out [T, nh*hd]; k and v go to the token's place in the paged cache (unless
// write_kv == 0, for a layer that reads another layer's keys and values).
// Tokens with position < 0 are padding: nothing is written for them.
// With ``parts`` the projection row is the sum of n_parts float32 partial rows
// parts[k][t][heads*hd] (split-K output of the skinny product) instead of qkv[t].
// With ``dense_out`` every head (q, k and v) goes to its place in dense_out [T, heads*hd] instead,
// and nothing else is written: the step between a norm and a position encoding that a part
// applies itself before the cache is written.
template <typename T>
__global__ void qk_norm_rope_write_kernel(const T* qkv, const float* parts, int n_parts, size_t part_stride, T* q_out,
                                          T* dense_out,
                                          const float* __restrict__ qn, const float* __restrict__ kn,
                                          const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                          const int* row_pos, const int* row_seq,
                                          const int* page_table, int pt_stride,
                                          T* k_store, T* v_store, int n_tok, int nh,
                                          int nkv, int hd, float eps, int write_kv) {
    // Positions, page ids, angles and norm weights never come from the kernel before this one (the
    // projection): they are fetched before the wait for it, and the projection row in one batch
    // after it, so that the wait is followed by one trip to memory, not five.
    const int lane = threadIdx.x & 31;
    const int heads = nh + 2 * nkv;
    const long long wid = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool live = wid < (long long)n_tok * heads;
    const int t = live ? (int)(wid / heads) : 0, hidx = live ? (int)(wid % heads) : 0;
    const int pos = live ? row_pos[t] : -1;
    const int half = hd >> 1;
    const bool is_q = hidx < nh, is_v = hidx >= nh + nkv;
    const bool work = pos >= 0 && (is_q || write_kv || dense_out != nullptr);
    T* dst = nullptr;
    if (work) {
        if (dense_out != nullptr) {
            dst = dense_out + ((size_t)t * heads + hidx) * hd;
        } else if (is_q) {
            dst = q_out + ((size_t)t * nh + hidx) * hd;
        } else {
            const int kvh = (hidx - nh) % nkv;
            const int page = page_table[(size_t)row_seq[t] * pt_stride + pos / DK_PAGE];
            dst = (is_v ? v_store : k_store) + kv_offset(page, nkv, kvh, pos % DK_PAGE, hd);
        }
    }
    const float* nw = is_q ? qn : kn;
    float c[4], sn[4], w1[4], w2[4];   // pairs (d, d + half), d = lane + 32*i; hd <= 256 gives at most 4 pairs a lane
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = lane + 32 * i;
        const bool on = work && !is_v && d < half;
        c[i] = on && cos_t ? cos_t[(size_t)pos * half + d] : 1.f;
        sn[i] = on && cos_t ? sin_t[(size_t)pos * half + d] : 0.f;
        w1[i] = on && nw ? nw[d] : 1.f;
        w2[i] = on && nw ? nw[d + half] : 1.f;
    }
    pdl_launch_dependents();   // before the wait (see pdl_launch_dependents): what decode attention does before its own wait
    pdl_wait();                // reads positions, page ids and cache pages of older tokens, none of them written in this step
    if (!work) return;
    const size_t x_off = (size_t)t * heads * hd + (size_t)hidx * hd;
    float x1[4] = {0.f, 0.f, 0.f, 0.f}, x2[4] = {0.f, 0.f, 0.f, 0.f};
    if (parts == nullptr) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int d = lane + 32 * i;
            if (d < half) x1[i] = to_f(qkv[x_off + d]), x2[i] = to_f(qkv[x_off + d + half]);
        }
    } else {
#pragma unroll 4
        for (int k = 0; k < n_parts; k++) {
            const float* pk = parts + (size_t)k * part_stride + x_off;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int d = lane + 32 * i;
                if (d < half) x1[i] += pk[d], x2[i] += pk[d + half];
            }
        }
    }
    if (is_v) {  // value head: plain copy
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int d = lane + 32 * i;
            if (d < half) dst[d] = from_f<T>(x1[i]), dst[d + half] = from_f<T>(x2[i]);
        }
        return;
    }
    if (nw) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) ss += pair_squares(x1[i], x2[i]);
        ss = warp_sum(ss);
        const float rs = rsqrtf(ss / (float)hd + eps);
#pragma unroll
        for (int i = 0; i < 4; i++) x1[i] = x1[i] * rs * w1[i], x2[i] = x2[i] * rs * w2[i];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = lane + 32 * i;
        if (d < half) {
            float o1 = x1[i], o2 = x2[i];
            if (cos_t) {
                o1 = x1[i] * c[i] - x2[i] * sn[i];
                o2 = x2[i] * c[i] + x1[i] * sn[i];
            }
            dst[d] = from_f<T>(o1);
            dst[d + half] = from_f<T>(o2);
        }
    }
}

// The head's sum of squares in the order of qk_norm_rope_write_kernel, whose lane L holds the pairs L and (heads of 128) L + 32: here
// pairs 4 l + c lie with lane l of each half of the head, c = 0..3. The 8 lanes of a quarter of the head (heads of 64: of a half) add
// up one c (two): 6 (7) shuffles where four columns a lane one by one would take 20 (16).
template <int HDT>
__device__ __forceinline__ float head_squares(const float4& first, const float4& other, int lane) {
    const float t[4] = {pair_squares(first.x, other.x), pair_squares(first.y, other.y), pair_squares(first.z, other.z),
                        pair_squares(first.w, other.w)};
    const bool odd = (lane & 8) != 0, high = (lane & 16) != 0;
    float s;
    if constexpr (HDT == 128) {                               // quarters 0 and 2 hold pairs 0..31 and c = 0, 2; 1 and 3 32..63 and c = 1, 3
        const float a = high ? t[2] : t[0], b = high ? t[3] : t[1];
        s = odd ? b : a;
        s += __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);    // pair L + 32 to pair L
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        s += __shfl_xor_sync(0xffffffffu, s, 16);             // c with c ^ 2
    } else {                                                  // halves 0 and 1: c = 0, 2 and c = 1, 3
        float u = odd ? t[3] : t[2];
        s = odd ? t[1] : t[0];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o), u += __shfl_xor_sync(0xffffffffu, u, o);
        s += u;
    }
    return s + __shfl_xor_sync(0xffffffffu, s, 8);            // c with c ^ 1
}

// The same for heads of 64 or 128 whose rows are float32 (parts of a projection, or a float32 projection as its only part): a lane has 4
// consecutive columns of a head and reads them as one float4 of every part, up to eight parts on their way at a time; the other half
// of the rotation comes from the lane half a head further. Every sum, the squares' among them, is added up as above, so that a row's
// result does not depend on where its tensors lie. Bound by the trip to the L2 after the wait. In a chain of its own, with
// scalar loads before: 4 parts of one row of 48 heads of 128 2.3 -> 1.4 us, 9 parts of 64 rows 4.6 -> 3.0; 544 float32 rows 11.0 either
// way. (64 registers: with the other half's norm weights kept instead of a second exchange 72, 2.8 us at 64 rows but 11.9 at 544.)
template <typename T, int HDT>
__global__ void qk_norm_rope_write_quad_kernel(const float* parts, int n_parts, size_t part_stride, float zero, T* q_out, T* dense_out,
                                               const float* __restrict__ qn, const float* __restrict__ kn,
                                               const float* __restrict__ cos_t, const float* __restrict__ sin_t, const int* row_pos,
                                               const int* row_seq, const int* page_table, int pt_stride, T* k_store, T* v_store,
                                               int n_tok, int nh, int nkv, float eps, int write_kv) {
    constexpr int G = HDT / 4, HALF = HDT / 2;                // lanes a head
    const int lane = threadIdx.x & 31, d = (lane % G) * 4;
    const int heads = nh + 2 * nkv;
    const long long item = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / G) + lane / G;
    const bool live = item < (long long)n_tok * heads;
    const int t = live ? (int)(item / heads) : 0, hidx = live ? (int)(item % heads) : 0;
    const int pos = live ? row_pos[t] : -1;
    const bool is_q = hidx < nh, is_v = hidx >= nh + nkv;
    const bool work = pos >= 0 && (is_q || write_kv || dense_out != nullptr);
    T* dst = nullptr;
    float4 c = make_float4(1.f, 1.f, 1.f, 1.f), sn = make_float4(0.f, 0.f, 0.f, 0.f), w = c;
    const float* nw = is_v ? nullptr : is_q ? qn : kn;
    const bool turn = cos_t != nullptr && !is_v;
    if (work) {
        if (dense_out != nullptr) {
            dst = dense_out + ((size_t)t * heads + hidx) * HDT;
        } else if (is_q) {
            dst = q_out + ((size_t)t * nh + hidx) * HDT;
        } else {
            const int page = page_table[(size_t)row_seq[t] * pt_stride + pos / DK_PAGE];
            dst = (is_v ? v_store : k_store) + kv_offset(page, nkv, (hidx - nh) % nkv, pos % DK_PAGE, HDT);
        }
        if (turn) {
            c = *reinterpret_cast<const float4*>(cos_t + (size_t)pos * HALF + d % HALF);
            sn = *reinterpret_cast<const float4*>(sin_t + (size_t)pos * HALF + d % HALF);
        }
        if (nw) w = *reinterpret_cast<const float4*>(nw + d);
    }
    pdl_launch_dependents();   // before the wait, as in qk_norm_rope_write_kernel
    pdl_wait();
    float4 x = make_float4(zero, zero, zero, zero);
    if (work) {
        const float* p = parts + (size_t)t * heads * HDT + (size_t)hidx * HDT + d;
        for (int k = 0; k < n_parts; k += 8) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (k + u < n_parts) v[u] = *reinterpret_cast<const float4*>(p + (size_t)(k + u) * part_stride);
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (k + u < n_parts) x.x += v[u].x, x.y += v[u].y, x.z += v[u].z, x.w += v[u].w;
        }
    }
    const bool second = d >= HALF;
    // the same columns of the head's other half
    auto other = [](const float4& a) {
        return make_float4(__shfl_xor_sync(0xffffffffu, a.x, G / 2), __shfl_xor_sync(0xffffffffu, a.y, G / 2),
                           __shfl_xor_sync(0xffffffffu, a.z, G / 2), __shfl_xor_sync(0xffffffffu, a.w, G / 2));
    };
    float4 y = other(x);
    const float ss = head_squares<HDT>(second ? y : x, second ? x : y, lane);
    if (nw) {
        const float rs = rsqrtf(ss / (float)HDT + eps);
        x.x = x.x * rs * w.x, x.y = x.y * rs * w.y, x.z = x.z * rs * w.z, x.w = x.w * rs * w.w;
    }
    y = other(x);
    if (!work) return;
    if (turn) {
        if (!second)
            x = make_float4(x.x * c.x - y.x * sn.x, x.y * c.y - y.y * sn.y, x.z * c.z - y.z * sn.z, x.w * c.w - y.w * sn.w);
        else
            x = make_float4(x.x * c.x + y.x * sn.x, x.y * c.y + y.y * sn.y, x.z * c.z + y.z * sn.z, x.w * c.w + y.w * sn.w);
    }
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst + d) = x;
    } else {
        uint2 pk;
        *reinterpret_cast<__nv_bfloat162*>(&pk.x) = __floats2bfloat162_rn(x.x, x.y);
        *reinterpret_cast<__nv_bfloat162*>(&pk.y) = __floats2bfloat162_rn(x.z, x.w);
        *reinterpret_cast<uint2*>(dst + d) = pk;
    }
}

// ---------------------------------------------------------------------------------------------
// out[i] = src[rows[i]] for rows of H floats (positions whose logits are wanted)
__global__ void gather_rows_f32_kernel(const float* src, const int* rows,
                                       float* out, int H) {
    pdl_wait();
    pdl_launch_dependents();
    const float* s = src + (size_t)rows[blockIdx.x] * H;
    float* o = out + (size_t)blockIdx.x * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) o[i] = s[i];
}

// ---------------------------------------------------------------------------------------------
// Wide variants for many rows of bfloat16 (prefill): 16-byte accesses instead of 2-byte ones.
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 t = __bfloat1622float2(p[i]);
        f[2 * i] = t.x, f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 v;
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; i++) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return v;
}

// silu(gate) * up, 8 outputs a thread; I % 8 == 0.
__global__ void silu_mul_wide_kernel(const bf16* gu, bf16* out, size_t n8, int I8) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n8) return;
    const size_t r = idx / I8, c = idx % I8;
    const uint4* row = reinterpret_cast<const uint4*>(gu) + r * 2 * I8;
    float g[8], u[8], o[8];
    unpack8(row[c], g);
    unpack8(row[I8 + c], u);
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = g[i] / (1.f + expf(-g[i])) * u[i];
    reinterpret_cast<uint4*>(out)[idx] = pack8(o);
}

// h += delta; a = rmsnorm(h) * w for bfloat16 delta / a, 8 elements a thread per pass, values kept
// in registers between the two passes. H % 8 == 0 and H <= 8 * 4 * blockDim.x.
__global__ void add_rmsnorm_wide_kernel(float* h, const bf16* delta, const float* __restrict__ w, float eps, int H, bf16* a) {
    __shared__ float red[33];
    pdl_wait();
    pdl_launch_dependents();
    const size_t row = blockIdx.x;
    float4* hr = reinterpret_cast<float4*>(h + row * H);
    const uint4* dr = delta ? reinterpret_cast<const uint4*>(delta + row * H) : nullptr;
    const int n8 = H / 8;
    float v[4][8];
    float ss = 0.f;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int i = threadIdx.x + it * blockDim.x;
        if (i < n8) {
            const float4 x0 = hr[2 * i], x1 = hr[2 * i + 1];
            v[it][0] = x0.x, v[it][1] = x0.y, v[it][2] = x0.z, v[it][3] = x0.w;
            v[it][4] = x1.x, v[it][5] = x1.y, v[it][6] = x1.z, v[it][7] = x1.w;
            if (dr) {
                float d[8];
                unpack8(dr[i], d);
#pragma unroll
                for (int k = 0; k < 8; k++) v[it][k] += d[k];
                hr[2 * i] = make_float4(v[it][0], v[it][1], v[it][2], v[it][3]);
                hr[2 * i + 1] = make_float4(v[it][4], v[it][5], v[it][6], v[it][7]);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) ss += v[it][k] * v[it][k];
        }
    }
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)H + eps);
    uint4* ar = reinterpret_cast<uint4*>(a + row * H);
    const float4* wr = reinterpret_cast<const float4*>(w);
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int i = threadIdx.x + it * blockDim.x;
        if (i < n8) {
            const float4 w0 = wr[2 * i], w1 = wr[2 * i + 1];
            float o[8] = {v[it][0] * rs * w0.x, v[it][1] * rs * w0.y, v[it][2] * rs * w0.z, v[it][3] * rs * w0.w,
                          v[it][4] * rs * w1.x, v[it][5] * rs * w1.y, v[it][6] * rs * w1.z, v[it][7] * rs * w1.w};
            ar[i] = pack8(o);
        }
    }
}

// The same with one warp per row (H % 256 == 0, H <= 4096): every load of the row is requested
// before any is used, the sum of squares needs shuffles only, and no block barrier is on the path.
template <int CH>   // CH = H / 256 chunks of 8 elements per lane
__global__ void __launch_bounds__(256)
add_rmsnorm_warp_kernel(float* h, const bf16* delta, const float* __restrict__ w, float eps, int n_rows, bf16* a) {
    constexpr int H = CH * 256;
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= (size_t)n_rows) return;
    float4* hr = reinterpret_cast<float4*>(h + row * H);
    const uint4* dr = delta ? reinterpret_cast<const uint4*>(delta + row * H) : nullptr;
    float v[CH][8];
    uint4 d8[CH];
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const int i = c * 32 + lane;          // index of this lane's 8 elements
        const float4 x0 = hr[2 * i], x1 = hr[2 * i + 1];
        v[c][0] = x0.x, v[c][1] = x0.y, v[c][2] = x0.z, v[c][3] = x0.w;
        v[c][4] = x1.x, v[c][5] = x1.y, v[c][6] = x1.z, v[c][7] = x1.w;
        if (dr) d8[c] = dr[i];
    }
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const int i = c * 32 + lane;
        if (dr) {
            float d[8];
            unpack8(d8[c], d);
#pragma unroll
            for (int k = 0; k < 8; k++) v[c][k] += d[k];
            hr[2 * i] = make_float4(v[c][0], v[c][1], v[c][2], v[c][3]);
            hr[2 * i + 1] = make_float4(v[c][4], v[c][5], v[c][6], v[c][7]);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) ss += v[c][k] * v[c][k];
    }
    ss = warp_sum(ss);
    const float rs = rsqrtf(ss / (float)H + eps);
    uint4* ar = reinterpret_cast<uint4*>(a + row * H);
    const float4* wr = reinterpret_cast<const float4*>(w);
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const int i = c * 32 + lane;
        const float4 w0 = wr[2 * i], w1 = wr[2 * i + 1];
        float o[8] = {v[c][0] * rs * w0.x, v[c][1] * rs * w0.y, v[c][2] * rs * w0.z, v[c][3] * rs * w0.w,
                      v[c][4] * rs * w1.x, v[c][5] * rs * w1.y, v[c][6] * rs * w1.z, v[c][7] * rs * w1.w};
        ar[i] = pack8(o);
    }
}

// q/k norm + rotation + cache write for bfloat16 with head sizes that are multiples of 16. A group
// of GS lanes (GS = the power of two >= head_dim / 16) takes one (token, head); a warp takes 32 / GS
// of them. Lane j of a group holds elements [8j, 8j+8) of each half of the head.
template <int GS>
__global__ void qk_norm_rope_write_wide_kernel(const bf16* qkv, bf16* q_out, bf16* dense_out, const float* __restrict__ qn,
                                               const float* __restrict__ kn, const float* __restrict__ cos_t,
                                               const float* __restrict__ sin_t, const int* row_pos, const int* row_seq,
                                               const int* page_table, int pt_stride, bf16* k_store, bf16* v_store,
                                               int n_tok, int nh, int nkv, int hd, float eps, int write_kv) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, j = lane % GS;
    const int heads = nh + 2 * nkv;
    const long long item = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / GS) + lane / GS;
    const bool live = item < (long long)n_tok * heads;
    const int t = live ? (int)(item / heads) : 0, hidx = live ? (int)(item % heads) : 0;
    const int pos = live ? row_pos[t] : -1;
    const int half = hd >> 1, half8 = hd >> 4;
    const bool is_v = hidx >= nh + nkv;
    const bool work = pos >= 0 && (hidx < nh || write_kv || dense_out != nullptr);
    const bf16* x = qkv + (size_t)t * heads * hd + (size_t)hidx * hd;
    bf16* dst = nullptr;
    if (work) {
        if (dense_out != nullptr) {
            dst = dense_out + ((size_t)t * heads + hidx) * hd;
        } else if (hidx < nh) {
            dst = q_out + ((size_t)t * nh + hidx) * hd;
        } else {
            const int kvh = (hidx - nh) % nkv;
            const int page = page_table[(size_t)row_seq[t] * pt_stride + pos / DK_PAGE];
            dst = (hidx < nh + nkv ? k_store : v_store) + kv_offset(page, nkv, kvh, pos % DK_PAGE, hd);
        }
    }
    const bool on = work && j < half8;
    float x1[8], x2[8];
    float ss = 0.f;
    if (on) {
        const uint4 r1 = reinterpret_cast<const uint4*>(x)[j], r2 = reinterpret_cast<const uint4*>(x + half)[j];
        if (is_v) {  // value head: plain copy
            reinterpret_cast<uint4*>(dst)[j] = r1;
            reinterpret_cast<uint4*>(dst + half)[j] = r2;
        }
        unpack8(r1, x1);
        unpack8(r2, x2);
#pragma unroll
        for (int i = 0; i < 8; i++) ss += x1[i] * x1[i] + x2[i] * x2[i];
    }
#pragma unroll
    for (int o = GS / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);   // within the group of GS lanes
    if (!on || is_v) return;
    const float* nw = hidx < nh ? qn : kn;
    const float rs = nw ? rsqrtf(ss / (float)hd + eps) : 1.f;
    // weights and angles of this lane's 8 + 8 elements: 16-byte loads (hd % 16 == 0 keeps them aligned)
    float w1[8], w2[8], cs[8], sn[8];
    auto load8 = [](const float* p, float (&f)[8]) {
        const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    };
    if (nw) load8(nw + 8 * j, w1), load8(nw + half + 8 * j, w2);
    if (cos_t) load8(cos_t + (size_t)pos * half + 8 * j, cs), load8(sin_t + (size_t)pos * half + 8 * j, sn);
    float o1[8], o2[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float a1 = x1[i] * rs, a2 = x2[i] * rs;
        if (nw) a1 *= w1[i], a2 *= w2[i];
        o1[i] = a1, o2[i] = a2;
        if (cos_t) {
            o1[i] = a1 * cs[i] - a2 * sn[i];
            o2[i] = a2 * cs[i] + a1 * sn[i];
        }
    }
    reinterpret_cast<uint4*>(dst)[j] = pack8(o1);
    reinterpret_cast<uint4*>(dst + half)[j] = pack8(o2);
}

// ---------------------------------------------------------------------------------------------
#define DISPATCH_T(dtype, ...)                         \
    if ((dtype) == 0) { typedef float T; __VA_ARGS__; } \
    else { typedef bf16 T; __VA_ARGS__; }

static inline int row_threads(int H) { return H >= 2048 ? 512 : (H >= 512 ? 256 : 128); }

DK_EXPORT int dk_embed_rmsnorm(int dtype, const int* tok, const void* embed, const float* w, float eps,
                               int n_tok, int H, int V, float* h, void* a, cudaStream_t st) {
    DISPATCH_T(dtype, return dk_launch(embed_rmsnorm_kernel<T>, dim3(n_tok), dim3(row_threads(H)), 0, st, tok,
                                       (const T*)embed, w, eps, H, V, h, (T*)a));
}

DK_EXPORT int dk_add_rmsnorm(int dtype, float* h, const void* delta, const float* parts, int n_parts,
                             long long part_stride, const int* rows, const float* w, float eps, int n_rows, int H,
                             void* a, cudaStream_t st) {
    if (dtype == 1 && parts == nullptr && rows == nullptr && H % 256 == 0 && H <= 4096 && n_rows > 64) {
        // warps a block: eight when the rows are many; fewer when blocks of eight would leave the SMs
        // with one or two blocks each (2,048 rows: 256 blocks on 148 SMs, a quarter of them idle half the time)
        int sms = 0, dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        int wpb = 8;
        while (wpb > 1 && (n_rows + wpb - 1) / wpb < 8 * sms) wpb >>= 1;
        const dim3 grid((n_rows + wpb - 1) / wpb), block(32 * wpb);
#define NORM_WARP(CH)                                                                                                   \
    if (H == CH * 256)                                                                                                  \
        return dk_launch_whole(add_rmsnorm_warp_kernel<CH>, grid, block, 0, st, h, (const bf16*)delta, w, eps, n_rows, (bf16*)a)
        NORM_WARP(1); NORM_WARP(2); NORM_WARP(3); NORM_WARP(4); NORM_WARP(5); NORM_WARP(6); NORM_WARP(7); NORM_WARP(8);
        NORM_WARP(9); NORM_WARP(10); NORM_WARP(11); NORM_WARP(12); NORM_WARP(13); NORM_WARP(14); NORM_WARP(15); NORM_WARP(16);
#undef NORM_WARP
    }
    if (dtype == 1 && parts == nullptr && rows == nullptr && H % 8 == 0 && H <= 8 * 4 * row_threads(H) && n_rows > 64)
        return dk_launch_whole(add_rmsnorm_wide_kernel, dim3(n_rows), dim3(row_threads(H)), 0, st, h, (const bf16*)delta, w, eps,
                         H, (bf16*)a);
    // float32: this kernel at any number of rows and with or without parts, so that a row's sum of squares is added up in one
    // order however many rows are beside it (its products are planned to leave parts at some row counts and not at others)
    const bool dense32 = dtype == 0 && (((uintptr_t)h | (uintptr_t)delta | (uintptr_t)parts | (uintptr_t)w | (uintptr_t)a) & 15) == 0;
    if ((n_rows <= 64 || parts != nullptr || dense32) && H % 4 == 0 && H <= 8192 && part_stride % 4 == 0) {
        if (H <= 4096) {
            DISPATCH_T(dtype, return dk_launch(add_rmsnorm_quad_kernel<T, 1>, dim3(n_rows), dim3((H / 4 + 31) / 32 * 32), 0, st, h,
                                               (const T*)delta, parts, n_parts, (size_t)part_stride, rows, w, eps, H, (T*)a));
        }
        DISPATCH_T(dtype, return dk_launch(add_rmsnorm_quad_kernel<T, 2>, dim3(n_rows), dim3((H / 8 + 31) / 32 * 32), 0, st, h,
                                           (const T*)delta, parts, n_parts, (size_t)part_stride, rows, w, eps, H, (T*)a));
    }
    size_t smem = rows ? (size_t)H * sizeof(float) : 0;
    if (smem > 48 * 1024) {
        DISPATCH_T(dtype, cudaFuncSetAttribute(add_rmsnorm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem));
    }
    DISPATCH_T(dtype, return dk_launch(add_rmsnorm_kernel<T>, dim3(n_rows), dim3(row_threads(H)), smem, st, h,
                                       (const T*)delta, parts, n_parts, (size_t)part_stride, rows, w, eps, H, (T*)a));
}

DK_EXPORT int dk_silu_mul(int dtype, const void* gu, void* out, long long n_rows, int I, cudaStream_t st) {
    size_t n = (size_t)n_rows * I;
    if (dtype == 1 && I % 8 == 0)
        return dk_launch(silu_mul_wide_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, st, (const bf16*)gu,
                         (bf16*)out, n / 8, I / 8);
    DISPATCH_T(dtype, return dk_launch(silu_mul_kernel<T>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st,
                                       (const T*)gu, (T*)out, n, I));
}

DK_EXPORT int dk_qk_norm_rope_write(int dtype, const void* qkv, const float* parts, int n_parts, long long part_stride,
                                    void* q_out, void* dense_out, const float* qn, const float* kn,
                                    const float* cos_t, const float* sin_t, const int* row_pos, const int* row_seq,
                                    const int* page_table, int pt_stride, void* k_store, void* v_store, int n_tok,
                                    int nh, int nkv, int hd, float eps, int write_kv, cudaStream_t st) {
    if (hd % 2 != 0 || hd > 256) return (int)cudaErrorInvalidValue;
    long long warps = (long long)n_tok * (nh + 2 * nkv);
    unsigned blocks = (unsigned)((warps + 3) / 4);
    if (dtype == 1 && parts == nullptr && hd % 16 == 0 && n_tok > 64) {
        const int half8 = hd / 16;
        const int gs = half8 <= 1 ? 1 : half8 <= 2 ? 2 : half8 <= 4 ? 4 : half8 <= 8 ? 8 : 16;
        const unsigned wblocks = (unsigned)((warps + 4LL * (32 / gs) - 1) / (4LL * (32 / gs)));
#define ROPE_WIDE(GS)                                                                                                  \
    return dk_launch_whole(qk_norm_rope_write_wide_kernel<GS>, dim3(wblocks), dim3(128), 0, st, (const bf16*)qkv, (bf16*)q_out, \
                     (bf16*)dense_out, qn, kn, cos_t, sin_t, row_pos, row_seq, page_table, pt_stride, (bf16*)k_store, (bf16*)v_store, n_tok, \
                     nh, nkv, hd, eps, write_kv)
        if (gs == 1) ROPE_WIDE(1);
        if (gs == 2) ROPE_WIDE(2);
        if (gs == 4) ROPE_WIDE(4);
        if (gs == 8) ROPE_WIDE(8);
        ROPE_WIDE(16);
#undef ROPE_WIDE
    }
    // float32 rows, whatever their number and whether in parts or not, so that a row's sum of squares is added up in one order
    const float* rows32 = parts != nullptr ? parts : dtype == 0 ? (const float*)qkv : nullptr;
    if ((hd == 64 || hd == 128) && rows32 != nullptr && part_stride % 4 == 0 &&
        (((uintptr_t)rows32 | (uintptr_t)q_out | (uintptr_t)dense_out | (uintptr_t)qn | (uintptr_t)kn | (uintptr_t)cos_t |
          (uintptr_t)sin_t | (uintptr_t)k_store | (uintptr_t)v_store) & 15) == 0) {
        const int n = parts != nullptr ? n_parts : 1;
#define ROPE_QUAD(HDT)                                                                                                   \
    DISPATCH_T(dtype, return dk_launch(qk_norm_rope_write_quad_kernel<T, HDT>, dim3((unsigned)((warps * HDT + 511) / 512)), dim3(128), 0, st, \
                                       rows32, n, (size_t)part_stride, parts != nullptr ? 0.f : -0.f, (T*)q_out, (T*)dense_out, qn, kn, cos_t, sin_t, row_pos,        \
                                       row_seq, page_table, pt_stride, (T*)k_store, (T*)v_store, n_tok, nh, nkv, eps, write_kv))
        if (hd == 128) ROPE_QUAD(128);
        ROPE_QUAD(64);
#undef ROPE_QUAD
    }
    DISPATCH_T(dtype, return dk_launch(qk_norm_rope_write_kernel<T>, dim3(blocks), dim3(128), 0, st, (const T*)qkv,
                                       parts, n_parts, (size_t)part_stride, (T*)q_out, (T*)dense_out, qn, kn, cos_t, sin_t, row_pos, row_seq, page_table, pt_stride,
                                       (T*)k_store, (T*)v_store, n_tok, nh, nkv, hd, eps, write_kv));
}

DK_EXPORT int dk_gather_rows_f32(const float* src, const int* rows, float* out, int n_rows, int H, cudaStream_t st) {
    return dk_launch(gather_rows_f32_kernel, dim3(n_rows), dim3(256), 0, st, src, rows, out, H);
}

// ---------------------------------------------------------------------------------------------
// Embedding with a scale and an absolute sinusoidal position vector:
//   h[row][2i] = embed[tok][2i] * scale + sin(p * f_i),  h[row][2i+1] = embed[tok][2i+1] * scale + cos(p * f_i)
// with p the row's position and f_i = inv_freq[i] (float64, made on the host). The angle is formed and
// brought into [-pi, pi] in float64, so that it is right to float32 rounding at any position; sine and
// cosine are the float32 functions. Without a table (inv_freq == nullptr) only the scale applies.
// a[row] = rmsnorm(h[row]) * w when w is given. Rows with position < 0 (padding) get position 0.
template <typename T>
__global__ void embed_position_rmsnorm_kernel(const int* tok, const T* __restrict__ embed, float scale,
                                              const int* row_pos, const double* __restrict__ inv_freq,
                                              const float* __restrict__ w, float eps, int H, int V, float* h, T* a) {
    __shared__ float red[33];
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = blockIdx.x;
    int t = tok[row];
    t = t < 0 ? 0 : (t >= V ? V - 1 : t);
    const int p = inv_freq ? max(row_pos[row], 0) : 0;
    const T* e = embed + (size_t)t * H;
    float* hr = h + row * H;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float v = __fmul_rn(to_f(e[i]), scale);
        if (inv_freq && (i >> 1) < H / 2) {
            double ang = (double)p * inv_freq[i >> 1];
            ang -= 6.283185307179586476925 * rint(ang * 0.15915494309189533577);
            v = __fadd_rn(v, (i & 1) ? cosf((float)ang) : sinf((float)ang));
        }
        hr[i] = v;
        ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, red);
    if (w == nullptr) return;
    const float rs = rsqrtf(ss / (float)H + eps);
    T* ar = a + row * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) ar[i] = from_f<T>(hr[i] * rs * w[i]);
}

// The same for widths that are multiples of 4, up to 8,192, on 16-byte boundaries: a thread holds up to four fours of columns, and an
// angle's sine and cosine are worked out together, once. The bits are those of the kernel above: product and sine are rounded apart,
// and the squares, handed over in shared memory, are added up in its order (a row's start does not depend on where its tensors lie).
// Bound by its instructions (issue slots 60 % busy, float64 and special functions 3 and 16 % of their pipes) and the waits at its three
// barriers: 16,000 rows of 2,560, bfloat16, 193 us with every number's angle worked out by itself, now 131; 8 rows 5.3 and 3.2.
template <typename T>
__global__ void __launch_bounds__(512)
embed_position_rmsnorm_wide_kernel(const int* tok, const T* __restrict__ embed, float scale, const int* row_pos,
                                   const double* __restrict__ inv_freq, const float* __restrict__ w, float eps, int H, int V, float* h,
                                   T* a) {
    __shared__ float red[33];
    extern __shared__ __align__(16) float vrow[];        // [H]
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = blockIdx.x;
    int t = tok[row];
    t = t < 0 ? 0 : (t >= V ? V - 1 : t);
    const int p = inv_freq ? max(row_pos[row], 0) : 0;
    const T* e = embed + (size_t)t * H;
    float v[4][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = (k * blockDim.x + threadIdx.x) * 4;
        if (i >= H) continue;
        alignas(16) T x[4];
        if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(e + i);
        else *reinterpret_cast<uint2*>(x) = *reinterpret_cast<const uint2*>(e + i);
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            v[k][c] = __fmul_rn(to_f(x[c]), scale), v[k][c + 1] = __fmul_rn(to_f(x[c + 1]), scale);
            if (inv_freq) {
                double ang = (double)p * inv_freq[(i + c) >> 1];
                ang -= 6.283185307179586476925 * rint(ang * 0.15915494309189533577);
                float s, co;
                sincosf((float)ang, &s, &co);
                v[k][c] = __fadd_rn(v[k][c], s), v[k][c + 1] = __fadd_rn(v[k][c + 1], co);
            }
        }
        const float4 f = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
        *reinterpret_cast<float4*>(h + row * H + i) = f;
        *reinterpret_cast<float4*>(vrow + i) = f;
    }
    if (w == nullptr) return;
    __syncthreads();
    float ss = 0.f;
#pragma unroll 4
    for (int i = threadIdx.x; i < H; i += blockDim.x) ss = fmaf(vrow[i], vrow[i], ss);
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)H + eps);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = (k * blockDim.x + threadIdx.x) * 4;
        if (i >= H) continue;
        const float4 wv = *reinterpret_cast<const float4*>(w + i);
        alignas(16) T y[4] = {from_f<T>(v[k][0] * rs * wv.x), from_f<T>(v[k][1] * rs * wv.y), from_f<T>(v[k][2] * rs * wv.z), from_f<T>(v[k][3] * rs * wv.w)};
        if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(a + row * H + i) = *reinterpret_cast<const float4*>(y);
        else *reinterpret_cast<uint2*>(a + row * H + i) = *reinterpret_cast<const uint2*>(y);
    }
}

DK_EXPORT int dk_embed_position_rmsnorm(int dtype, const int* tok, const void* embed, float scale, const int* row_pos,
                                        const double* inv_freq, const float* w, float eps, int n_tok, int H, int V,
                                        float* h, void* a, cudaStream_t st) {
    if (H % 4 == 0 && H <= 8192 && (((uintptr_t)embed | (uintptr_t)w | (uintptr_t)h | (uintptr_t)a) & 15) == 0) {
        // as many threads as the general kernel: a thread's squares are then the same ones
        DISPATCH_T(dtype, return dk_launch(embed_position_rmsnorm_wide_kernel<T>, dim3(n_tok), dim3(row_threads(H)), H * sizeof(float), st, tok,
                                           (const T*)embed, scale, row_pos, inv_freq, w, eps, H, V, h, (T*)a));
    }
    DISPATCH_T(dtype, return dk_launch(embed_position_rmsnorm_kernel<T>, dim3(n_tok), dim3(row_threads(H)), 0, st, tok,
                                       (const T*)embed, scale, row_pos, inv_freq, w, eps, H, V, h, (T*)a));
}

// h[row] += other[row] (if other) + vec (if vec): what a schedule adds to the residual stream before a
// layer (a saved copy of the stream, a learned vector). All float32.
__global__ void stream_add_kernel(float* h, const float* other, const float* __restrict__ vec, size_t n, int H) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v = h[i];
    if (other) v += other[i];
    if (vec) v += vec[i % H];
    h[i] = v;
}

DK_EXPORT int dk_stream_add(float* h, const float* other, const float* vec, long long n_rows, int H, cudaStream_t st) {
    const size_t n = (size_t)n_rows * H;
    return dk_launch(stream_add_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, h, other, vec, n, H);
}

// x = cap * tanh(factor * x / cap) in place (float32 logits); cap 0: x = factor * x
__global__ void softcap_kernel(float* x, size_t n, float cap, float factor) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float v = x[i] * factor;
        x[i] = cap > 0.f ? cap * tanhf(v / cap) : v;
    }
}

DK_EXPORT int dk_softcap(float* x, long long n, float cap, float factor, cudaStream_t st) {
    return dk_launch(softcap_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, x, (size_t)n, cap, factor);
}

// xIELU (common.cuh) as a kernel of its own, for the products that do not have it in their epilogue.

template <typename T>
__global__ void xielu_kernel(const T* z, T* out, size_t n, float ap, float an) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = from_f<T>(xielu_f(to_f(z[i]), ap, an));
}

__global__ void xielu_wide_kernel(const bf16* z, bf16* out, size_t n8, float ap, float an) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    uint4 raw = reinterpret_cast<const uint4*>(z)[i];
    bf16* v = reinterpret_cast<bf16*>(&raw);
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = __float2bfloat16_rn(xielu_f(__bfloat162float(v[k]), ap, an));
    reinterpret_cast<uint4*>(out)[i] = raw;
}

DK_EXPORT int dk_xielu(int dtype, const void* z, void* out, long long n, float ap, float an, cudaStream_t st) {
    if (dtype == 1 && n % 8 == 0 && ((uintptr_t)z % 16 == 0) && ((uintptr_t)out % 16 == 0))
        return dk_launch(xielu_wide_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, st, (const bf16*)z,
                         (bf16*)out, (size_t)(n / 8), ap, an);
    DISPATCH_T(dtype, return dk_launch(xielu_kernel<T>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, (const T*)z,
                                       (T*)out, (size_t)n, ap, an));
}

// ---------------------------------------------------------------------------------------------
// Norm after the sum: h[row] = rmsnorm(alpha * h[row] + delta[row]) * w, written back to the float32
// stream, and a[row] = the same in the storage type (what the next sublayer reads). delta as a tensor
// or as n_parts float32 partial sums. The sum, its mean square and the scaling are float32.
template <typename T>
__global__ void scale_add_rmsnorm_kernel(float* h, float alpha, const T* delta, const float* parts, int n_parts,
                                         size_t part_stride, const float* __restrict__ w, float eps, int H, T* a) {
    __shared__ float red[33];
    pdl_wait();
    pdl_launch_dependents();
    const size_t row = blockIdx.x;
    float* hr = h + row * H;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float d = delta ? to_f(delta[row * H + i]) : 0.f;
        for (int k = 0; k < n_parts; k++) d += parts[(size_t)k * part_stride + row * H + i];
        const float v = fmaf(alpha, hr[i], d);
        hr[i] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = 1.f / sqrtf(ss / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = hr[i] * rs * w[i];
        hr[i] = v;
        a[row * H + i] = from_f<T>(v);
    }
}

// The same in one pass for widths that are multiples of 4 up to 8,192: a thread keeps NV groups of 4 columns in
// registers between the sum of squares and the scaling, every load requested before any is used, the norm's weight
// before the wait for the kernel in front.
template <typename T, int NV>
__global__ void __launch_bounds__(256)
scale_add_rmsnorm_regs_kernel(float* h, float alpha, const T* delta, const float* parts, int n_parts, size_t part_stride,
                              const float* __restrict__ w, float eps, int H, T* a) {
    __shared__ float red[33];
    float4 wv[NV], v[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        wv[q] = c < H ? ld4(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    pdl_launch_dependents();
    const size_t row = blockIdx.x;
    float* hr = h + row * H;
    float4 d[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        v[q] = c < H ? ld4(hr + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        d[q] = (c < H && delta) ? ld4(delta + row * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int k = 0; k < n_parts; k++)
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const int c = (threadIdx.x + q * 256) * 4;
            if (c < H) {
                const float4 p = ld4(parts + (size_t)k * part_stride + row * H + c);
                d[q].x += p.x, d[q].y += p.y, d[q].z += p.z, d[q].w += p.w;
            }
        }
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        v[q].x = fmaf(alpha, v[q].x, d[q].x), v[q].y = fmaf(alpha, v[q].y, d[q].y);
        v[q].z = fmaf(alpha, v[q].z, d[q].z), v[q].w = fmaf(alpha, v[q].w, d[q].w);
        ss += v[q].x * v[q].x + v[q].y * v[q].y + v[q].z * v[q].z + v[q].w * v[q].w;
    }
    ss = block_sum(ss, red);
    const float rs = 1.f / sqrtf(ss / (float)H + eps);
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        if (c < H) {
            const float4 o = make_float4(v[q].x * rs * wv[q].x, v[q].y * rs * wv[q].y, v[q].z * rs * wv[q].z, v[q].w * rs * wv[q].w);
            st4(hr + c, o);
            st4(a + row * H + c, o);
        }
    }
}

DK_EXPORT int dk_scale_add_rmsnorm(int dtype, float* h, float alpha, const void* delta, const float* parts, int n_parts,
                                   long long part_stride, const float* w, float eps, int n_rows, int H, void* a,
                                   cudaStream_t st) {
    if (H % 4 == 0 && H <= 8192 && part_stride % 4 == 0) {
#define SAN_REGS(NV)                                                                                                      \
    if (H <= 1024 * NV) {                                                                                                 \
        DISPATCH_T(dtype, return dk_launch(scale_add_rmsnorm_regs_kernel<T, NV>, dim3(n_rows), dim3(256), 0, st, h, alpha, \
                                           (const T*)delta, parts, n_parts, (size_t)part_stride, w, eps, H, (T*)a));      \
    }
        SAN_REGS(1) SAN_REGS(2) SAN_REGS(3) SAN_REGS(4) SAN_REGS(6) SAN_REGS(8)
#undef SAN_REGS
    }
    DISPATCH_T(dtype, return dk_launch(scale_add_rmsnorm_kernel<T>, dim3(n_rows), dim3(row_threads(H)), 0, st, h, alpha,
                                       (const T*)delta, parts, n_parts, (size_t)part_stride, w, eps, H, (T*)a));
}

// ---------------------------------------------------------------------------------------------
// A sublayer's output normed before it joins the stream, and the next norm behind the sum:
//   h[row] += rmsnorm(delta[row]) * wb (eps_b);   a[out_row] = rmsnorm(h[row]) * w (eps).
// delta as a tensor or as n_parts float32 partial sums. With `rows` the kernel gathers (out_row = blockIdx.x,
// row = rows[blockIdx.x]) and leaves h as it is. Sums, mean squares and scalings are float32.
// The generic form keeps the row in shared memory (H floats); any width.
template <typename T>
__global__ void normed_add_rmsnorm_kernel(float* h, const T* delta, const float* parts, int n_parts, size_t part_stride,
                                          const int* rows, const float* __restrict__ wb, float eps_b,
                                          const float* __restrict__ w, float eps, int H, T* a) {
    __shared__ float red[33];
    extern __shared__ float vals[];
    pdl_wait();
    pdl_launch_dependents();
    const size_t out_row = blockIdx.x;
    const size_t row = rows ? (size_t)rows[out_row] : out_row;
    float* hr = h + row * H;
    float ssd = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float d = delta ? to_f(delta[row * H + i]) : 0.f;
        for (int k = 0; k < n_parts; k++) d += parts[(size_t)k * part_stride + row * H + i];
        vals[i] = d;
        ssd += d * d;
    }
    ssd = block_sum(ssd, red);
    const float rd = 1.f / sqrtf(ssd / (float)H + eps_b);
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = hr[i] + vals[i] * rd * wb[i];
        vals[i] = v;
        if (!rows) hr[i] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = 1.f / sqrtf(ss / (float)H + eps);
    T* ar = a + out_row * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) ar[i] = from_f<T>(vals[i] * rs * w[i]);
}

// The same in one pass for widths that are multiples of 4 up to 8,192: NV groups of 4 columns a thread stay in
// registers between the two sums of squares and the scaling; both weights are fetched before the wait.
template <typename T, int NV>
__global__ void __launch_bounds__(256)
normed_add_rmsnorm_regs_kernel(float* h, const T* delta, const float* parts, int n_parts, size_t part_stride,
                               const int* rows, const float* __restrict__ wb, float eps_b, const float* __restrict__ w,
                               float eps, int H, T* a) {
    __shared__ float red[33];
    float4 wv[NV], wbv[NV], v[NV], d[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        wv[q] = c < H ? ld4(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        wbv[q] = c < H ? ld4(wb + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    pdl_launch_dependents();
    const size_t out_row = blockIdx.x;
    const size_t row = rows ? (size_t)rows[out_row] : out_row;
    float* hr = h + row * H;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        v[q] = c < H ? ld4(hr + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        d[q] = (c < H && delta) ? ld4(delta + row * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int k = 0; k < n_parts; k++)
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const int c = (threadIdx.x + q * 256) * 4;
            if (c < H) {
                const float4 p = ld4(parts + (size_t)k * part_stride + row * H + c);
                d[q].x += p.x, d[q].y += p.y, d[q].z += p.z, d[q].w += p.w;
            }
        }
    float ssd = 0.f;
#pragma unroll
    for (int q = 0; q < NV; q++) ssd += d[q].x * d[q].x + d[q].y * d[q].y + d[q].z * d[q].z + d[q].w * d[q].w;
    ssd = block_sum(ssd, red);
    const float rd = 1.f / sqrtf(ssd / (float)H + eps_b);
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        v[q].x += d[q].x * rd * wbv[q].x, v[q].y += d[q].y * rd * wbv[q].y;
        v[q].z += d[q].z * rd * wbv[q].z, v[q].w += d[q].w * rd * wbv[q].w;
        ss += v[q].x * v[q].x + v[q].y * v[q].y + v[q].z * v[q].z + v[q].w * v[q].w;
    }
    ss = block_sum(ss, red);
    const float rs = 1.f / sqrtf(ss / (float)H + eps);
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const int c = (threadIdx.x + q * 256) * 4;
        if (c < H) {
            if (!rows) st4(hr + c, v[q]);
            st4(a + out_row * H + c, make_float4(v[q].x * rs * wv[q].x, v[q].y * rs * wv[q].y, v[q].z * rs * wv[q].z,
                                                 v[q].w * rs * wv[q].w));
        }
    }
}

DK_EXPORT int dk_normed_add_rmsnorm(int dtype, float* h, const void* delta, const float* parts, int n_parts,
                                    long long part_stride, const int* rows, const float* wb, float eps_b, const float* w,
                                    float eps, int n_rows, int H, void* a, cudaStream_t st) {
    if (H % 4 == 0 && H <= 8192 && part_stride % 4 == 0) {
#define NAN_REGS(NV)                                                                                                       \
    if (H <= 1024 * NV) {                                                                                                  \
        DISPATCH_T(dtype, return dk_launch(normed_add_rmsnorm_regs_kernel<T, NV>, dim3(n_rows), dim3(256), 0, st, h,       \
                                           (const T*)delta, parts, n_parts, (size_t)part_stride, rows, wb, eps_b, w, eps,  \
                                           H, (T*)a));                                                                     \
    }
        NAN_REGS(1) NAN_REGS(2) NAN_REGS(3) NAN_REGS(4) NAN_REGS(6) NAN_REGS(8)
#undef NAN_REGS
    }
    const size_t smem = (size_t)H * sizeof(float);
    if (smem > 48 * 1024) {
        DISPATCH_T(dtype, cudaFuncSetAttribute(normed_add_rmsnorm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem));
    }
    DISPATCH_T(dtype, return dk_launch(normed_add_rmsnorm_kernel<T>, dim3(n_rows), dim3(row_threads(H)), smem, st, h,
                                       (const T*)delta, parts, n_parts, (size_t)part_stride, rows, wb, eps_b, w, eps, H,
                                       (T*)a));
}

// a[row] = h[row] in the storage type (the stream as a sublayer's input, where no kernel before left it).
template <typename T>
__global__ void cast_rows_kernel(const float* h, T* a, size_t n) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = from_f<T>(h[i]);
}

DK_EXPORT int dk_cast_rows(int dtype, const float* h, void* a, long long n, cudaStream_t st) {
    DISPATCH_T(dtype, return dk_launch(cast_rows_kernel<T>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, h, (T*)a,
                                       (size_t)n));
}

// out[r, c] = act(gu[r, c]) * gu[r, I + c] for rows [gate | up]; act 0: SiLU, 1: the tanh form of GELU,
// 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))); 2: with g' = min(g, limit) and u' = clamp(u, -limit, limit),
// g' sigmoid(1.702 g') (u' + 1). Arithmetic in float32.
__device__ __forceinline__ float gelu_tanh_f(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
template <typename T>
__global__ void act_mul_kernel(const T* gu, T* out, size_t n, int I, int act, float limit) {
    pdl_wait();
    pdl_launch_dependents();
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    size_t r = idx / I, c = idx % I;
    float g = to_f(gu[r * 2 * I + c]);
    float u = to_f(gu[r * 2 * I + I + c]);
    if (act == 2) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        out[idx] = from_f<T>(g / (1.f + expf(-1.702f * g)) * (u + 1.f));
        return;
    }
    out[idx] = from_f<T>((act == 1 ? gelu_tanh_f(g) : g / (1.f + expf(-g))) * u);
}

DK_EXPORT int dk_act_mul(int dtype, const void* gu, void* out, long long n_rows, int I, int act, float limit, cudaStream_t st) {
    size_t n = (size_t)n_rows * I;
    DISPATCH_T(dtype, return dk_launch(act_mul_kernel<T>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st,
                                       (const T*)gu, (T*)out, n, I, act, limit));
}
