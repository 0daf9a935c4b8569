// Attention of the prompt path: causal grouped-query attention of a long run of consecutive tokens on the tensor cores, in FP32 precision.
//
// Two kernels. rope_split_kernel rotates queries and keys (ops/Rope.java:125-149), appends keys and values to the FP32 cache, and writes every
// row of hd values that the attention reads as two halves, hi + lo (22 significant bits), times a power of two of its own (exact).
// prompt_attention_kernel multiplies those with mma.sync.m16n8k16, three products for one (hi.hi + hi.lo + lo.hi), FP32 accumulation, and
// streaming softmax in FP32 (ops/FlashAttention.java:538-626 of the reference), and writes its result rounded to bfloat16, which is what
// the linear behind it takes.
//
// Why: with FP32 arithmetic on the CUDA cores this took 300 us a layer for 512 tokens of 32 heads, more than the layer's linears; the rotation,
// with two values per thread, another 53. Bound now by the issue of mma.sync: 384 for 16 queries x 64 keys at head size 128.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "jq_prompt.cuh"

namespace jq {

namespace {

// The largest magnitude of a row goes to [2^9, 2^10): the lo halves of values down to 2^-13 of it stay normal numbers.
__device__ __forceinline__ void row_scale(float amax, float& up, float& down) {
    uint32_t e = __float_as_uint(amax) >> 23;
    const bool bad = e == 255u;  // a NaN or an Inf: the row's scale becomes NaN and reaches every result that uses it (its halves are zeros)
    e = e < 20u ? 20u : (e > 250u ? 250u : e);
    up = __uint_as_float((263u - e) << 23);
    down = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((e - 9u) << 23);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

// One warp per row of HD values: queries [token][head], then keys and values [kv head][key], keys up to a multiple of 64 (zeros beyond).
template <int HD>
__global__ void __launch_bounds__(256) rope_split_kernel(PromptAttention p) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int HALF = HD / 2, N = HD / 64;  // a lane has N neighbouring values of either half
    const int lane = threadIdx.x & 31;
    const int keys = p.pos0 + p.T;
    int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int64_t q_rows = (int64_t)p.T * p.heads, k_rows = (int64_t)p.kv_heads * p.keys_pad;
    const float* src = nullptr;
    float* cache = nullptr;
    __half* hi;
    __half* lo;
    float* scale;
    int pos = -1;  // where to rotate
    float factor = 1.0f;
    const int kv_dim = p.kv_heads * HD;
    if (row < q_rows) {
        src = p.q + row * HD;
        pos = p.pos0 + (int)(row / p.heads);
        hi = p.qh + row * HD;
        lo = p.ql + row * HD;
        scale = p.qs + row;
        factor = p.scale;
    } else {
        row -= q_rows;
        const bool is_v = row >= k_rows;
        row -= is_v ? k_rows : 0;
        if (row >= k_rows) {
            return;
        }
        const int kvh = (int)(row / p.keys_pad), key = (int)(row % p.keys_pad);
        float* const c = (is_v ? p.v_cache : p.k_cache) + (int64_t)key * kv_dim + kvh * HD;
        if (key >= p.pos0 && key < keys) {
            src = (is_v ? p.v : p.k) + (int64_t)(key - p.pos0) * kv_dim + kvh * HD;
            cache = c;
            pos = is_v ? -1 : key;
        } else if (key < p.pos0) {
            src = c;
        }
        hi = (is_v ? p.vh : p.kh) + row * HD;
        lo = (is_v ? p.vl : p.kl) + row * HD;
        scale = (is_v ? p.vs : p.ks) + row;
    }
    float a[N], b[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        a[i] = src != nullptr ? src[lane * N + i] : 0.0f;
        b[i] = src != nullptr ? src[HALF + lane * N + i] : 0.0f;
    }
    if (pos >= 0) {
#pragma unroll
        for (int i = 0; i < N; i++) {
            const float c = p.cos_t[pos * HALF + lane * N + i], s = p.sin_t[pos * HALF + lane * N + i];
            const float r0 = a[i] * c - b[i] * s, r1 = a[i] * s + b[i] * c;
            a[i] = r0;
            b[i] = r1;
        }
    }
    uint32_t am = 0;  // magnitudes as bits: a NaN is larger than any number
#pragma unroll
    for (int i = 0; i < N; i++) {
        am = max(am, max(__float_as_uint(a[i]) & 0x7fffffffu, __float_as_uint(b[i]) & 0x7fffffffu));
        if (cache != nullptr) {
            cache[lane * N + i] = a[i];
            cache[HALF + lane * N + i] = b[i];
        }
    }
    am = __reduce_max_sync(0xffffffffu, am);
    float up, down;
    row_scale(__uint_as_float(am), up, down);
    if (am >= 0x7f800000u) {  // the scale says it: a NaN among the halves of a value row would reach queries that do not see the key, as 0 x NaN
#pragma unroll
        for (int i = 0; i < N; i++) {
            a[i] = b[i] = 0.0f;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        __half hv[N], lv[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const float v = (h == 0 ? a[i] : b[i]) * up;
            hv[i] = __float2half_rn(v);
            lv[i] = __float2half_rn(v - __half2float(hv[i]));
        }
        const int at = h * HALF + lane * N;
        if constexpr (N == 2) {
            *reinterpret_cast<__half2*>(hi + at) = __halves2half2(hv[0], hv[1]);
            *reinterpret_cast<__half2*>(lo + at) = __halves2half2(lv[0], lv[1]);
        } else {
            hi[at] = hv[0];
            lo[at] = lv[0];
        }
    }
    if (lane == 0) {
        *scale = src != nullptr ? down * factor : 0.0f;
    }
}

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void hmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

constexpr int QT = 64, KT = 64, THREADS = 128;  // queries and keys per tile; a warp has 16 queries

template <int HD>
constexpr size_t attention_smem() {
    return (size_t)4 * KT * HD * 2 + 2 * KT * 4;
}

// CTA = (64 queries, head), the tiles with the most keys first. 64 queries rather than 128: two CTAs share an SM, a long tile beside a short one.
// Keys and values are single-buffered, each loaded while the other is used.
template <int HD>
__global__ void __launch_bounds__(THREADS, 2) prompt_attention_kernel(PromptAttention p) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int ROW = HD * 2, CH = HD / 8;  // bytes and 16-byte pieces per row; pieces are swizzled by (row & 7)
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t kh_s = s0, kl_s = s0 + KT * ROW, vh_s = s0 + 2 * KT * ROW, vl_s = s0 + 3 * KT * ROW;
    float* const ks_s = reinterpret_cast<float*>(smem + 4 * KT * ROW);
    float* const vs_s = ks_s + KT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.x, kvh = h / (p.heads / p.kv_heads);
    const int t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * QT;  // longest first
    const int last = p.pos0 + (t0 + QT < p.T ? t0 + QT : p.T) - 1;  // the last key any query of the tile sees
    const int tiles = last / KT + 1;
    const __half* const kh = p.kh + (int64_t)kvh * p.keys_pad * HD;
    const __half* const kl = p.kl + (int64_t)kvh * p.keys_pad * HD;
    const __half* const vh = p.vh + (int64_t)kvh * p.keys_pad * HD;
    const __half* const vl = p.vl + (int64_t)kvh * p.keys_pad * HD;
    auto load = [&](const __half* a, const __half* b, const float* sc, uint32_t da, uint32_t db, float* ds, int tile) {
        const int64_t at = (int64_t)tile * KT * HD;
#pragma unroll 4
        for (int i = tid; i < KT * CH; i += THREADS) {
            const int r = i / CH, c = i % CH;
            const uint32_t to = (uint32_t)(r * ROW + (((c & ~7) | ((c ^ r) & 7)) << 4));
            cp16(da + to, a + at + i * 8);
            cp16(db + to, b + at + i * 8);
        }
        if (tid < KT / 4) {
            cp16((uint32_t)__cvta_generic_to_shared(ds + tid * 4), sc + (int64_t)kvh * p.keys_pad + tile * KT + tid * 4);
        }
        cp_commit();
    };
    load(kh, kl, p.ks, kh_s, kl_s, ks_s, 0);
    load(vh, vl, p.vs, vh_s, vl_s, vs_s, 0);
    // this warp's queries as A fragments: rows g and g + 8
    const int r0 = t0 + warp * 16 + g, r1 = r0 + 8;
    uint32_t qa[HD / 16][4], qb[HD / 16][4];
    {
        const int64_t o0 = ((int64_t)(r0 < p.T ? r0 : 0) * p.heads + h) * HD, o1 = ((int64_t)(r1 < p.T ? r1 : 0) * p.heads + h) * HD;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ks++) {
            const int c = ks * 16 + 2 * t;
            qa[ks][0] = *reinterpret_cast<const uint32_t*>(p.qh + o0 + c);
            qa[ks][1] = *reinterpret_cast<const uint32_t*>(p.qh + o1 + c);
            qa[ks][2] = *reinterpret_cast<const uint32_t*>(p.qh + o0 + c + 8);
            qa[ks][3] = *reinterpret_cast<const uint32_t*>(p.qh + o1 + c + 8);
            qb[ks][0] = *reinterpret_cast<const uint32_t*>(p.ql + o0 + c);
            qb[ks][1] = *reinterpret_cast<const uint32_t*>(p.ql + o1 + c);
            qb[ks][2] = *reinterpret_cast<const uint32_t*>(p.ql + o0 + c + 8);
            qb[ks][3] = *reinterpret_cast<const uint32_t*>(p.ql + o1 + c + 8);
        }
    }
    const float sq0 = p.qs[(int64_t)(r0 < p.T ? r0 : 0) * p.heads + h], sq1 = p.qs[(int64_t)(r1 < p.T ? r1 : 0) * p.heads + h];
    float acc[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; i++) {
        acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    float vmax0 = 7.8886091e-31f, vmax1 = vmax0;  // 2^-100; a query's acc is in units of this power of two, the largest scale of the values it has seen
    // ldmatrix rows: K fragments of 16 keys (two n-blocks) x 16 d; V fragments of 16 keys x 16 d (transposed)
    const int k_row = (lane & 7) + ((lane >> 4) << 3), k_ch = (lane >> 3) & 1;
    const int v_row = (lane & 7) + (((lane >> 3) & 1) << 3), v_ch = lane >> 4;
    for (int tile = 0; tile < tiles; tile++) {
        cp_wait<1>();
        __syncthreads();
        // ---- scores
        float s[KT / 8][4];
#pragma unroll
        for (int nb = 0; nb < KT / 16; nb++) {
            s[2 * nb][0] = s[2 * nb][1] = s[2 * nb][2] = s[2 * nb][3] = 0.0f;
            s[2 * nb + 1][0] = s[2 * nb + 1][1] = s[2 * nb + 1][2] = s[2 * nb + 1][3] = 0.0f;
            const int row = nb * 16 + k_row;
#pragma unroll
            for (int ks = 0; ks < HD / 16; ks++) {
                const int c = 2 * ks + k_ch;
                const uint32_t at = (uint32_t)(row * ROW + (((c & ~7) | ((c ^ row) & 7)) << 4));
                uint32_t bh[4], bl[4];
                ldm4(bh, kh_s + at);
                ldm4(bl, kl_s + at);
                hmma(s[2 * nb], qa[ks], bh[0], bh[1]);
                hmma(s[2 * nb + 1], qa[ks], bh[2], bh[3]);
                hmma(s[2 * nb], qa[ks], bl[0], bl[1]);
                hmma(s[2 * nb + 1], qa[ks], bl[2], bl[3]);
                hmma(s[2 * nb], qb[ks], bh[0], bh[1]);
                hmma(s[2 * nb + 1], qb[ks], bh[2], bh[3]);
            }
        }
        const int key0 = tile * KT;
        const bool edge = key0 + KT - 1 > p.pos0 + t0 + warp * 16;  // some query of this warp does not see all of the tile's keys
        float x0 = m0, x1 = m1;
#pragma unroll
        for (int nb = 0; nb < KT / 8; nb++) {
            const float2 sk = *reinterpret_cast<const float2*>(ks_s + nb * 8 + 2 * t);
            s[nb][0] *= sq0 * sk.x; s[nb][1] *= sq0 * sk.y;
            s[nb][2] *= sq1 * sk.x; s[nb][3] *= sq1 * sk.y;
            if (edge) {
                const int key = key0 + nb * 8 + 2 * t;
                s[nb][0] = key <= p.pos0 + r0 ? s[nb][0] : -INFINITY;
                s[nb][1] = key + 1 <= p.pos0 + r0 ? s[nb][1] : -INFINITY;
                s[nb][2] = key <= p.pos0 + r1 ? s[nb][2] : -INFINITY;
                s[nb][3] = key + 1 <= p.pos0 + r1 ? s[nb][3] : -INFINITY;
            }
            x0 = fmaxf(x0, fmaxf(s[nb][0], s[nb][1]));
            x1 = fmaxf(x1, fmaxf(s[nb][2], s[nb][3]));
        }
        __syncthreads();  // every warp is done with the keys
        if (tile + 1 < tiles) {
            load(kh, kl, p.ks, kh_s, kl_s, ks_s, tile + 1);
        } else {
            cp_commit();
        }
        // ---- softmax statistics: a row's columns sit in the four lanes of a quad
        x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
        x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
        // (no key of a later tile seen yet cannot happen: key 0 is in the first tile and every query sees it)
        const float al0 = expf(m0 - x0), al1 = expf(m1 - x1);
        m0 = x0;
        m1 = x1;
        l0 *= al0;
        l1 *= al1;
        cp_wait<1>();
        __syncthreads();  // the tile's values are here
        // every value row has a scale of its own, which goes into the weights, relative to the largest one that the query has seen so far
        float vm0 = vmax0, vm1 = vmax1;
        if (!edge) {
            const float vm = warp_max(fmaxf(vs_s[lane], vs_s[lane + 32]));
            vm0 = fmaxf(vm0, vm);
            vm1 = fmaxf(vm1, vm);
        } else {
#pragma unroll
            for (int nb = 0; nb < KT / 8; nb++) {
                const float2 sv = *reinterpret_cast<const float2*>(vs_s + nb * 8 + 2 * t);
                const int key = key0 + nb * 8 + 2 * t;
                vm0 = fmaxf(vm0, fmaxf(key <= p.pos0 + r0 ? sv.x : 0.0f, key + 1 <= p.pos0 + r0 ? sv.y : 0.0f));
                vm1 = fmaxf(vm1, fmaxf(key <= p.pos0 + r1 ? sv.x : 0.0f, key + 1 <= p.pos0 + r1 ? sv.y : 0.0f));
            }
            vm0 = fmaxf(vm0, __shfl_xor_sync(0xffffffffu, vm0, 1));
            vm0 = fmaxf(vm0, __shfl_xor_sync(0xffffffffu, vm0, 2));
            vm1 = fmaxf(vm1, __shfl_xor_sync(0xffffffffu, vm1, 1));
            vm1 = fmaxf(vm1, __shfl_xor_sync(0xffffffffu, vm1, 2));
        }
        const float inv0 = 1024.0f / vm0, inv1 = 1024.0f / vm1;  // powers of two; weights of up to 2^10
        const float b0 = al0 * (vmax0 / vm0), b1 = al1 * (vmax1 / vm1);
        vmax0 = vm0;
        vmax1 = vm1;
#pragma unroll
        for (int i = 0; i < HD / 8; i++) {
            acc[i][0] *= b0; acc[i][1] *= b0;
            acc[i][2] *= b1; acc[i][3] *= b1;
        }
#pragma unroll
        for (int kb = 0; kb < KT / 16; kb++) {
            uint32_t pa[4], pb[4];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                float(&e)[4] = s[2 * kb + j];
                const float2 sv = *reinterpret_cast<const float2*>(vs_s + kb * 16 + j * 8 + 2 * t);
                e[0] = expf(e[0] - m0); e[1] = expf(e[1] - m0);
                e[2] = expf(e[2] - m1); e[3] = expf(e[3] - m1);
                l0 += e[0] + e[1];
                l1 += e[2] + e[3];
                e[0] *= sv.x * inv0; e[1] *= sv.y * inv0;
                e[2] *= sv.x * inv1; e[3] *= sv.y * inv1;
                if (edge) {  // a key that the query does not see has the weight zero, and its scale may be a NaN
                    const int key = key0 + kb * 16 + j * 8 + 2 * t;
                    e[0] = key <= p.pos0 + r0 ? e[0] : 0.0f;
                    e[1] = key + 1 <= p.pos0 + r0 ? e[1] : 0.0f;
                    e[2] = key <= p.pos0 + r1 ? e[2] : 0.0f;
                    e[3] = key + 1 <= p.pos0 + r1 ? e[3] : 0.0f;
                }
                split2(e[0], e[1], pa[2 * j], pb[2 * j]);
                split2(e[2], e[3], pa[2 * j + 1], pb[2 * j + 1]);
            }
            const int row = kb * 16 + v_row;
#pragma unroll
            for (int db = 0; db < HD / 16; db++) {
                const int c = 2 * db + v_ch;
                const uint32_t at = (uint32_t)(row * ROW + (((c & ~7) | ((c ^ row) & 7)) << 4));
                uint32_t bh[4], bl[4];
                ldm4t(bh, vh_s + at);
                ldm4t(bl, vl_s + at);
                hmma(acc[2 * db], pa, bh[0], bh[1]);
                hmma(acc[2 * db + 1], pa, bh[2], bh[3]);
                hmma(acc[2 * db], pa, bl[0], bl[1]);
                hmma(acc[2 * db + 1], pa, bl[2], bl[3]);
                hmma(acc[2 * db], pb, bh[0], bh[1]);
                hmma(acc[2 * db + 1], pb, bh[2], bh[3]);
            }
        }
        __syncthreads();  // every warp is done with the values
        if (tile + 1 < tiles) {
            load(vh, vl, p.vs, vh_s, vl_s, vs_s, tile + 1);
        } else {
            cp_commit();
        }
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float f0 = vmax0 * 0.0009765625f / l0, f1 = vmax1 * 0.0009765625f / l1;
    __nv_bfloat16* const o0 = p.out + ((int64_t)r0 * p.heads + h) * HD + 2 * t;
    __nv_bfloat16* const o1 = p.out + ((int64_t)r1 * p.heads + h) * HD + 2 * t;
#pragma unroll
    for (int i = 0; i < HD / 8; i++) {
        if (r0 < p.T) {
            *reinterpret_cast<__nv_bfloat162*>(o0 + i * 8) = __floats2bfloat162_rn(acc[i][0] * f0, acc[i][1] * f0);
        }
        if (r1 < p.T) {
            *reinterpret_cast<__nv_bfloat162*>(o1 + i * 8) = __floats2bfloat162_rn(acc[i][2] * f1, acc[i][3] * f1);
        }
    }
}

template <int HD>
int run(const PromptAttention& p, cudaStream_t s) {
    static std::atomic<uint64_t> configured{0};  // the opt-in for large dynamic shared memory is per device
    int dev = 0;
    JQ_CUDA(cudaGetDevice(&dev));
    if ((configured.load(std::memory_order_relaxed) >> (dev & 63) & 1) == 0) {
        JQ_CUDA(cudaFuncSetAttribute(prompt_attention_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attention_smem<HD>()));
        configured.fetch_or((uint64_t)1 << (dev & 63));
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = s;
    const int64_t rows = (int64_t)p.T * p.heads + 2 * (int64_t)p.kv_heads * p.keys_pad;
    cfg.gridDim = dim3((unsigned)((rows + 7) / 8));
    cfg.blockDim = dim3(256);
    JQ_CUDA(cudaLaunchKernelEx(&cfg, rope_split_kernel<HD>, p));
    count_launch();
    cfg.gridDim = dim3((unsigned)p.heads, (unsigned)((p.T + QT - 1) / QT));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = attention_smem<HD>();
    JQ_CUDA(cudaLaunchKernelEx(&cfg, prompt_attention_kernel<HD>, p));
    count_launch();
    return JQ_OK;
}

}  // namespace

size_t prompt_attention_bytes(int T, int keys, int heads, int kv_heads, int hd) {
    const size_t pad = (size_t)(keys + KT - 1) / KT * KT;
    return ((size_t)T * heads + 2 * (size_t)kv_heads * pad) * ((size_t)hd * 4 + 4) + 8 * 256;
}

void prompt_attention_layout(PromptAttention& p, uint8_t* scratch, int hd) {
    p.keys_pad = (p.pos0 + p.T + KT - 1) / KT * KT;
    const size_t q = (size_t)p.T * p.heads, k = (size_t)p.kv_heads * p.keys_pad;
    auto take = [&](size_t bytes) {
        uint8_t* at = scratch;
        scratch += (bytes + 255) / 256 * 256;
        return at;
    };
    p.qh = reinterpret_cast<__half*>(take(q * hd * 2));
    p.ql = reinterpret_cast<__half*>(take(q * hd * 2));
    p.kh = reinterpret_cast<__half*>(take(k * hd * 2));
    p.kl = reinterpret_cast<__half*>(take(k * hd * 2));
    p.vh = reinterpret_cast<__half*>(take(k * hd * 2));
    p.vl = reinterpret_cast<__half*>(take(k * hd * 2));
    p.qs = reinterpret_cast<float*>(take(q * 4));
    p.ks = reinterpret_cast<float*>(take(k * 4));
    p.vs = reinterpret_cast<float*>(take(k * 4));
}

int launch_prompt_attention(const PromptAttention& p, int hd, cudaStream_t s) { return hd == 128 ? run<128>(p, s) : run<64>(p, s); }

}  // namespace jq
