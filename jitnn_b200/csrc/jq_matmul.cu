// Host side of the matrix kernel (jq_matmul.cuh): the split of FP32 activations, the choice of tiles, the launches.
#include <cuda_bf16.h>

#include <cstring>
#include <memory>
#include <mutex>

#include "jq_matmul_launch.cuh"

namespace jq {

namespace mm {

// x [m, k] FP32 (or silu(x) * up) -> two planes of halves [2][m][width] (hi, lo) and a scale per (BLK values of k, row of x): the block's values times a power of
// two that brings the largest to [2^9, 2^10), hi = that rounded to half precision, lo = the rest rounded to half precision: 22
// significant bits for everything down to 2^-13 of the largest. A block that holds a NaN or an Inf gets the scale NaN, which reaches
// every output of that row. One warp per 256 values of a row; memory bound (8 bytes moved per value, 4 of them to L2).
// EXT: 16 more columns follow every 256, the sums over the eight runs of 32 values, twice (hi plane: their hi parts, lo plane: their lo
// parts).
template <int BLK, bool EXT>
__global__ void __launch_bounds__(256) split_kernel(const float* x, const float* up, int m, int64_t k, int per_row, uint4* __restrict__ planes,
                                                    float* __restrict__ scales, int stride, int vec) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t task = (int64_t)blockIdx.x * 8 + warp;
    const int row = (int)(task / per_row), b = (int)(task - (int64_t)row * per_row);
    if (row >= m) {
        return;
    }
    const int64_t i0 = (int64_t)b * 256 + lane * 8;
    const float* src = x + (int64_t)row * k + i0;
    float v[8];
    if (vec && i0 + 8 <= k) {
        const float4 a = *reinterpret_cast<const float4*>(src), c = *(reinterpret_cast<const float4*>(src) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = i0 + i < k ? src[i] : 0.0f;
        }
    }
    if (up != nullptr) {  // x is the gate of a feed-forward block
        const float* us = up + (src - x);
        float u[8];
        if (vec && i0 + 8 <= k) {
            const float4 a = *reinterpret_cast<const float4*>(us), c = *(reinterpret_cast<const float4*>(us) + 1);
            u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w;
            u[4] = c.x; u[5] = c.y; u[6] = c.z; u[7] = c.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                u[i] = i0 + i < k ? us[i] : 0.0f;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = (v[i] / (1.0f + expf(-v[i]))) * u[i];
        }
    }
    uint32_t am = 0;  // the largest magnitude as bits: an Inf or a NaN is larger than any number
#pragma unroll
    for (int i = 0; i < 8; i++) {
        am = max(am, __float_as_uint(v[i]) & 0x7fffffffu);
    }
#pragma unroll
    for (int o = BLK / 16; o > 0; o >>= 1) {
        am = max(am, __shfl_xor_sync(0xffffffffu, am, o));
    }
    const bool bad = am >= 0x7f800000u;
    uint32_t e = am >> 23;
    e = e < 14u ? 14u : (e > 254u ? 254u : e);
    const float f = __uint_as_float((263u - e) << 23);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        split_pair(v[2 * i] * f, v[2 * i + 1] * f, hi[i], lo[i]);
    }
    constexpr int BLOCK = EXT ? 272 : 256;
    const int64_t row_at = ((int64_t)row * per_row + b) * BLOCK, at = (row_at >> 3) + lane, plane = ((int64_t)m * per_row * BLOCK) >> 3;
    planes[at] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    planes[at + plane] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    if constexpr (EXT) {
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&hi[i])), c = __half22float2(*reinterpret_cast<const __half2*>(&lo[i]));
            sum += (a.x + c.x) + (a.y + c.y);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const __half h = __float2half_rn(sum), l = __float2half_rn(sum - __half2float(h));
        if ((lane & 3) == 0) {  // sums of up to 2^15
            __half* to = reinterpret_cast<__half*>(planes) + row_at + 256 + (lane >> 2);
            to[0] = h;
            to[8] = h;
            to[plane * 8] = l;
            to[plane * 8 + 8] = l;
        }
    }
    if ((lane & (BLK / 8 - 1)) == 0) {
        scales[(int64_t)(i0 / BLK) * stride + row] = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((e - 9u) << 23);
    }
}

static long long wait_clocks() { return (long long)g_opt_wait_limit_us.load(std::memory_order_relaxed) * 2000; }  // about 2 GHz

static int unit_bytes(int type) { return TILE_ROWS * (plane_q_bytes(type) + plane_aux_bytes(type)) * 256 / block_values(type); }

static Facts facts(int type, bool fp32, bool bwd, int nmax) {
    switch (type) {
        case JQ_TYPE_Q4_K: return facts_format<JQ_TYPE_Q4_K>(fp32, bwd, nmax);
        case JQ_TYPE_Q5_K: return facts_format<JQ_TYPE_Q5_K>(fp32, bwd, nmax);
        case JQ_TYPE_Q6_K: return facts_format<JQ_TYPE_Q6_K>(fp32, bwd, nmax);
        case JQ_TYPE_Q8_0: return facts_format<JQ_TYPE_Q8_0>(fp32, bwd, nmax);
        case JQ_TYPE_Q4_0: return facts_format<JQ_TYPE_Q4_0>(fp32, bwd, nmax);
        default: return facts_format<JQ_TYPE_Q4_1>(fp32, bwd, nmax);
    }
}

// Ring depths for a tile of nt rows of x: at least as many weight operands as there are groups of dequantiser warps, two activation entries and
// two raw units (or one per group); then the activations' ring grows first. False if not even those fit.
static bool configure(int type, bool fp32, bool bwd, int nt, int ksplit, Args& a, Plan& plan) {
    plan.fp32 = fp32;
    plan.bwd = bwd;
    plan.nmax = !fp32 ? (nt <= 128 ? 128 : 256) : (nt <= 32 ? 32 : 128);
    a.nt = nt;
    a.ksplit = ksplit;
    const Facts f = facts(type, fp32, bwd, plan.nmax);
    const int at = a_bytes(bwd), bt = f.b_tiles * tile_bytes(fp32, nt), rb = unit_bytes(type), tail = TAIL_BYTES + f.scales, room = 227 * 1024 - 1024 - tail;
    // tensor memory: as many accumulators as fit beside the groups' operands; operands behind them
    a.cols = f.columns * nt;
    a.bufs = fp32 ? MAX_BUFS : 2;
    while (a.bufs > 1 && a.bufs * a.cols + f.operands * f.a_cols > 512) {
        a.bufs--;
    }
    if (f.paired && a.bufs < 2) {
        return false;  // (two parts and the 16 more columns: tiles of up to 112 rows)
    }
    int max_a = 4;
    if (!bwd) {
        max_a = (512 - a.bufs * a.cols) / f.a_cols;
        max_a = max_a > MAX_A ? MAX_A : max_a;
    }
    const int raw_step = f.owned ? f.groups : 1;
    a.sa = bwd ? f.groups : max_a;
    a.sb = 2;
    a.raw = f.owned ? f.groups : 2;
    int left = room - a.sa * at - a.sb * bt - a.raw * rb;
    if (left < 0 || a.sa < f.groups) {
        return false;
    }
    auto grow = [&](int& depth, int most, int bytes, int step) {
        while (depth + step <= most && left >= bytes * step) {
            depth += step;
            left -= bytes * step;
        }
    };
    grow(a.sb, bwd ? 3 : (f.b_tiles > 1 ? 3 : 6), bt, 1);
    if (at > 0) {
        grow(a.sa, max_a, at, 1);
    }
    grow(a.raw, f.owned ? MAX_RAW : 3, rb, raw_step);
    grow(a.sb, f.b_tiles > 1 ? 6 : MAX_B, bt, 1);
    grow(a.raw, f.owned ? MAX_RAW : 4, rb, raw_step);
    a.tmem = 32;
    while (a.tmem < a.bufs * a.cols + (bwd ? 0 : a.sa * f.a_cols)) {
        a.tmem *= 2;
    }
    plan.smem = (size_t)(room - left) + tail + 1024;
    return true;
}

// What one unit of the contraction takes a CTA in nanoseconds, by the tile's width (measured on long contractions): the dequantiser warps and
// the barriers between the roles up to a width, the tensor pipe beyond it.
static double unit_ns(int type, bool fp32, bool bwd, int nt) {
    if (bwd) {
        return nt < 64 ? 1040.0 : 570.0 + 8.6 * nt;
    }
    if (!fp32) {
        return nt <= 128 ? 950.0 : 350.0 + 4.5 * ((nt + 63) / 64 * 64);  // (a tile of 208 or 240 is no faster than one of 256)
    }
    if (nt <= 32) {
        return one_part(type) ? 1270.0 : 1430.0;
    }
    const double t = one_part(type) ? 1330.0 + 6.5 * nt : 1450.0 + 8.6 * nt;
    return one_part(type) || t > 1960.0 ? t : 1960.0;
}

// Clusters of ks CTAs that run at a time, one CTA per SM (cudaOccupancyMaxActiveClusters; the SMs of a GPC are not all a multiple of 4 or 8).
static int clusters_of(int ks) { return ks == 1 ? 148 : (ks == 2 ? 74 : (ks == 4 ? 33 : 15)); }

// Tile width and ranges of the contraction for a product of `ftiles` tiles of features x m over `units` units.
static double choose(int type, bool fp32, bool bwd, int64_t ftiles, int units, int m, Args& a, Plan& plan) {
    const int nmax = fp32 ? 128 : 256;
    double best = 1e30;
    int best_nt = 16, best_ks = 1;
    int last_nt = 0;
    for (int tt = (m + nmax - 1) / nmax; tt <= (m + nmax - 1) / nmax + 6; tt++) {
        const int nt = ((m + tt - 1) / tt + 15) / 16 * 16;
        if (nt == last_nt || (fp32 && !bwd && nt <= 16)) {  // (16 rows of x are the rows kernel's)
            continue;
        }
        last_nt = nt;
        const int64_t tiles = ftiles * ((m + nt - 1) / nt);
        const double unit = unit_ns(type, fp32, bwd, nt);
        for (int ks = 1; ks <= 8; ks *= 2) {
            if (ks > 1 && units < 2 * ks) {
                break;
            }
            const int slots = clusters_of(ks);  // clusters at a time
            if (ks > 1 && tiles > slots) {
                break;  // more than one wave of whole tiles: nothing to gain
            }
            if (!configure(type, fp32, bwd, nt, ks, a, plan)) {
                continue;
            }
            // (a last wave that leaves SMs idle is a little faster: there is more of L2 and of the power for each CTA)
            const double part = (double)(tiles % slots) / slots, waves = (double)(tiles / slots) + (part > 0.0 ? 0.9 + 0.1 * part : 0.0);
            const double cost = waves * (((units + ks - 1) / ks) * unit + 1500.0 + 12.0 * nt) + (ks > 1 ? 1500.0 + 6.0 * nt : 0.0);
            if (cost < best) {
                best = cost;
                best_nt = nt;
                best_ks = ks;
            }
        }
    }
    configure(type, fp32, bwd, best_nt, best_ks, a, plan);
    a.ftiles = (int)ftiles;
    a.ttiles = (m + best_nt - 1) / best_nt;
    const int tiles = a.ftiles * a.ttiles;
    plan.ctas = best_ks > 1 || tiles < 148 ? tiles * best_ks : 148;
    a.units = units;
    a.m = m;
    return best;
}

// A product may be cut by features into up to three launches, each with its own tiles: whole waves first, then what is left, which alone would
// leave most of the chip idle for a whole contraction, with its contraction split over clusters. (Q4_K 11008 x 4096, 200 rows: 63.3 us in one launch,
// 56.5 in two; backward 4096 x 11008, 128 rows: 67.9 and 57.9.) The launch behind waits for the one in front, fills and drains: GAP_NS, measured at 5 to 7 us. Finding the cut takes 10 to 35 us.
constexpr int MAX_PARTS = 3;
constexpr double GAP_NS = 7000.0;
struct Part {
    Args a;
    Plan plan;
};
struct Parts {
    int count;
    Part part[MAX_PARTS];
};
static double cut(int type, bool fp32, bool bwd, int first_ft, int ftiles, int units, int m, int most, Parts& out) {
    Parts best;
    best.count = 1;
    best.part[0] = Part{};
    double cost = choose(type, fp32, bwd, ftiles, units, m, best.part[0].a, best.part[0].plan);
    best.part[0].a.first_ft = first_ft;
    if (most > 1) {
        const int nmax = fp32 ? 128 : 256, least = (m + nmax - 1) / nmax;
        for (int tt = least; tt <= least + 2; tt++) {  // tiles of rows of x in front
            for (int ks = 1; ks <= 4; ks *= 2) {
                const int slots = clusters_of(ks), waves = ks == 1 ? ftiles * tt / slots : 1, front = waves * slots / tt;
                if (front < 1 || front >= ftiles) {
                    continue;
                }
                Parts rest;
                Part lead{};
                const double c = choose(type, fp32, bwd, front, units, m, lead.a, lead.plan) + GAP_NS +
                                 cut(type, fp32, bwd, first_ft + front, ftiles - front, units, m, most - 1, rest);
                if (c < cost) {
                    cost = c;
                    lead.a.first_ft = first_ft;
                    best.count = 1 + rest.count;
                    best.part[0] = lead;
                    for (int i = 0; i < rest.count; i++) {
                        best.part[1 + i] = rest.part[i];
                    }
                }
            }
        }
    }
    out = best;
    return cost;
}

// The same from a small table of the thread: a user's program asks for the same shapes again and again.
static const Parts& parts_of(int type, bool fp32, bool bwd, int ftiles, int units, int m) {
    struct Entry {
        int key[6];
        Parts parts;
    };
    constexpr int ENTRIES = 64;
    static thread_local std::unique_ptr<Entry[]> table;
    if (table == nullptr) {
        table.reset(new Entry[ENTRIES]());
    }
    const int key[6] = {type + 1, fp32, bwd, ftiles, units, m};
    uint32_t h = 0;
    for (int v : key) {
        h = (h ^ (uint32_t)v) * 0x9E3779B1u;
        h ^= h >> 15;
    }
    Entry& e = table[h % ENTRIES];
    if (memcmp(e.key, key, sizeof(key)) != 0) {
        cut(type, fp32, bwd, 0, ftiles, units, m, MAX_PARTS, e.parts);
        memcpy(e.key, key, sizeof(key));
    }
    return e.parts;
}

static int launch_any(int type, const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) {
    switch (type) {
        case JQ_TYPE_Q4_K: return launch_q4_k(plan, args, map, s);
        case JQ_TYPE_Q5_K: return launch_q5_k(plan, args, map, s);
        case JQ_TYPE_Q6_K: return launch_q6_k(plan, args, map, s);
        case JQ_TYPE_Q8_0: return launch_q8_0(plan, args, map, s);
        case JQ_TYPE_Q4_0: return launch_q4_0(plan, args, map, s);
        case JQ_TYPE_Q4_1: return launch_q4_1(plan, args, map, s);
        default: return fail(JQ_ERR_UNSUPPORTED, "matrix product: type %d has no kernel", type);
    }
}

// The activations as a tensor of [planes][rows][width] 16-bit values.
static int activation_map(CUtensorMap* map, bool bf16, const void* x, int64_t width, int64_t rows, int planes, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (enc == nullptr) {
        return fail(JQ_ERR_CUDA, "matrix product: cuTensorMapEncodeTiled is not available from this driver");
    }
    const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)width * 2, (cuuint64_t)width * 2 * (cuuint64_t)rows};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)planes};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? JQ_OK : fail(JQ_ERR_CUDA, "matrix product: cuTensorMapEncodeTiled failed with code %d", (int)r);
}

// Puts `count` weights (one format and k) into the arguments; returns their tiles of features.
static int weight_args(const View* vs, int count, bool bwd, float* const* ys, Args& a) {
    int end = 0;
    for (int i = 0; i < MAX_WEIGHTS; i++) {
        const View& v = vs[i < count ? i : 0];
        a.q[i] = v.q;
        a.aux[i] = v.aux;
        a.y[i] = ys[i < count ? i : 0];
        a.features[i] = bwd ? v.k : v.n;
        end += i < count ? (int)((a.features[i] + 127) / 128) : 0;
        a.ft_end[i] = end;
    }
    a.kb = (int)tiled_steps(vs[0].k);
    return end;
}

constexpr int SPLIT_SLOT = 6;  // scratch slots 6 and 7: split activations without and with the 16 more columns

// ys[i] [m, features_i] = the FP32 products of `count` weights with the same x (backward: one weight); x has `width` values per row.
static int product_f32(const View* vs, int count, bool bwd, const float* x, const float* up, int64_t m, const float* bias, float* const* ys, cudaStream_t s) {
    const int64_t width = bwd ? vs[0].n : vs[0].k;
    const int per_row = (int)((width + 255) / 256), blk = bwd ? 128 : 256;
    constexpr int64_t GROUP = 4096;  // rows at a time: bounds the scratch
    int* status = nullptr;
    int rc = status_word(&status);
    for (int64_t m0 = 0; m0 < m && rc == JQ_OK; m0 += GROUP) {
        const int rows = (int)(m - m0 < GROUP ? m - m0 : GROUP);
        const int stride = (rows + 128 + 15) / 16 * 16;  // tiles of rows reach at most this far
        const float* xg = x + m0 * width;
        const float* ug = up != nullptr ? up + m0 * width : nullptr;
        if (!bwd && rows <= 16) {
            float* at[MAX_WEIGHTS];
            for (int i = 0; i < count; i++) {
                at[i] = ys[i] + m0 * vs[i].n;
            }
            rc = launch_rows(vs, count, xg, ug, rows, bias, at, s);
            continue;
        }
        const int vec = width % 4 == 0 && (((uintptr_t)xg | (uintptr_t)ug) & 15) == 0;
        // weights with the 16 more columns per unit and weights without: one split each
        for (int ext = 0; ext < 2 && rc == JQ_OK; ext++) {
            const int64_t wpad = (int64_t)per_row * (ext ? 272 : 256);
            const size_t plane_bytes = (size_t)2 * rows * wpad * 2;
            uint8_t* scratch = nullptr;
            float* scales = nullptr;
            for (int i = 0; i < count && rc == JQ_OK; i++) {
                // the weights of one format in one launch, with the first of them
                const int type = vs[i].type;
                View like[MAX_WEIGHTS];
                float* like_y[MAX_WEIGHTS];
                int n_like = 0;
                bool first = true;
                for (int j = 0; j < count; j++) {
                    if (vs[j].type == type) {
                        first = first && j >= i;
                        like[n_like] = vs[j];
                        like_y[n_like++] = ys[j] + m0 * (bwd ? vs[j].k : vs[j].n);
                    }
                }
                if (!first || facts(type, true, bwd, 16).ext != (ext != 0)) {
                    continue;
                }
                if (scratch == nullptr) {
                    rc = scratch_for_slot(s, SPLIT_SLOT + ext, plane_bytes + (size_t)(per_row * 256 / blk) * stride * sizeof(float), &scratch);
                    if (rc != JQ_OK) {
                        break;
                    }
                    scales = reinterpret_cast<float*>(scratch + plane_bytes);
                    cudaLaunchConfig_t cfg = {};
                    cudaLaunchAttribute attr[1];
                    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
                    attr[0].val.programmaticStreamSerializationAllowed = 1;
                    cfg.attrs = attr;
                    cfg.numAttrs = 1;
                    cfg.stream = s;
                    cfg.gridDim = dim3((unsigned)(((int64_t)rows * per_row + 7) / 8));
                    cfg.blockDim = dim3(256);
                    auto split = bwd ? split_kernel<128, false> : (ext ? split_kernel<256, true> : split_kernel<256, false>);
                    JQ_CUDA(cudaLaunchKernelEx(&cfg, split, xg, ug, rows, width, per_row, reinterpret_cast<uint4*>(scratch), scales, stride, vec));
                    count_launch();
                }
                Args w = {};
                const int ftiles = weight_args(like, n_like, bwd, like_y, w);
                const Parts& parts = parts_of(type, true, bwd, ftiles, bwd ? (int)(tiled_rows(vs[i].n) / TILE_ROWS) : w.kb, rows);
                for (int c = 0; c < parts.count && rc == JQ_OK; c++) {
                    Args a = parts.part[c].a;
                    weight_args(like, n_like, bwd, like_y, a);
                    CUtensorMap map;
                    rc = activation_map(&map, false, scratch, wpad, rows, 2, a.nt);
                    if (rc == JQ_OK) {
                        a.xscale = scales;
                        a.xstride = stride;
                        a.bias = bias;
                        a.status = status;
                        a.wait_clocks = wait_clocks();
                        rc = launch_any(type, parts.part[c].plan, a, map, s);
                    }
                }
            }
        }
    }
    return rc;
}

}  // namespace mm

int launch_matmul_f32(const View& v, const float* x, int64_t m, const float* bias, float* y, cudaStream_t s) {
    return mm::product_f32(&v, 1, false, x, nullptr, m, bias, &y, s);
}

int launch_matmul_f32_swiglu(const View& v, const float* gate, const float* up, int64_t m, float* y, cudaStream_t s) {
    return mm::product_f32(&v, 1, false, gate, up, m, nullptr, &y, s);
}

int launch_matmul_f32_multi(const View* vs, int count, const float* x, int64_t m, float* const* ys, cudaStream_t s) {
    return mm::product_f32(vs, count, false, x, nullptr, m, nullptr, ys, s);
}

// More than 16 rows of x always: the weight is read once for all of them. Up to 16 rows (the rows kernel's) take the time of 8 or of 16, so the line lies where
// the decode kernels need another pass. Measured with 4096 and 32000 output rows, k = 4096, last row count in front of the line / first behind it / the
// rows kernel, us: Q4_K (8 rows in a pass) 6.9 / 11.2 / 9.0 and 24.3 / 38.8 / 24.4; Q5_K 7.2 / 12.5 / 10.6 and 26.5 / 43.8 / 33.4; Q6_K (4) 7.6 / 14.4 / 9.4
// and 33.8 / 55.3 / 32.1; the 32-element formats (2) Q8_0 4.7 / 9.2 / 8.4 and 23.4 / 46.8 / 25.7, Q4_0 4.6 / 8.8 / 8.2 and 16.2 / 31.1 / 23.8, Q4_1 4.4 / 8.6 / 8.8
// and 17.0 / 32.8 / 27.7. With k = 1024 alike: Q4_K 5.0 / 7.2 / 5.7 and 15.1 / 21.6 / 9.9, Q8_0 with 1024 output rows 3.1 / 5.8 / 5.9. (Q4_K from 3 to 8 rows, both us,
// the decode kernel 6.8 and 25.0, the rows kernel 8.0 and 21.8: that crosses with the number of output rows.)
// The line must not depend on the number of output rows, and neither do the sums, so a row shard gives bitwise the outputs of the whole weight.
// Where the decode kernels decline (k no multiple of 256, or too wide) there is only the CUDA-core kernel besides, whose time grows with rows x k and
// with the output rows. At 4096 of them the rows kernel is the faster one from a little less on than the lines below say: Q8_0 k = 288 from 5 rows (5.6 us
// against 5.2), 1056 from 3 (9.2, 8.4), 2080 from 2 (11.1, 10.0); Q4_0 and Q4_1 288 from 3 (7.4, 5.1), 1056 from 2 (10.7, 8.1), 2080 from one (10.6, 9.4).
// In front of the lines a call needs no scratch buffer, so that a program may capture one that it has not made before.
bool matmul_takes(const View& v, int64_t rows) {
    if (rows > 16) {
        return true;
    }
    if (v.type == JQ_TYPE_Q4_K || v.type == JQ_TYPE_Q5_K) {
        return rows >= 9;
    }
    if (v.type == JQ_TYPE_Q6_K) {
        return rows >= 5;
    }
    if (gemv_blk32_i8_scratch_bytes(v.type, v.k, rows < 2 ? 1 : 2) > 0) {
        return rows >= (v.k <= 28672 ? 3 : 5);  // (a wider k's image of x may not fit the scratch buffer that calls with one or two rows have left)
    }
    return rows * v.k >= (v.type == JQ_TYPE_Q8_0 ? 4096 : 2048);
}

// gx [m, k] = g [m, n] . dequant(W) (ops/Gguf.java:208-212, ops/Quant.java:191-197); device pointers; n >= 1, m >= 1.
int launch_linear_backward(const View& v, const float* g, int64_t m, float* gx, cudaStream_t s) { return mm::product_f32(&v, 1, true, g, nullptr, m, nullptr, &gx, s); }

bool prefill_supported(const View& v) { return has_linear_kernel(v.type) && v.k % 64 == 0 && v.n > 0 && v.k > 0; }

// ys[i] [m, n_i] = x_bf16[m, k] . W_i^T (+ bias for the first) for up to three weights of one k; x 16-byte aligned device memory.
int launch_prefill_bf16_multi(const View* vs, int count, const uint16_t* x_bf16, int64_t m, const float* bias, float* const* ys, cudaStream_t s) {
    using namespace mm;
    int* status = nullptr;
    int rc = status_word(&status);
    for (int i = 0; i < count && rc == JQ_OK; i++) {
        if (!prefill_supported(vs[i])) {
            return fail(JQ_ERR_UNSUPPORTED, "prefill: the tensor-core kernel needs k to be a multiple of 64 (k = %lld)", (long long)vs[i].k);
        }
        // the weights of one format in one launch, with the first of them
        View like[MAX_WEIGHTS];
        float* like_y[MAX_WEIGHTS];
        int n_like = 0;
        bool first = true;
        for (int j = 0; j < count; j++) {
            if (vs[j].type == vs[i].type) {
                first = first && j >= i;
                like[n_like] = vs[j];
                like_y[n_like++] = ys[j];
            }
        }
        if (!first) {
            continue;
        }
        Args w = {};
        const int ftiles = weight_args(like, n_like, false, like_y, w);
        const Parts& parts = parts_of(vs[i].type, false, false, ftiles, w.kb, (int)m);
        for (int c = 0; c < parts.count && rc == JQ_OK; c++) {
            Args a = parts.part[c].a;
            weight_args(like, n_like, false, like_y, a);
            CUtensorMap map;
            rc = activation_map(&map, true, x_bf16, vs[i].k, m, 1, a.nt);
            if (rc == JQ_OK) {
                a.bias = i == 0 ? bias : nullptr;
                a.status = status;
                a.wait_clocks = wait_clocks();
                rc = launch_any(vs[i].type, parts.part[c].plan, a, map, s);
            }
        }
    }
    return rc;
}

int launch_prefill_bf16(const View& v, const uint16_t* x_bf16, int64_t m, const float* bias, float* y, cudaStream_t s) {
    return launch_prefill_bf16_multi(&v, 1, x_bf16, m, bias, &y, s);
}

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    });
    return fn;
}

// fp32 -> bf16 (round to nearest even, as the reference's LowPrecision.java:36-46), for jq_linear_f32's prefill option
static __global__ void f32_to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out, int64_t count) {
    int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i + 3 < count) {
        const float4 v = *reinterpret_cast<const float4*>(x + i);
        __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(out + i) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    } else {
        for (; i < count; i++) {
            out[i] = __float2bfloat16_rn(x[i]);
        }
    }
}

int launch_f32_to_bf16(const float* x, uint16_t* out, int64_t count, cudaStream_t s) {
    if (count == 0) {
        return JQ_OK;
    }
    const int64_t threads = (count + 3) / 4;
    f32_to_bf16_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(x, reinterpret_cast<__nv_bfloat16*>(out), count);
    count_launch();
    return check_launch("f32_to_bf16_kernel");
}

}  // namespace jq
