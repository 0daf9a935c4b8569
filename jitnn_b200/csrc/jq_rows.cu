// Host side of the rows kernel (jq_rows.cuh): the image of x, the launches (their choice: jq_rows_cut.cuh).
#include "jq_rows_cut.cuh"
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

// x [m, k] FP32 (or silu(x) * up) -> per 256-wide step of k its image (jq_rows.cuh) and a scale per row: the row's 256 values times a power of two that
// brings the largest to [2^9, 2^10), hi = that rounded to half precision, lo = the rest rounded to half precision: 22 significant bits for
// everything down to 2^-13 of the largest. NT: 8 or 16 rows. A row's 256 that hold a NaN or an Inf get the scale NaN, which reaches every output of that row. One
// warp per row and step, eight values a lane; rows from m on are zeros. Memory bound: 4 bytes read and 4.5 written (to L2) a value.
template <int NT>
__global__ void __launch_bounds__(128) image_kernel(const float* __restrict__ x, const float* __restrict__ up, int m, int64_t k, int units, uint8_t* __restrict__ image,
                                                    float* __restrict__ scales, int vec) {
    constexpr int N = 2 * NT, STEP = step_bytes(NT);
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t task = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, u = (int)(task / NT), row = (int)(task % NT);
    if (u >= units) {
        return;
    }
    const int64_t i0 = (int64_t)u * 256 + lane * 8, at = (int64_t)row * k + i0;
    float v[8];
    if (row < m && vec && i0 + 8 <= k) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(x + at)), c = __ldg(reinterpret_cast<const float4*>(x + at) + 1);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = row < m && i0 + i < k ? __ldg(x + at + i) : 0.0f;
        }
    }
    if (up != nullptr) {  // x is the gate of a feed-forward block
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float g = row < m && i0 + i < k ? __ldg(up + at + i) : 0.0f;
            v[i] = (v[i] / (1.0f + expf(-v[i]))) * g;
        }
    }
    uint32_t am = 0;  // the largest magnitude as bits: an Inf or a NaN is larger than any number
#pragma unroll
    for (int i = 0; i < 8; i++) {
        am = max(am, __float_as_uint(v[i]) & 0x7fffffffu);
    }
    am = __reduce_max_sync(0xffffffffu, am);
    const bool bad = am >= 0x7f800000u;
    uint32_t e = am >> 23;
    e = e < 14u ? 14u : (e > 254u ? 254u : e);
    const float f = __uint_as_float((263u - e) << 23);
    uint32_t hi[4], lo[4];  // of four values 0 and 2, 1 and 3
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = v[(i >> 1) * 4 + (i & 1)] * f, c = v[(i >> 1) * 4 + (i & 1) + 2] * f;
        mm::split_pair(a, c, hi[i], lo[i]);
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i])), l = __half22float2(*reinterpret_cast<const __half2*>(&lo[i]));
        sum += (h.x + l.x) + (h.y + l.y);
    }
    // lane = step of 16 and half of it; columns row (hi) and NT + row (lo), 128 bytes per eight columns
    uint8_t* const unit = image + (int64_t)u * image_bytes(NT);
    const int col = (row >> 3) * 128 + (row & 7) * 16;
    uint8_t* const to = unit + (lane >> 1) * STEP + (lane & 1) * (N * 16) + col;
    *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(to + NT * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    // the sums over runs of 32 (four lanes), up to 2^15, twice
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const __half sh = __float2half_rn(sum), sl = __float2half_rn(sum - __half2float(sh));
    if ((lane & 3) == 0) {
        __half* const run = reinterpret_cast<__half*>(unit + 16 * STEP + col) + (lane >> 2);
        run[0] = run[N * 8] = sh;
        run[NT * 8] = run[(N + NT) * 8] = sl;
    }
    if (lane == 0) {
        scales[(int64_t)u * NT + row] = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((e - 9u) << 23);
    }
}

static int launch_any(int type, Args& a, int ctas, bool after, cudaStream_t s) {
    switch (type) {
        case JQ_TYPE_Q4_K: return launch_q4_k(a, ctas, after, s);
        case JQ_TYPE_Q5_K: return launch_q5_k(a, ctas, after, s);
        case JQ_TYPE_Q6_K: return launch_q6_k(a, ctas, after, s);
        case JQ_TYPE_Q8_0: return launch_q8_0(a, ctas, after, s);
        case JQ_TYPE_Q4_0: return launch_q4_0(a, ctas, after, s);
        case JQ_TYPE_Q4_1: return launch_q4_1(a, ctas, after, s);
        default: return fail(JQ_ERR_UNSUPPORTED, "rows product: type %d has no kernel", type);
    }
}

// Scratch for image and scales. Up to four rows the slot is that of the decode kernels' images, so that a program that has made a call with one or two rows may
// capture one with three or four (matmul_takes sends no wider k here than the slot's least size holds).
constexpr int SLOT = 8;
constexpr int slot_of(int m) { return m < 5 ? 0 : SLOT; }

}  // namespace rows

// ys[i] [rows, n_i] = x . W_i^T (+ bias for the first), x [rows, k] or silu(x) * up, for up to three weights of one k: one image, the weights of one
// format in one launch.
int launch_rows(const View* vs, int count, const float* x, const float* up, int m, const float* bias, float* const* ys, cudaStream_t s) {
    using namespace rows;
    const int64_t k = vs[0].k;
    const int units = (int)tiled_steps(k);
    int* status = nullptr;
    uint8_t* image = nullptr;
    int rc = status_word(&status);
    if (rc == JQ_OK) {
        rc = scratch_for_slot(s, slot_of(m), (size_t)units * (image_bytes(m < 5 ? 8 : MAX_NT) + MAX_NT * sizeof(float)), &image);
    }
    if (rc != JQ_OK) {
        return rc;
    }
    const int nt = m <= 8 ? 8 : 16;
    float* const scales = reinterpret_cast<float*>(image + (size_t)units * image_bytes(nt));
    {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.stream = s;
        cfg.gridDim = dim3((unsigned)((int64_t)units * nt / 4));
        cfg.blockDim = dim3(128);
        const int vec = k % 4 == 0 && (((uintptr_t)x | (uintptr_t)up) & 15) == 0;
        JQ_CUDA(cudaLaunchKernelEx(&cfg, nt == 8 ? image_kernel<8> : image_kernel<16>, x, up, m, k, units, image, scales, vec));
        count_launch();
    }
    for (int i = 0; i < count && rc == JQ_OK; i++) {
        // the weights of one format in one launch, with the first of them
        Args a = {};
        int like = 0, end = 0;
        bool first = true;
        for (int j = 0; j < count; j++) {
            if (vs[j].type == vs[i].type) {
                first = first && j >= i;
                a.q[like] = vs[j].q;
                a.aux[like] = vs[j].aux;
                a.y[like] = ys[j];
                a.n[like] = vs[j].n;
                end += (int)((vs[j].n + 127) / 128);
                a.ft_end[like++] = end;
            }
        }
        if (!first) {
            continue;
        }
        for (int j = like; j < MAX_WEIGHTS; j++) {
            a.q[j] = a.q[0], a.aux[j] = a.aux[0], a.y[j] = a.y[0], a.n[j] = a.n[0], a.ft_end[j] = end;
        }
        a.image = image;
        a.scales = scales;
        a.bias = i == 0 ? bias : nullptr;
        a.units = units;
        a.m = m;
        a.status = status;
        a.wait_clocks = (long long)g_opt_wait_limit_us.load(std::memory_order_relaxed) * 2000;  // about 2 GHz
        Parts parts;
        cut(end, units, unit_ns(vs[i].type), MAX_PARTS, parts);
        for (int c = 0, at = 0; c < parts.count && rc == JQ_OK; c++) {
            a.first_ft = at;
            a.ftiles = at += parts.tiles[c];
            a.ksplit = parts.ksplit[c];
            a.followed = c + 1 < parts.count;
            rc = launch_any(vs[i].type, a, a.ksplit > 1 ? parts.tiles[c] * a.ksplit : (parts.tiles[c] < 148 ? parts.tiles[c] : 148), c > 0, s);
        }
    }
    return rc;
}

}  // namespace jq
