// Host side of the rows kernel (jq_rows.cuh): the image of x, the launches (their choice: jq_rows_cut.cuh).
#include "jq_rows_cut.cuh"
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

// x [m, k] FP32 (or silu(x) * up) -> its image (jq_rows_image.cuh), rows from m on zeros. One warp per row and 256-wide step of k, eight values a lane. Memory bound:
// 4 bytes read and 4.5 written (to L2) a value.
template <int NT>
__global__ void __launch_bounds__(128) image_kernel(const float* x, const float* up, int m, int64_t k, int units, uint8_t* __restrict__ image,
                                                    float* __restrict__ scales, int vec) {
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
        const float4 a = *reinterpret_cast<const float4*>(x + at), c = *(reinterpret_cast<const float4*>(x + at) + 1);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = row < m && i0 + i < k ? x[at + i] : 0.0f;
        }
    }
    if (up != nullptr) {  // x is the gate of a feed-forward block
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float g = row < m && i0 + i < k ? up[at + i] : 0.0f;
            v[i] = (v[i] / (1.0f + expf(-v[i]))) * g;
        }
    }
    store_image<NT>(v, u, row, image, scales, lane);
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

// Scratch for image and scales: one slot, sized for 16 rows, so that a program that has made a call may capture one with another number of rows. Three and four rows of
// which the decode kernels take two in a pass use the slot of those kernels' images, whose least size holds theirs, so that a call with one or two rows is enough in front of a
// capture and the other way round. A capture that finds its slot too small takes the other one, for three and four rows of every k that fits there.
constexpr int SLOT = 8, DECODE_SLOT = 0;
static_assert((28672 / 256) * (image_bytes(8) + MAX_NT * sizeof(float)) <= (1 << 20), "the least size of a scratch buffer");

}  // namespace rows

// Where the image of m rows of x for the next product on `s` goes, whose first weight has that type, for a kernel that writes it itself. (Asked again it says the same.)
int rows_image(cudaStream_t s, int type, int m, int64_t k, uint8_t** image, float** scales) {
    using namespace rows;
    const size_t units = (size_t)tiled_steps(k), few = units * (image_bytes(8) + MAX_NT * sizeof(float)), any = units * (image_bytes(MAX_NT) + MAX_NT * sizeof(float));
    const bool either = (m == 3 || m == 4) && k <= 28672 && gemv_blk32_i8_scratch_bytes(type, k, 1) > 0, decode = either && gemv_blk32_i8_scratch_bytes(type, k, 2) > 0;
    *image = either ? scratch_held(s, decode ? DECODE_SLOT : SLOT, decode ? few : any) : nullptr;
    if (either && *image == nullptr && capturing(s)) {
        *image = scratch_held(s, decode ? SLOT : DECODE_SLOT, decode ? any : few);
    }
    const int rc = *image != nullptr ? JQ_OK : scratch_for_slot(s, decode ? DECODE_SLOT : SLOT, decode ? few : any, image);
    *scales = reinterpret_cast<float*>(*image + units * image_bytes(nt_of(m)));
    return rc;
}

// ys[i] [rows, n_i] = x . W_i^T (+ bias for the first), x [rows, k] or silu(x) * up, for up to three weights of one k: one image, the weights of one
// format in one launch. x null: the kernel in front has written the image. Only the first launch waits for it; the others, further tiles or another format, start as SMs
// become free.
int launch_rows(const View* vs, int count, const float* x, const float* up, int m, const float* bias, float* const* ys, cudaStream_t s) {
    using namespace rows;
    const int64_t k = vs[0].k;
    const int units = (int)tiled_steps(k), nt = nt_of(m);
    int* status = nullptr;
    uint8_t* image = nullptr;
    float* scales = nullptr;
    int rc = status_word(&status);
    if (rc == JQ_OK) {
        rc = rows_image(s, vs[0].type, m, k, &image, &scales);
    }
    if (rc != JQ_OK) {
        return rc;
    }
    if (x != nullptr) {
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
    bool after = false;
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
        bool more = false;  // another format is behind
        for (int j = i + 1; j < count; j++) {
            bool fresh = true;
            for (int h = 0; h < j; h++) {
                fresh = fresh && vs[h].type != vs[j].type;
            }
            more = more || fresh;
        }
        Parts parts;
        cut(end, units, unit_ns(vs[i].type), MAX_PARTS, parts);
        for (int c = 0, at = 0; c < parts.count && rc == JQ_OK; c++) {
            a.first_ft = at;
            a.ftiles = at += parts.tiles[c];
            a.ksplit = parts.ksplit[c];
            a.followed = more || c + 1 < parts.count;
            rc = launch_any(vs[i].type, a, a.ksplit > 1 ? parts.tiles[c] * a.ksplit : (parts.tiles[c] < 148 ? parts.tiles[c] : 148), after, s);
            after = true;
        }
    }
    return rc;
}

}  // namespace jq
