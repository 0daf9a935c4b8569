// Shared declarations of the library: error reporting, the weight handle, launch bookkeeping.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/jitnn_b200.h"

namespace jq {

// ---- error reporting (thread-local message behind jq_last_error) ------------------------------
int fail(int code, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

#define JQ_CUDA(call)                                   \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) {                        \
            return ::jq::cuda_fail(e_, #call);          \
        }                                               \
    } while (0)

extern std::atomic<int64_t> g_launches;
inline void count_launch(int n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// Checks the launch that was just issued.
int check_launch(const char* kernel);

// ---- block geometry (DType.java:75-98 of the reference) ---------------------------------------
inline int block_values(int type) {
    switch (type) {
        case JQ_TYPE_Q8_0: case JQ_TYPE_Q4_0: case JQ_TYPE_Q4_1: case JQ_TYPE_Q5_0: case JQ_TYPE_Q5_1: return 32;
        case JQ_TYPE_Q4_K: case JQ_TYPE_Q5_K: case JQ_TYPE_Q6_K: case JQ_TYPE_Q2_K: case JQ_TYPE_Q3_K: return 256;
        default: return 0;
    }
}

inline int block_bytes(int type) {
    switch (type) {
        case JQ_TYPE_Q8_0: return 34;
        case JQ_TYPE_Q4_0: return 18;
        case JQ_TYPE_Q4_1: return 20;
        case JQ_TYPE_Q4_K: return 144;
        case JQ_TYPE_Q5_K: return 176;
        case JQ_TYPE_Q6_K: return 210;
        case JQ_TYPE_Q5_0: return 22;
        case JQ_TYPE_Q5_1: return 24;
        case JQ_TYPE_Q2_K: return 84;
        case JQ_TYPE_Q3_K: return 110;
        default: return 0;
    }
}

// Bytes per block of the quant plane and of the scale plane in the device layout. Formats whose
// blocks are 16-byte multiples (Q4_K, Q5_K) and the dequantise-only formats stay verbatim (aux = 0).
inline int plane_q_bytes(int type) {
    switch (type) {
        case JQ_TYPE_Q8_0: return 32;
        case JQ_TYPE_Q4_0: return 16;
        case JQ_TYPE_Q4_1: return 16;
        case JQ_TYPE_Q6_K: return 208;
        default: return block_bytes(type);
    }
}

inline int plane_aux_bytes(int type) {
    switch (type) {
        case JQ_TYPE_Q8_0: return 2;
        case JQ_TYPE_Q4_0: return 2;
        case JQ_TYPE_Q4_1: return 4;
        case JQ_TYPE_Q6_K: return 2;
        default: return 0;
    }
}

// Q4_K and Q5_K weights are stored tile by tile: 128 consecutive rows form a tile, and within a tile the blocks of one
// 256-element super-block of k lie together, row after row: [tile][super-block b][row in tile][block bytes]. One
// (tile, super-block) unit is then a single contiguous run of 128 x block bytes, which the copy engine moves with one bulk copy.
// The last tile is padded with zero rows. No byte of a block changes; jq_weight_download restores GGUF's order.
constexpr int TILE_ROWS = 128;
__host__ __device__ inline bool tiled_layout(int type) { return type == JQ_TYPE_Q4_K || type == JQ_TYPE_Q5_K; }
// The formats with two planes (quants; fp16 scales) order the blocks of each plane the same way. Q6_K: 16 rows x one super-block are
// 3328 contiguous bytes of the quant plane and 32 of the d plane. The formats with 32-element blocks take eight blocks (256 values
// of k) where the K-quants have a super-block; a k that is no multiple of 256 is padded with zero blocks, and the 16-byte pieces of
// a row's eight blocks are stored with the low three bits of their number XORed by (row & 7), so that eight rows read at the same
// place of their rows fall into different shared-memory banks after a plain copy.
__host__ __device__ inline bool tiled_planes(int type) {
    return type == JQ_TYPE_Q6_K || type == JQ_TYPE_Q8_0 || type == JQ_TYPE_Q4_0 || type == JQ_TYPE_Q4_1;
}
__host__ __device__ inline int64_t tiled_rows(int64_t n) { return (n + TILE_ROWS - 1) / TILE_ROWS * TILE_ROWS; }
// 256-wide steps of k of a tiled weight.
__host__ __device__ inline int64_t tiled_steps(int64_t k) { return (k + 255) >> 8; }
// Position of super-block b of `row` among the super-blocks of a tiled plane with kb of them per row.
__host__ __device__ inline int64_t tiled_index(int64_t row, int64_t b, int64_t kb) {
    return ((row >> 7) * kb + b) * TILE_ROWS + (row & (TILE_ROWS - 1));
}
// Position of 32-element block b of `row` in a tiled plane of kb 256-wide steps per row.
__host__ __device__ inline int64_t tiled_index32(int64_t row, int64_t b, int64_t kb) { return tiled_index(row, b >> 3, kb) * 8 + (b & 7); }
// Where 16-byte piece c of a row's 256-wide step lies within that row's run of the quant plane.
__host__ __device__ inline int swizzle_piece(int c, int64_t row) { return (c & ~7) | ((c ^ (int)row) & 7); }
// Byte offset of block b of `row` in a tiled weight with kb blocks of `bytes` bytes per row.
__host__ __device__ inline int64_t tiled_offset(int64_t row, int64_t b, int64_t kb, int bytes) {
    return ((row >> 7) * kb + b) * (int64_t)(TILE_ROWS * bytes) + (row & (TILE_ROWS - 1)) * bytes;
}

inline bool has_linear_kernel(int type) {
    return type == JQ_TYPE_Q8_0 || type == JQ_TYPE_Q4_0 || type == JQ_TYPE_Q4_1 || type == JQ_TYPE_Q4_K ||
           type == JQ_TYPE_Q5_K || type == JQ_TYPE_Q6_K;
}

// What the kernels see of a weight.
struct View {
    const uint8_t* q;    // quant plane, tiled blocks (Q4_K, Q5_K) or verbatim blocks, 256-byte aligned
    const uint8_t* aux;  // scale plane, or nullptr
    int64_t n;           // output rows
    int64_t k;           // input features
    int type;
};

// ---- kernel launchers (one translation unit each) ----------------------------------------------
// kb: blocks per row; the planes hold their blocks in tiled order (tiled_rows(n) rows).
int launch_repack(int type, const uint8_t* verbatim, uint8_t* q, uint8_t* aux, int64_t blocks, int64_t kb, cudaStream_t s);
int launch_unpack(int type, const uint8_t* q, const uint8_t* aux, uint8_t* verbatim, int64_t blocks, int64_t kb, cudaStream_t s);
// Verbatim blocks [n, kb] <-> the tiled layout of Q4_K and Q5_K (`tiled` holds tiled_rows(n) rows).
int launch_tile(int type, const uint8_t* verbatim, uint8_t* tiled, int64_t n, int64_t kb, bool inverse, cudaStream_t s);
int launch_dequantize(const View& v, float* dst, cudaStream_t s);
// x_remote: x lies in host memory that the GPU reads across PCIe; kernels then read it once instead of once per thread block.
int launch_gemv(const View& v, const float* x, int rows, const float* bias, float* y, cudaStream_t s, bool x_remote = false);
// gx [m, k] = g [m, n] . dequant(W) (jq_matmul.cu).
int launch_linear_backward(const View& v, const float* g, int64_t m, float* gx, cudaStream_t s);
int launch_quantize_q8_0(const float* x, int64_t blocks, uint8_t* out, cudaStream_t s);
// Where a GEMV's outputs go besides (or instead of) y when the linear is sharded by rows over several GPUs: every
// rank's copy of the full output and flag words (jq_peer.cu). world = 0: no peers.
struct PeerOut {
    float* y[8];         // every rank's y [m, n_total] (this rank's included)
    uint32_t* flags[8];  // every rank's flag words
    unsigned long long* stage[8];  // every rank's staging words [m, n_total] (value and exchange number in one 8-byte word), or null:
                                   // the outputs then go straight into y and the exchange is announced through the arrival counters
    int world, rank;
    int64_t n_total, col0;  // this rank's rows are columns col0 .. of y
    int64_t n_own;          // how many of them: rows of this rank's shard
    const PeerOut* table;   // host side only: where a copy of this struct lives in device memory
    int wait_first;         // the kernel's input is what this rank's latest exchange delivered: wait for all ranks' parts before reading it
    int wait_after;         // the kernel ends only when all ranks' parts of its own exchange have arrived in this rank's y (bounded wait by one CTA)
    long long wait_clocks;  // clocks a thread waits in all for the other ranks' marked words
};
// Integer tensor-core GEMV (mma.sync) for Q4_K and Q5_K, rows <= 8 (jq_gemv_q4k_i8.cu); *handled = false leaves the call to
// another kernel. `image` is scratch of gemv_q4k_i8_scratch_bytes(k, rows) bytes.
int launch_gemv_q4k_i8(const View& v, const float* x, int rows, const float* bias, float* y, cudaStream_t s, uint8_t* image, bool* handled,
                       const PeerOut* peer = nullptr, bool x_remote = false);
size_t gemv_q4k_i8_scratch_bytes(int64_t k, int rows);
int launch_gemv_q4k_i8_multi(const View* vs, int count, const float* x, int rows, float* const* ys, cudaStream_t s, uint8_t* image, bool* handled);
// The same for one row of x whose activation image (jq_q4k_image.cuh) a kernel earlier in the stream has already written; a
// second Q4_K weight with the same k can ride in the same launch.
size_t q4k_image_bytes_one_row(int64_t k);
// What a GEMV of one row needs to make its activation image from RMSNorm(x + delta) itself. It also leaves x + delta in x_out (not x: other
// thread blocks still read it).
struct NormInput {
    const float *x, *delta, *w;
    float eps;
    float* x_out;  // receives x + delta; null where the launch in front does that
    bool followed;  // a launch on the same input is behind, which does not wait for this one: it may start when this one knows that the input is complete
};
int launch_gemv_q4k_i8_normed(const View* vs, int count, const NormInput& norm, float* const* ys, cudaStream_t s, bool* handled);
// The launch behind it, of one Q6_K weight: it starts as SMs become free and ends after the one in front.
bool gemv_q6k_i8_normed_takes(const View& v);
int launch_gemv_q6k_i8_normed(const View& v, const NormInput& norm, float* y, cudaStream_t s);
int launch_gemv_q4k_i8_imaged(const View& v, const View* v2, const uint8_t* image, const float* bias, float* y, float* y2, cudaStream_t s, bool* handled,
                              const PeerOut* peer = nullptr, const View* v3 = nullptr, float* y3 = nullptr);
// Status word of the waits a GEMV makes itself for a peer exchange (peer_wait_inline): 0 or 32 + rank, cleared by the call.
int gemv_peer_status(int* status);
// Pieces of the peer exchange (jq_peer.cu) for the row-sharded decoder: the bounded wait for all ranks' flags of this
// rank's latest exchange, and a Q4_K row shard applied to an activation image that is already complete, its outputs
// stored into every rank's y [1, n_total] at payload_offset, followed by that wait.
// staging_offset >= 0: the outputs travel as marked words through that area of the payload and the kernel ends when this
// rank's y is complete (wait_after is then moot); < 0: straight into every rank's y, announced through the arrival counters.
int peer_linear_q4k_imaged(const jq_weight* w, const uint8_t* image, int64_t n_total, int64_t col0, void* const* peer_buffers, int64_t payload_offset,
                           int64_t staging_offset, int rank, int world, cudaStream_t s, bool wait_first, bool wait_after);
// Status word of the waits that the decoder's kernels make themselves (peer_wait_inline): 0 or 32 + rank, cleared by the call.
int decoder_peer_status(int* status);
// Q6_K for one row of x whose activation image (jq_q6k_image.cuh) a kernel earlier in the stream has written.
size_t q6k_image_bytes_one_row(int64_t k);
int launch_gemv_q6k_i8_imaged(const View& v, const uint8_t* image, const float* bias, float* y, cudaStream_t s, bool* handled);
// Whether the GEMV of one or two rows of x in Q6_K or a 32-element format makes the image of x itself (the bits are those of the image kernel's). Every thread block then
// makes all of it, so not for more than 8192 values (four blocks a warp), nor where x lies in host memory, which is read once. Up to 6144 values, up to 32 tiles of rows
// and with more tiles than SMs it saves 0.3 to 1.6 us of the GPU's time and a launch of 1.6 us on the host. Between, thread blocks read the same values all at once with no
// weights behind to hide it. Weights from device memory, inside / image kernel, us, replayed from a graph and (launched one after the other):
//   one row of 8192, n = 1024    Q8_0 5.6 / 4.9 (5.6 / 5.7), Q4_0 5.3 / 4.3 (6.1 / 5.6), Q4_1 5.1 / 4.7 (6.2 / 5.6), Q6_K 6.3 / 6.9 (8.0 / 7.3)
//                    n = 2048    Q8_0 6.1 / 5.6 (6.6 / 6.9), Q4_0 6.0 / 4.9 (6.3 / 5.7), Q4_1 6.0 / 5.5 (6.5 / 5.7), Q6_K 7.6 / 7.5 (8.2 / 8.4)
//   two rows of 4096, n = 1024   Q8_0 4.4 / 3.9 (5.5 / 6.8), Q4_0 4.1 / 4.0 (3.8 / 5.5), Q4_1 4.0 / 3.5 (3.8 / 5.8), Q6_K 5.3 / 5.1 (5.5 / 5.9)
//                    n = 2048    Q8_0 4.8 / 4.3 (5.2 / 5.7), Q4_0 4.5 / 3.8 (4.9 / 5.8), Q4_1 4.5 / 4.5 (4.9 / 5.7), Q6_K 5.7 / 5.3 (6.0 / 5.9)
//   and on either side of that, one row of 8192: n = 256 Q8_0 4.5 / 4.6, Q6_K 5.2 / 5.9; n = 4096 Q8_0 7.7 / 8.4, Q6_K 7.9 / 8.2.
// So one row of Q4_0 and Q4_1 has the image kernel there; one row of Q8_0, and two rows, have it where a graph is captured, whose replays cost the host nothing.
bool gemv_image_inside(const View& v, int rows, bool x_remote, cudaStream_t s);
// The same for Q6_K, rows <= 4.
int launch_gemv_q6k_i8(const View& v, const float* x, int rows, const float* bias, float* y, cudaStream_t s, uint8_t* image, bool* handled, bool x_remote);
size_t gemv_q6k_i8_scratch_bytes(int64_t k, int rows);
// The same for Q8_0, Q4_0 and Q4_1 (jq_gemv_blk32_i8.cu): rows <= 2, k a multiple of 256.
int launch_gemv_blk32_i8(const View& v, const float* x, int rows, const float* bias, float* y, cudaStream_t s, uint8_t* image, bool* handled, bool x_remote);
size_t gemv_blk32_i8_scratch_bytes(int type, int64_t k, int rows);

// Scratch memory of at least `bytes` on the current device, private to work enqueued on `s` (one buffer per
// device and stream, grown on demand and kept until the library is unloaded).
int scratch_for(cudaStream_t s, size_t bytes, uint8_t** out);
// A second, third ... scratch buffer of the same (device, stream), for a caller that needs one while a kernel launcher uses slot 0.
int scratch_for_slot(cudaStream_t s, int slot, size_t bytes, uint8_t** out);
uint8_t* scratch_held(cudaStream_t s, int slot, size_t bytes);

inline bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) != cudaSuccess) {
        cudaGetLastError();  // (the default stream while another is captured: the launch itself says so)
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

// The same for words that kernels use as counters and leave at zero: a new allocation starts out zeroed (in stream order).
int scratch_zeroed_for_slot(cudaStream_t s, int slot, size_t bytes, uint8_t** out);
// For a stream of the library's own that is about to be destroyed.
void scratch_release(cudaStream_t s);
// Status words: where kernels record that a bounded wait gave up. Page-locked host memory that the device writes, so that reading one costs
// no copy. A call that waits for its own result gives its kernels a word of its own (StatusScope) and learns of its own failures alone; the
// kernels of calls that only enqueue work write to the word of their device, which jq_device_status reads.
int status_word(int** word);          // for the kernels launched now, on the current device
int take_status_word(int** word);     // a zeroed word; give_status_word returns it
void give_status_word(int* word);
int* device_status_word(int device);  // nullptr before the first weight of that device
// The code in a word (0: no wait gave up), which is cleared. After the work that may write it has ended.
inline int read_status(int* word) {
    volatile int* v = word;
    const int code = *v;
    if (code != 0) {
        *v = 0;
    }
    return code;
}
struct StatusScope {
    int* before;
    explicit StatusScope(int* word);
    ~StatusScope();
};

// Decode GEMV on tcgen05 (jq_gemv_umma.cu): Q4_K and Q5_K, 1 to 16 rows of x in one pass over the weights.
bool gemv_umma_takes(int type, int64_t k, int rows);  // under option gemv_tcgen05 = 1
bool gemv_umma_fallback(int type, int64_t k, int rows);  // may stand in for the mma.sync kernel on a shape that one declines
size_t gemv_umma_image_bytes(int64_t k, int rows);
inline size_t gemv_umma_image_bytes_one_row(int64_t k) { return gemv_umma_image_bytes(k, 1); }
int launch_gemv_umma_image(const float* x, int rows, int64_t k, uint8_t* image, cudaStream_t s);
int launch_gemv_umma(const View& v, const View* v2, const float* x, uint8_t* image, int rows, const float* bias, float* y, float* y2, cudaStream_t s,
                     const PeerOut* peer = nullptr, bool no_scratch = false);
int launch_gemv_umma_multi(const View* vs, int count, const float* x, uint8_t* image, int rows, const float* bias, float* const* ys, cudaStream_t s,
                           const PeerOut* peer = nullptr, bool no_scratch = false);
int gemv_umma_peer_status(int* status);  // 0, or 32 + rank once a wait of its peer exchange has given up
// Option "gemv_tcgen05": 1 sends Q4_K and Q5_K decode (1 to 16 rows) to the tcgen05 GEMV, 2 never, 0 where the mma.sync kernel declines.
extern std::atomic<int64_t> g_opt_gemv_umma;
// Option "wait_limit_us": microseconds after which a bounded device-side wait of the tcgen05 GEMV gives up.
extern std::atomic<int64_t> g_opt_wait_limit_us;
extern std::atomic<int64_t> g_opt_peer_wait_us;  // microseconds a thread waits in all for the other ranks' values of a sharded linear

// Rows of zero padding behind every uploaded weight plane: kernels that work on 16-row tiles read past n.
constexpr int PAD_ROWS = 16;

// The matrix kernel (jq_matmul.cu): the FP32 product with many rows of x, and the bfloat16 product.
int launch_matmul_f32(const View& v, const float* x, int64_t m, const float* bias, float* y, cudaStream_t s);
// The same for x = silu(gate) * up, made where x is split into halves.
int launch_matmul_f32_swiglu(const View& v, const float* gate, const float* up, int64_t m, float* y, cudaStream_t s);
// Up to three weights of one k on the same x: the split of x into halves is shared, weights of one format are one launch.
int launch_matmul_f32_multi(const View* vs, int count, const float* x, int64_t m, float* const* ys, cudaStream_t s);
// The rows kernel (jq_rows.cu): the same for up to 16 rows of x (up: x is silu(x) * up).
int launch_rows(const View* vs, int count, const float* x, const float* up, int m, const float* bias, float* const* ys, cudaStream_t s);
int rows_image(cudaStream_t s, int type, int m, int64_t k, uint8_t** image, float** scales);  // for a kernel that writes x's image itself: then x is null
bool matmul_takes(const View& v, int64_t rows);  // where it is the fastest of the FP32 kernels
bool prefill_supported(const View& v);
int launch_prefill_bf16(const View& v, const uint16_t* x_bf16, int64_t m, const float* bias, float* y, cudaStream_t s);
int launch_prefill_bf16_multi(const View* vs, int count, const uint16_t* x_bf16, int64_t m, const float* bias, float* const* ys, cudaStream_t s);
int launch_f32_to_bf16(const float* x, uint16_t* out, int64_t count, cudaStream_t s);
// Same for the bounded waits of the peer gather (jq_peer.cu): 0, or 32 + the rank whose slice did not arrive.
int peer_status(int* status);

// Option "gemv_generic": non-zero routes every GEMV to the generic CUDA-core kernel (for comparisons).
extern std::atomic<int64_t> g_opt_gemv_generic;
// Option "decoder_graph": zero keeps the decoder's single-token step on eager launches (for comparisons).
extern std::atomic<int64_t> g_opt_decoder_graph;
// Option "decoder_fused": zero keeps the decoder's single-token step on the general kernels (one per operator).
extern std::atomic<int64_t> g_opt_decoder_fused;

}  // namespace jq

// The opaque handle of the C ABI.
struct jq_weight {
    uint32_t magic;
    int device;
    int type;
    int layout;
    int64_t n;
    int64_t k;
    uint8_t* q;
    uint8_t* aux;
    int64_t q_bytes;
    int64_t aux_bytes;
};

#define JQ_WEIGHT_MAGIC 0x4a515754u
