// The matrix kernel: products of a quantised weight with many rows of activations on the 5th-generation tensor cores.
//
//   forward   y[m, n]  = x[m, k] . W[n, k]^T (+ bias)     features = rows of W,  contraction over k
//   backward  gx[m, k] = g[m, n] . W[n, k]                features = k,          contraction over the rows of W
//
// Two operand precisions. BF16: x is bfloat16, weights are rounded to bfloat16, one product. FP32: x is split into two halves (hi + lo, 22
// significant bits), and so are weights that one half cannot hold (jq_matmul_dequant.cuh); the products hi.hi + hi.lo + lo.hi (or
// the first two) are taken, so that results keep FP32's accuracy; sums leave the tensor core every 128 (backward: 64) terms and are added
// up in registers, rounded to nearest (see Shape::ACC).
//
// A CTA owns 128 features and a tile of up to 256 (FP32: 128) rows of x and walks the contraction in stages of 64. (Pairs of CTAs under one
// tcgen05.mma, cta_group::2, read each activation tile from L2 once for 256 features; measured equal within 3 % on every shape and
// dearer to synchronise, so not kept.) Roles:
//   warp 0       one thread brings activation tiles in by TMA (128-byte swizzle, no multicast). From "free" to "full" a tile takes more than a
//                microsecond (L2), several stages' worth, so this ring is deeper than that of the weight operands
//   warp 1       issues tcgen05.mma
//   warp 2       one thread brings raw units in (128 rows x 256 k, one contiguous run of the tiled weight, cp.async.bulk)
//   then         groups of four warps that dequantise. The groups take stages in turn, so that what a stage costs a warp besides its
//                instructions (barrier round trips) overlaps with the other groups' work. Forward: a thread turns 64 weights of its
//                row into 32 columns of its lane of the operand in tensor memory. In shared memory, writing and reading the weights took
//                more of its 128 bytes per clock than the rest together, and bound the kernel. Backward: the weights are the transposed
//                operand, which only shared memory can hold: a thread makes a 128-byte row of 64 features of one contraction index
//   last         four or sixteen warps take finished accumulators from tensor memory (up to four buffers), add them up, store y
// A cluster may also split the contraction (ksplit ranges); the ranges' sums then meet through distributed shared memory, in range
// order. Grid: one cluster per tile and range, or, without ranges, as many CTAs as the GPU has SMs walking the tiles.
//
// What bounds it: the tensor pipe for BF16 tiles of 200 and more rows of x (1.5 us per unit at 256, the measured rate of a dense BF16 product). Below
// that a BF16 unit takes 0.95 us whatever the number of rows. FP32, one unit: 1.4 us for 32 MMAs (two parts,
// up to 32 rows), 1.3 us + 6.5 ns a row for 34 (Q4_K). That is not the tensor pipe (an MMA of up to 32 columns whose weights lie in tensor memory takes
// 16 clocks) but the instructions of the roles and their hand-overs; the FP32 product of up to 16 rows has a kernel of its own (jq_rows.cuh).
//
// Every wait is bounded: one that runs out records a code, raises the CTA's abort flag and all roles fall through to the exit.
#pragma once

#include <cuda_bf16.h>

#include "jq_matmul_dequant.cuh"
#include "jq_tc.cuh"

namespace jq {
namespace mm {

// How an instance splits its work. TURN: chunks of 64 k that a group of dequantiser warps makes at a time, one operand in tensor memory; what a
// turn costs besides its instructions (barrier round trips, stores' completion) is several hundred clocks, so longer turns pay wherever
// tensor memory holds an operand for every group beside the accumulator. JOINED: x's hi and lo rows are one operand of 2 nt columns
// (fewer of the small MMAs, whose issue would bound), and an operand's activation tiles arrive together.
// The FP32 instance for more than 32 rows of x reads its accumulators with sixteen warps, 32 columns per thread (with eight, their loads' latency
// bound the kernel: Q4_K 32000 x 4096, 128 rows 114 us, now 87), and has registers for two groups only.
__host__ __device__ constexpr bool one_part(int type) { return type == JQ_TYPE_Q4_K || type == JQ_TYPE_Q5_K; }
template <int TYPE, bool FP32, bool BWD, int NMAX>
struct Shape {
    static constexpr bool JOINED = FP32 && NMAX <= 32;
    static constexpr int TURN = BWD ? 1 : (!FP32 ? (NMAX <= 128 ? 4 : 1) : (JOINED || one_part(TYPE) ? 2 : 1));
    static constexpr int GROUPS = FP32 && !JOINED ? 2 : (BWD || (!FP32 && NMAX > 128) ? 4 : 3), FOLD = FP32 && !JOINED ? 16 : 4, THREADS = (3 + 4 * GROUPS + FOLD) * 32;
    static constexpr int CHUNKS = BWD ? 2 : 4;                           // chunks of 64 of the contraction in a unit
    static constexpr int TURNS = CHUNKS / TURN;
    static constexpr bool EXT = FP32 && !BWD && (one_part(TYPE) || TYPE == JQ_TYPE_Q4_1);  // 16 more columns of the contraction per unit
    static constexpr int PARTS = FP32 && !BWD && !one_part(TYPE) ? 2 : 1;                    // operand columns per value
    static constexpr int A_COLS = BWD ? 0 : 32 * PARTS * TURN + (EXT ? 8 : 0);              // tensor-memory columns of an operand
    static constexpr int B_TILES = JOINED && !BWD ? TURN + (EXT ? 1 : 0) : 1;               // activation tiles of 64 that arrive together
    static constexpr bool OWNED = TURNS == 1;                           // a raw unit is one group's own
    // FP32: ACC chunks' products go into one accumulator before the fold adds it up. The tensor core cuts every sum off towards zero, so the error
    // grows with the MMAs that add to an accumulator of full size. Products with a lo part are small: they go first (PAIRED: two chunks' operands
    // and activation tiles are waited for and used together) or into columns of their own (JOINED); then 4 (backward) or 8 are left.
    // Relative to the result's norm at k = 4096: 1.5e-7 (backward) and 1.8 to 2.3e-7. All products of 256 terms as they come left 4e-7 to 2.4e-6.
    static constexpr int ACC = BWD ? 1 : 2, ACCS = CHUNKS / ACC;
    static constexpr bool PAIRED = FP32 && !BWD && !JOINED;
    static constexpr int AHEAD = BWD && !JOINED ? 8 : 1;                // units whose scales of x the fold fetches at a time
    static constexpr int SCALES = 8 * 2 * 64 * 4 * AHEAD;               // bytes for them
    static constexpr int OPERANDS = PAIRED ? 2 / TURN + 2 : GROUPS;     // to have at least
    static_assert(!FP32 || PAIRED || TURN % ACC == 0, "");
};
constexpr int A_TILE = 128 * 128;  // 128 rows of 128 bytes
constexpr int MAX_A = 6, MAX_B = 12, MAX_RAW = 6;
constexpr int MAX_BUFS = 4;
constexpr int FACTORS = 8;   // units whose factors the fold may still need, see where they are written

constexpr int MAX_WEIGHTS = 3;

struct Args {
    // Up to three weights of one format and k, whose tiles of features follow one another. Linears on one x (q, k and v; gate and up) leave
    // the chip partly idle one by one: 32 or 86 tiles of features on 148 SMs, each launch with a fill and a drain. Together: prompt of 512
    // tokens, 8 layers of the 7B width, 2529 -> 2437 us.
    const uint8_t* q[MAX_WEIGHTS];
    const uint8_t* aux[MAX_WEIGHTS];
    float* y[MAX_WEIGHTS];
    int64_t features[MAX_WEIGHTS];  // valid features, and the row length of y
    int ft_end[MAX_WEIGHTS];        // tiles of features up to and including each weight
    int kb;           // 256-wide steps of k in the weight
    int units;        // units along the contraction
    int first_ft, ftiles;  // tiles of 128 features: those of this launch
    int ttiles, nt;   // tiles of nt rows of x
    int m;
    int ksplit;
    int sa, sb, raw;  // ring depths: weight operands, activation tiles, raw units
    int cols;         // tensor-memory columns of one accumulator
    int bufs;         // accumulators: as many as fit, up to MAX_BUFS
    int tmem;         // columns to allocate
    const float* xscale;  // FP32: scale of (contraction block, row of x): [block][xstride]
    int xstride;
    const float* bias;    // of the first weight, or null
    int* status;      // receives the code of a wait that gives up: 1 operand free, 2 weights ready, 3 activations ready or their tile free,
                      // 4 accumulator ready, 5 accumulator free, 6 raw blocks, 8 raw blocks read by all
    long long wait_clocks;  // after which a wait gives up
};

// Shared-memory matrix descriptors, 128-byte swizzle (layout type 2), descriptor version 1 (sm_100). The high word is the same for all: 1024
// bytes from one group of eight 128-byte rows to the next. K-major rows hold 64 values of the contraction; feature-major rows 64 features
// of one contraction index, and the next 64 features follow 8 KB further.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_k(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_mn(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | ((8192u >> 4) << 16); }

// D (tensor memory, lane = feature) = or += A (shared memory) . B (shared memory); descriptors by their low words
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "r"(DESC_HI)
        : "memory");
}

// The same with the A operand in tensor memory (lane = feature, two values of the contraction per column).
__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "r"(DESC_HI)
        : "memory");
}

// Which weight a tile of features belongs to, and the first tile of that weight.
__device__ __forceinline__ int weight_of(const Args& p, int ft, int& ft0) {
    const int w = ft < p.ft_end[0] ? 0 : (ft < p.ft_end[1] ? 1 : 2);
    ft0 = w == 0 ? 0 : (w == 1 ? p.ft_end[0] : p.ft_end[1]);
    return w;
}
template <typename T>
__device__ __forceinline__ T pick(const T (&v)[MAX_WEIGHTS], int w) {
    return w == 0 ? v[0] : (w == 1 ? v[1] : v[2]);
}

__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A bounded wait, as tc::mbar_wait. (A try_wait with a time limit of its own becomes a sleep in software that wakes late.) Most roles start
// before the kernel in front of this one has ended, and in the end all of them wait for what it writes: the limit counts from its end on. The
// roles that have waited for it already (AFTER) need no second turn.
template <bool AFTER = false, typename A>
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, const A& p, int code) {
    if (tc::mbar_try(bar, parity)) {
        return true;
    }
    for (int turn = AFTER ? 1 : 0; turn < 2; turn++) {
        const long long t0 = clock64();
        do {
            if (tc::mbar_try(bar, parity)) {
                return true;
            }
            if (*abort_flag != 0) {
                return false;
            }
        } while (clock64() - t0 <= p.wait_clocks);
        if (turn == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }
    }
    tc::record_status(p.status, code);
    *abort_flag = 1;
    return false;
}

// The same for a whole warp that goes on to warp-wide instructions: all lanes or none.
template <bool AFTER = false, typename A>
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, const A& p, int code) {
    return __all_sync(0xffffffffu, wait<AFTER>(bar, parity, abort_flag, p, code));
}

// Different barriers for lanes 0 .. n - 1 of a warp: one round trip for all of them (a poll takes over a hundred clocks even when the phase is
// complete, and more when all lanes poll the same barrier).
__device__ __forceinline__ bool wait_lanes(int n, int lane, uint32_t bar, uint32_t parity, volatile int* abort_flag, const Args& p, int code) {
    const bool ok = __all_sync(0xffffffffu, lane < n ? wait(bar, parity, abort_flag, p, code) : true);
    __syncwarp();
    return ok;
}

__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(c0),
                 "r"(c1), "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void ld_tmem8(float (&r)[8], uint32_t addr) {
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) {
        r[i] = __uint_as_float(u[i]);
    }
}
__device__ __forceinline__ void ld_tmem16(float (&r)[16], uint32_t addr) {
    uint32_t u[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]),
                   "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(addr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) {
        r[i] = __uint_as_float(u[i]);
    }
}
__device__ __forceinline__ void ld_tmem_done() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void st_tmem8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]),
                 "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ void sts16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// A run of 16 weights as operand values: bfloat16 (hi), or halves hi and lo.
template <bool FP32>
__device__ __forceinline__ void operand_run(const f2 (&w)[8], uint32_t (&hi)[8], uint32_t (&lo)[8]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float a, b;
        unpack2(w[i], a, b);
        if constexpr (FP32) {
            const __half2 h = __floats2half2_rn(a, b);
            hi[i] = *reinterpret_cast<const uint32_t*>(&h);
            float c, d;  // what is left: exact
            asm("{\n\t.reg .f16 l, h, m;\n\t.reg .b16 minus_one;\n\tmov.b32 {l, h}, %2;\n\tmov.b16 minus_one, 0xBC00;\n\tmov.b16 m, minus_one;\n\t"
                "fma.rn.f32.f16 %0, l, m, %3;\n\tfma.rn.f32.f16 %1, h, m, %4;\n\t}"
                : "=f"(c), "=f"(d)
                : "r"(hi[i]), "f"(a), "f"(b));
            const __half2 l = __floats2half2_rn(c, d);
            lo[i] = *reinterpret_cast<const uint32_t*>(&l);
        } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            hi[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
    }
}

// A run into this lane's row of an operand in tensor memory: pieces p, p + 1 of the row's eight are columns 4 p .. 4 p + 7.
__device__ __forceinline__ void run_to_tmem(const f2 (&w)[8], uint32_t a, int p) {
    uint32_t hi[8], lo[8];
    operand_run<false>(w, hi, lo);
    st_tmem8(a + 4 * p, hi);
}

// A run into the row at `row_addr` of an operand in shared memory (pieces p, p + 1, swizzled by row & 7; lo A_TILE further).
template <bool FP32>
__device__ __forceinline__ void run_to_smem(const f2 (&w)[8], uint32_t row_addr, int p, int swz) {
    uint32_t hi[8], lo[8];
    operand_run<FP32>(w, hi, lo);
    const uint32_t at0 = row_addr + (uint32_t)((p ^ swz) << 4), at1 = row_addr + (uint32_t)(((p + 1) ^ swz) << 4);
    sts16(at0, hi[0], hi[1], hi[2], hi[3]);
    sts16(at1, hi[4], hi[5], hi[6], hi[7]);
    if constexpr (FP32) {
        sts16(at0 + A_TILE, lo[0], lo[1], lo[2], lo[3]);
        sts16(at1 + A_TILE, lo[4], lo[5], lo[6], lo[7]);
    }
}

// A scale of x or a bias, behind the wait for the kernel that writes it: not a read-only load, which might be moved in front of that wait.
__device__ __forceinline__ float load_behind_wait(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

// Bytes of the parts of a CTA's shared memory.
template <int TYPE>
__host__ __device__ constexpr int raw_bytes() {
    return Dq<TYPE>::UNIT_Q + Dq<TYPE>::UNIT_A;
}
__host__ __device__ inline int a_bytes(bool bwd) { return bwd ? 2 * A_TILE : 0; }  // the forward product's weights go to tensor memory
__host__ __device__ inline int tile_bytes(bool fp32, int nt) { return (fp32 ? 2 * nt : nt) * 128; }
constexpr int TAIL_BYTES = FACTORS * 128 * 4 + 1024;  // row factors, barriers

// NMAX: largest tile of rows of x an FP32 instance adds up in registers.
template <int TYPE, bool FP32, bool BWD, int NMAX>
__global__ void __launch_bounds__((Shape<TYPE, FP32, BWD, NMAX>::THREADS), 1) matmul_kernel(const __grid_constant__ Args p, const __grid_constant__ CUtensorMap xmap) {
    using D = Dq<TYPE>;
    using W = Shape<TYPE, FP32, BWD, NMAX>;
    using H = Half<TYPE>;
    static_assert(FP32 || !BWD, "the backward product is FP32");
    constexpr bool HALF = FP32 && !BWD;  // weights by half arithmetic, see there
    constexpr bool EXT = W::EXT, JOINED = W::JOINED, OWNED = W::OWNED;
    constexpr int G = W::GROUPS, TURN = W::TURN, TURNS = W::TURNS, A_COLS = W::A_COLS, BT = W::B_TILES;
    static_assert(!HALF || (W::PARTS == H::TILES && EXT == H::EXT), "");
    constexpr int X_UNIT = BWD ? 128 : 256 + (EXT ? 16 : 0);  // columns of the activations per unit
    extern __shared__ uint8_t smem_unaligned[];
    const uint32_t base = (tc::smem_u32(smem_unaligned) + 1023u) & ~1023u;  // swizzled tiles start on 1024-byte boundaries
    const int SA = p.sa, SB = p.sb, R = p.raw, nt = p.nt;
    const uint32_t tile_st = (uint32_t)tile_bytes(FP32, nt), a_st = (uint32_t)a_bytes(BWD), b_st = (uint32_t)BT * tile_st;
    const uint32_t a0 = base, b0 = a0 + (uint32_t)SA * a_st, raw0 = b0 + (uint32_t)SB * b_st;
    const uint32_t fac0 = raw0 + (uint32_t)R * raw_bytes<TYPE>();
    const uint32_t scl0 = fac0 + FACTORS * 128 * 4, full_a = scl0 + W::SCALES, free_a = full_a + 8 * MAX_A, full_b = free_a + 8 * MAX_A, free_b = full_b + 8 * MAX_B;
    const uint32_t raw_full = free_b + 8 * MAX_B, raw_read = raw_full + 8 * MAX_RAW;
    const uint32_t acc_full = raw_read + 8 * MAX_RAW, acc_empty = acc_full + 8 * MAX_BUFS, fac_full = acc_empty + 8 * MAX_BUFS, max_full = fac_full + 8 * FACTORS, slot_s = max_full + 64;
    uint8_t* const generic = smem_unaligned + (slot_s - tc::smem_u32(smem_unaligned));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(generic);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(generic + 4);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int range = p.ksplit == 1 ? 0 : (int)cluster_rank();  // which range of the contraction
    const int cluster_id = (int)blockIdx.x / p.ksplit, clusters = (int)gridDim.x / p.ksplit;
    const int u0 = (int)((int64_t)range * p.units / p.ksplit), u1 = (int)((int64_t)(range + 1) * p.units / p.ksplit);
    const int tiles = p.ftiles * p.ttiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; s++) {
            tc::mbar_init(full_a + 8 * s, 4);  // a group's four warps
            tc::mbar_init(free_a + 8 * s, 1);
        }
        for (int s = 0; s < SB; s++) {
            tc::mbar_init(full_b + 8 * s, 1);
            tc::mbar_init(free_b + 8 * s, 1);
        }
        for (int r = 0; r < R; r++) {
            tc::mbar_init(raw_full + 8 * r, 1);
            tc::mbar_init(raw_read + 8 * r, OWNED ? 4 : 4 * G);
        }
        for (int i = 0; i < MAX_BUFS; i++) {
            tc::mbar_init(acc_full + 8 * i, 1);
            tc::mbar_init(acc_empty + 8 * i, W::FOLD);
        }
        for (int i = 0; i < FACTORS; i++) {
            tc::mbar_init(fac_full + 8 * i, BWD ? 2 : 4);
        }
        for (int i = 0; i < 8; i++) {
            tc::mbar_init(max_full + 8 * i, 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_s), "r"(p.tmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    if (p.ksplit > 1) {
        cluster_sync();
    }
    tc::fence_after_sync();
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t tmem_a = tmem + (uint32_t)(p.bufs * p.cols);  // the ring of weight operands behind the accumulators

    if (warp == 0) {
        // ---- activation tiles -------------------------------------------------------------------------------------------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // x is written by the kernel in front
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
                const int t0 = (tile % p.ttiles) * nt;
                for (int u = u0; u < u1 && ok; u++) {
                    constexpr int ALL = W::CHUNKS + (EXT ? 1 : 0);  // tiles per unit; the last one is the 16 more columns
                    for (int i = 0; i < ALL;) {
                        const int last = BT > 1 ? (i + TURN == W::CHUNKS ? ALL : i + TURN) : i + 1;
                        if (!(ok = wait<true>(free_b + 8 * s, ph, abort_flag, p, 3))) {
                            break;
                        }
                        const uint32_t bar = full_b + 8 * s;
                        uint32_t dst = b0 + (uint32_t)s * b_st;
                        tc::mbar_expect_tx(bar, (uint32_t)(last - i) * tile_st);
                        for (; i < last; i++, dst += tile_st) {  // FP32: hi rows, then lo rows
                            tma_3d(dst, &xmap, bar, u * X_UNIT + i * 64, t0, 0);
                        }
                        if (++s == SB) {
                            s = 0;
                            ph ^= 1;
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issue: the warp goes through the loop together, so that addresses and descriptors stay in uniform registers, and one elected
        // lane issues. (A lone lane's loop, converting every operand, took 300 clocks a stage beside busy dequantiser warps.)
        const uint32_t fmt = FP32 ? 0u : ((1u << 7) | (1u << 10));  // halves or bfloat16
        const uint32_t id = (1u << 4) | fmt | (BWD ? 1u << 15 : 0u) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t id_n = id | ((uint32_t)(nt >> 3) << 17), id_2n = id | ((uint32_t)(2 * nt >> 3) << 17);
        const uint32_t lo_rows = (uint32_t)(nt * 128) >> 4;  // from x's hi rows to its lo rows, in descriptor units
        int s = 0, sb = 0, buf = 0;
        uint32_t ph = 0, phb = 0, aph = 0;
        bool ok = true, ready = false, ready_b = false;
        if constexpr (W::PAIRED) {
            constexpr int OPS = 2 / TURN;        // operands of two chunks
            constexpr bool TWO = W::PARTS == 2;  // the weights have a lo part
            for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
                for (int u = u0; u < u1 && ok; u++) {
#pragma unroll
                    for (int pair = 0; pair < 2; pair++) {
                        // lane 0 (and 1) waits for the operand(s), the next two for an activation tile each, the last one for the accumulator
                        uint32_t a_at[OPS], a_bar[OPS], b_at[2], b_bar[2], bar = 0, parity = 0;
#pragma unroll
                        for (int o = 0; o < OPS; o++) {
                            a_at[o] = tmem_a + (uint32_t)(s * A_COLS);
                            a_bar[o] = free_a + 8 * s;
                            bar = lane == o ? full_a + 8 * s : bar;
                            parity = lane == o ? ph : parity;
                            if (++s == SA) {
                                s = 0;
                                ph ^= 1;
                            }
                        }
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            b_at[b] = desc_k(b0 + (uint32_t)sb * b_st);
                            b_bar[b] = free_b + 8 * sb;
                            bar = lane == OPS + b ? full_b + 8 * sb : bar;
                            parity = lane == OPS + b ? phb : parity;
                            if (++sb == SB) {
                                sb = 0;
                                phb ^= 1;
                            }
                        }
                        bar = lane == OPS + 2 ? acc_empty + 8 * buf : bar;
                        parity = lane == OPS + 2 ? aph ^ 1u : parity;
                        if (!(ok = wait_lanes(OPS + 3, lane, bar, parity, abort_flag, p, lane < OPS ? 2 : (lane < OPS + 2 ? 3 : 5)))) {
                            break;
                        }
                        tc::fence_after_sync();
                        const uint32_t d = tmem + (uint32_t)(buf * p.cols), d_bar = acc_full + 8 * buf;
                        if (++buf == p.bufs) {
                            buf = 0;
                            aph ^= 1;
                        }
                        if (elect_one()) {
                            // first all products with a lo part
#pragma unroll
                            for (int c = 0; c < 2; c++) {
                                const uint32_t ta = a_at[c / TURN] + (uint32_t)(c % TURN * 32 * W::PARTS);  // 16 of the contraction are 8 columns
#pragma unroll
                                for (uint32_t ks = 0; ks < 4; ks++) {
                                    mma_ta(d, ta + 8 * ks, b_at[c] + lo_rows + 2 * ks, id_n, (uint32_t)c | ks);
                                    if constexpr (TWO) {
                                        mma_ta(d, ta + 32 + 8 * ks, b_at[c] + 2 * ks, id_n, 1u);
                                    }
                                }
                            }
#pragma unroll
                            for (int c = 0; c < 2; c++) {
                                const uint32_t ta = a_at[c / TURN] + (uint32_t)(c % TURN * 32 * W::PARTS);
#pragma unroll
                                for (uint32_t ks = 0; ks < 4; ks++) {
                                    mma_ta(d, ta + 8 * ks, b_at[c] + 2 * ks, id_n, 1u);
                                }
                                tc::umma_commit(b_bar[c]);
                            }
                        }
                        __syncwarp();
                        if (EXT && pair == 1) {  // the 16 more columns; their tile is not waited for with the others, which it would keep from being refilled
                            const uint32_t bd = desc_k(b0 + (uint32_t)sb * b_st), be = free_b + 8 * sb;
                            if (!(ok = wait_lanes(1, lane, full_b + 8 * sb, phb, abort_flag, p, 3))) {
                                break;
                            }
                            tc::fence_after_sync();
                            if (++sb == SB) {
                                sb = 0;
                                phb ^= 1;
                            }
                            if (elect_one()) {
                                const uint32_t te = a_at[OPS - 1] + TURN * 32 * W::PARTS;
                                mma_ta(d, te, bd + lo_rows, id_n, 1u);
                                mma_ta(d, te, bd, id_n, 1u);
                                tc::umma_commit(be);
                            }
                            __syncwarp();
                        }
                        if (elect_one()) {
#pragma unroll
                            for (int o = 0; o < OPS; o++) {
                                tc::umma_commit(a_bar[o]);
                            }
                            tc::umma_commit(d_bar);
                        }
                        __syncwarp();
                    }
                }
            }
        }
        for (int tile = cluster_id; !W::PAIRED && tile < tiles && ok; tile += clusters) {
            bool first = true;
            for (int u = u0; u < u1 && ok; u++) {
                if (!FP32 && u == u0) {
                    if (!(ok = wait_warp(acc_empty + 8 * buf, aph ^ 1u, abort_flag, p, 5))) {
                        break;
                    }
                    first = true;
                }
#pragma unroll
                for (int turn = 0; turn < TURNS; turn++) {
                    if (FP32 && !(ok = wait_warp(acc_empty + 8 * buf, aph ^ 1u, abort_flag, p, 5))) {
                        break;
                    }
                    if (!(ok = __all_sync(0xffffffffu, ready) || wait_warp(full_a + 8 * s, ph, abort_flag, p, 2))) {
                        break;
                    }
                    // asked before this operand's MMAs are issued: the answer takes over a hundred clocks even when it is yes
                    const int sn = s + 1 == SA ? 0 : s + 1;
                    const uint32_t phn = sn == 0 ? ph ^ 1 : ph;
                    ready = tc::mbar_test(full_a + 8 * sn, phn);
                    constexpr int LAST = TURN + (EXT ? 1 : 0);
#pragma unroll
                    for (int c = 0; c < LAST; c++) {
                        const bool ext = c == TURN;
                        if (ext && turn < TURNS - 1) {
                            break;
                        }
                        if (BT == 1 || c == 0) {
                            if (!(ok = __all_sync(0xffffffffu, ready_b) || wait_warp(full_b + 8 * sb, phb, abort_flag, p, 3))) {
                                break;
                            }
                            ready_b = tc::mbar_test(full_b + 8 * (sb + 1 == SB ? 0 : sb + 1), sb + 1 == SB ? phb ^ 1 : phb);
                            tc::fence_after_sync();
                        }
                        if (FP32 && !ext && c % W::ACC == 0) {  // the next accumulator (the turn's first one is waited for above)
                            if (c > 0 && !(ok = wait_warp(acc_empty + 8 * buf, aph ^ 1u, abort_flag, p, 5))) {
                                break;
                            }
                            first = true;
                            tc::fence_after_sync();
                        }
                        const uint32_t d = tmem + (uint32_t)(buf * p.cols), d_lo = d + (uint32_t)nt;  // JOINED: sums with a lo part in columns of their own
                        // x: hi, lo; 16 of the contraction are 32 bytes
                        const uint32_t bd = desc_k(b0 + (uint32_t)sb * b_st + (BT == 1 ? 0u : (uint32_t)c * tile_st)), bl = bd + lo_rows;
                        const bool b_done = BT == 1 || c == LAST - 1 || (turn < TURNS - 1 && c == TURN - 1);
                        const bool a_done = turn < TURNS - 1 ? c == TURN - 1 : c == LAST - 1;
                        const bool d_done = FP32 ? (ext || ((c + 1) % W::ACC == 0 && !(EXT && turn == TURNS - 1 && c == TURN - 1)))
                                                 : a_done && turn == TURNS - 1 && u == u1 - 1;
                        if (elect_one()) {
                            const uint32_t acc = first ? 0u : 1u;
                            if constexpr (BWD) {
                                // feature-major weights: 16 of the contraction are two 1024-byte groups
                                const uint32_t ad = desc_mn(a0 + (uint32_t)s * a_st), al = ad + (A_TILE >> 4);
#pragma unroll
                                for (uint32_t ks = 0; ks < 4; ks++) {
                                    if constexpr (JOINED) {
                                        mma(d, ad + 128 * ks, bd + 2 * ks, id_2n, acc | ks);  // hi x (hi | lo)
                                        mma(d_lo, al + 128 * ks, bd + 2 * ks, id_n, 1u);      // lo x hi
                                    } else {
                                        mma(d, al + 128 * ks, bd + 2 * ks, id_n, acc | ks);
                                        mma(d, ad + 128 * ks, bl + 2 * ks, id_n, 1u);
                                    }
                                }
                                if constexpr (!JOINED) {
#pragma unroll
                                    for (uint32_t ks = 0; ks < 4; ks++) {
                                        mma(d, ad + 128 * ks, bd + 2 * ks, id_n, 1u);
                                    }
                                }
                            } else {
                                constexpr bool TWO = W::PARTS == 2;                                        // the weights have a lo part
                                const uint32_t ta = tmem_a + (uint32_t)(s * A_COLS + c * 32 * W::PARTS);  // 16 of the contraction are 8 columns
#pragma unroll
                                for (uint32_t ks = 0; ks < (ext ? 1 : 4); ks++) {
                                    if constexpr (JOINED) {
                                        mma_ta(d, ta + 8 * ks, bd + 2 * ks, id_2n, acc | ks);  // hi x (hi | lo)
                                        if (TWO && !ext) {
                                            mma_ta(d_lo, ta + 32 + 8 * ks, bd + 2 * ks, id_n, 1u);
                                        }
                                    } else {
                                        mma_ta(d, ta + 8 * ks, bd + 2 * ks, id_n, acc | ks);
                                    }
                                }
                            }
                            if (b_done) {
                                tc::umma_commit(free_b + 8 * sb);
                            }
                            if (a_done) {
                                tc::umma_commit(free_a + 8 * s);
                            }
                            if (d_done) {
                                tc::umma_commit(acc_full + 8 * buf);
                            }
                        }
                        __syncwarp();
                        first = false;
                        if (d_done && ++buf == p.bufs) {
                            buf = 0;
                            aph ^= 1;
                        }
                        if (b_done && ++sb == SB) {
                            sb = 0;
                            phb ^= 1;
                        }
                    }
                    if (!ok) {
                        break;
                    }
                    s = sn;
                    ph = phn;
                }
            }
        }
    } else if (warp == 2) {
        // ---- raw units, in the order in which they are used: tile after tile, u0 .. u1 - 1 ---------------------------------------
        if (lane == 0) {
            int r = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
                const int ft = p.first_ft + tile / p.ttiles;
                int ft0;
                const int wi = weight_of(p, ft, ft0);
                const uint8_t* const wq = pick(p.q, wi);
                const uint8_t* const wa = pick(p.aux, wi);
                for (int u = u0; u < u1; u++) {
                    const int64_t at = BWD ? (int64_t)u * p.kb + (ft >> 1) : (int64_t)(ft - ft0) * p.kb + u;
                    if (!(ok = wait(raw_read + 8 * r, ph, abort_flag, p, 8))) {
                        break;
                    }
                    const uint32_t dst = raw0 + (uint32_t)r * raw_bytes<TYPE>(), bar = raw_full + 8 * r;
                    tc::mbar_expect_tx(bar, raw_bytes<TYPE>());
                    tc::bulk_load(dst, wq + at * D::UNIT_Q, D::UNIT_Q, bar);
                    if constexpr (D::UNIT_A > 0) {
                        tc::bulk_load(dst + D::UNIT_Q, wa + at * D::UNIT_A, D::UNIT_A, bar);
                    }
                    if (++r == R) {
                        r = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp < 3 + 4 * G) {
        // ---- dequantise ------------------------------------------------------------------------------------------------------------
        const int tid = (threadIdx.x - 96) & 127, group = (warp - 3) >> 2;
        // forward: a thread has one row of the unit; backward: 64 rows x the two 64-feature halves of this CTA's 128 features
        // (the warp's place among tensor memory's lanes, 32 (warp % 4) .., decides which)
        const int row0 = BWD ? (tid & 63) : (warp & 3) * 32 + lane;
        const uint32_t my_lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t row_at = (BWD ? (uint32_t)(tid >> 6) * 8192u : 0u) + (uint32_t)row0 * 128u;  // of the thread's row in the operand tile
        int s = group, r = 0, at_unit = 0;
        uint32_t ph = 1, rph = 0;  // SA >= G: the barrier of a group's next operand is never two phases behind
        bool ok = true, raw_ready = false;
        int first = OWNED ? 0 : group;  // the group's first turn of the unit, or of a later one
        for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
            const int h = (p.first_ft + tile / p.ttiles) & 1;  // backward: which 128 of the super-block's features
            for (int u = u0; u < u1; u++, at_unit++) {
                // Units of the whole ring in turn, where they are the group's own (R is a multiple of G, so a slot belongs to one group); else
                // every group waits for and gives back every unit. Either way no group is a turn of the ring away from a barrier it tests.
                const int rn = r + 1 == R ? 0 : r + 1;
                const uint32_t rphn = rn == 0 ? rph ^ 1 : rph;
                const bool mine = OWNED ? at_unit % G == group : first < TURNS;
                if (OWNED && !mine) {
                    r = rn;
                    rph = rphn;
                    continue;
                }
                if (!__all_sync(0xffffffffu, raw_ready) && !(ok = wait_warp(raw_full + 8 * r, rph, abort_flag, p, 6))) {
                    break;
                }
                if constexpr (OWNED) {
                    const int ro = r + G >= R ? r + G - R : r + G;  // the group's next unit
                    raw_ready = tc::mbar_test(raw_full + 8 * ro, r + G >= R ? rph ^ 1 : rph);
                } else {
                    raw_ready = tc::mbar_test(raw_full + 8 * rn, rphn);
                }
                if (!mine) {
                    __syncwarp();
                    if (lane == 0) {
                        tc::mbar_arrive(raw_read + 8 * r);
                    }
                } else {
                    const uint32_t uq = raw0 + (uint32_t)r * raw_bytes<TYPE>(), ua = uq + D::UNIT_Q;
                    typename D::Head head;
                    float f0 = 1.0f, f1 = 1.0f;
                    uint32_t unit_factor = 0, unit_factor1 = 0;  // what the fold multiplies the unit's sums by
                    if constexpr (!BWD) {
                        head = D::head(uq, ua, row0);
                    }
                    if constexpr (HALF) {
                        unit_factor = __float_as_uint(H::factor(head));
                    }
                    if constexpr (BWD) {
                        // For every 32 features a power of two brings the largest weight that their blocks can hold to [2^13, 2^14); the fold
                        // multiplies by its inverse. (Features are outputs of their own: with one power of two for all 128, blocks 2^-20 times
                        // their neighbours' lost bits.) The unit's maxima [block][warp] lie behind its factors.
                        const int slot = at_unit & 7;  // a group is at most four turns, so fewer than eight units, ahead of another
                        const uint32_t maxima = fac0 + (uint32_t)slot * 512u + 64u;
                        if (first == 0) {
                            float b[4];
                            D::bounds(D::head(uq, ua, tid), h, b);
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(b[i]));
                                if (lane == 0) {
                                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(maxima + 16u * i + 4u * (uint32_t)(tid >> 5)), "r"(m) : "memory");
                                }
                            }
                            if (lane == 0) {
                                tc::mbar_arrive(max_full + 8 * slot);
                            }
                        }
                        if (!(ok = wait_warp(max_full + 8 * slot, (uint32_t)(at_unit >> 3) & 1u, abort_flag, p, 8))) {
                            break;
                        }
                        auto exponent = [&](int block) {
                            const uint4 m = lds16(maxima + 16u * (uint32_t)block);
                            const uint32_t e = max(max(m.x, m.y), max(m.z, m.w)) >> 23;
                            return e < 40u ? 40u : (e > 254u ? 254u : e);
                        };
                        const uint32_t e0 = exponent(2 * (tid >> 6)), e1 = exponent(2 * (tid >> 6) + 1);
                        f0 = __uint_as_float((267u - e0) << 23);
                        f1 = __uint_as_float((267u - e1) << 23);
                        unit_factor = (e0 - 13u) << 23;
                        unit_factor1 = (e1 - 13u) << 23;
                    }
                    for (int turn = first; turn < TURNS; turn += G) {
                        const bool ready = tc::mbar_test(free_a + 8 * s, ph);  // asked early: the answer takes longer than it looks
                        const int row = BWD ? row0 + 64 * turn : row0, c0 = BWD ? 2 * h + (tid >> 6) : turn * TURN;
                        if constexpr (BWD) {
                            head = D::head(uq, ua, row);
                        }
                        typename D::Raw raw[TURN];
#pragma unroll
                        for (int j = 0; j < TURN; j++) {
                            raw[j] = D::load(uq, row, c0 + j);
                        }
                        // This warp has read all it needs of the unit once its loads are done. Program order alone does not see to that: with an arrival right
                        // behind loads whose values are used later, the next unit was copied over what they had yet to read (backward, 11008 x 4096
                        // Q4_0, 128 rows: wrong weights in 179 of 200 calls). FP32 forward gives the unit back when its values have gone to tensor
                        // memory; the others, which use theirs behind another wait, behind a fence. (A vote on a word of every load, in all forms:
                        // Q8_0 11008 x 4096, 200 rows 65.7 us, now 63.8; Q4_K 57.6 and 57.4; BF16 Q4_K 512 rows 46.1 and 45.3; backward Q6_K 4096 x 4096,
                        // 128 rows 28.4 and 27.9. Only Q4_1 was faster with it: 300 rows 92.2 and 92.9.)
                        const bool done = OWNED || turn + G >= TURNS;
                        if (!HALF && done) {
                            tc::reads_before_refill();
                            if (lane == 0) {
                                tc::mbar_arrive(raw_read + 8 * r);
                            }
                        }
                        // the first values while it is on its way
                        f2 w0[8], w1[8];
                        if constexpr (!HALF) {
                            D::values(head, raw[0], c0, 0, f0, f1, w0, w1);
                        }
                        if (!__all_sync(0xffffffffu, ready) && !(ok = wait_warp(free_a + 8 * s, ph, abort_flag, p, 1))) {
                            break;
                        }
                        if (FP32 && turn == 0) {
                            // The unit's factors for the fold, into a ring of FACTORS units. This operand's slot is free, so what it held SA
                            // operands ago went through the tensor core, into an accumulator that the fold had emptied: the fold has
                            // finished the accumulator `bufs` before that one, and with it the unit eight before this one as
                            // SA TURN / ACC + bufs <= 7 ACCS + 1 (at most 6 + 4 and 15).
                            const uint32_t fa = fac0 + (uint32_t)(at_unit & (FACTORS - 1)) * 512u;
                            if constexpr (!BWD) {
                                asm volatile("st.shared.u32 [%0], %1;" ::"r"(fa + 4u * (uint32_t)row0), "r"(unit_factor) : "memory");
                            } else if ((tid & 63) == 0) {  // one for every 32 features
                                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(fa + 8u * (uint32_t)(tid >> 6)), "r"(unit_factor), "r"(unit_factor1) : "memory");
                            }
                            __syncwarp();
                            if (lane == 0 && (!BWD || (tid & 63) == 0)) {
                                tc::mbar_arrive(fac_full + 8 * (at_unit & (FACTORS - 1)));
                            }
                        }
                        if constexpr (BWD) {  // operand row = contraction index, 64 features a row
                            const uint32_t to = a0 + (uint32_t)s * a_st + row_at;
                            run_to_smem<FP32>(w0, to, D::piece(0, 0), row0 & 7);
                            run_to_smem<FP32>(w1, to, D::piece(0, 1), row0 & 7);
                            D::values(head, raw[0], c0, 1, f0, f1, w0, w1);
                            run_to_smem<FP32>(w0, to, D::piece(1, 0), row0 & 7);
                            run_to_smem<FP32>(w1, to, D::piece(1, 1), row0 & 7);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic stores -> visible to the tensor core
                        } else {
                            const uint32_t to = tmem_a + my_lanes + (uint32_t)(s * A_COLS);
                            tc::fence_after_sync();
#pragma unroll
                            for (int j = 0; j < TURN; j++) {
                                const uint32_t tj = to + (uint32_t)(j * 32 * W::PARTS);
                                if constexpr (HALF) {
                                    const typename H::Scales sc = H::scales(head, c0 + j);
#pragma unroll
                                    for (int i = 0; i < 4; i++) {
                                        uint32_t hi[8], lo[8];
                                        H::values(head, raw[j], sc, c0 + j, i >> 1, i & 1, hi, lo);
                                        st_tmem8(tj + 4 * D::piece(i >> 1, i & 1), hi);
                                        if constexpr (W::PARTS == 2) {
                                            st_tmem8(tj + 32 + 4 * D::piece(i >> 1, i & 1), lo);
                                        }
                                    }
                                } else {
                                    if (j > 0) {
                                        D::values(head, raw[j], c0 + j, 0, f0, f1, w0, w1);
                                    }
                                    run_to_tmem(w0, tj, D::piece(0, 0));
                                    run_to_tmem(w1, tj, D::piece(0, 1));
                                    D::values(head, raw[j], c0 + j, 1, f0, f1, w0, w1);
                                    run_to_tmem(w0, tj, D::piece(1, 0));
                                    run_to_tmem(w1, tj, D::piece(1, 1));
                                }
                            }
                            if constexpr (EXT) {
                                if (turn == TURNS - 1) {
                                    uint32_t v[8];
                                    H::ext(head, v);
                                    st_tmem8(to + TURN * 32 * W::PARTS, v);
                                }
                            }
                            if (HALF && done) {
                                __syncwarp();
                                if (lane == 0) {
                                    tc::mbar_arrive(raw_read + 8 * r);
                                }
                            }
                            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                            tc::fence_before_sync();
                        }
                        __syncwarp();
                        if (lane == 0) {
                            tc::mbar_arrive(full_a + 8 * s);
                        }
                        if ((s += G) >= SA) {
                            s -= SA;
                            ph ^= 1;
                        }
                        first += G;
                    }
                    if (!ok) {
                        break;
                    }
                }
                first = OWNED ? 0 : first - TURNS;
                r = rn;
                rph = rphn;
            }
        }
    } else {
        // ---- accumulators to y -----------------------------------------------------------------------------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the scales of x; and y may be read by the kernel in front
        constexpr int PARTS = W::FOLD / 4;
        const int group = warp & 3, part = (warp - 3 - 4 * G) >> 2;  // a warp may only read lanes 32 (warp % 4) .. of tensor memory
        const int lane_row = group * 32 + lane;
        const uint32_t lanes = (uint32_t)(group * 32) << 16;
        // this warp's columns of the tile, a multiple of 16: up to NMAX / PARTS in registers (BF16: all)
        const int c0 = part * (FP32 ? NMAX / PARTS : nt / PARTS), cols = FP32 ? max(0, min(NMAX / PARTS, nt - c0)) : nt / PARTS;
        int chunk = 0, buf = 0;
        uint32_t aph = 0;
        bool ok = true;
        auto release = [&] {  // the accumulator is read: the next one
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                tc::mbar_arrive(acc_empty + 8 * buf);
            }
            if (++buf == p.bufs) {
                buf = 0;
                aph ^= 1;
            }
        };
        for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
            const int ft = p.first_ft + tile / p.ttiles, t0 = (tile % p.ttiles) * nt;
            int ft0;
            const int wi = weight_of(p, ft, ft0);
            const int64_t feature = (int64_t)(ft - ft0) * 128 + lane_row, features = pick(p.features, wi);
            const bool valid = feature < features;
            const float bias = p.bias != nullptr && wi == 0 && valid ? load_behind_wait(p.bias + feature) : 0.0f;
            // Columns c .. c + 7 of the tile are finished: to y, or (contraction split over the cluster) to this CTA's own partial tile
            // [column][128]. One warp per scheduler does this, so it is kept short: no test per value where the tile is whole.
            const int64_t row_bytes = features * 4;
            uint8_t* const yt = reinterpret_cast<uint8_t*>(pick(p.y, wi) + (int64_t)t0 * features + feature);
            const bool whole = t0 + nt <= p.m;
            auto emit8 = [&](int c, const float (&v)[8]) {
                if (p.ksplit > 1) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + (uint32_t)((c + i) * 128 + lane_row) * 4u), "f"(v[i]) : "memory");
                    }
                } else if (valid) {
                    uint8_t* at = yt + (int64_t)c * row_bytes;
                    if (whole) {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            *reinterpret_cast<float*>(at) = v[i] + bias;
                            at += row_bytes;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            if (t0 + c + i < p.m) {
                                *reinterpret_cast<float*>(at) = v[i] + bias;
                            }
                            at += row_bytes;
                        }
                    }
                }
            };
            if constexpr (FP32) {
                constexpr int C = NMAX / PARTS, C32 = C < 32 ? 32 : C;  // columns per thread
                f2 sum[C / 2];
#pragma unroll
                for (int i = 0; i < C / 2; i++) {
                    sum[i] = 0;
                }
                // The scales of a unit's columns: fetched by the lanes AHEAD units at a time, read back as broadcasts. (A load takes up to 2000 clocks while the
                // weights stream: one unit ahead, the backward form's units waited for it: Q4_K 32000 x 4096, 128 rows 147 us, now 138; 4096 x 4096
                // 28.5 and 27.2. The forward forms do not wait for it.)
                constexpr int AHEAD = W::AHEAD, NEXT = (C * AHEAD + 31) / 32;
                const uint32_t scl = scl0 + (uint32_t)(warp - 3 - 4 * G) * (8u * C32 * AHEAD);
                float next[NEXT];
                const float* xs = p.xscale + (int64_t)u0 * p.xstride + t0 + c0 + lane;  // of the units that are fetched next
                auto fetch = [&](int u) {
#pragma unroll
                    for (int i = 0; i < NEXT; i++) {
                        const int on = AHEAD > 1 ? i : 0, off = AHEAD > 1 ? 0 : 32 * i;  // (AHEAD > 1: 32 columns)
                        next[i] = lane + off < cols && (AHEAD == 1 || u + on < u1) ? load_behind_wait(xs + (int64_t)on * p.xstride + off) : 0.0f;
                    }
                    xs += (int64_t)AHEAD * p.xstride;
                };
                fetch(u0);
                for (int u = u0; u < u1; u++, chunk++) {
                    const int step = (u - u0) % AHEAD, block = (u - u0) / AHEAD & 1;
                    const uint32_t sb = scl + (uint32_t)((block * AHEAD + step) * C32) * 4u;
                    if (step == 0) {
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < NEXT; i++) {
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(sb + (uint32_t)(lane + 32 * i) * 4u), "f"(next[i]) : "memory");
                        }
                        if (u + AHEAD < u1) {
                            fetch(u + AHEAD);
                        }
                        __syncwarp();
                    }
                    if (!(ok = wait_warp<true>(fac_full + 8 * (chunk & (FACTORS - 1)), (uint32_t)(chunk / FACTORS) & 1u, abort_flag, p, 6))) {
                        break;
                    }
                    float f;
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(fac0 + (uint32_t)(chunk & (FACTORS - 1)) * 512u + 4u * (uint32_t)(BWD ? group : lane_row)));
                    const f2 ff = pack2(f, f);
#pragma unroll 1
                    for (int a = 0; a < W::ACCS; a++) {
                        if (!(ok = wait_warp<true>(acc_full + 8 * buf, aph, abort_flag, p, 4))) {
                            break;
                        }
                        tc::fence_after_sync();
                        const uint32_t d = tmem + lanes + (uint32_t)(buf * p.cols + c0);
#pragma unroll
                        for (int c = 0; c < C / 16; c++) {
                            if (c * 16 < cols) {
                                float hi[16], lo[16];
                                ld_tmem16(hi, d + c * 16);
                                if constexpr (JOINED) {
                                    ld_tmem16(lo, d + nt + c * 16);
                                }
                                ld_tmem_done();
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const uint4 x4 = lds16(sb + c * 64 + j * 16);
                                    const f2 sc[2] = {pack2(__uint_as_float(x4.x), __uint_as_float(x4.y)), pack2(__uint_as_float(x4.z), __uint_as_float(x4.w))};
#pragma unroll
                                    for (int i = 2 * j; i < 2 * j + 2; i++) {
                                        f2 v = mul2(pack2(hi[2 * i], hi[2 * i + 1]), ff);
                                        if constexpr (JOINED) {
                                            v = fma2(pack2(lo[2 * i], lo[2 * i + 1]), ff, v);
                                        }
                                        sum[c * 8 + i] = fma2(v, sc[i & 1], sum[c * 8 + i]);
                                    }
                                }
                            }
                        }
                        release();
                    }
                    if (!ok) {
                        break;
                    }
                }
                if (!ok) {
                    break;
                }
                // (the last accumulator is complete: every tile in shared memory is used up and may hold the partial tile)
#pragma unroll
                for (int c = 0; c < C / 8; c++) {
                    if (c * 8 < cols) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            unpack2(sum[c * 4 + i], v[2 * i], v[2 * i + 1]);
                        }
                        emit8(c0 + c * 8, v);
                    }
                }
            } else {
                if (!(ok = wait_warp<true>(acc_full + 8 * buf, aph, abort_flag, p, 4))) {
                    break;
                }
                tc::fence_after_sync();
                const uint32_t d = tmem + lanes + (uint32_t)(buf * p.cols + c0);
                for (int c = 0; c < cols; c += 16) {
                    float v[8], w[8];
                    ld_tmem8(v, d + c);
                    ld_tmem8(w, d + c + 8);
                    ld_tmem_done();
                    emit8(c0 + c, v);
                    emit8(c0 + c + 8, w);
                }
                release();
            }
        }
    }

    // ---- exit -----------------------------------------------------------------------------------------------------------------------
    tc::fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        for (int i = 0; i < 1000; i++) {
            __nanosleep(1000);  // copies that may still be in flight land long before this millisecond is over
        }
    }
    __syncthreads();
    if (p.ksplit > 1) {
        cluster_sync();  // partial tiles are complete
    }
    if (p.ksplit > 1 && *abort_flag == 0) {
        // columns range, range + ksplit, .. of the tile: the ranges' sums in order
        const int ft = p.first_ft + cluster_id / p.ttiles, t0 = (cluster_id % p.ttiles) * nt;
        int ft0;
        const int wi = weight_of(p, ft, ft0);
        const int64_t f0 = (int64_t)(ft - ft0) * 128, features = pick(p.features, wi);
        float* const y = pick(p.y, wi);
        const float* const bias = wi == 0 ? p.bias : nullptr;
        const int mine = (nt - range + p.ksplit - 1) / p.ksplit * 32;  // pieces of four features of a column
        constexpr int BATCH = 2, MOST = 4;  // pieces and ranges in flight: another CTA's memory is most of a microsecond away
        for (int i0 = threadIdx.x; i0 < mine; i0 += BATCH * W::THREADS) {
            float4 sum[BATCH];
#pragma unroll
            for (int j = 0; j < BATCH; j++) {
                sum[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            for (int g0 = 0; g0 < p.ksplit; g0 += MOST) {
                float4 v[MOST][BATCH];
#pragma unroll
                for (int g = 0; g < MOST; g++) {
                    const int part = g0 + g;
                    const bool there = part < p.ksplit;
                    const uint32_t from = map_rank(base, (uint32_t)(there ? part : 0));
#pragma unroll
                    for (int j = 0; j < BATCH; j++) {
                        const int i = i0 + j * W::THREADS, col = range + (i >> 5) * p.ksplit;
                        v[g][j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // a missing range adds an exact zero
                        if (there && i < mine) {
                            asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                         : "=f"(v[g][j].x), "=f"(v[g][j].y), "=f"(v[g][j].z), "=f"(v[g][j].w)
                                         : "r"(from + (uint32_t)(col * 128 + (i & 31) * 4) * 4u));
                        }
                    }
                }
#pragma unroll
                for (int g = 0; g < MOST; g++) {
#pragma unroll
                    for (int j = 0; j < BATCH; j++) {
                        sum[j].x += v[g][j].x; sum[j].y += v[g][j].y; sum[j].z += v[g][j].z; sum[j].w += v[g][j].w;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < BATCH; j++) {
                const int i = i0 + j * W::THREADS, col = range + (i >> 5) * p.ksplit;
                const int64_t f = f0 + (i & 31) * 4;
                if (i >= mine || t0 + col >= p.m) {
                    continue;
                }
                float* const at = y + (int64_t)(t0 + col) * features + f;
                const float one[4] = {sum[j].x, sum[j].y, sum[j].z, sum[j].w};
                if (f + 4 <= features && ((uintptr_t)at & 15) == 0) {
                    float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (bias != nullptr) {
                        b = make_float4(load_behind_wait(bias + f), load_behind_wait(bias + f + 1), load_behind_wait(bias + f + 2), load_behind_wait(bias + f + 3));
                    }
                    *reinterpret_cast<float4*>(at) = make_float4(one[0] + b.x, one[1] + b.y, one[2] + b.z, one[3] + b.w);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (f + q < features) {
                            at[q] = one[q] + (bias != nullptr ? load_behind_wait(bias + f + q) : 0.0f);
                        }
                    }
                }
            }
        }
    }
    if (p.ksplit > 1) {
        __syncthreads();
        cluster_sync();  // no CTA leaves while another still reads its partial tile
    }
    if (warp == 1) {
        tc::fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem) : "memory");
    }
}

}  // namespace mm
}  // namespace jq
