// Q8_0-weight matrix products next to attention: the QKV projections before it and the output projection
// after it (flare-core/src/model.rs:2016-2136, 2249-2291), for `batch` input vectors at once.
//
// The arithmetic is the reference's, operation for operation, so that the result is the CPU's bit for bit
// (flare-core/src/model.rs, the branch compiled on x86_64):
//   quantize_input_q8_0 (5507-5527)     per 32 inputs: amax, d = amax / 127, id = 127 / amax (0 when d == 0),
//                                       q = round(x * id) as i8; the block scale d stays f32
//   matvec_q8_0_preq_into (8066-8100)   per row, blocks in ascending order:
//                                       sum += (w_scale * x_scale[block]) * (int32 dot of the 32 int8 pairs) as f32
//                                       with w_scale the block's f16 scale widened exactly; separate multiplies and add
// The integer dot is exact in any order (one int8 MMA per block of 32); the f32 sum over a row's blocks is the only
// order-sensitive part and stays sequential.
#include "common.cuh"
#include "q8_input.cuh"
#include "tma.cuh"
#include <algorithm>
#include <mutex>

// The GGUF block stream (f16 scale + 32 x i8 per 34 bytes) taken apart at upload into the order the product reads:
// tiles of 16 rows, per tile its blocks in ascending order, per block BLK bytes: the 16 x 32 codes as the int8 MMA's A
// operand (16 bytes per lane), then the 16 scales as (row g, row g + 8) pairs.  A run of blocks of a tile is one
// contiguous piece on a 16-byte boundary whatever the width, and the bytes are the stream's own 34 per 32 values.
struct flare_weight {
    flare_attn_ctx* ctx = nullptr;
    int rows = 0, cols = 0;
    int paired = 0;              // rows are [gate | up]: tiles go gate 0-15, gate 16-31, up 0-15, up 16-31 of each 32 channels
    unsigned char* packed = nullptr;
};

namespace {

constexpr int BLK = 16 * 34;         // bytes of one block column of a tile
constexpr int WARPS = 8;             // multiplying warps of a CTA
constexpr int CHUNK = 64;            // blocks of a tile handled per step, at most: eight per warp
constexpr int PER_WARP = CHUNK / WARPS;
constexpr int MAX_STAGES = 8;
constexpr int ROW1 = CHUNK + 8;      // floats per row of the one-vector kernel's products (8 extra: rows on other banks)

// a thread per 16 bytes of the packed form: lane (g, t) of a block holds rows g and g + 8, channels 4t.. and 16 + 4t..
__global__ void repack_q8_0_kernel(const unsigned char* __restrict__ blocks, int rows, int nb, int paired, size_t n_items,
                                   unsigned char* __restrict__ packed) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_items; i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i & 31), g = lane >> 2, t = lane & 3;
        const size_t tb = i >> 5;
        const int blk = (int)(tb % nb);
        const size_t tile = tb / nb;
        const size_t row0 = paired ? (tile >> 2) * 32 + (tile & 1) * 16 + ((tile >> 1) & 1) * (size_t)(rows / 2) : tile * 16;
        unsigned char* dst = packed + tb * BLK;
        uint32_t v[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {                 // a0: row g, a1: row g + 8, a2 / a3: the same, upper 16 channels
            const size_t row = row0 + g + 8 * (r & 1);
            v[r] = 0;
            if (row < (size_t)rows) {
                const uint16_t* s = reinterpret_cast<const uint16_t*>(blocks + (row * nb + blk) * 34) + 1 + 8 * (r >> 1) + 2 * t;
                v[r] = (uint32_t)s[0] | (uint32_t)s[1] << 16;
            }
        }
        *reinterpret_cast<uint4*>(dst + lane * 16) = make_uint4(v[0], v[1], v[2], v[3]);
        if (t < 2) {
            const size_t row = row0 + g + 8 * t;
            *reinterpret_cast<uint16_t*>(dst + 512 + g * 4 + t * 2) =
                row < (size_t)rows ? *reinterpret_cast<const uint16_t*>(blocks + (row * nb + blk) * 34) : (uint16_t)0;
        }
    }
}

// quantize_input_q8_0: one warp per 32-value block, lane = element
__global__ void quantize_input_kernel(const float* __restrict__ x, size_t n_blocks, int8_t* __restrict__ xq,
                                      float* __restrict__ xs) {
    flare_pdl_wait();
    flare_pdl_trigger();
    const int lane = threadIdx.x & 31;
    for (size_t w = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5; w < n_blocks; w += ((size_t)gridDim.x * blockDim.x) >> 5)
        flare_quantize_block_of_32(x[w * 32 + lane], lane, xq + w * 32, xs + w);
}

struct ProductParams {
    const unsigned char* w;
    Q8Input in;
    Q8Output out;
    int rows, nb, batch;
    int n_units;                 // tiles, or groups of four tiles of a paired matrix
    int chunks, cb;              // steps per tile and blocks per step (the last one may have fewer)
    int n_stages, stage_bytes;
    int col_groups;              // groups of eight input vectors; neighbouring CTAs take the groups of the same tiles
    int* err;
};

__device__ __forceinline__ void mma_s8(int (&d)[4], const uint4& a, uint32_t b0, uint32_t b1, const int (&c)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
__device__ __forceinline__ float silu_mul(float gate, float up) {
    return __fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), up);
}

// Both kernels below walk steps of (16 rows) x (up to 64 blocks) of packed weights, 35 KB each, that one thread keeps
// requesting as bulk copies into a ring.  In a step every warp multiplies its (up to) eight blocks by int8 MMAs, whose K
// is exactly a block, and leaves the scaled products in shared memory; other threads add them in block order.
//
// What bounds them is HBM, and at a model's sizes (4 to 35 MB a matrix) the time until the first bytes arrive.  The
// weights belong to no kernel of the stream, so the ring is filled before the wait for the predecessor, and the successor
// is let in at once: its ring fills while this kernel works (two CTAs fit on an SM).  It reads nothing else before its
// own wait.
struct Steps {
    int cta, n_cta, steps_per_unit, n_steps;
    __device__ Steps(const ProductParams& p, int tiles) {
        cta = blockIdx.x / p.col_groups; n_cta = gridDim.x / p.col_groups;
        steps_per_unit = tiles * p.chunks;
        n_steps = (cta < p.n_units ? (p.n_units - cta + n_cta - 1) / n_cta : 0) * steps_per_unit;
    }
};
__device__ __forceinline__ void issue_step(const ProductParams& p, const Steps& st, int tiles, unsigned char* ring, uint64_t* bars, int s) {
    const int unit = st.cta + s / st.steps_per_unit * st.n_cta, r = s % st.steps_per_unit, c0 = r % p.chunks * p.cb;
    const size_t tile = (size_t)unit * tiles + r / p.chunks;
    const uint32_t bytes = (uint32_t)min(p.cb, p.nb - c0) * BLK;
    uint64_t* bar = &bars[s % p.n_stages];
    ptx::mbar_expect_tx(bar, bytes);
    ptx::bulk_load(ring + (size_t)(s % p.n_stages) * p.stage_bytes, p.w + (tile * p.nb + c0) * BLK, bytes, bar);
}
__device__ __forceinline__ void start_ring(const ProductParams& p, const Steps& st, int tiles, unsigned char* ring, uint64_t* bars) {
    for (int s = 0; s < p.n_stages; s++) ptx::mbar_init(&bars[s], 1);
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    for (int s = 0; s < p.n_stages && s < st.n_steps; s++) issue_step(p, st, tiles, ring, bars, s);
}
// A copy never arrived: those in flight land (or give up) before the shared memory goes, and the host is told.
__device__ __noinline__ void give_up(const ProductParams& p, const Steps& st, uint64_t* bars, int s) {
    if (threadIdx.x != 0) return;
    for (int k = s; k < s + p.n_stages && k < st.n_steps; k++) ptx::mbar_wait(&bars[k % p.n_stages], (uint32_t)((k / p.n_stages) & 1));
    flare_report(p.err, FLARE_ERR_TIMEOUT);
}

// Up to eight input vectors (as codes): they are the MMA's eight columns.  128 threads add, one per (row, vector).
template <int OUT>
__global__ void __launch_bounds__(32 * WARPS, 2) product_q8_0_kernel(const ProductParams p) {
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ uint64_t full_bar[MAX_STAGES];
    __shared__ float s_hid[8][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    constexpr int TILES = OUT == OUT_SILU_Q8 ? 4 : 1;
    float* terms = reinterpret_cast<float*>(ring + (size_t)p.n_stages * p.stage_bytes);
    const int col0 = 8 * (blockIdx.x % p.col_groups);
    const Steps st(p, TILES);
    if (threadIdx.x == 0) start_ring(p, st, TILES, ring, full_bar);
    flare_pdl_trigger();
    flare_pdl_wait();

    // B operand and scales of this warp's blocks of the current chunk: vector g's codes, the scales of vectors 2t, 2t + 1
    uint32_t b[PER_WARP][2];
    float xs[PER_WARP][2];
    const int col = col0 + g;
    auto load_codes = [&](int c0) {
        const int cn = min(p.cb, p.nb - c0), per = (cn + WARPS - 1) / WARPS;
#pragma unroll
        for (int j = 0; j < PER_WARP; j++) {
            const int i = warp * per + j;
            b[j][0] = b[j][1] = 0; xs[j][0] = xs[j][1] = 0.0f;
            if (j < per && i < cn) {
                if (col < p.batch) {
                    const int8_t* src = p.in.xq + ((size_t)col * p.nb + c0 + i) * 32 + 4 * t;
                    b[j][0] = *reinterpret_cast<const uint32_t*>(src);
                    b[j][1] = *reinterpret_cast<const uint32_t*>(src + 16);
                }
#pragma unroll
                for (int k = 0; k < 2; k++)
                    if (col0 + 2 * t + k < p.batch) xs[j][k] = p.in.xs[(size_t)(col0 + 2 * t + k) * p.nb + c0 + i];
            }
        }
    };
    load_codes(0);
    __syncthreads();                                   // the barriers are initialised

    // the (row, vector) whose sum this thread keeps (threads 0 .. 127): an accumulator register of lane tid / 4
    const int srow = (threadIdx.x >> 4) + 8 * ((threadIdx.x >> 1) & 1), svec = 2 * ((threadIdx.x >> 2) & 3) + (threadIdx.x & 1);
    const bool summing = threadIdx.x < 128 && col0 + svec < p.batch;
    float sum = 0.0f, kept[TILES] = {};
    const int none[4] = {0, 0, 0, 0};
    for (int s = 0; s < st.n_steps; s++) {
        const int stage = s % p.n_stages, r = s % st.steps_per_unit, chunk = r % p.chunks, c0 = chunk * p.cb;
        const int unit = st.cta + s / st.steps_per_unit * st.n_cta, cn = min(p.cb, p.nb - c0), per = (cn + WARPS - 1) / WARPS;
        const bool failed = !ptx::mbar_wait(&full_bar[stage], (uint32_t)((s / p.n_stages) & 1));
        const unsigned char* buf = ring + (size_t)stage * p.stage_bytes;
        auto scaled = [&](int i, const uint4& a, __half2 wsh, uint32_t b0, uint32_t b1, float xs0, float xs1) {
            const float2 ws = __half22float2(wsh);
            int d[4];
            mma_s8(d, a, b0, b1, none);
            float4 v;
            v.x = __fmul_rn(__fmul_rn(ws.x, xs0), (float)d[0]);
            v.y = __fmul_rn(__fmul_rn(ws.x, xs1), (float)d[1]);
            v.z = __fmul_rn(__fmul_rn(ws.y, xs0), (float)d[2]);
            v.w = __fmul_rn(__fmul_rn(ws.y, xs1), (float)d[3]);
            *reinterpret_cast<float4*>(terms + FLARE_CK(i * 128 + lane * 4, 4, p.cb * 128, p.err)) = v;
        };
        if (cn == CHUNK) {                             // no bounds inside: the blocks' loads and MMAs run side by side
            const unsigned char* mine = buf + warp * PER_WARP * BLK;
            uint4 a[PER_WARP];
            __half2 ws[PER_WARP];
#pragma unroll
            for (int j = 0; j < PER_WARP; j++) {
                a[j] = *reinterpret_cast<const uint4*>(mine + j * BLK + lane * 16);
                ws[j] = *reinterpret_cast<const __half2*>(mine + j * BLK + 512 + g * 4);
            }
#pragma unroll
            for (int j = 0; j < PER_WARP; j++) scaled(warp * PER_WARP + j, a[j], ws[j], b[j][0], b[j][1], xs[j][0], xs[j][1]);
        } else {
#pragma unroll
            for (int j = 0; j < PER_WARP; j++) {
                const int i = warp * per + j;
                if (j < per && i < cn) {
                    const unsigned char* at = buf + FLARE_CK(i * BLK, BLK, p.stage_bytes, p.err);
                    scaled(i, *reinterpret_cast<const uint4*>(at + lane * 16), *reinterpret_cast<const __half2*>(at + 512 + g * 4),
                           b[j][0], b[j][1], xs[j][0], xs[j][1]);
                }
            }
        }
        if (p.chunks > 1 && s + 1 < st.n_steps) load_codes((s + 1) % p.chunks * p.cb);     // on their way during the sums
        if (__syncthreads_or(failed)) { give_up(p, st, full_bar, s); return; }
        // the products are there and the stage has been read
        if (threadIdx.x == 0 && s + p.n_stages < st.n_steps) { ptx::fence_proxy_async(); issue_step(p, st, TILES, ring, full_bar, s + p.n_stages); }
        if (threadIdx.x < 128) {
            if (chunk == 0) sum = 0.0f;
            if (summing) {
                const float* tp = terms + threadIdx.x;
                int i = 0;
                for (; i + 16 <= cn; i += 16) {
                    float v[16];
#pragma unroll
                    for (int k = 0; k < 16; k++) v[k] = tp[(i + k) * 128];
#pragma unroll
                    for (int k = 0; k < 16; k++) sum = __fadd_rn(sum, v[k]);
                }
                for (; i < cn; i++) sum = __fadd_rn(sum, tp[i * 128]);
            }
            if (chunk == p.chunks - 1) {
                if constexpr (OUT == OUT_SILU_Q8) {
                    const int tile = r / p.chunks;
#pragma unroll
                    for (int k = 0; k < TILES; k++) if (k == tile) kept[k] = sum;
                    if (tile == TILES - 1) {           // uniform over the CTA
                        s_hid[svec][srow] = silu_mul(kept[0], kept[2]);
                        s_hid[svec][16 + srow] = silu_mul(kept[1], kept[3]);
                        asm volatile("bar.sync 1, 128;" ::: "memory");
                        const int n_blocks = p.rows / 64;              // blocks of a hidden vector
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const int c = 2 * warp + k;
                            if (col0 + c < p.batch) {
                                const size_t at = (size_t)(col0 + c) * n_blocks + unit;
                                flare_quantize_block_of_32(s_hid[c][lane], lane, p.out.oq + at * 32, p.out.os + at);
                            }
                        }
                    }
                } else {
                    const size_t out_row = (size_t)unit * 16 + srow;
                    if (summing && out_row < (size_t)p.rows) {
                        float* o = p.out.out + (size_t)(col0 + svec) * p.rows + out_row;
                        *o = p.out.accumulate ? __fadd_rn(*o, sum) : sum;
                    }
                }
            }
        }
        __syncthreads();                               // the sums have read the products
    }
}

// One input vector: the MMA's columns are eight consecutive blocks instead.  MMA j of a warp multiplies block j by its
// input codes in column j and zeros elsewhere and adds to the same accumulators, so that eight MMAs leave 16 rows x 8
// block dots, all of them wanted, for one round of scaling: a seventh of the instructions per step of a body like the
// kernel's above with one column in use (which took 76 us for 128256 x 2048, issue bound; this one 45.7 = 6.1 TB/s).  A ninth warp adds, a lane per
// row, while the others are at the next step.  The input's norm and quantisation run here while the first weights travel,
// instead of in a kernel of their own.
template <int IN, int OUT>
__global__ void __launch_bounds__(32 * WARPS + 32, 2) product1_q8_0_kernel(const ProductParams p) {
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ uint64_t full_bar[MAX_STAGES];
    __shared__ float s_sq[WARPS];
    __shared__ uint32_t s_codes[IN == IN_CODES ? 1 : CHUNK * 8];
    __shared__ float s_xs[IN == IN_CODES ? 1 : CHUNK];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    constexpr int TILES = OUT == OUT_SILU_Q8 ? 4 : 1;
    float* terms = reinterpret_cast<float*>(ring + (size_t)p.n_stages * p.stage_bytes);      // [2][16][ROW1]
    const Steps st(p, TILES);
    if (threadIdx.x == 0) start_ring(p, st, TILES, ring, full_bar);
    flare_pdl_trigger();
    flare_pdl_wait();

    if constexpr (IN != IN_CODES) {                    // one chunk: p.nb <= CHUNK
        float inv_rms = 1.0f;
        if constexpr (IN != IN_F32) {
            if (warp < WARPS) {
                const float sq = flare_sum_sq_of_warp(p.in.x, p.nb * 32, warp, lane);
                if (lane == 0) s_sq[warp] = sq;
            }
            __syncthreads();
            inv_rms = flare_inv_rms(s_sq, p.nb * 32, p.in.eps);
        }
        for (int u = threadIdx.x; u < (p.nb * 8 + 31) / 32 * 32; u += 32 * WARPS + 32) {
            float n[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (u < p.nb * 8) {
                const float4 xv = *reinterpret_cast<const float4*>(p.in.x + 4 * u);
                n[0] = xv.x; n[1] = xv.y; n[2] = xv.z; n[3] = xv.w;
                if constexpr (IN != IN_F32) flare_norm_quad(n, p.in.norm + 4 * u, inv_rms, IN == IN_NORM_Q8);
            }
            float d;
            const uint32_t c = flare_q8_quad(n, d);
            if (u < p.nb * 8) {
                s_codes[u] = c;
                if ((u & 7) == 0) s_xs[u >> 3] = d;
            }
        }
    }
    __syncthreads();                                   // the codes are there, the barriers initialised

    if (warp == WARPS) {                               // the adding warp: lane = row
        float sum = 0.0f, kept[TILES] = {};
        for (int s = 0; s < st.n_steps; s++) {
            const int r = s % st.steps_per_unit, chunk = r % p.chunks, cn = min(p.cb, p.nb - chunk * p.cb);
            const int unit = st.cta + s / st.steps_per_unit * st.n_cta;
            if (__syncthreads_or(0)) return;
            const float* tp = terms + (s & 1) * 16 * ROW1 + (lane & 15) * ROW1;
            if (chunk == 0) sum = 0.0f;
            int i = 0;
            for (; i + 16 <= cn; i += 16) {
                float4 v[4];
#pragma unroll
                for (int k = 0; k < 4; k++) v[k] = *reinterpret_cast<const float4*>(tp + i + 4 * k);
#pragma unroll
                for (int k = 0; k < 4; k++) sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v[k].x), v[k].y), v[k].z), v[k].w);
            }
            for (; i < cn; i++) sum = __fadd_rn(sum, tp[i]);
            if (chunk != p.chunks - 1) continue;
            if constexpr (OUT == OUT_SILU_Q8) {
                const int tile = r / p.chunks;
#pragma unroll
                for (int k = 0; k < TILES; k++) if (k == tile) kept[k] = sum;
                if (tile == TILES - 1) {               // lanes 16 .. 31 hold the same sums as 0 .. 15
                    const float h = lane < 16 ? silu_mul(kept[0], kept[2]) : silu_mul(kept[1], kept[3]);
                    flare_quantize_block_of_32(h, lane, p.out.oq + (size_t)unit * 32, p.out.os + unit);
                }
            } else {
                const size_t row = (size_t)unit * 16 + lane;
                if (lane < 16 && row < (size_t)p.rows) p.out.out[row] = p.out.accumulate ? __fadd_rn(p.out.out[row], sum) : sum;
            }
        }
        return;
    }

    // lane (g, t): codes of block g of this warp's eight, scales of blocks 2t and 2t + 1
    uint32_t b0, b1;
    float xs0, xs1;
    auto load_codes = [&](int c0) {
        const int cn = min(p.cb, p.nb - c0), i = warp * 8;
        b0 = b1 = 0; xs0 = xs1 = 0.0f;
        const uint32_t* codes = IN == IN_CODES ? reinterpret_cast<const uint32_t*>(p.in.xq) : s_codes;
        const float* scales = IN == IN_CODES ? p.in.xs : s_xs;
        if (i + g < cn) { b0 = codes[(c0 + i + g) * 8 + t]; b1 = codes[(c0 + i + g) * 8 + 4 + t]; }
        if (i + 2 * t < cn) xs0 = scales[c0 + i + 2 * t];
        if (i + 2 * t + 1 < cn) xs1 = scales[c0 + i + 2 * t + 1];
    };
    load_codes(0);
    for (int s = 0; s < st.n_steps; s++) {
        const int stage = s % p.n_stages, chunk = s % p.chunks, cn = min(p.cb, p.nb - chunk * p.cb);
        const bool failed = !ptx::mbar_wait(&full_bar[stage], (uint32_t)((s / p.n_stages) & 1));
        const int n = min(8, cn - warp * 8);           // this warp's blocks (none or fewer: none)
        if (n > 0) {
            const unsigned char* mine = ring + FLARE_CK((uint32_t)stage * p.stage_bytes + warp * 8 * BLK, n * BLK, p.n_stages * p.stage_bytes, p.err);
            int d[2][4] = {};                          // two chains
            float2 w0 = make_float2(0.0f, 0.0f), w1 = w0;
            if (n == 8) {
                uint4 a[8];
#pragma unroll
                for (int j = 0; j < 8; j++) a[j] = *reinterpret_cast<const uint4*>(mine + j * BLK + lane * 16);
#pragma unroll
                for (int j = 0; j < 8; j++) mma_s8(d[j & 1], a[j], g == j ? b0 : 0u, g == j ? b1 : 0u, d[j & 1]);
            } else {
#pragma unroll
                for (int j = 0; j < 7; j++)
                    if (j < n) mma_s8(d[j & 1], *reinterpret_cast<const uint4*>(mine + j * BLK + lane * 16), g == j ? b0 : 0u, g == j ? b1 : 0u, d[j & 1]);
            }
            if (2 * t < n) w0 = __half22float2(*reinterpret_cast<const __half2*>(mine + 2 * t * BLK + 512 + g * 4));
            if (2 * t + 1 < n) w1 = __half22float2(*reinterpret_cast<const __half2*>(mine + (2 * t + 1) * BLK + 512 + g * 4));
            float* row = terms + (s & 1) * 16 * ROW1 + g * ROW1 + warp * 8 + 2 * t;
            *reinterpret_cast<float2*>(row) = make_float2(__fmul_rn(__fmul_rn(w0.x, xs0), (float)(d[0][0] + d[1][0])),
                                                          __fmul_rn(__fmul_rn(w1.x, xs1), (float)(d[0][1] + d[1][1])));
            *reinterpret_cast<float2*>(row + 8 * ROW1) = make_float2(__fmul_rn(__fmul_rn(w0.y, xs0), (float)(d[0][2] + d[1][2])),
                                                                     __fmul_rn(__fmul_rn(w1.y, xs1), (float)(d[0][3] + d[1][3])));
        }
        if (p.chunks > 1 && s + 1 < st.n_steps) load_codes((s + 1) % p.chunks * p.cb);
        if (__syncthreads_or(failed)) { give_up(p, st, full_bar, s); return; }
        if (threadIdx.x == 0 && s + p.n_stages < st.n_steps) { ptx::fence_proxy_async(); issue_step(p, st, TILES, ring, full_bar, s + p.n_stages); }
    }
}

}  // namespace

// paired: the rows are [gate | up] halves of a feed-forward matrix (rows a multiple of 64)
int flare_weight_upload(flare_attn_ctx* ctx, const void* blocks, int rows, int cols, int paired, flare_weight** out_w) {
    if (!ctx) return FLARE_ERR_INVALID_ARG;
    if (!out_w) return flare_set_error(ctx, FLARE_ERR_INVALID_ARG, "out_w is null");
    *out_w = nullptr;
    if (!blocks || rows < 1 || cols < 32 || cols % 32 || (paired && rows % 64))
        return flare_set_error(ctx, FLARE_ERR_INVALID_ARG, "flare_weight_upload_q8_0: %d x %d (cols must be a positive multiple of 32)", rows, cols);
    FLARE_CUDA_OK(ctx, cudaSetDevice(ctx->device));
    flare_weight* w = new (std::nothrow) flare_weight();
    if (!w) return FLARE_ERR_OOM;
    w->ctx = ctx; w->rows = rows; w->cols = cols; w->paired = paired;
    const int nb = cols / 32;
    const size_t tile_blocks = (size_t)((rows + 15) / 16) * nb, bytes = (size_t)rows * nb * 34;
    unsigned char* raw = nullptr;
    cudaError_t e = cudaMalloc(&raw, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&w->packed, tile_blocks * BLK);
    if (e == cudaSuccess) e = cudaMemcpyAsync(raw, blocks, bytes, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        const size_t g = std::min<size_t>((tile_blocks * 32 + 255) / 256, 148 * 32);
        repack_q8_0_kernel<<<(int)g, 256, 0, ctx->stream>>>(raw, rows, nb, paired, tile_blocks * 32, w->packed);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(raw);
    if (e != cudaSuccess) {
        const int code = e == cudaErrorMemoryAllocation ? FLARE_ERR_OOM : FLARE_ERR_CUDA;
        flare_set_error(ctx, code, "flare_weight_upload_q8_0: %zu bytes: %s", bytes, cudaGetErrorString(e));
        cudaGetLastError();
        cudaFree(w->packed);
        delete w;
        return code;
    }
    *out_w = w;
    return FLARE_OK;
}

extern "C" {

int flare_weight_upload_q8_0(flare_attn_ctx* ctx, const void* blocks, int rows, int cols, flare_weight** out_w) {
    return flare_weight_upload(ctx, blocks, rows, cols, 0, out_w);
}

int flare_weight_free(flare_weight* w) {
    if (!w) return FLARE_OK;
    cudaSetDevice(w->ctx->device);
    cudaStreamSynchronize(w->ctx->stream);
    cudaFree(w->packed);
    delete w;
    return FLARE_OK;
}

int flare_matvec_q8_0(flare_attn_ctx* ctx, const flare_weight* w, const float* x, int batch, float* out, int on_device) {
    if (!ctx) return FLARE_ERR_INVALID_ARG;
    if (!w || w->ctx != ctx) return flare_set_error(ctx, FLARE_ERR_STATE, "the weight matrix does not belong to this context");
    if (!x || !out || batch < 1 || batch > 256)
        return flare_set_error(ctx, FLARE_ERR_INVALID_ARG, "flare_matvec_q8_0: null buffer or batch %d outside [1, 256]", batch);
    FLARE_CUDA_OK(ctx, cudaSetDevice(ctx->device));
    const size_t xn = (size_t)batch * w->cols, on = (size_t)batch * w->rows, nblk = xn / 32;
    // scratch: quantised inputs and their scales (and, with host buffers, x and out themselves)
    const size_t q_off = 0, s_off = (xn + 255) / 256 * 256, x_off = s_off + (nblk * 4 + 255) / 256 * 256;
    const size_t o_off = x_off + (on_device ? 0 : (xn * 4 + 255) / 256 * 256);
    const size_t need = o_off + (on_device ? 0 : on * 4);
    FLARE_TRY(flare_ensure(ctx, &ctx->d_conv, &ctx->conv_bytes, need + 256));
    char* d = (char*)ctx->d_conv;
    const float* dx = x;
    float* dout = out;
    if (!on_device) {
        FLARE_CUDA_OK(ctx, cudaMemcpyAsync(d + x_off, x, xn * 4, cudaMemcpyHostToDevice, ctx->stream));
        dx = (const float*)(d + x_off); dout = (float*)(d + o_off);
    }
    Q8Input in;
    Q8Output to;
    to.out = dout;
    if (flare_product_quantises(w, batch) && ((uintptr_t)dx & 15) == 0) { in.kind = IN_F32; in.x = dx; }
    else {
        FLARE_TRY(flare_launch_quantize_input(ctx, dx, nblk, (int8_t*)(d + q_off), (float*)(d + s_off)));
        in.xq = (const int8_t*)(d + q_off); in.xs = (const float*)(d + s_off);
    }
    FLARE_TRY(flare_launch_product_q8_0(ctx, w, in, batch, to));
    if (!on_device) {
        FLARE_CUDA_OK(ctx, cudaMemcpyAsync(out, dout, on * 4, cudaMemcpyDeviceToHost, ctx->stream));
        FLARE_CUDA_OK(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return FLARE_OK;
}

}  // extern "C"

// quantize_input_q8_0 of n_blocks blocks of 32 values, all on the device
int flare_launch_quantize_input(flare_attn_ctx* ctx, const float* d_x, size_t n_blocks, int8_t* d_xq, float* d_xs) {
    const int threads = 256;
    size_t g = (n_blocks * 32 + threads - 1) / threads;
    if (g > 148 * 16) g = 148 * 16;
    if (g < 1) g = 1;
    ctx->last_launch_overlappable = false;
    FLARE_CUDA_OK(ctx, flare_launch_pdl(quantize_input_kernel, dim3((unsigned)g), dim3(threads), 0, ctx->stream, d_x, n_blocks, d_xq, d_xs));
    FLARE_LAUNCH_CHECK(ctx);
    return FLARE_OK;
}

// One vector of at most 64 blocks is quantised by the product itself.  (With eight vectors each CTA would spend 9 us on
// what a kernel of its own does in 2.5, most of it hidden behind the first weights.)
bool flare_product_quantises(const flare_weight* w, int batch) { return batch == 1 && w->cols <= CHUNK * 32; }

using ProductKernel = void (*)(const ProductParams);
static ProductKernel product_kernel(int in, int out, bool one) {
    if (!one) return out == OUT_SILU_Q8 ? product_q8_0_kernel<OUT_SILU_Q8> : product_q8_0_kernel<OUT_F32>;
    if (out == OUT_SILU_Q8) return in == IN_CODES ? product1_q8_0_kernel<IN_CODES, OUT_SILU_Q8> : product1_q8_0_kernel<IN_NORM_Q8, OUT_SILU_Q8>;
    switch (in) {
        case IN_CODES: return product1_q8_0_kernel<IN_CODES, OUT_F32>;
        case IN_F32: return product1_q8_0_kernel<IN_F32, OUT_F32>;
        case IN_NORM_Q8: return product1_q8_0_kernel<IN_NORM_Q8, OUT_F32>;
        default: return product1_q8_0_kernel<IN_NORM_F32, OUT_F32>;
    }
}

// matvec_q8_0_preq_into for `batch` input vectors, all on the device, with what precedes and follows it in a forward pass
int flare_launch_product_q8_0(flare_attn_ctx* ctx, const flare_weight* w, const Q8Input& in, int batch, const Q8Output& out) {
    const int kind = out.oq ? OUT_SILU_Q8 : OUT_F32;
    if ((in.kind != IN_CODES && !flare_product_quantises(w, batch)) || (kind == OUT_SILU_Q8) != (w->paired != 0) ||
        (kind == OUT_SILU_Q8 && in.kind != IN_CODES && in.kind != IN_NORM_Q8))
        return flare_set_error(ctx, FLARE_ERR_STATE, "Q8_0 product: input form %d, output form %d for a matrix of %d x %d", in.kind, kind, w->rows, w->cols);
    const bool one = batch == 1;
    ProductParams p;
    p.w = w->packed; p.in = in; p.out = out;
    p.rows = w->rows; p.nb = w->cols / 32; p.batch = batch;
    p.n_units = w->paired ? w->rows / 64 : (w->rows + 15) / 16;
    p.chunks = (p.nb + CHUNK - 1) / CHUNK;
    p.cb = (p.nb + p.chunks - 1) / p.chunks;
    p.stage_bytes = p.cb * BLK;
    p.n_stages = std::max(2, std::min(MAX_STAGES, 2 * CHUNK * BLK / p.stage_bytes));
    p.col_groups = (batch + 7) / 8;
    p.err = ctx->d_err;
    const int smem = p.n_stages * p.stage_bytes + (one ? 2 * 16 * ROW1 * 4 : p.cb * 512), max_smem = 2 * CHUNK * BLK + CHUNK * 512;
    ProductKernel kernel = product_kernel(in.kind, kind, one);
    {
        static std::mutex m;
        static bool done[64][2][2][4] = {};
        std::lock_guard<std::mutex> lock(m);
        bool& d = done[ctx->device & 63][one][kind][in.kind];
        if (!d) FLARE_CUDA_OK(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
        d = true;
    }
    // two CTAs fit on an SM; what does not fit at once is walked by those that do
    const int n_cta = std::min(p.n_units, std::max(1, 2 * ctx->sm_count / p.col_groups));
    ctx->last_launch_overlappable = false;
    FLARE_CUDA_OK(ctx, flare_launch_pdl(kernel, dim3(n_cta * p.col_groups), dim3(32 * WARPS + (one ? 32 : 0)), (size_t)smem, ctx->stream, p));
    FLARE_LAUNCH_CHECK(ctx);
    return FLARE_OK;
}

void flare_weight_dims(const flare_weight* w, int* rows, int* cols) { *rows = w->rows; *cols = w->cols; }
