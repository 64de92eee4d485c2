// Q8_0 split-KV decode attention, the bandwidth-bound fast path (head_dim 64 / 128, up to 8 KV heads).
//
// One CTA = one (sequence, slot range, group of NI items), one warp per KV head.  An item is a query together with up
// to 4 of the query heads that share a KV head.  Whole 32-slot tiles — every head's int8 K and V payload and the f16
// scales, i.e. contiguous 16 KB + 1 KB pieces of each plane, which keeps DRAM pages open — stream into a ring of
// shared-memory stages through cp.async.bulk.tensor (landing as [128 bytes of heads][slot], 128B swizzle) and cp.async.bulk, each stage guarded by an mbarrier.  There is no producer warp and no wait for a free stage: the last
// warp to finish with a stage (a shared-memory ticket) refills it.
//
// Dequantise-then-FMA on CUDA cores costs ~10 instructions per KV byte and cannot keep up with HBM, so both contractions
// run on tensor cores, transposed: the cache is the 16-row operand A and the (at most 4) query heads are the 8 columns,
// with the Q8_0 scales hoisted out of the sums:
//   scores  S[slot, head] = qs_head * sum_blk ks[slot, blk] * (Kint[slot, blk, :] . Qint[blk, :, head])
//           as an exact int8 MMA (m16n8k32): Qint is q * log2e/sqrt(d) in 15-bit fixed point per head, carried as two
//           int8 limbs in columns 2h and 2h + 1, so a lane ends up with both limbs of 2 slots of one head and no
//           lane holds a duplicate.
//   output  O[d, head] = sum_slot Vint[slot, d] * (p * vs[slot, blk(d)])
//           as an f16 MMA (m16n8k16, f32 accumulate): the weight p*vs is rounded to f16 and moved into operand layout by
//           movmatrix; the columns hold the two channel blocks of 4 heads (NI == 1) or two items of 4 heads.  Vint bytes
//           become exact f16 values 1024 + (v + 128) with one xor and one byte-permute per pair (V is transposed by
//           ldmatrix.trans on the swizzled tile); the constant 1152 * sum(weights) is subtracted at the end.
// What a tile's K and V cost to unpack is paid once for all NI items.  Instruction issue used to pace this kernel (480
// warp instructions per 32-slot tile with the heads as rows, half of the lanes holding copies).
//
// Softmax is the single-pass online recurrence of flare-core/src/model.rs:9914-9966, applied to 32 slots at a time with
// lazy rescaling; slot ranges are merged by log-sum-exp, through distributed shared memory when they form a cluster.
//
// A decode step can hand its new K/V rows to this kernel (StepFusion): the warp of a KV head quantises its slice, writes
// it to the cache and patches it into the tile that its range reads, so a step is one launch and not two.
#include "common.cuh"
#include "q8_input.cuh"
#include "tma.cuh"
#include <algorithm>
#include <math_constants.h>
#include <mutex>

namespace {

// Guards the per-device tables below: two contexts on two host threads may make their first call at once.
std::mutex g_table_mutex;

constexpr int T = 32;            // slots per tile
constexpr int STAGES = 3;
constexpr int MAX_CLUSTER = 16;       // 9 .. 16 CTAs per cluster are beyond the portable size: opted into per kernel
constexpr int SMALL = 64;             // sequences whose lengths travel as launch parameters
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kQFix = 16256.0f;     // 127 * 128: |Qint| <= 16256 = 128 * limb0 + limb1

struct Q8Params {
    const float* q;
    size_t q_seq_stride;        // floats
    float* out;
    float* work;
    const int* attend_len;      // device arrays, used when n_small == 0
    const int2* ring;
    const __half* k_scale;      // layer base, sequence 0
    const __half* v_scale;
    size_t scale_seq_stride;    // halves between sequences
    int layer_seq0;             // layer * batch: TMA coordinate of sequence 0
    int batch, num_heads, nkv, G, max_seq, slot_begin, slot_end, want_partial;
    int n_split, n_ranges;   // CTAs per sequence; those of them that have a slot range (all, or one of a cluster of two)
    int n_small;             // > 0: the arrays below hold the lengths (no global load before the first TMA request)
    int n_q, causal_q, hgroups;   // items of a sequence: n_q queries x hgroups groups of up to 4 heads per kv head
    int cluster;             // the n_split CTAs of a sequence form one thread-block cluster and merge through shared memory
    int rec_off;             // byte offset of the cluster's record buffer in dynamic shared memory
    int wait_first;          // the stream may still be writing tiles of this layer: wait before the first tile request
    // the new rows (null: none), the cache planes they go to, and the rotation applied on the way
    const float *new_k, *new_v;
    size_t new_stride;
    int8_t *kq, *vq;
    __half *ks_w, *vs_w;
    size_t payload_seq_stride;
    const float *cos, *sin;
    const long long* positions;
    int8_t* oq;              // quantised output blocks instead of f32
    float* os;
    int* err;
    int attend_small[SMALL];
    int pos_small[SMALL];    // ring position of each sequence (only read with new rows)
};

// Byte offset of 16-byte chunk `chunk` of slot `row` of KV head kvh within a K (or V) tile.  The tile is made of 128-byte
// rows — one head of 128 channels or two of 64 — because the copy engine pays per row: with 64-byte rows it delivered 26
// bytes per cycle and SM.  128-byte hardware swizzle: the chunk index is XORed with the row's low three bits.
template <int HD> __device__ __forceinline__ uint32_t tile_at(int kvh, int row, int chunk) {
    const int panel = HD == 64 ? kvh >> 1 : kvh, c = HD == 64 ? (kvh & 1) * 4 + chunk : chunk;
    return (uint32_t)(panel * (T * 128) + row * 128 + ((c ^ (row & 7)) << 4));
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    // the zero addend is an operand of its own: tying it to d costs four register moves per product
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
// register-only conversions (no address is taken, so nothing is forced into local memory)
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    uint32_t u;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(u) : "f"(hi), "f"(lo));
    return u;
}
__device__ __forceinline__ float2 unpack_half2(uint32_t u) {
    float2 f;
    asm("{\n\t.reg .f16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.f32.f16 %0, lo;\n\tcvt.f32.f16 %1, hi;\n\t}"
        : "=f"(f.x), "=f"(f.y) : "r"(u));
    return f;
}

// Thread-block cluster: the split barrier over all threads of all CTAs of the cluster, and stores into a peer's shared
// memory that count themselves in on an mbarrier of that peer.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_map(uint32_t smem_addr, uint32_t cta_rank) {
    uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(cta_rank)); return r;
}
__device__ __forceinline__ void cluster_st_async(uint32_t addr, uint32_t bar, float x, float y) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                 ::"r"(addr), "f"(x), "f"(y), "r"(bar) : "memory");
}

// Channel `lane` of 32-channel block `blk` of a new key row, rotated for table row `pos` (apply_rope_with_table,
// flare-core/src/model.rs:7256-7292: element i pairs with i + head_dim/2; two multiplies and a subtract / an add, not fused).
template <int HD>
__device__ __forceinline__ float rotated(const float* __restrict__ head, int e, const float* __restrict__ cos,
                                         const float* __restrict__ sin, long long pos) {
    constexpr int H2 = HD / 2;
    const float* cr = cos + (size_t)pos * H2;
    const float* sr = sin + (size_t)pos * H2;
    if (e < H2) return __fsub_rn(__fmul_rn(__ldg(head + e), __ldg(cr + e)), __fmul_rn(__ldg(head + e + H2), __ldg(sr + e)));
    const int i = e - H2;
    return __fadd_rn(__fmul_rn(__ldg(head + i), __ldg(sr + i)), __fmul_rn(__ldg(head + e), __ldg(cr + i)));
}

// What a CTA keeps of the new row of its sequence: each warp its own head's codes (lane = channel of a block) and scales.
template <int HD> struct NewRow {
    int k[HD / 32], v[HD / 32];
    float ks[HD / 32], vs[HD / 32];
};

// NI: items per CTA (1, or an even number: pairs share the columns of the output product).
// NKV: the number of KV heads when it is known (8: every address within a tile is then a constant offset), else 0.
template <int HD, int NI, int NKV>
__global__ void __launch_bounds__(256, HD == 64 ? 2 : 1)
decode_q8_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                 const __grid_constant__ Q8Params p) {
    constexpr int NB = HD / 32;             // Q8_0 blocks per head row
    constexpr int NC = HD / 16;             // 16-channel tiles of the output product
    constexpr int NP = NI == 1 ? 1 : NI / 2;        // column sets: one item with two channel blocks, or pairs of items
    constexpr int NSET = NI == 1 ? NB / 2 : NB;     // B operands per column set and k-step
    constexpr int TILE = T * HD;            // bytes of one head's K (or V) tile
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full_bar[STAGES];
    __shared__ uint64_t rec_bar;
    __shared__ int done_cnt[STAGES];        // warps that have finished with the stage's current tile

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int nkv = NKV ? NKV : p.nkv, kvh = warp;
    const int split = blockIdx.x, b = blockIdx.y, n_ranges = p.n_ranges;
    // stage layout: K payload [nkv][T][HD], V payload [nkv][T][HD], K scales [T][nkv*NB] f16, V scales
    const int payload = nkv * TILE;
    const int scale_tile = T * nkv * NB * 2;
    const int stage_bytes = 2 * payload + 2 * scale_tile;     // a multiple of 1024 (checked on the host)
    unsigned char* sbase = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const int n_items = p.n_q * p.hgroups;
    const int item0 = NI * (int)blockIdx.z;
    // slots that item `it` of this CTA reads: query i of a causally ordered group sees n_q - 1 - i slots fewer
    const int attend_b = p.n_small ? p.attend_small[b] : p.attend_len[b];
    auto item_hi = [&](int it) {
        const int qi = min(item0 + it, n_items - 1) / p.hgroups;
        int h = max(0, attend_b - (p.causal_q ? (p.n_q - 1 - qi) : 0));
        return p.slot_end >= 0 ? min(h, p.slot_end) : h;
    };
    const int lo = p.slot_end >= 0 ? max(0, p.slot_begin) : 0;
    const int hi = item_hi(NI - 1), hi_short = item_hi(0);
    // slot range of this split, in whole tiles of the longest item's range
    const int t_first = lo / T, t_last = hi > lo ? (hi + T - 1) / T : t_first;
    const int n_tiles_seq = t_last - t_first;
    const int t_begin = t_first + (int)(((long long)min(split, n_ranges) * n_tiles_seq) / n_ranges);
    const int t_end = t_first + (int)(((long long)min(split + 1, n_ranges) * n_tiles_seq) / n_ranges);
    const int n_tiles = t_end - t_begin;

    const int bpr = nkv * NB;       // scale entries per slot row
    const unsigned char* ksg = reinterpret_cast<const unsigned char*>(p.k_scale + (size_t)b * p.scale_seq_stride);
    const unsigned char* vsg = reinterpret_cast<const unsigned char*>(p.v_scale + (size_t)b * p.scale_seq_stride);
    auto issue = [&](int i) {       // one thread: tile i of this CTA -> stage i % STAGES
        const int s = i % STAGES;
        unsigned char* st = sbase + (size_t)s * stage_bytes;
        const int slot0 = (t_begin + i) * T;
        const int rows = min(T, p.max_seq - slot0);            // scale rows that exist in the plane
        const uint32_t sbytes = (uint32_t)rows * bpr * 2;
        ptx::mbar_expect_tx(&full_bar[s], 2 * payload + 2 * sbytes);
        ptx::tma_load_4d(st, &kmap, &full_bar[s], 0, slot0, 0, p.layer_seq0 + b);
        ptx::tma_load_4d(st + payload, &vmap, &full_bar[s], 0, slot0, 0, p.layer_seq0 + b);
        ptx::bulk_load(st + 2 * payload, ksg + (size_t)slot0 * bpr * 2, sbytes, &full_bar[s]);
        ptx::bulk_load(st + 2 * payload + scale_tile, vsg + (size_t)slot0 * bpr * 2, sbytes, &full_bar[s]);
    };
    // Launched as a programmatic dependent in every case: unless the predecessor may be writing this layer's rows, the
    // first tiles are requested while it drains.
    if (p.wait_first) flare_pdl_wait();
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { ptx::mbar_init(&full_bar[s], 1); done_cnt[s] = 0; }
        if (p.cluster) ptx::mbar_init(&rec_bar, 1);
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
        for (int i = 0; i < STAGES && i < n_tiles; i++) issue(i);
    }
    // heads whose records this CTA merges: h % n_split == rank
    const uint32_t rank = p.cluster ? cluster_ctarank() : 0;
    const int my_heads = p.cluster ? (p.num_heads - (int)rank + p.n_split - 1) / p.n_split : 0;
    __syncthreads();
    if (p.cluster) {
        if (threadIdx.x == 0 && my_heads > 0) ptx::mbar_expect_tx(&rec_bar, (uint32_t)(p.n_split * my_heads * (HD + 2) * 4));
        cluster_arrive();               // this CTA's record barrier is ready; waited for before the first record is sent
    }
    // K/V tiles requested above do not depend on the previous kernel in the stream; q and the new rows do.
    flare_pdl_wait();
    // From here on the next kernel may be scheduled: its CTAs take the places this grid's CTAs leave one by one (and
    // the free places at once) and request their first tiles.  The trigger comes after the wait, so whatever ran before
    // this kernel's predecessor has completed by the time the successor starts: a successor has to keep its early
    // requests clear of this kernel's rows only.
    flare_pdl_trigger();

    // q (and the new rows below) are needed at once: all loads are issued before the first is used
    float qv[NI][NB][8];
    const float* rope_c = p.cos ? p.cos + (size_t)p.positions[b] * (HD / 2) + tig * 4 : nullptr;
    const float* rope_s = p.cos ? p.sin + (size_t)p.positions[b] * (HD / 2) + tig * 4 : nullptr;
#pragma unroll
    for (int it = 0; it < NI; it++) {
        const int item = min(item0 + it, n_items - 1), qi = item / p.hgroups, hg = item % p.hgroups, hq = g >> 1;
        const float* qrow = p.q + (size_t)b * p.q_seq_stride + ((size_t)qi * p.num_heads + kvh * p.G + 4 * hg + (hq < p.G - 4 * hg ? hq : 0)) * HD;
#pragma unroll
        for (int blk = 0; blk < NB; blk++) {
            const float4* qp = reinterpret_cast<const float4*>(qrow + blk * 32 + tig * 4);
            const float4 x = __ldg(qp), y = __ldg(qp + 4);              // channels 4 tig .. + 3 of both 16-channel halves
            qv[it][blk][0] = x.x; qv[it][blk][1] = x.y; qv[it][blk][2] = x.z; qv[it][blk][3] = x.w;
            qv[it][blk][4] = y.x; qv[it][blk][5] = y.y; qv[it][blk][6] = y.z; qv[it][blk][7] = y.w;
        }
    }

    // ---- the new row of this sequence ------------------------------------------------------------------------
    int new_tile = -1, new_row = 0;         // tile of this CTA's range that holds the new slot, and its row there
    NewRow<HD> nr;
    if (p.new_k) {
        const int pos = p.n_small ? p.pos_small[b] : p.ring[b].x;
        const int tile = pos / T;
        const bool in_seq = tile >= t_first && tile < t_last;
        if (tile >= t_begin && tile < t_end) { new_tile = tile - t_begin; new_row = pos % T; }
        const bool writer = blockIdx.z == 0 && (new_tile >= 0 || (!in_seq && split == 0));
        if (new_tile >= 0 || writer) {
            const float* krow = p.new_k + (size_t)b * p.new_stride + kvh * HD;
            const float* vrow = p.new_v + (size_t)b * p.new_stride + kvh * HD;
            const long long rp = p.cos ? p.positions[b] : 0;
#pragma unroll
            for (int blk = 0; blk < NB; blk++) {
                const float kx = p.cos ? rotated<HD>(krow, blk * 32 + lane, p.cos, p.sin, rp) : __ldg(krow + blk * 32 + lane);
                const float vx = __ldg(vrow + blk * 32 + lane);
                nr.k[blk] = flare_q8_code(kx, nr.ks[blk]);
                nr.v[blk] = flare_q8_code(vx, nr.vs[blk]);
            }
            if (writer) {
                const size_t row = (size_t)b * p.payload_seq_stride + ((size_t)pos * nkv + kvh) * HD;
                const size_t srow = (size_t)b * p.scale_seq_stride + (size_t)pos * bpr + kvh * NB;
#pragma unroll
                for (int blk = 0; blk < NB; blk++) {
                    p.kq[row + blk * 32 + lane] = (int8_t)nr.k[blk];
                    p.vq[row + blk * 32 + lane] = (int8_t)nr.v[blk];
                    if (lane == 0) { p.ks_w[srow + blk] = __float2half_rn(nr.ks[blk]); p.vs_w[srow + blk] = __float2half_rn(nr.vs[blk]); }
                }
            }
        }
    }

    // ---- q as two int8 limbs per head: B operand of m16n8k32, column g = limb g & 1 of head g >> 1 -------------
    uint32_t qb[NI][NB][2];
    float qs[NI];                                   // of head tig: score = qs * sum_blk ks * (int dot)
#pragma unroll
    for (int it = 0; it < NI; it++) {
        const int item = item0 + it, hg = min(item, n_items - 1) % p.hgroups, hq = g >> 1;
        const bool ok = item < n_items && hq < p.G - 4 * hg;
        const float sc = rsqrtf((float)HD) * kLog2e;
        float amax = 0.0f;
        if (rope_c) {
#pragma unroll
            for (int blk = 0; blk < NB / 2; blk++)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int ch = blk * 32 + (i >> 2) * 16 + (i & 3);
                    const float c = __ldg(rope_c + ch), s = __ldg(rope_s + ch), x0 = qv[it][blk][i], x1 = qv[it][blk + NB / 2][i];
                    qv[it][blk][i] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
                    qv[it][blk + NB / 2][i] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
                }
        }
#pragma unroll
        for (int blk = 0; blk < NB; blk++)
#pragma unroll
            for (int i = 0; i < 8; i++) { qv[it][blk][i] *= sc; amax = fmaxf(amax, fabsf(qv[it][blk][i])); }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float inv = amax > 0.0f ? kQFix / amax : 0.0f;
#pragma unroll
        for (int blk = 0; blk < NB; blk++) {
            uint32_t l[2] = {0, 0};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int Q = __float2int_rn(qv[it][blk][i] * inv);
                const int lo_limb = ((Q + 64) & 127) - 64;          // [-64, 63]
                const int hi_limb = (Q - lo_limb) >> 7;              // exact: Q = 128 * hi + lo
                l[i >> 2] |= (uint32_t)(((g & 1) ? lo_limb : hi_limb) & 0xFF) << (8 * (i & 3));
            }
            qb[it][blk][0] = ok ? l[0] : 0u;
            qb[it][blk][1] = ok ? l[1] : 0u;
        }
        qs[it] = __shfl_sync(0xffffffffu, amax / kQFix, 8 * tig);      // lane with g = 2 tig holds head tig
    }

    // ---- running state: the lane's column pair belongs to head tig -----------------------------------------------
    float acc[NP][NC][4];           // channels 16 c + 2 g (elements 0, 1) and + 1 (elements 2, 3)
    float lb[NP][NSET];             // sum of the rounded weights of column g (head g >> 1) over this lane's slots
    float m_run[NI], l_run[NI];
#pragma unroll
    for (int pr = 0; pr < NP; pr++) {
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[pr][c][k] = 0.0f;
#pragma unroll
        for (int s = 0; s < NSET; s++) lb[pr][s] = 0.0f;
    }
#pragma unroll
    for (int it = 0; it < NI; it++) { m_run[it] = -CUDART_INF_F; l_run[it] = 0.0f; }

    // lane-constant shared-memory offsets.  The swizzle XORs the 16-byte chunk index with row bits that are the same
    // for every 8-slot step (rows advance by 8), so each address is base(lane) + constant.
    uint32_t koff[2 * NB];          // K bytes of slot g, channels c*16 + 4*tig .. +3
#pragma unroll
    for (int c = 0; c < 2 * NB; c++) koff[c] = tile_at<HD>(kvh, g, c) + tig * 4;
    uint32_t voff[NC / 2];          // ldmatrix row address: V slot 8 * (mi & 1) + r, chunk 2 cp + (mi >> 1)
#pragma unroll
    for (int cp = 0; cp < NC / 2; cp++)
        voff[cp] = payload + tile_at<HD>(kvh, ((lane >> 3) & 1) * 8 + (lane & 7), 2 * cp + (lane >> 4));
    const uint32_t ksoff = 2 * payload + (g * bpr + kvh * NB) * 2;         // scales of slot g, this head: [slot][nkv*NB] f16

    bool failed = false;
    for (int i = 0; i < n_tiles; i++) {
        const int s = i % STAGES;
        const int slot0 = (t_begin + i) * T;
        if (!ptx::mbar_wait(&full_bar[s], (uint32_t)((i / STAGES) & 1))) { failed = true; break; }
        unsigned char* kt = sbase + (size_t)s * stage_bytes;
        const uint32_t vt = ptx::smem_u32(kt);
        if (i == new_tile) {        // the slot written by this very call: its codes straight into the tile (this head's slice only)
#pragma unroll
            for (int blk = 0; blk < NB; blk++) {
                const uint32_t off = tile_at<HD>(kvh, new_row, blk * 2 + (lane >> 4)) + (lane & 15);
                kt[off] = (unsigned char)nr.k[blk];
                kt[payload + off] = (unsigned char)nr.v[blk];
                if (lane == 0) {
                    __half* sr = reinterpret_cast<__half*>(kt + 2 * payload) + new_row * bpr + kvh * NB + blk;
                    *sr = __float2half_rn(nr.ks[blk]);
                    *reinterpret_cast<__half*>(reinterpret_cast<unsigned char*>(sr) + scale_tile) = __float2half_rn(nr.vs[blk]);
                }
            }
            ptx::fence_proxy_async();       // before a later copy into this stage
            __syncwarp();
        }

        // ---- scores of slots 16 mt + g and + 8 for head tig: int8 MMA per 16 slots and 32-channel block --------
        float sc[NI][4], vs[4][NB];          // sc[][2 mt + r]: integer-domain scores (score = qs * sc, qs >= 0)
        const bool edge_tile = (slot0 < lo) || (slot0 + T > hi_short);      // warp-uniform
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
            float ks[2][NB];
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int h = 0; h < NB / 2; h++) {
                    const uint32_t so = ksoff + ((16 * mt + 8 * r) * bpr + 2 * h) * 2;
                    const float2 kf = unpack_half2(*reinterpret_cast<const uint32_t*>(kt + FLARE_CK(so, 4, stage_bytes, p.err)));
                    const float2 vf = unpack_half2(*reinterpret_cast<const uint32_t*>(kt + FLARE_CK(so + scale_tile, 4, stage_bytes, p.err)));
                    ks[r][2 * h] = kf.x; ks[r][2 * h + 1] = kf.y;
                    vs[2 * mt + r][2 * h] = vf.x; vs[2 * mt + r][2 * h + 1] = vf.y;
                }
#pragma unroll
            for (int it = 0; it < NI; it++) { sc[it][2 * mt] = 0.0f; sc[it][2 * mt + 1] = 0.0f; }
#pragma unroll
            for (int blk = 0; blk < NB; blk++) {
                // A fragment: slots g and g + 8, channels blk*32 + 4*tig .. +3 and 16 further (the four words of a quad
                // row are one 16-byte chunk: no bank conflicts in the swizzled tile)
                uint32_t ka[4];
#pragma unroll
                for (int w = 0; w < 4; w++)
                    ka[w] = *reinterpret_cast<const uint32_t*>(kt + FLARE_CK(koff[2 * blk + (w >> 1)] + (2 * mt + (w & 1)) * 8 * 128, 4, payload, p.err));
#pragma unroll
                for (int it = 0; it < NI; it++) {
                    int d[4];
                    mma_s8(d, ka[0], ka[1], ka[2], ka[3], qb[it][blk][0], qb[it][blk][1]);
                    sc[it][2 * mt] = fmaf(ks[0][blk], (float)(d[0] * 128 + d[1]), sc[it][2 * mt]);
                    sc[it][2 * mt + 1] = fmaf(ks[1][blk], (float)(d[2] * 128 + d[3]), sc[it][2 * mt + 1]);
                }
            }
        }
        if (edge_tile) {       // only the first and last tile of a range hold slots outside it
            // A slot outside the range gets weight exp2(-inf) = 0, but its V scale may be anything: rows past the end of
            // the plane are never copied, so that part of the stage keeps what an earlier kernel left in shared memory
            // (possibly Inf or NaN bit patterns, and 0 * NaN = NaN).  Zero it as well.
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int slot = slot0 + 8 * r + g;
#pragma unroll
                for (int it = 0; it < NI; it++)
                    if (slot < lo || slot >= item_hi(it)) sc[it][r] = -CUDART_INF_F;
                if (slot < lo || slot >= hi)
#pragma unroll
                    for (int blk = 0; blk < NB; blk++) vs[r][blk] = 0.0f;
            }
        }
        // Lazy rescaling: the reference maximum m_run only moves when a score exceeds it by more than 2^8, so
        // exponentials stay below 256 and the accumulators are rarely rescaled.  The test is a vote; the maximum over
        // the 8 lanes of a head is only reduced when it has to move.
        float tmax[NI];
        bool bump = false;
#pragma unroll
        for (int it = 0; it < NI; it++) {
            tmax[it] = fmaxf(fmaxf(sc[it][0], sc[it][1]), fmaxf(sc[it][2], sc[it][3])) * qs[it];
            bump = bump || tmax[it] > m_run[it] + 8.0f;          // also true for the first valid slots (m_run = -inf)
        }
        if (__any_sync(0xffffffffu, bump)) {
            float alpha[NI];
#pragma unroll
            for (int it = 0; it < NI; it++) {
                float t = tmax[it];
#pragma unroll
                for (int off = 4; off <= 16; off <<= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, off));
                const bool up = t > m_run[it] + 8.0f;
                alpha[it] = up ? fast_exp2(m_run[it] - t) : 1.0f;      // m_run = -inf -> 0 (nothing accumulated yet)
                if (up) m_run[it] = t;
                l_run[it] *= alpha[it];
            }
#pragma unroll
            for (int pr = 0; pr < NP; pr++) {
                const float a0 = alpha[NI == 1 ? 0 : 2 * pr], a1 = alpha[NI == 1 ? 0 : 2 * pr + 1];
#pragma unroll
                for (int c = 0; c < NC; c++) { acc[pr][c][0] *= a0; acc[pr][c][1] *= a1; acc[pr][c][2] *= a0; acc[pr][c][3] *= a1; }
                // the weight sums belong to column g: item g & 1 of head g >> 1, which other lanes of the quad row look after
                const float c0 = __shfl_sync(0xffffffffu, a0, (lane & ~3) | (g >> 1)), c1 = __shfl_sync(0xffffffffu, a1, (lane & ~3) | (g >> 1));
#pragma unroll
                for (int s2 = 0; s2 < NSET; s2++) lb[pr][s2] *= (g & 1) ? c1 : c0;
            }
        }
#pragma unroll
        for (int it = 0; it < NI; it++) {
            // an item whose own range ends before this CTA's first tile has seen nothing yet (m_run = -inf)
            const float neg_m = (NI > 1 && m_run[it] == -CUDART_INF_F) ? 0.0f : -m_run[it];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                sc[it][r] = fast_exp2(fmaf(sc[it][r], qs[it], neg_m));
                // two neighbouring slots in order, as lanes g and g ^ 1 hold them (only even g end up with the sum)
                l_run[it] = (l_run[it] + sc[it][r]) + __shfl_xor_sync(0xffffffffu, sc[it][r], 4);
            }
        }

        // ---- output: f16 MMA, weights p * vs rounded to f16 (relative error 2^-12, well inside the output tolerance);
        //      the bias term uses the rounded weights so that it cancels exactly -----------------------------
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
            uint32_t bw[NP][NSET][2];
#pragma unroll
            for (int pr = 0; pr < NP; pr++)
#pragma unroll
                for (int s2 = 0; s2 < NSET; s2++) {
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const int sl = 2 * mt + r;
                        const float w0 = NI == 1 ? sc[0][sl] * vs[sl][2 * s2] : sc[2 * pr][sl] * vs[sl][s2];
                        const float w1 = NI == 1 ? sc[0][sl] * vs[sl][(2 * s2 + 1) % NB] : sc[NI == 1 ? 0 : 2 * pr + 1][sl] * vs[sl][s2];
                        bw[pr][s2][r] = movmatrix_trans(pack_half2(w0, w1));       // column g, slots 2 tig and 2 tig + 1
                        const float2 wf = unpack_half2(bw[pr][s2][r]);
                        lb[pr][s2] += wf.x + wf.y;
                    }
                }
#pragma unroll
            for (int cp = 0; cp < NC / 2; cp++) {          // pairs of 16-channel tiles
                uint32_t rr[4];
                // a row of 16 bytes per lane, inside this head's V tile
                ldmatrix_x4_trans(rr, vt + FLARE_CK(voff[cp] + mt * 16 * 128, 16, 2 * payload, p.err));
#pragma unroll
                for (int k = 0; k < 4; k++) rr[k] ^= 0x80808080u;     // int8 -> uint8 (v + 128)
#pragma unroll
                for (int cc = 0; cc < 2; cc++) {
                    // bytes (slot a, ch 0), (slot a, ch 1), (slot a+1, ch 0), (slot a+1, ch 1) ->
                    // half2 (1024 + u[a][ch], 1024 + u[a+1][ch]): even channels are rows 0-7 of A, odd ones rows 8-15
                    const uint32_t a0 = __byte_perm(rr[2 * cc], 0x64646464u, 0x4240);
                    const uint32_t a1 = __byte_perm(rr[2 * cc], 0x64646464u, 0x4341);
                    const uint32_t a2 = __byte_perm(rr[2 * cc + 1], 0x64646464u, 0x4240);
                    const uint32_t a3 = __byte_perm(rr[2 * cc + 1], 0x64646464u, 0x4341);
                    const int c = 2 * cp + cc, s2 = NI == 1 ? c / 4 : c / 2;
#pragma unroll
                    for (int pr = 0; pr < NP; pr++) mma_f16(acc[pr][c], a0, a1, a2, a3, bw[pr][s2][0], bw[pr][s2][1]);
                }
            }
        }

        // ---- the last warp to finish with this stage refills it -------------------------------
        __syncwarp();
        if (lane == 0 && i + STAGES < n_tiles) {
            if (atomicAdd(&done_cnt[s], 1) == nkv - 1) {
                done_cnt[s] = 0;
                ptx::fence_proxy_async();
                issue(i + STAGES);
            }
        }
    }
    if (failed && lane == 0) flare_report(p.err, FLARE_ERR_TIMEOUT);

    // ---- finish: the sums over the lanes of a head (of a column), remove the 1152 bias, merge or write -------------
#pragma unroll
    for (int it = 0; it < NI; it++) {
        l_run[it] += __shfl_xor_sync(0xffffffffu, l_run[it], 8);
        l_run[it] += __shfl_xor_sync(0xffffffffu, l_run[it], 16);
        l_run[it] = __shfl_sync(0xffffffffu, l_run[it], tig);                  // from g = 0
    }
    float bias[NP][NSET][2];        // of columns 2 tig and 2 tig + 1
#pragma unroll
    for (int pr = 0; pr < NP; pr++)
#pragma unroll
        for (int s2 = 0; s2 < NSET; s2++) {
            lb[pr][s2] += __shfl_xor_sync(0xffffffffu, lb[pr][s2], 1);
            lb[pr][s2] += __shfl_xor_sync(0xffffffffu, lb[pr][s2], 2);
            bias[pr][s2][0] = 1152.0f * __shfl_sync(0xffffffffu, lb[pr][s2], 8 * tig);
            bias[pr][s2][1] = 1152.0f * __shfl_sync(0xffffffffu, lb[pr][s2], 8 * tig + 4);
        }
    // channels 16 c + 2 g and + 1 of head tig, unnormalised
    auto channel_pair = [&](int it, int c) {
        const int pr = NI == 1 ? 0 : it / 2, blk = c / 2;
        const int col = NI == 1 ? (blk & 1) : (it & 1), set = NI == 1 ? blk / 2 : blk;
        const float bs = bias[pr][set][col];
        return make_float2(acc[pr][c][col] - bs, acc[pr][c][2 + col] - bs);
    };
    if (NI == 1 && p.cluster) {
        // The splits of this sequence are the CTAs of one cluster.  The record (m, l, o) of a head goes to the CTA that
        // merges the head, by asynchronous stores that count themselves in on that CTA's barrier: no barrier over the
        // whole cluster stands between the last tile and the merge.  (Two cluster barriers around loads from the
        // peers' memory cost 2.6 us per call at 8 CTAs.)
        const float* rec = reinterpret_cast<const float*>(sbase + p.rec_off);       // [local head][source][HD + 2]
        cluster_wait();                                     // every peer's record barrier is ready
        if (tig < p.G) {
            const uint32_t h = (uint32_t)(kvh * p.G + tig), n = (uint32_t)p.n_split, owner = h % n;
            const uint32_t bar = cluster_map(ptx::smem_u32(&rec_bar), owner);
            const uint32_t dst = cluster_map(ptx::smem_u32(rec) + ((h / n) * n + rank) * (HD + 2) * 4, owner);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const float2 o = channel_pair(0, c);
                cluster_st_async(dst + (2 + 16 * c + 2 * g) * 4, bar, o.x, o.y);
            }
            if (g == 0) cluster_st_async(dst, bar, m_run[0], failed ? 0.0f : l_run[0]);
        }
        if (my_heads == 0) return;
        if (!ptx::mbar_wait(&rec_bar, 0)) {                 // a peer never delivered: report, write nothing
            if (lane == 0) flare_report(p.err, FLARE_ERR_TIMEOUT);
            return;
        }
        for (int idx = threadIdx.x; idx < my_heads * HD; idx += blockDim.x) {
            const int lh = idx / HD, d = idx % HD;
            const float* r = rec + (size_t)lh * p.n_split * (HD + 2);
            float mm = -CUDART_INF_F;
            for (int s2 = 0; s2 < p.n_split; s2++) if (r[s2 * (HD + 2) + 1] > 0.0f) mm = fmaxf(mm, r[s2 * (HD + 2)]);
            float ll = 0.0f, o = 0.0f;
            for (int s2 = 0; s2 < p.n_split; s2++) {
                const float l2 = r[s2 * (HD + 2) + 1];
                const float w = l2 > 0.0f ? fast_exp2(r[s2 * (HD + 2)] - mm) : 0.0f;
                ll = fmaf(l2, w, ll);
                o = fmaf(r[s2 * (HD + 2) + 2 + d], w, o);
            }
            o = ll > 0.0f ? (p.n_ranges == 1 ? o * (1.0f / ll) : o / ll) : 0.0f;       // one range: as the path below writes it
            const size_t at = ((size_t)b * p.num_heads + rank + (size_t)lh * p.n_split) * HD + d;
            if (p.oq) {                                     // 32 consecutive channels are one warp: an input block of the next product
                float bs;
                p.oq[at] = (int8_t)flare_q8_code(o, bs);
                if (lane == 0) p.os[at / 32] = bs;
            } else p.out[at] = o;
        }
        return;
    }
    if (failed) return;
    const bool final_out = (p.n_split == 1) && !p.want_partial;
#pragma unroll
    for (int it = 0; it < NI; it++) {
        const int item = item0 + it, qi = item / p.hgroups, hg = item % p.hgroups;
        if (item >= n_items || tig >= p.G - 4 * hg) continue;
        const size_t row = ((size_t)b * p.n_q + qi) * p.num_heads + kvh * p.G + 4 * hg + tig;
        const float inv_l = l_run[it] > 0.0f ? 1.0f / l_run[it] : 0.0f;
        float* wrec = p.work + (row * p.n_split + split) * (HD + 2);
#ifdef FLARE_DEBUG_BOUNDS
        if (row >= (size_t)p.batch * p.n_q * p.num_heads || split >= p.n_split) { flare_report(p.err, FLARE_ERR_BOUNDS); return; }
#endif
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const float2 o = channel_pair(it, c);
            if (final_out) *reinterpret_cast<float2*>(p.out + row * HD + 16 * c + 2 * g) = make_float2(o.x * inv_l, o.y * inv_l);
            else *reinterpret_cast<float2*>(wrec + 2 + 16 * c + 2 * g) = o;
        }
        if (!final_out && g == 0) { wrec[0] = m_run[it]; wrec[1] = l_run[it]; }
    }
}

}  // namespace

static size_t q8_stage_bytes(int nkv, int hd) {
    return (size_t)nkv * 2 * T * hd + 2 * (size_t)T * nkv * (hd / 32) * 2;
}
// Items of a sequence: queries x groups of up to 4 query heads per KV head.
static int q8_items(const DecodeArgs& a) { return a.n_q * ((a.num_heads / a.kv.num_kv_heads + 3) / 4); }

bool flare_decode_q8_supported(const DecodeArgs& a) {
    const int hd = a.kv.head_dim, nkv = a.kv.num_kv_heads;
    if (a.kv.dtype != FLARE_KV_Q8_0 || (hd != 64 && hd != 128) || nkv > 8 || a.window != 0 || !a.kmap || q8_items(a) > 64) return false;
    // every stage must start on a 1024-byte boundary (swizzle) and the scale tile on 16 bytes; other shapes keep the
    // f32 arithmetic of the general kernel
    return q8_stage_bytes(nkv, hd) % 1024 == 0;
}

using Q8Kernel = void (*)(const CUtensorMap, const CUtensorMap, const Q8Params);
template <int NKV> static Q8Kernel q8_kernel_of(int hd, int ni) {
    if (hd == 64) return ni == 1 ? decode_q8_kernel<64, 1, NKV> : decode_q8_kernel<64, 2, NKV>;
    return ni == 1 ? decode_q8_kernel<128, 1, NKV> : decode_q8_kernel<128, 2, NKV>;
}
static Q8Kernel q8_kernel(int hd, int ni, int nkv) { return nkv == 8 ? q8_kernel_of<8>(hd, ni) : q8_kernel_of<0>(hd, ni); }

// The opt-ins to large dynamic shared memory and to large clusters, once per device and instantiation (table mutex held).
static int q8_opt_in(flare_attn_ctx* ctx, int hd, int ni, int nkv, int smem) {
    static bool done[64][2][8][2] = {};
    bool& d = done[ctx->device & 63][hd == 128][ni][nkv == 8];
    if (d) return FLARE_OK;
    FLARE_CUDA_OK(ctx, cudaFuncSetAttribute(q8_kernel(hd, ni, nkv), cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (ni == 1) FLARE_CUDA_OK(ctx, cudaFuncSetAttribute(q8_kernel(hd, ni, nkv), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    d = true;
    return FLARE_OK;
}

int flare_launch_decode_q8(flare_attn_ctx* ctx, const DecodeArgs& a) {
    const int hd = a.kv.head_dim, nkv = a.kv.num_kv_heads;
    const int rows = a.batch * a.n_q * a.num_heads;
    if (rows == 0) return FLARE_OK;
    Q8Params p;
    p.q = a.q; p.out = a.out;
    p.q_seq_stride = a.q_seq_stride ? a.q_seq_stride : (size_t)a.n_q * a.num_heads * hd;
    p.k_scale = reinterpret_cast<const __half*>(a.kv.plane[FLARE_PLANE_K_SCALE]);
    p.v_scale = reinterpret_cast<const __half*>(a.kv.plane[FLARE_PLANE_V_SCALE]);
    p.scale_seq_stride = a.kv.stride[FLARE_PLANE_K_SCALE] / 2;
    p.layer_seq0 = a.layer * a.batch;
    p.batch = a.batch; p.num_heads = a.num_heads; p.nkv = nkv; p.G = a.num_heads / nkv; p.max_seq = a.kv.max_seq_len;
    p.n_q = a.n_q; p.causal_q = a.causal_q; p.hgroups = (p.G + 3) / 4;
    p.n_small = 0; p.attend_len = nullptr; p.ring = nullptr;
    const StepFusion* f = a.fuse;
    if (a.h_attend && a.batch <= SMALL) {
        p.n_small = a.batch;
        for (int b = 0; b < a.batch; b++) p.attend_small[b] = a.h_attend[b];
        if (f && f->k) for (int b = 0; b < a.batch; b++) p.pos_small[b] = a.h_ring[b].x;
    } else FLARE_TRY(flare_small_on_device(ctx, a, &p.attend_len, &p.ring));
    p.new_k = f ? f->k : nullptr; p.new_v = f ? f->v : nullptr; p.new_stride = f ? f->row_stride : 0;
    p.cos = f ? f->cos : nullptr; p.sin = f ? f->sin : nullptr; p.positions = f ? f->positions : nullptr;
    p.oq = nullptr; p.os = nullptr;
    p.kq = (int8_t*)a.kv.plane[FLARE_PLANE_K_Q]; p.vq = (int8_t*)a.kv.plane[FLARE_PLANE_V_Q];
    p.ks_w = (__half*)a.kv.plane[FLARE_PLANE_K_SCALE]; p.vs_w = (__half*)a.kv.plane[FLARE_PLANE_V_SCALE];
    p.payload_seq_stride = a.kv.stride[FLARE_PLANE_K_Q];
    p.slot_begin = a.slot_begin; p.slot_end = a.slot_end; p.want_partial = a.want_partial;
    int range_max = a.slot_end >= 0 ? (a.slot_end - a.slot_begin) : a.max_attend;
    if (range_max < 0) range_max = 0;
    p.err = ctx->d_err;

    const int items = q8_items(a);
    // Several items go two to a CTA.  (Four or six at once, a warp per head and CTA, leave one CTA of 8 warps on an SM: six
    // queries x 32 sequences x 3000 slots 58 us against 66.)
    const int ni = items == 1 ? 1 : 2;
    const int zdim = (items + ni - 1) / ni;
    const size_t smem_plain = STAGES * q8_stage_bytes(nkv, hd) + 1024;
    const int ctas_per_sm = smem_plain <= 110 * 1024 ? 2 : 1;
    const int places = ctx->sm_count * ctas_per_sm;
    // at least two tiles per CTA (slot-range calls and calls whose records another kernel merges keep four: twice the
    // ranges are twice the records for that kernel)
    int min_tiles = (a.defer_merge || a.want_partial || a.slot_end >= 0) ? 4 : 2;
    const int max_split = std::max(1, ((range_max + T - 1) / T + min_tiles - 1) / min_tiles), max_tiles = (range_max + T - 1) / T;
    // one wave: as many splits as fit without a second, partly filled one
    const int units = a.batch * zdim, fit = std::max(1, std::min({places / units, max_split, 256}));
    // Cluster mode: when a handful of splits per sequence fill the GPU anyway, the splits of a sequence become one
    // thread-block cluster (2 .. 16 CTAs; more than 8 is the non-portable size, opted into) and merge through distributed
    // shared memory: no second kernel, no round trip of the records through global memory.  The size is the largest one,
    // not far below the number of splits that would fit, for which every sequence's cluster is resident at once.
    int cluster = 0, n_split = 1, n_ranges = 1;
    // a CTA of a cluster of c merges every c-th head and receives c records for each
    auto rec_bytes = [&](int c) { return (size_t)((p.num_heads + c - 1) / c * c) * (hd + 2) * 4; };
    const size_t smem_limit = 226 * 1024;                // of 227 KB; the barriers are static shared memory
    size_t smem = smem_plain;
    if (!a.want_partial && a.slot_end < 0 && ni == 1) {
        // [device][hd == 128][nkv][size]: clusters resident at once; 0 = not asked yet
        static int max_clusters[64][2][9][MAX_CLUSTER + 1] = {};
        std::lock_guard<std::mutex> lock(g_table_mutex);
        // (two at least: the cluster's remote stores need a real cluster, and a CTA without tiles costs nothing)
        int c_first = fit > MAX_CLUSTER ? MAX_CLUSTER : fit < 2 ? 2 : fit;
        for (int c = c_first; c >= 2 && !cluster; c--) {
            // Far fewer CTAs than places: the merge kernel is cheaper (a CTA alone needs 0.65 us per tile: one sequence x
            // 4096 slots 7.7 us with 64 ranges and the second kernel, 9.4 with a cluster of 16), unless the ranges are
            // so short that the call is over before the second kernel would have done its work (2048 slots: 6.5 us in a
            // cluster, 8.0 with the merge kernel), or the wave of ranges would load every SM twice (8 sequences x 3000
            // slots: 9.9 and 11.4).  Outputs that are about to become 8-bit codes keep to a fixed line: where the
            // ranges are cut shows in an output's last bits, and in a code now and then.
            const int short_range = fit * a.batch > ctx->sm_count ? 10 : 5;
            if (f && f->oq ? c * 5 < fit * 4 : c * 9 < fit * 5 && (max_tiles + c - 1) / c > short_range) break;
            if (smem_plain + rec_bytes(c) > smem_limit) continue;
            int& mc = max_clusters[ctx->device & 63][hd == 128][nkv][c];
            if (mc == 0) {
                FLARE_TRY(q8_opt_in(ctx, hd, ni, nkv, (int)smem_limit));
                cudaLaunchAttribute ca[1];
                ca[0].id = cudaLaunchAttributeClusterDimension;
                ca[0].val.clusterDim.x = c; ca[0].val.clusterDim.y = 1; ca[0].val.clusterDim.z = 1;
                cudaLaunchConfig_t qc = {};
                qc.gridDim = dim3(c, 1); qc.blockDim = dim3(32 * nkv); qc.dynamicSmemBytes = smem_plain + rec_bytes(c);
                qc.attrs = ca; qc.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, q8_kernel(hd, ni, nkv), &qc) != cudaSuccess) { cudaGetLastError(); n = 0; }
                mc = n > 0 ? n : -1;
            }
            if (mc >= a.batch) cluster = c;
        }
    }
    if (cluster) {
        n_split = cluster; n_ranges = std::min(cluster, max_split);
        p.rec_off = (int)(STAGES * q8_stage_bytes(nkv, hd));
        smem = smem_plain + rec_bytes(cluster);
        if (f && f->oq) { p.oq = f->oq; p.os = f->os; }
    } else {
        p.rec_off = 0;
        n_split = fit;
        // Several items per sequence and a wave filled to less than three quarters: two full waves of shorter ranges keep
        // every SM loaded twice
        const int two_waves = 2 * places / units;
        if (items > 1 && fit * units * 4 < places * 3 && two_waves > fit && two_waves <= max_split) n_split = std::min(two_waves, 256);
    }
    if (f && f->quantised) *f->quantised = p.oq != nullptr;
    p.n_split = n_split;
    p.n_ranges = cluster ? n_ranges : n_split;
    p.cluster = cluster;
    p.work = nullptr;
    const bool merge = !cluster && (n_split > 1 || a.want_partial);
    if (merge) {
        // two workspaces used alternately: the merge of one call may still be reading while the next call's decode
        // kernel (started early, see below) writes
        size_t need = ((size_t)rows * n_split * (hd + 2) * sizeof(float) + 255) / 256 * 256;
        FLARE_TRY(flare_ensure(ctx, &ctx->d_work, &ctx->work_bytes, 2 * need));
        ctx->work_phase ^= 1;
        p.work = (float*)((char*)ctx->d_work + (size_t)ctx->work_phase * need);
    }
    Q8Kernel kernel = q8_kernel(hd, ni, nkv);
    { std::lock_guard<std::mutex> lock(g_table_mutex); FLARE_TRY(q8_opt_in(ctx, hd, ni, nkv, (int)smem_limit)); }
    // Programmatic dependent launch: when the previous kernel on this stream is one that stores no cache rows, or stores
    // those of another layer, this kernel requests its first K/V tiles while the predecessor drains; it waits before
    // touching q or the new rows.
    p.wait_first = (ctx->last_launch_overlappable && ctx->last_written_layer != a.kv.plane[FLARE_PLANE_K_Q]) ? 0 : 1;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster ? cluster : 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_split, a.batch, zdim);
    cfg.blockDim = dim3(32 * nkv);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cfg.attrs = attr;
    cfg.numAttrs = cluster ? 2 : 1;
    FLARE_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, kernel, *a.kmap, *a.vmap, p));
    FLARE_LAUNCH_CHECK(ctx);
    const void* written = p.new_k ? a.kv.plane[FLARE_PLANE_K_Q] : nullptr;
    ctx->last_launch_overlappable = true;
    ctx->last_written_layer = written;
    if (a.defer_merge && a.want_partial) {          // the caller merges: tell it where the records are
        *a.work_out = p.work; *a.n_split_out = n_split;
        return FLARE_OK;
    }
    if (merge) {
        // log-sum-exp merge of the slot ranges, chained with programmatic dependent launch (multi.cu).  Its successor may
        // start before the kernel above has completed, so what that kernel stores stays on record.
        FLARE_TRY(flare_launch_merge_splits(ctx, p.work, n_split, rows, hd, a.out, a.want_partial));
        ctx->last_launch_overlappable = true;
        ctx->last_written_layer = written;
    }
    return FLARE_OK;
}
