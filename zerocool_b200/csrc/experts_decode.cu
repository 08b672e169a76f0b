// Decode family: the routed and shared experts for short token batches.
//
// Replaces, for every expert that received work, the reference's per-expert launches
//   gated_linear -> q4_gate_mv_r2 / q4_gate_up (kernels/metal/qwen.metal:333-376, 71-81)
//   linear_into  -> q4_mv_r* / q4_mm           (qwen.metal:289-330, 63-70), scatter_experts :800-803
// issued by encode_expert_rows (src/engine/pipeline.cpp:7-31), and the shared expert of
// Model::moe (src/engine/model.cpp:482-484), with two grouped launches per layer of one kernel
// template:
//   NMAT = 2 (gate/up): h[row, f]  = silu(gate_e . x_row) * (up_e . x_row)    for every (expert, row)
//   NMAT = 1 (down):    y[slot, c] = down_e . h_row, written at the slot's router position
//
// Each launch streams every selected record once per eight rows (a pass). What bounds it is HBM as long as a weight costs few
// enough instructions: at 6.5 TB/s an SM receives ~46 4-bit weights per clock and can issue four warp instructions, so 1,024
// weights (16 rows x 64 k, one quantisation group of a tile) have ~88 issue slots at best. With everything around the products
// the item kernels execute 68 instructions on them (ncu, gate/up at 64 tokens), this one 61. Layers measured against the item
// kernels (us): 5 tokens 59 -> 50, 64 tokens 181 -> 172, 128 tokens 241 -> 231, 256 tokens 304 -> 264, 256 tokens at hidden 4096
// 605 -> 484; 700 tokens with Zipf-skewed loads 1816 -> 438 (the passes of one long item are spread over the machine instead of two CTAs).
// The 4-bit instantiations use all 128 registers a thread can have here and spill 4 to 48 bytes, the 8-bit ones with two-term rows 82 to 106.
// What is left at 64 tokens: ~8 us per launch until the first product (item list, tables, rows, then the first 128 KB per SM),
// and ends of the CTAs' runs that differ by up to a tenth.
//  * The multiply-accumulates run on the tensor cores as m16n8k16 FP16 MMAs with up to eight token
//    rows in the N dimension. Integer codes are exact in
//    FP16, a BF16 activation converts exactly, an FP32 activation is split into two FP16 terms, and products are
//    accumulated in FP32 per 64-wide quantisation group. The group's scale is applied to that FP32 sum; the bias term is
//    a product of its own:
//        acc += scale[row, g] * sum_k(q * x);     acc += bias[row, :] . group sums of x
//    which is the reference's affine_dot form (qwen.metal:46-62) with an exact inner sum. The bias product is an
//    TF32 MMA over a pair of stages (eight Q4 or four Q8 groups): a 16-bit bias is exact in TF32, and the FP32 group sum enters
//    as three TF32 terms, all of its 24 bits, smallest term first. It has accumulators of its own, which are added to acc in
//    FP32: the MMA's adder does not round to nearest, and in acc it would do so once per product. The product stands
//    between the two stages of its pair, where it cancels against the codes' part soonest. Error against 64 bits beside the item
//    kernels' FMA per group (two-term rows): gate/up 8.3e-6 / 8.3e-6 and down 2.26e-5 / 2.30e-5 (folded Q4), 2.29e-7 / 2.31e-7
//    and 3.7e-7 / 4.2e-7 (not folded), a Q8 layer 2.8e-7 / 3.1e-7; biases alone 1.9e-7 / 2.0e-7, and 1.3e-7 / 0.5e-7 where all
//    terms have one sign.
//  * Q4 codes become FP16 with one logic operation per two weights: (w & 0x000f000f) | 0x6400 is the
//    half2 (1024+q_lo, 1024+q_hi), and (w & 0x00f000f0) | 0x6400 is (1024+16 q, 1024+16 q). With FOLD
//    those values go into the MMA as they are: the activations that meet a "q" slot are staged multiplied by 16
//    (exact; the finished sum is divided by 16), and the 1024 offset is removed from the FP32 group sum, which starts
//    from -1024 * sum(x as staged).
//    Without FOLD the offset and the factor 16 are removed in FP16 before the MMA (exact, 4 more ops per
//    word).
//  * Codes reach a warp through its own ring of two 4 KB stages, filled by one TMA instruction per stage (a box of 32 rows
//    x 128 bytes: 16 rows of gate and of up, or 32 rows of down), so a copy costs no address arithmetic and no L1. The
//    128-byte swizzle exchanges 16-byte pieces by row mod 8; MMA row g reads tile row pi(g) = 0,4,2,6,1,5,3,7, with which
//    the 8-byte (Q4) and 16-byte (Q8) fragment reads of a warp hit every bank once.
//  * Scales and biases are read straight from global memory into registers, one stage ahead: the four lanes of a row share
//    an 8-byte read of four scales, and each lane fetches the one bias it supplies to the bias product.
//  * The grid is one persistent CTA per SM. The passes of all items are laid end to end (a block-wide scan of the
//    permutation's item list, which every CTA does for itself), every pass is cut into units of RT row tiles, and CTA b
//    takes the b-th of gridDim.x equal runs of units: no last wave, and the copies of the next unit are in flight while a
//    unit is finished. KS warps share a row tile by taking every KS-th stage of K; their partial sums are added in warp
//    order by one of them (a different one for each unit).
//  * Lanes whose token row is absent skip the activation reads.
//  * Because a dot product does not care about the order of k, the MMA's k slots are bound to whatever
//    k values fall out of the cheapest extraction; the activations are staged in the matching order.
// Activations must stay inside FP16 after the factor 16 (|x| < 4094 for Q4 projections, < 65504 for Q8); hidden
// states after a norm are O(1..100). A value beyond that raises ZC_STATUS_RANGE in the status word (the output of
// that row is then not meaningful); the same holds for the SwiGLU rows the down projection reads.
#include <cmath>

#include "experts_common.cuh"

namespace zc {
namespace {

constexpr int NROW = 8;               // token rows of a pass (the N of m16n8k16)
constexpr int MAX_WARPS = 16;
constexpr int MAX_THREADS = MAX_WARPS * 32;
constexpr int STAGES = 2;             // ring stages per warp
constexpr int STAGE_BYTES = 4096;     // 32 rows x 128 code bytes
constexpr int TABLE = 32;             // passes whose descriptors and rows a CTA keeps at a time
constexpr uint32_t PERM_CACHE = 1024;  // a permutation up to this long is fetched whole while the item list is read
constexpr uint32_t POLL_LIMIT = 1u << 18;     // attempts of a bounded wait, each suspended for at most about a microsecond

// D(16x8, fp32) += A(16x4, tf32) * B(4x8, tf32): a0: A[g][c], a1: A[g+8][c], b0: B[c][g].
__device__ __forceinline__ void mma_tf32_1684(float (&d)[4], float a0, float a1, float b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(b0)));
}

// D(16x8, fp32) += A(16x8, tf32) * B(8x8, tf32): a0: A[g][c], a1: A[g+8][c], a2: A[g][c+4], a3: A[g+8][c+4], b0: B[c][g], b1: B[c+4][g].
__device__ __forceinline__ void mma_tf32_1688(float (&d)[4], float a0, float a1, float a2, float a3, float b0, float b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)), "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// v as three TF32 values (11 + 11 + 2 significant bits: exact).
__device__ __forceinline__ void tf32_terms(float v, float& h, float& m, float& l) {
    h = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
    const float r = v - h;
    m = __uint_as_float(__float_as_uint(r) & 0xffffe000u);
    l = r - m;
}

// How a launch is cut (chosen on the host, stream_plan): warps per CTA, warps that share a row tile, staged passes,
// and what follows from them.
struct StreamPlan {
    uint32_t warps, ks, nbuf;
    uint32_t rt, ks_shift;           // warps / ks; log2(ks)
    uint32_t tiles_per_pass;         // row tiles of one pass: N / TILE
    uint32_t pairs;                  // stage pairs of a row's K, the last one padded
    uint32_t own;                    // item-list entries per thread
    float inv_tiles, inv_grid;
};

// The TMA view of one projection (pair) of all records: [expert][matrix][row][byte], and the same of the shared record.
struct StreamMaps { CUtensorMap routed, shared; };

__device__ __forceinline__ void ring_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int row, int expert) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(STAGE_BYTES) : "memory");
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(row), "r"(0), "r"(expert), "r"(bar) : "memory");
}
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void group_sync(uint32_t id, uint32_t threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void group_arrive(uint32_t id, uint32_t threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// n / d by a reciprocal and one correction (quotients below 2^20: the estimate is off by one at most).
__device__ __forceinline__ uint32_t quick_div(uint32_t n, uint32_t d, float inverse) {
    uint32_t q = __float2uint_rz(__uint2float_rn(n) * inverse);
    const int r = int(n - q * d);
    if (r < 0) --q;
    else if (uint32_t(r) >= d) ++q;
    return q;
}

__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// Stage this warp's share of the valid source rows (n < nvalid) of K elements into shared memory (convert8: hi, lo, and per group)
//   sx[n][grp] = sx;
//   offs[grp][n / 2][4] = -1024 * sf (nothing without FOLD), laid out as the four accumulators of a lane: the MMA starts from it,
//   which removes the folded 1024 offset of the codes.
// Rows n >= nvalid are left as they are: an MMA column only depends on its own B column.
// A warp takes 256 consecutive elements of a row at a time (eight per lane), pieces `first`, `first + stride`, ...
template <bool Q4ORDER, bool SPLIT, bool FOLD, typename RowOf>
__device__ __forceinline__ void stage_rows(const void* src, bool src_f32, RowOf row_of, uint32_t nvalid, uint32_t K, uint32_t RS, uint32_t GP,
                                           bool ref, __half* hi, __half* lo, float* sx_out, float* offs, uint32_t* status, uint32_t first, uint32_t stride) {
    const uint32_t per_row = (K + 255) / 256, lane = threadIdx.x % 32;
    bool beyond = false;
    uint32_t n = 0, piece = first;
    while (n < nvalid) {
        while (piece >= per_row) { piece -= per_row; ++n; }
        if (n >= nvalid) break;
        const uint32_t q = piece * 32 + lane;
        const bool live = q * 8 < K;           // a row's last piece may be short; its idle lanes carry zeros through the shuffles
        const size_t row = row_of(n);
        float v[8];
        if (!live) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        } else if (src_f32) {
            const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(src) + row * K + q * 8);
            const float4 a = __ldcg(p), b = __ldcg(p + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(src) + row * K + q * 8));
            const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(r[i] << 16); v[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u); }
        }
        uint4 ph, pl;
        float sx, sf;
        convert8<Q4ORDER, SPLIT, FOLD>(v, ref, ph, pl, sx, sf, beyond);
        if (live) {
            if ((lane & 7) == 0) {
                sx_out[n * GP + q / 8] = sx;
                if (FOLD) {                    // the MMA's addend of a lane: {tokens 2c, 2c + 1} for row g, the same for row g + 8
                    float* o = offs + (q / 8) * (2 * NROW) + (n / 2) * 4 + n % 2;
                    o[0] = o[2] = -1024.0f * sf;
                }
            }
            *reinterpret_cast<uint4*>(hi + n * RS + q * 8) = ph;
            if (SPLIT) *reinterpret_cast<uint4*>(lo + n * RS + q * 8) = pl;
        }
        piece += stride;
    }
    if (beyond) atomicOr(status, ZC_STATUS_RANGE);
}

// d[m] (16 rows x 8 tokens) = off + sum over one 64-wide group of code * x, for the two 16-row fragments m of a stage (the
// lane's rows g: w[m][0], g+8: w[m][1]). The fragments' independent MMA chains are interleaved. The low terms of a word follow its high
// terms, as in the item kernels: the adder drops bits relative to the running sum, which the high terms bring down from the folded offset.
template <int BITS, bool SPLIT, bool FOLD>
__device__ __forceinline__ void group_mma(float (&d)[2][4], const float4& off, const uint32_t (&w)[2][2][BITS / 2],
                                          const uint4 (&bh)[2], const uint4 (&bl)[2], bool q8_signed) {
    constexpr int PER = BITS == 4 ? 2 : 1, STEPS = BITS == 4 ? 2 : 4;      // MMAs per code word, code words
#pragma unroll
    for (int i = 0; i < STEPS; ++i) {
        uint32_t p[2][2][2 * PER];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if constexpr (BITS == 4) dequant_q4<FOLD>(w[m][r][i], p[m][r]);
                else dequant_q8(w[m][r][i], q8_signed, p[m][r]);
            }
#pragma unroll
        for (int t = 0; t < (SPLIT ? 2 : 1); ++t)                          // the low terms after the word's high terms
#pragma unroll
            for (int h = 0; h < PER; ++h) {
                const int step = i * PER + h;                              // of the group's four
                const uint4 v = t ? bl[step / 2] : bh[step / 2];
                const uint32_t b0 = step % 2 ? v.z : v.x, b1 = step % 2 ? v.w : v.y;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    if (step == 0 && t == 0) mma_f16_16816_c(d[m], p[m][0][0], p[m][1][0], p[m][0][1], p[m][1][1], b0, b1, off.x, off.y, off.z, off.w);
                    else mma_f16_16816(d[m], p[m][0][2 * h], p[m][1][2 * h], p[m][0][2 * h + 1], p[m][1][2 * h + 1], b0, b1);
                }
            }
    }
}

// Two 16-bit metadata values of a word as FP32.
template <bool META_F16>
__device__ __forceinline__ float2 meta_pair(uint32_t w) {
    if constexpr (META_F16) return __half22float2(*reinterpret_cast<const __half2*>(&w));
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// ---------------------------------------------------------------------------------------------
// The streaming kernel.
//   KS: warps that share one row tile, splitting K; the CTA works on RT = warps / KS tiles at a time.
//   NBUF: staged passes (2: the next pass's rows are converted while this one is multiplied).
// ---------------------------------------------------------------------------------------------
template <int BITS, bool SPLIT, bool FOLD, bool META_F16, int NMAT>
__global__ void __launch_bounds__(MAX_THREADS, 1) stream_kernel(const Call c, const __grid_constant__ StreamMaps maps, const StreamPlan plan) {
    constexpr int GPS = BITS == 4 ? 4 : 2;           // quantisation groups of one stage (128 code bytes of a row)
    constexpr int TILE = NMAT == 2 ? 16 : 32;        // matrix rows of a warp's tile; a stage holds two 16-row fragments either way
    constexpr int WORDS = BITS / 2;                  // 32-bit words per lane per row per group
    constexpr bool FOLDQ = FOLD && BITS == 4;
    constexpr int SW = GPS / 2;                      // words of a row's scales in one stage
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(16) uint64_t ring_bar[MAX_WARPS][STAGES];
    __shared__ __align__(16) uint64_t rows_full[2], rows_done[2];      // per staged pass: every warp has converted its share / has finished its tiles
    __shared__ int4 table[TABLE];                    // {expert (-1: shared), first position, rows, first row in hbuf}
    __shared__ int slots[TABLE][NROW];               // gate/up: token of every row; down: its router slot (routed) or token (shared); -1: absent
    __shared__ uint32_t warp_sums[MAX_WARPS];
    __shared__ int perm_s[PERM_CACHE];

    const uint32_t W = plan.warps, KS = plan.ks, RT = plan.rt, NBUF = plan.nbuf, UB = plan.tiles_per_pass, pairs = plan.pairs;
    const uint32_t tid = threadIdx.x, lane = tid % 32, g = lane / 4, cq = lane % 4;
    const uint32_t warp = __shfl_sync(0xffffffffu, tid / 32, 0);       // warp-uniform for the compiler too
    const uint32_t ks = warp & (KS - 1), rt = warp >> plan.ks_shift;
    const uint32_t K = NMAT == 2 ? c.H : c.F, N = NMAT == 2 ? c.F : c.H, G = K / 64;
    const uint32_t GPAD = pairs * 2 * GPS, RS = GPAD * 64 + ROW_PAD, GP = GPAD + 8;
    const uint32_t buf_bytes = (SPLIT ? 2 : 1) * NROW * RS * 2 + NROW * GP * 4 + GPAD * NROW * 8;
    uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* rows_base = ring + W * STAGES * STAGE_BYTES;                             // [NBUF]: hi [NROW][RS], lo, sx [NROW][GP], offs [GPAD][NROW / 2][4]
    float* red = reinterpret_cast<float*>(rows_base + NBUF * buf_bytes);              // [RT][KS - 1][2][32] float4
    auto hi_of = [&](uint32_t buf) { return reinterpret_cast<__half*>(rows_base + buf * buf_bytes); };
    auto sx_of = [&](uint32_t buf) { return reinterpret_cast<float*>(rows_base + buf * buf_bytes + (SPLIT ? 2 : 1) * NROW * RS * 2); };
    const uint32_t ring_base = smem_u32(ring) + warp * (STAGES * STAGE_BYTES), bar_base = smem_u32(&ring_bar[0][0]) + warp * (STAGES * 8);
    const uint32_t full_base = smem_u32(&rows_full[0]), done_base = smem_u32(&rows_done[0]);
    if (tid < W * STAGES + 4) {
        const uint32_t at = tid < W * STAGES ? smem_u32(&ring_bar[0][0]) + tid * 8 : tid < W * STAGES + 2 ? full_base + (tid - W * STAGES) * 8 : done_base + (tid - W * STAGES - 2) * 8;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(at), "r"(tid < W * STAGES ? 1u : W) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (GPAD != G) {                                 // k past the matrix: codes arrive as zeros and meet zeros
        for (uint32_t buf = 0; buf < NBUF; ++buf) {
            __half* xh = hi_of(buf);
            float* sx = sx_of(buf);
            float* offs = sx + NROW * GP;
            for (uint32_t i = tid; i < (SPLIT ? 2 : 1) * NROW * (GPAD - G) * 64; i += blockDim.x)
                xh[(i / ((GPAD - G) * 64)) * RS + G * 64 + i % ((GPAD - G) * 64)] = __ushort_as_half(0);
            for (uint32_t i = tid; i < NROW * (GPAD - G); i += blockDim.x) {
                const uint32_t n = i / (GPAD - G), grp = G + i % (GPAD - G);
                sx[n * GP + grp] = 0.0f;
                offs[grp * 2 * NROW + n] = offs[grp * 2 * NROW + NROW + n] = 0.0f;
            }
        }
    }

    // gate/up follows the routing kernel and needs its lists at once. down follows gate/up, whose own wait has
    // already seen the routing kernel complete: the passes, the row lists and the first weight stages of down are
    // set up while gate/up is still draining (on SMs that it has left), and only the read of the SwiGLU rows waits for it.
    uint32_t limit = POLL_LIMIT, parity0 = 0, parity1 = 0, done_tiles = 0, fin = rt & (KS - 1);
    if constexpr (NMAT == 2) { pdl_wait(); pdl_launch_dependents(); }

    // ---- the passes: the shared expert's blocks of NROW tokens, then every listed expert's blocks of NROW rows ----
    const uint32_t shared_passes = c.has_shared ? (c.T + NROW - 1) / NROW : 0;
    // A thread owns `own` consecutive entries of the item list; the first stays in registers, others (more experts than
    // threads) are read again when the table is filled.
    const uint32_t own = plan.own;
    auto entry_at = [&](uint32_t q) {
        int4 e = make_int4(-1, 0, 0, 0);
        if (tid * own + q < c.E) e = __ldcg(c.items + tid * own + q);                  // x = -1 past the list's end
        if (e.x < 0 || (c.item_rows_max && uint32_t(e.z) > c.item_rows_max)) e.z = 0;  // those rows go to the tensor-core family
        return e;
    };
    const uint32_t slots_total = c.T * c.K;
    const bool perm_cached = slots_total <= PERM_CACHE;
    int perm_mine[2] = {0, 0};
    if (perm_cached) {
#pragma unroll
        for (int q = 0; q < 2; ++q) if (tid + q * blockDim.x < slots_total) perm_mine[q] = __ldcg(c.perm + tid + q * blockDim.x);
    }
    const int4 entry0 = entry_at(0);
    uint32_t mine = (uint32_t(entry0.z) + NROW - 1) / NROW;
    for (uint32_t q = 1; q < own; ++q) mine += (uint32_t(entry_at(q).z) + NROW - 1) / NROW;
    if (perm_cached) {
#pragma unroll
        for (int q = 0; q < 2; ++q) if (tid + q * blockDim.x < slots_total) perm_s[tid + q * blockDim.x] = perm_mine[q];
        for (uint32_t i = tid + 2 * blockDim.x; i < slots_total; i += blockDim.x) perm_s[i] = __ldcg(c.perm + i);
    }
    uint32_t before = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, before, off);
        if (lane >= uint32_t(off)) before += v;
    }
    if (lane == 31) warp_sums[warp] = before;
    __syncthreads();
    uint32_t total_passes = shared_passes;
    before += shared_passes - mine;
    {
        const uint32_t v = lane < W ? warp_sums[lane] : 0;
        total_passes += __reduce_add_sync(0xffffffffu, v);
        before += __reduce_add_sync(0xffffffffu, lane < warp ? v : 0);
    }
    // Tiles of all passes end to end; this CTA takes [t_first, t_last), its group rt every RT-th of them.
    const uint32_t tiles = total_passes * UB, each = quick_div(tiles, gridDim.x, plan.inv_grid), extra = tiles - each * gridDim.x;
    const uint32_t t_first = blockIdx.x * each + min(blockIdx.x, extra), t_last = t_first + each + (blockIdx.x < extra ? 1u : 0u);
    if (t_first == t_last) { if (NMAT == 1) pdl_wait(); return; }

    const uint32_t pi = ((g & 1) << 2) | (g & 2) | (g >> 2);                          // tile row of MMA row g
    const uint32_t lane_off = BITS == 4 ? pi * 128 + ((((cq >> 1) ^ pi) << 4) | ((cq & 1) << 3)) : pi * 128 + ((cq ^ pi) << 4);
    const uint8_t* code_at[GPS];                     // the lane's codes of row g of the first fragment, per group of a stage
#pragma unroll
    for (int j = 0; j < GPS; ++j) code_at[j] = ring + warp * (STAGES * STAGE_BYTES) + (BITS == 4 ? (lane_off ^ uint32_t(j << 5)) : (lane_off ^ uint32_t(j << 6)));
    const bool q8s = c.q8_signed;
    bool waited = NMAT == 2;
    const uint32_t meta_at = NMAT == 2 ? uint32_t(c.gate.scales) : uint32_t(c.down.scales);
    const uint32_t meta_frag = NMAT == 2 ? uint32_t(c.up.scales - c.gate.scales) : 16 * G * 2;       // second fragment: the same rows of up, or the next 16 rows of down
    const uint32_t bias_at = N * G * 2 + cq * (BITS == 4 ? 4 : 2), lane_scale = pi * (G * 2), step_bytes = KS * (2 * GPS) * 2;
    const bool whole_pairs = G % (2 * GPS) == 0;
    const uint32_t stages = (G + GPS - 1) / GPS;     // of a row's K; odd: the last pair has one
    auto wait_bar = [&](uint32_t bar, uint32_t ph) {       // bounded; a second full wait lets a late copy land before its buffer is used again
        if (ring_wait(bar, ph, limit)) return;
        atomicOr(c.status, ZC_STATUS_TIMEOUT);
        ring_wait(bar, ph, limit);
        limit = 16;
    };

    const uint32_t p_first = quick_div(t_first, UB, plan.inv_tiles), p_last = quick_div(t_last - 1, UB, plan.inv_tiles);
    for (uint32_t pw = p_first; pw <= p_last; pw += TABLE) {
        const uint32_t np = min(p_last - pw + 1, uint32_t(TABLE));                    // passes of this window
        const uint32_t ta = max(t_first, pw * UB), tb = min(t_last, (pw + np) * UB);  // its tiles
        if (pw != p_first) __syncthreads();                                           // the previous window's entries have been read
        if (tid < np && pw + tid < shared_passes) {
            const uint32_t p0 = (pw + tid) * NROW;
            table[tid] = make_int4(-1, int(p0), int(min(uint32_t(NROW), c.T - p0)), int(c.T * c.K + p0));
        }
        {
            uint32_t first = before;
            for (uint32_t q = 0; q < own; ++q) {
                const int4 e = q == 0 ? entry0 : entry_at(q);
                const uint32_t n = (uint32_t(e.z) + NROW - 1) / NROW;
                for (uint32_t p = max(first, pw); p < min(first + n, pw + np); ++p) {
                    const uint32_t r0 = (p - first) * NROW, pos = uint32_t(e.y) + r0;
                    table[p - pw] = make_int4(e.x - int(c.first_expert), int(pos), int(min(uint32_t(NROW), uint32_t(e.z) - r0)), int(pos));
                }
                first += n;
            }
        }
        __syncthreads();

        // ---- the sequence of this warp: pairs of stages (2 GPS groups) of its tiles. While a pair is multiplied, each of its
        // two ring slots is refilled with the next pair's stage as soon as it has been read, and the stage's scales and the
        // pair's biases are fetched for the next pair into the registers they leave ----
        struct Cursor { uint32_t t, blk, ps; };      // tile of the window's sequence, its place in its pass, its pass in the table
        auto next_tile = [&](Cursor& k) { k.t += RT; k.blk += RT; while (k.blk >= UB) { k.blk -= UB; ++k.ps; } };
        Cursor now{ta, pw == p_first ? t_first - p_first * UB : 0, 0};
        now.t += rt; now.blk += rt;
        while (now.blk >= UB) { now.blk -= UB; ++now.ps; }
        Cursor ahead = now;                          // the tile of the next pair, and the pair
        uint32_t ahead_pair = ks;
        int ahead_e = 0;
        const CUtensorMap* ahead_map = &maps.routed;
        const uint8_t* mp[2][2];                     // the lane's scale pointers: [fragment][row g / g+8] of the next pair
        auto enter_tile = [&]() {                    // ahead.t < tb
            const int e = __shfl_sync(0xffffffffu, table[ahead.ps].x, 0);
            ahead_e = max(e, 0);
            ahead_map = e < 0 ? &maps.shared : &maps.routed;
            const uint8_t* rec = (e < 0 ? c.shared_record : c.records + size_t(e) * c.record_stride) + (meta_at + ahead.blk * TILE * (G * 2) + ks * (2 * GPS * 2)) + lane_scale;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int r = 0; r < 2; ++r) mp[m][r] = rec + (m * meta_frag + r * G * 16);
        };
        uint32_t sc[2][2][2][SW];                    // [stage of the pair][fragment][row g / g+8]: the scales of the stage's groups, two per word
        uint32_t bi[2][2];                           // the biases this lane supplies to the pair's bias product
        auto issue = [&](int half) {
            if (lane == 0 && ahead_pair * 2 + half < stages) ring_load(ring_base + half * STAGE_BYTES, ahead_map, bar_base + half * 8, int((ahead_pair * 2 + half) * 128), int(ahead.blk * TILE), ahead_e);
        };
        auto fetch_scales = [&](int half) {
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint8_t* p = mp[m][r] + half * (GPS * 2);
                    if (whole_pairs) {
                        if constexpr (GPS == 4) {
                            const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
                            sc[half][m][r][0] = v.x; sc[half][m][r][SW - 1] = v.y;
                        } else sc[half][m][r][0] = __ldg(reinterpret_cast<const uint32_t*>(p));
                    } else {                         // rows of an even number of groups: words are 4-byte aligned, those past the row are zero
#pragma unroll
                        for (int w = 0; w < SW; ++w)
                            sc[half][m][r][w] = (ahead_pair * 2 + half) * GPS + 2 * w < G ? __ldg(reinterpret_cast<const uint32_t*>(p) + w) : 0u;
                    }
                }
        };
        auto fetch_biases = [&]() {
            const bool on = whole_pairs || ahead_pair * (2 * GPS) + (BITS == 4 ? 2 * cq : cq) < G;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if constexpr (BITS == 4) bi[m][r] = on ? __ldg(reinterpret_cast<const uint32_t*>(mp[m][r] + bias_at)) : 0u;
                    else bi[m][r] = on ? uint32_t(__ldg(reinterpret_cast<const uint16_t*>(mp[m][r] + bias_at))) : 0u;
                }
        };
        auto step = [&]() {                          // `ahead` to the pair after it
            ahead_pair += KS;
            if (ahead_pair < pairs) {
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int r = 0; r < 2; ++r) mp[m][r] += step_bytes;
                return;
            }
            ahead_pair = ks;
            next_tile(ahead);
            if (ahead.t < tb) enter_tile();
        };
        // rows of this window's passes
        for (uint32_t i = tid; i < np * NROW; i += blockDim.x) {
            const int4 d = table[i / NROW];
            const uint32_t n = i % NROW;
            int v = -1;
            if (int(n) < d.z) {
                if (d.x < 0) v = d.y + int(n);
                else {
                    v = perm_cached ? perm_s[d.y + n] : __ldcg(c.perm + d.y + n);
                    if (NMAT == 2) v = int(uint32_t(v) / c.K);
                }
            }
            slots[i / NROW][n] = v;
        }
        __syncthreads();

        // This warp's share of the rows of pass q (counted from p_first), once the pass that used the buffer before is done.
        auto stage_share = [&](uint32_t ps) {
            const uint32_t q = pw + ps - p_first, buf = q & (NBUF - 1), use = NBUF == 2 ? q >> 1 : q;
            if (use) wait_bar(done_base + buf * 8, (use - 1) & 1);
            const int4 d = table[ps];
            __half* hi = hi_of(buf);
            float* sx = sx_of(buf);
            stage_rows<BITS == 4, SPLIT, FOLDQ>(NMAT == 2 ? c.x : static_cast<const void*>(c.hbuf), NMAT == 2 ? c.act_dtype == ZC_F32 : true,
                [&](uint32_t n) { return NMAT == 2 ? size_t(slots[ps][n]) : size_t(d.w) + n; },
                uint32_t(d.z), K, RS, GP, c.ref && BITS == 4, hi, hi + NROW * RS, sx, sx + NROW * GP, c.status, warp, W);
            __syncwarp();
            if (lane == 0) bar_arrive(full_base + buf * 8);
        };
        // down's first window: its weights depend on nothing that gate/up writes, so the ring, the scales and the biases of the
        // first tile are under way while gate/up drains (64 tokens 173.3 -> 171.9 us a layer, 16 tokens 81.9 -> 80.6).
        // Otherwise the rows of the first pass are requested before the first weights, which would stand in front of
        // them in the memory system (128 KB per SM at once); those of the second pass (two blocks) behind them.
        const bool any = ahead.t < tb, early = !waited;
        auto first_weights = [&]() { issue(1); fetch_scales(0); fetch_scales(1); fetch_biases(); step(); };
        if (any) { enter_tile(); issue(0); }
        if (early) {
            if (any) first_weights();
            pdl_wait(); pdl_launch_dependents();
            waited = true;
        }
#pragma unroll 1
        for (uint32_t ps = 0; ps < min(np, NBUF); ++ps) stage_share(ps);
        if (any && !early) first_weights();
        for (uint32_t ps = 0; ps < np; ++ps) {
            const uint32_t q = pw + ps - p_first, buf = q & (NBUF - 1), use = NBUF == 2 ? q >> 1 : q;
            bool next_staged = ps + 1 == np || (NBUF == 2 && ps == 0);   // the window's second pass already is
            wait_bar(full_base + buf * 8, use & 1);
            const uint32_t nvalid = uint32_t(__shfl_sync(0xffffffffu, table[ps].z, 0));
            const __half* xhi = hi_of(buf);
            const __half* xlo = xhi + NROW * RS;
            const float* sx = sx_of(buf);
            const float* offs = sx + NROW * GP;
            const uint32_t row_at = g < nvalid ? g : 0;                  // the lane's token row in the staged block; lanes without one read row 0 (their MMA columns are never stored)
            bool more = now.ps == ps && now.t < tb, left = false;
            do {
                if (more) {
                    float acc[2][4] = {};
                    for (uint32_t pair = ks; pair < pairs; pair += KS) {
                        const float4* op = reinterpret_cast<const float4*>(offs) + pair * (2 * GPS) * (NROW / 2) + cq;
                        const __half* xb = xhi + row_at * RS + pair * (2 * GPS * 64) + cq * 16;
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            if (half == 1) {         // the bias product of the pair's groups
                                const float* sp = sx + row_at * GP + pair * (2 * GPS);
                                float add[2][4] = {};
                                if constexpr (BITS == 4) {           // k slots cq and cq + 4 of the MMA are groups 2 cq and 2 cq + 1
                                    const float2 v = *reinterpret_cast<const float2*>(sp + 2 * cq);
                                    float h0, m0, l0, h1, m1, l1;
                                    tf32_terms(v.x, h0, m0, l0);
                                    tf32_terms(v.y, h1, m1, l1);
#pragma unroll
                                    for (int m = 0; m < 2; ++m) {
                                        const float2 b0 = meta_pair<META_F16>(bi[m][0]), b1 = meta_pair<META_F16>(bi[m][1]);
                                        mma_tf32_1688(add[m], b0.x, b1.x, b0.y, b1.y, l0, l1);
                                        mma_tf32_1688(add[m], b0.x, b1.x, b0.y, b1.y, m0, m1);
                                        mma_tf32_1688(add[m], b0.x, b1.x, b0.y, b1.y, h0, h1);
                                    }
                                } else {                             // k slot cq is group cq
                                    float h0, m0, l0;
                                    tf32_terms(sp[cq], h0, m0, l0);
#pragma unroll
                                    for (int m = 0; m < 2; ++m) {
                                        const float b0 = meta_pair<META_F16>(bi[m][0]).x, b1 = meta_pair<META_F16>(bi[m][1]).x;
                                        mma_tf32_1684(add[m], b0, b1, l0);
                                        mma_tf32_1684(add[m], b0, b1, m0);
                                        mma_tf32_1684(add[m], b0, b1, h0);
                                    }
                                }
#pragma unroll
                                for (int m = 0; m < 2; ++m)
#pragma unroll
                                    for (int i = 0; i < 4; ++i) acc[m][i] += add[m][i];
                            }
                            if (half == 0 || pair * 2 + 1 < stages) {
                                wait_bar(bar_base + half * 8, half ? parity1 : parity0);
                                if (half) parity1 ^= 1; else parity0 ^= 1;
#pragma unroll
                                for (int j = 0; j < GPS; ++j) {
                                    const __half* x = xb + (half * GPS + j) * 64;
                                    const uint4 bh[2] = {*reinterpret_cast<const uint4*>(x), *reinterpret_cast<const uint4*>(x + 8)};
                                    uint4 bl[2] = {};
                                    if constexpr (SPLIT) {
                                        bl[0] = *reinterpret_cast<const uint4*>(x + NROW * RS);
                                        bl[1] = *reinterpret_cast<const uint4*>(x + NROW * RS + 8);
                                    }
                                    const float4 off = FOLDQ ? op[(half * GPS + j) * (NROW / 2)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                    uint32_t w[2][2][WORDS];
#pragma unroll
                                    for (int m = 0; m < 2; ++m)
#pragma unroll
                                        for (int r = 0; r < 2; ++r) {
                                            const uint8_t* at = code_at[j] + half * STAGE_BYTES + m * 2048 + r * 1024;
                                            if constexpr (BITS == 4) {
                                                const uint2 v = *reinterpret_cast<const uint2*>(at);
                                                w[m][r][0] = v.x; w[m][r][1] = v.y;
                                            } else {
                                                const uint4 v = *reinterpret_cast<const uint4*>(at);
                                                w[m][r][0] = v.x; w[m][r][1] = v.y; w[m][r][WORDS - 2] = v.z; w[m][r][WORDS - 1] = v.w;
                                            }
                                        }
                                    float d[2][4];
                                    group_mma<BITS, SPLIT, FOLDQ>(d, off, w, bh, bl, q8s);
#pragma unroll
                                    for (int m = 0; m < 2; ++m) {
                                        const float2 p0 = meta_pair<META_F16>(sc[half][m][0][j / 2]), p1 = meta_pair<META_F16>(sc[half][m][1][j / 2]);
                                        const float s0 = j % 2 ? p0.y : p0.x, s1 = j % 2 ? p1.y : p1.x;
                                        acc[m][0] = __fmaf_rn(s0, d[m][0], acc[m][0]); acc[m][1] = __fmaf_rn(s0, d[m][1], acc[m][1]);
                                        acc[m][2] = __fmaf_rn(s1, d[m][2], acc[m][2]); acc[m][3] = __fmaf_rn(s1, d[m][3], acc[m][3]);
                                    }
                                }
                            }
                            __syncwarp();            // every lane has read the stage: refill it
                            if (ahead.t < tb) {
                                issue(half);
                                fetch_scales(half);
                                if (half == 1) { fetch_biases(); step(); }
                            }
                        }
                    }
                    // ---- the KS partial sums of the tile, added in warp order by one of its warps ----
                    bool finisher = true;
                    if (KS > 1) {
                        const uint32_t threads = KS * 32;
                        finisher = ks == fin;
                        // Barrier 1 + 2 rt: the partials are written. Barrier 2 + 2 rt: those of the tile before have been read. All
                        // KS warps pass the second one before any of them arrives at the first again.
                        if (done_tiles) group_sync(2 + 2 * rt, threads);
                        float4* area = reinterpret_cast<float4*>(red) + size_t(rt) * (KS - 1) * 2 * 32 + lane;
                        if (!finisher) {
                            float4* to = area + size_t(ks < fin ? ks : ks - 1) * 2 * 32;
#pragma unroll
                            for (int m = 0; m < 2; ++m) to[m * 32] = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
                            group_arrive(1 + 2 * rt, threads);
                        } else {
                            group_sync(1 + 2 * rt, threads);
                            float sum[2][4] = {};
                            for (uint32_t k = 0; k < KS; ++k) {
                                const float4* from = area + size_t(k < fin ? k : k - 1) * 2 * 32;
#pragma unroll
                                for (int m = 0; m < 2; ++m) {
                                    const float4 v = k == fin ? make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]) : from[m * 32];
                                    sum[m][0] += v.x; sum[m][1] += v.y; sum[m][2] += v.z; sum[m][3] += v.w;
                                }
                            }
#pragma unroll
                            for (int m = 0; m < 2; ++m)
#pragma unroll
                                for (int i = 0; i < 4; ++i) acc[m][i] = sum[m][i];
                        }
                        fin = fin + 1 == KS ? 0 : fin + 1;
                        ++done_tiles;
                    }
                    if (finisher) {                  // lane: rows pi, pi + 8 of the tile, tokens 2 cq, 2 cq + 1
                        const uint32_t row0 = now.blk * TILE + pi;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t n = 2 * cq + i;
                            if (n >= nvalid) continue;
                            float a[2][2];
#pragma unroll
                            for (int m = 0; m < 2; ++m)
#pragma unroll
                                for (int r = 0; r < 2; ++r) a[m][r] = FOLDQ ? acc[m][2 * r + i] * 0.0625f : acc[m][2 * r + i];       // the rows were staged x 16
                            if constexpr (NMAT == 2) {
                                float* to = c.hbuf + size_t(uint32_t(table[ps].w) + n) * c.F + row0;
#pragma unroll
                                for (int r = 0; r < 2; ++r) {
                                    float h;
                                    if (c.ref) {   // qwen.metal:71-81
                                        const float gate = bf_round(a[0][r]), up = bf_round(a[1][r]);
                                        h = bf_round(bf_round(gate * sigmoid_bf(gate)) * up);
                                    } else {
                                        h = (a[0][r] * sigmoid_f(a[0][r])) * a[1][r];
                                    }
                                    to[8 * r] = h;
                                }
                            } else {
                                float* to = (table[ps].x < 0 ? c.shared_out : c.expert_out) + size_t(uint32_t(slots[ps][n])) * c.H + row0;
#pragma unroll
                                for (int m = 0; m < 2; ++m)
#pragma unroll
                                    for (int r = 0; r < 2; ++r) to[16 * m + 8 * r] = c.ref ? bf_round(a[m][r]) : a[m][r];
                            }
                        }
                    }
                    next_tile(now);
                    more = now.ps == ps && now.t < tb;
                }
                // The next pass's rows: after this warp's first tile of the pass (by then the others have left the pass before
                // it, whose block they go to), with one block only when every warp is done with this pass.
                if (!more && NBUF == 1) { left = true; __syncwarp(); if (lane == 0) bar_arrive(done_base + buf * 8); }
                if (!next_staged && (NBUF == 2 || !more)) { next_staged = true; stage_share(ps + 1); }
            } while (more);
            if (!left) { __syncwarp(); if (lane == 0) bar_arrive(done_base + buf * 8); }
        }
    }
}

// Shared memory of a launch.
size_t stream_smem(const StreamPlan& p, bool split, uint32_t K, uint32_t bits) {
    const uint32_t gpad = p.pairs * (bits == 4 ? 8 : 4);
    return 1024 + size_t(p.warps) * STAGES * STAGE_BYTES + size_t(p.warps / p.ks) * (p.ks - 1) * 2 * 32 * 16 +
           p.nbuf * (size_t(split ? 2 : 1) * NROW * (gpad * 64 + ROW_PAD) * 2 + size_t(NROW) * (gpad + 8) * 4 + size_t(gpad) * NROW * 8);
}
constexpr size_t STREAM_SMEM_MAX = 221 * 1024;      // 227 KB less the static tables

template <int BITS, bool SPLIT, bool FOLD, bool META_F16, int NMAT>
int launch_stream(zc_moe* m, const Call& c, const StreamPlan& p, cudaStream_t s) {
    const size_t smem = stream_smem(p, SPLIT, NMAT == 2 ? c.H : c.F, BITS);
    auto kernel = stream_kernel<BITS, SPLIT, FOLD, META_F16, NMAT>;
    static SmemOptIn configured;        // one per instantiation of this function template
    if (opt_in_smem(kernel, configured, m->device, smem) != cudaSuccess) return check_launch(m, "expert kernel attribute");
    const LayerMem& L = m->layers[c.layer];
    const StreamMaps maps{NMAT == 2 ? L.map_gate_up.m : L.map_down.m, NMAT == 2 ? L.map_shared_gate_up.m : L.map_shared_down.m};
    Timed t(m, s, NMAT == 2 ? KERNEL_GATE_UP : KERNEL_DOWN);
    const cudaError_t e = launch_chained(m, NMAT == 2 ? KERNEL_GATE_UP : KERNEL_DOWN, kernel, dim3(sm_count(m)), dim3(p.warps * 32), smem, s, nullptr, 0, c, maps, p);
    if (e != cudaSuccess) return fail(m, ZC_EEXEC, std::string("expert kernel launch: ") + cudaGetErrorString(e));
    return check_launch(m, NMAT == 2 ? "gate_up" : "down");
}

template <int BITS, bool FOLD, bool META_F16, int NMAT>
int dispatch_split(zc_moe* m, const Call& c, const StreamPlan& p, bool split, cudaStream_t s) {
    return split ? launch_stream<BITS, true, FOLD, META_F16, NMAT>(m, c, p, s) : launch_stream<BITS, false, FOLD, META_F16, NMAT>(m, c, p, s);
}
template <int NMAT>
int dispatch_expert(zc_moe* m, const Call& c, const StreamPlan& p, bool split, uint32_t bits, bool fold, cudaStream_t s) {
    if (bits == 8) return c.meta_f16 ? dispatch_split<8, false, true, NMAT>(m, c, p, split, s) : dispatch_split<8, false, false, NMAT>(m, c, p, split, s);
    if (fold) return c.meta_f16 ? dispatch_split<4, true, true, NMAT>(m, c, p, split, s) : dispatch_split<4, true, false, NMAT>(m, c, p, split, s);
    return c.meta_f16 ? dispatch_split<4, false, true, NMAT>(m, c, p, split, s) : dispatch_split<4, false, false, NMAT>(m, c, p, split, s);
}

}  // namespace

// TMA views of a layer's records (codes of gate and up together: the two projections have one geometry and lie one
// projection apart; codes of down), encoded once when the handle is created. Where they cannot be had - a driver without the
// encoder, or a geometry that it refuses - the handle stays with the item kernels.
void make_stream_maps(zc_moe* m, LayerMem& L) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
        if (e != cudaSuccess) cudaGetLastError();
        return reinterpret_cast<Encode>(e == cudaSuccess && q == cudaDriverEntryPointSuccess ? p : nullptr);
    }();
    if (!encode) { m->stream_maps = false; return; }
    auto make = [&](StreamMap& to, uint8_t* record, const Projection& pr, uint64_t pair_stride, uint32_t experts, uint64_t stride) {
        const uint64_t row = uint64_t(pr.K) * pr.bits / 8;
        const cuuint64_t dims[4] = {row, pr.N, pair_stride ? 2u : 1u, experts};
        const cuuint64_t strides[3] = {row, pair_stride ? pair_stride : row * pr.N, stride};
        const cuuint32_t box[4] = {128, pair_stride ? 16u : 32u, pair_stride ? 2u : 1u, 1}, elem[4] = {1, 1, 1, 1};
        return encode(&to.m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, record + pr.codes, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const zc_moe_desc& d = m->d;
    const Projection gate = projection_of(d, 0), up = projection_of(d, 1), down = projection_of(d, 2);
    bool ok = make(L.map_gate_up, L.records, gate, up.codes - gate.codes, d.local_experts, d.record_stride) &&
              make(L.map_down, L.records, down, 0, d.local_experts, d.record_stride);
    L.map_shared_gate_up = L.map_gate_up;
    L.map_shared_down = L.map_down;
    if (ok && d.has_shared) {
        const zc_moe_desc sd = shared_desc_of(d);
        const Projection sg = projection_of(sd, 0), su = projection_of(sd, 1), sdn = projection_of(sd, 2);
        const uint64_t stride = (record_bytes_of(sd) + 16383) / 16384 * 16384;
        ok = make(L.map_shared_gate_up, L.shared_record, sg, su.codes - sg.codes, 1, stride) && make(L.map_shared_down, L.shared_record, sdn, 0, 1, stride);
    }
    m->stream_maps = m->stream_maps && ok;
}

static int launch_experts_decode_one(zc_moe* m, const Call& c, cudaStream_t s);

// A shared expert whose record has other bit widths than the routed experts' (the reference's mixed artifact: routed Q4,
// shared Q8) cannot share a launch with them - the code width is a template parameter - so it runs as launches of its
// own over the same buffers (its rows of hbuf and shared_out are disjoint from the routed ones).
int launch_experts_decode(zc_moe* m, const Call& c, cudaStream_t s) {
    if (!(c.has_shared && c.shared_split)) return launch_experts_decode_one(m, c, s);
    int total = 0, n;
    if (c.items != m->empty_items) {
        Call routed = c;
        routed.has_shared = 0;
        if ((n = launch_experts_decode_one(m, routed, s)) < 0) return n;
        total += n;
    }
    Call shared = c;
    shared.gate = c.sgate; shared.up = c.sup; shared.down = c.sdown; shared.shared_split = 0;
    shared.items = m->empty_items; shared.counters = m->zero_counters;
    if ((n = launch_experts_decode_one(m, shared, s)) < 0) return n;
    return total + n;
}

static bool stream_plan(const ExpertLoad& l, uint32_t sms, int nmat, StreamPlan& p) {
    const uint32_t K = nmat == 2 ? l.hidden : l.ffn, bits = nmat == 2 ? l.gate_bits : l.down_bits;
    const bool split = nmat == 2 ? l.split_x : l.split_h;
    p.pairs = (K / 64 + (bits == 4 ? 7 : 3)) / (bits == 4 ? 8 : 4);
    auto fits = [&]() { return stream_smem(p, split, K, bits) <= STREAM_SMEM_MAX; };
    p.warps = MAX_WARPS; p.ks = 1; p.nbuf = 2;
    if (!fits()) p.nbuf = 1;
    // Four warps share a gate/up tile for the shortest batches (one tile per warp would leave most of the SMs without work) and
    // where only one row block fits (hidden above 2560): there the warps of a CTA meet at every pass, and with a quarter of
    // the tiles in flight they arrive closer together (256 tokens at hidden 4096: 492 us against 511 for the layer).
    if (nmat == 2 && p.pairs >= 4 && (p.nbuf == 1 || l.few)) p.ks = 4;
    if (!fits()) p.ks = 1;
    while (!fits() && p.warps > 4) p.warps /= 2;
    p.rt = p.warps / p.ks; p.ks_shift = p.ks == 4 ? 2 : 0;
    p.tiles_per_pass = nmat == 2 ? l.ffn / 16 : l.hidden / 32;
    p.own = (l.list + p.warps * 32 - 1) / (p.warps * 32);
    p.inv_tiles = 1.0f / float(p.tiles_per_pass); p.inv_grid = 1.0f / float(sms);
    return fits();
}

// Expected number of eight-row passes of `rows` rows that fall evenly on `experts` experts: experts x E[ceil(X / 8)], X Poisson.
static double expected_passes(double rows, double experts) {
    if (rows <= 0.0 || experts <= 0.0) return 0.0;
    const double mean = rows / experts;
    if (mean > 64.0) return rows / 8.0 + 0.5 * experts;
    double p = std::exp(-mean), sum = 0.0;
    for (int x = 1; x < 160; ++x) { p *= mean / x; sum += p * ((x + 7) / 8); }
    return experts * sum;
}

// Batches that stay with the item kernels (csrc/experts_item.cu), whose many small CTAs start faster. The figures are item / streaming,
// us a layer, for loads that fall evenly; `rounds` is how often a launch's gate/up tiles fill the streaming kernel's warps.
//  - Up to 64 rows and tokens the item kernels split K over eight warps and win while there is little to stream: 0.36 rounds (2 tokens
//    of 512 experts 35.5 / 37.0, hidden 2560 44.2 / 47.5; 3 tokens of 256 experts 35.2 / 35.1, hidden 2560 43.7 / 44.0), 0.17 rounds with
//    two-term rows (2 tokens, FP32 activations: streaming 8 - 10 % faster) and above hidden 2560 (hidden 3072: 1 token 36.3 / 38.8, 2 tokens
//    51.4 / 45.4; hidden 4096: 1 token 44.3 / 45.5 launched one by one though 44.2 / 44.0 from a graph, 2 tokens 62.5 / 52.5; the shared expert
//    alone 12.0 / 18.5).
//  - Beyond, where a round of the streaming kernel is nearly empty and few experts need a second pass: 1.7 to 1.97 rounds (14 / 15 / 16 /
//    17 tokens 77.7 / 77.0, 78.2 / 78.6, 78.6 / 80.7, 91.5 / 88.9; 14 tokens at ffn 768 of 256 experts 73.3 / 78.8). With a down
//    projection whose K is not whole stages (ffn 640: ten groups cost twelve) the streaming kernel loses more often: 0.8 to 2.5
//    rounds, except from 0.47 to 0.82 of a round (512 experts of 2560 / 640: 8 tokens 76.4 / 83.0, 10 tokens 93 / 93, 14 tokens 107.7 /
//    112.4, 18 tokens 130.2 / 128.8; 64 experts: 24 tokens 70.0 / 72.3, 48 tokens 84.0 / 80.8). Skewed loads (Zipf 1.1) would be better
//    off streaming there: 16 tokens 72.8 / 54.8, at 2560 / 640 72.2 / 69.8. Above 2.5 rounds even loads gain 1 to 2 % on the item
//    kernels (22 tokens 145.9 / 149.0) and skewed ones lose 10 (89.4 / 80.9): those batches stream.
//  - Experts with more rows take further passes, and the codes are dequantised for each: there the streaming kernel
//    wins (128 experts: 64 tokens 83.8 / 80.6, 128 tokens 119.5 / 109.9; 512 experts with skewed loads, 64 tokens 302 / 87).
bool item_kernels_pay(const ExpertLoad& l, uint32_t sms) {
    const double passes = expected_passes(l.rows, l.experts) + (l.shared_tokens + NROW - 1) / NROW;
    const double rounds = passes * (l.ffn / 16) / (double(sms) * MAX_WARPS);
    if (l.row_limit) return false;
    if (l.item_split) return rounds <= (l.hidden > 2560 || l.split_x ? 0.17 : 0.36);
    if (l.hidden > 2560 || !l.rows) return false;
    const double mean = double(l.rows) / l.experts;
    auto ragged = [](uint32_t K, uint32_t bits) { return (K / 64) % (bits == 4 ? 4 : 2) != 0; };
    if (!ragged(l.hidden, l.gate_bits) && !ragged(l.ffn, l.down_bits)) return mean <= 1.0 && rounds > 1.7 && rounds < 1.97;
    const double part = rounds - std::floor(rounds);
    return mean <= (rounds < 1.2 ? 4.0 : 1.5) && rounds > 0.8 && rounds < 2.5 && !(part > 0.47 && part < 0.82);
}
bool streaming_kernels_fit(const ExpertLoad& l) {
    StreamPlan p{};
    return stream_plan(l, 148, 2, p) && stream_plan(l, 148, 1, p);
}

static int launch_experts_decode_one(zc_moe* m, const Call& c, cudaStream_t s) {
    // A BF16 activation is exact as one FP16 term; an FP32 activation needs two, except under the
    // reference arithmetic, whose FP32 buffers hold BF16 values by contract.
    const bool split_x = c.act_dtype == ZC_F32 && !c.ref;
    // The SwiGLU rows h are FP32 in memory. By default the down product reads them as one FP16 term (11 significant
    // bits, against the 8 of the BF16 the reference rounds h to; measured 1.2e-3 x RMS max-abs at 64 tokens, inside the
    // 2e-3 bound); with the "exact_h" option as two FP16 terms, which costs a second MMA per fragment.
    // The reference arithmetic's h is BF16: exact in one term.
    const bool split_h = !c.ref && m->exact_h;
    ExpertLoad l{};
    l.rows = c.items == m->empty_items ? 0 : c.rows_expected ? c.rows_expected : c.T * c.K;
    l.shared_tokens = c.has_shared ? c.T : 0;
    l.experts = c.local_experts; l.list = c.E; l.hidden = c.H; l.ffn = c.F; l.gate_bits = c.gate.bits; l.down_bits = c.down.bits;
    l.split_x = split_x; l.split_h = split_h; l.row_limit = c.item_rows_max != 0;
    l.item_split = c.T * (c.K + (c.has_shared ? 1 : 0)) <= 64;
    // The shared expert alone is cut as in its layer's launch, so that its rows are the same bits on every path.
    l.few = c.rows_expected ? c.rows_expected <= 64 : l.item_split;
    StreamPlan gate_up{}, down{};
    const bool fits = m->stream_maps && stream_plan(l, sm_count(m), 2, gate_up) && stream_plan(l, sm_count(m), 1, down);
    if (m->expert_kernels == 2 && !fits) return fail(m, ZC_EINVAL, "expert_kernels = 2: the streaming kernels do not take this shape");
    if (m->expert_kernels == 1 || !fits || (m->expert_kernels == 0 && item_kernels_pay(l, sm_count(m)))) return launch_experts_item(m, c, s);
    int rc;
    if ((rc = dispatch_expert<2>(m, c, gate_up, split_x, c.gate.bits, m->fold_q4, s)) < 0) return rc;
    if ((rc = dispatch_expert<1>(m, c, down, split_h, c.down.bits, m->fold_q4, s)) < 0) return rc;
    return 2;
}

}  // namespace zc
