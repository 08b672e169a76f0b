// Router logits (and the shared-expert gate scalar) in fp32 with a pinned accumulation order.
//
// Replaces router_mm + router_accumulate (kernels/metal/qwen.metal:512-534, launched from
// src/engine/metal.mm:818-822) and keeps their arithmetic: K is cut into sixteen contiguous partitions,
// each partition is a k-ascending chain of fused multiply-adds that one thread owns, and the sixteen
// partials are added in order 0..15, starting from zero. The order is part of the contract
// because one last-bit change in a logit can flip a top-k decision; it reproduces the MLX bit patterns
// the reference's own test holds (tests/test_qwen.cpp:798-826).
//
// Layer calls use router_cluster_kernel up to 128 tokens and router_tile_kernel beyond (router_cut): their partials stay in
// shared memory. router_partial_kernel serves the entry point that may not allocate: grid (row tiles of 32, 16 partitions, token
// tiles); a CTA stages its slice of x (k-major) and of the router rows (k-major) in shared memory, every thread runs its chains,
// the partials go to memory as [16, T, rows], and the last of the sixteen CTAs of a tile to finish adds them.
#include "common.cuh"
#include <cooperative_groups.h>

namespace zc {
namespace {

constexpr int ROUTER_THREADS = 256;

// TT tokens x 32 rows per CTA: TT = 8 -> one output per thread, TT = 16 -> two.
template <int TT>
__global__ void __launch_bounds__(ROUTER_THREADS) router_partial_kernel(Call c, float* __restrict__ partial, uint32_t rows_padded,
                                                                         uint32_t* __restrict__ tile_done, uint32_t reduce) {
    constexpr int ROW_TILE = 32;
    extern __shared__ __align__(16) float smem[];
    const uint32_t H = c.H, part = H / 16;
    float* xs = smem;                    // [part][TT]
    float* ws = smem + part * TT;        // [part][ROW_TILE]
    const uint32_t e0 = blockIdx.x * ROW_TILE, p = blockIdx.y, t0 = blockIdx.z * TT;
    const uint32_t rows_total = c.E + (c.has_shared ? 1u : 0u);
    const uint32_t tid = threadIdx.x;
    const uint32_t k0 = p * part;
    pdl_wait();

    // x slice -> xs[k][t]
    for (uint32_t task = tid; task < TT * (part / 8); task += ROUTER_THREADS) {
        const uint32_t tt = task % TT, kb = task / TT, t = t0 + tt;
        float v[8];
        if (t < c.T) {
            if (c.act_dtype == ZC_F32) {
                const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(c.x) + size_t(t) * H + k0 + kb * 8);
                const float4 a = __ldg(src), b = __ldg(src + 1);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            } else {
                const uint4 raw = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(c.x) + size_t(t) * H + k0 + kb * 8));
                const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(r[i] << 16); v[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u); }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) xs[(kb * 8 + i) * TT + tt] = v[i];
    }
    // router rows -> ws[k][e]; four loads are issued before their stores so that a thread pays the memory
    // latency once per batch, not once per 16 bytes
    const uint32_t wtasks = ROW_TILE * (part / 4);
    for (uint32_t first = tid; first < wtasks; first += 4 * ROUTER_THREADS) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t task = first + u * ROUTER_THREADS;
            v[u] = make_float4(0, 0, 0, 0);
            if (task < wtasks) {
                const uint32_t el = task % ROW_TILE, kq = task / ROW_TILE, e = e0 + el;
                if (e < rows_total) {
                    const void* base = e < c.E ? c.router_w : c.shared_gate_w;
                    const size_t row = e < c.E ? e : 0;
                    if (c.router_dtype == ZC_F32) {
                        v[u] = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + row * H + k0 + kq * 4));
                    } else {
                        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + row * H + k0 + kq * 4));
                        v[u] = make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                                           __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t task = first + u * ROUTER_THREADS;
            if (task < wtasks) {
                const uint32_t el = task % ROW_TILE, kq = task / ROW_TILE;
                ws[(kq * 4 + 0) * ROW_TILE + el] = v[u].x;
                ws[(kq * 4 + 1) * ROW_TILE + el] = v[u].y;
                ws[(kq * 4 + 2) * ROW_TILE + el] = v[u].z;
                ws[(kq * 4 + 3) * ROW_TILE + el] = v[u].w;
            }
        }
    }
    __syncthreads();

    if constexpr (TT == 16) {
        const uint32_t tx = tid % 16, ty = tid / 16;        // rows 2tx, 2tx+1; token ty
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 8
        for (uint32_t k = 0; k < part; ++k) {
            const float xv = xs[k * TT + ty];
            const float2 wv = *reinterpret_cast<const float2*>(ws + k * ROW_TILE + tx * 2);
            a0 = __fmaf_rn(xv, wv.x, a0);
            a1 = __fmaf_rn(xv, wv.y, a1);
        }
        const uint32_t t = t0 + ty;
        if (t < c.T) *reinterpret_cast<float2*>(partial + (size_t(p) * c.T + t) * rows_padded + e0 + tx * 2) = make_float2(a0, a1);
    } else {
        const uint32_t el = tid % ROW_TILE, tt = tid / ROW_TILE;   // TT == 8
        float acc = 0.0f;
#pragma unroll 8
        for (uint32_t k = 0; k < part; ++k) acc = __fmaf_rn(xs[k * TT + tt], ws[k * ROW_TILE + el], acc);
        const uint32_t t = t0 + tt;
        if (t < c.T) partial[(size_t(p) * c.T + t) * rows_padded + e0 + el] = acc;
    }
    if (!reduce) return;
    // The last of the sixteen partition CTAs of this (row tile, token tile) adds the partials in order
    // 0..15, starting from zero like router_accumulate (qwen.metal:529-534).
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    uint32_t* counter = tile_done + blockIdx.z * gridDim.x + blockIdx.x;
    if (tid == 0) last = atomicAdd(counter, 1u) == 15u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (tid == 0) *counter = 0;
    constexpr int PER = TT * ROW_TILE / ROUTER_THREADS;      // outputs per thread: 1, 2 or 8
    constexpr int BATCH = PER < 4 ? PER : 4;                 // outputs whose 16 loads are in flight together
#pragma unroll 1
    for (int b = 0; b < PER; b += BATCH) {
        float v[BATCH][16];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const uint32_t o = tid + (b + i) * ROUTER_THREADS, tt = o / ROW_TILE, el = o % ROW_TILE, t = t0 + tt, e = e0 + el;
            const bool live = t < c.T && e < rows_total;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) v[i][q] = live ? __ldcg(partial + (size_t(q) * c.T + t) * rows_padded + e) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const uint32_t o = tid + (b + i) * ROUTER_THREADS, tt = o / ROW_TILE, el = o % ROW_TILE, t = t0 + tt, e = e0 + el;
            if (t >= c.T || e >= rows_total) continue;
            float sum = 0.0f;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) sum = __fadd_rn(sum, v[i][q]);
            if (e < c.E) c.logits[size_t(t) * c.E + e] = c.router_bias ? __fadd_rn(sum, c.router_bias[e]) : sum;
            else c.gate_logit[t] = sum;
        }
    }
}


// ---------------------------------------------------------------------------------------------------------
// Cluster form of the same computation, used whenever the device can host its clusters. A thread-block
// cluster of eight CTAs covers the sixteen partitions of one (row tile, token tile): CTA r computes
// partitions 2r and 2r+1. The partials never leave the chip: each CTA leaves its two [TT][rows] partial tiles in
// its shared memory, and after one cluster barrier every CTA adds, in order 0..15 from zero, the sixteen
// partials of its eighth of the outputs, read from its peers' shared memory. Compared with the global-memory
// form this removes the partial store, the fence, the arrival counter and the tail that one CTA ran alone.
//
// Staging: x and the router rows keep their row-major [row][k] layout in shared memory (leading dimension
// KC + 4 floats, which spreads eight consecutive rows over all banks for 16-byte reads), so fp32 rows are
// copied with 16-byte cp.async and everything is in flight at once: one memory round trip before the chains.
// Thread (tx = lane, ty = warp) owns rows tx (and tx + 32) x tokens ty*TPT.. x both partitions: up to 32
// independent chains, each still the k-ascending fused multiply-add chain of its partition.
namespace cg = cooperative_groups;
#ifndef ZC_ROUTER_SMALL_T
#define ZC_ROUTER_SMALL_T 128
#endif
constexpr int CLUSTER_PARTS = 2;                      // partitions per CTA
constexpr int CLUSTER_SIZE = 16 / CLUSTER_PARTS;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

template <int TT, int RPT>
__global__ void __launch_bounds__(ROUTER_THREADS) router_cluster_kernel(Call c) {
    constexpr int ROW_TILE = 32 * RPT, TPT = TT / 8;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float smem[];
    const uint32_t H = c.H, part = H / 16, KC = CLUSTER_PARTS * part, LD = KC + 4;
    float* ws = smem;                         // [ROW_TILE][LD]
    float* xs = ws + ROW_TILE * LD;           // [TT][LD]
    float* ps = xs + TT * LD;                 // [2][TT][ROW_TILE]
    const uint32_t e0 = blockIdx.x * ROW_TILE, cr = blockIdx.y, t0 = blockIdx.z * TT;
    const uint32_t rows_total = c.E + (c.has_shared ? 1u : 0u);
    const uint32_t tid = threadIdx.x, k0 = cr * KC;

    // ---- stage: the rows first (weights), then x (registers when it needs a conversion) ----
    constexpr int XB = 4;                     // x tasks (8 values each) a thread keeps in flight
    const uint32_t xtasks = TT * (KC / 8);
    const bool x32 = c.act_dtype == ZC_F32, w32 = c.router_dtype == ZC_F32;
    auto stage_rows = [&]() {
        const uint32_t wtasks = ROW_TILE * (KC / 4);
        if (w32) {
            for (uint32_t task = tid; task < wtasks; task += ROUTER_THREADS) {
                const uint32_t el = task / (KC / 4), kq = task % (KC / 4), e = e0 + el;
                float* dst = ws + el * LD + kq * 4;
                if (e < rows_total) {
                    const float* base = e < c.E ? static_cast<const float*>(c.router_w) + size_t(e) * H : static_cast<const float*>(c.shared_gate_w);
                    cp_async16(dst, base + k0 + kq * 4);
                } else {
                    *reinterpret_cast<float4*>(dst) = make_float4(0, 0, 0, 0);
                }
            }
        } else {
            for (uint32_t first = tid; first < wtasks; first += 4 * ROUTER_THREADS) {
                uint2 raw[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t task = first + u * ROUTER_THREADS;
                    raw[u] = make_uint2(0, 0);
                    if (task < wtasks) {
                        const uint32_t el = task / (KC / 4), kq = task % (KC / 4), e = e0 + el;
                        if (e < rows_total) {
                            const uint16_t* base = e < c.E ? static_cast<const uint16_t*>(c.router_w) + size_t(e) * H : static_cast<const uint16_t*>(c.shared_gate_w);
                            raw[u] = __ldg(reinterpret_cast<const uint2*>(base + k0 + kq * 4));
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t task = first + u * ROUTER_THREADS;
                    if (task < wtasks) {
                        const uint32_t el = task / (KC / 4), kq = task % (KC / 4);
                        *reinterpret_cast<float4*>(ws + el * LD + kq * 4) =
                            make_float4(__uint_as_float(raw[u].x << 16), __uint_as_float(raw[u].x & 0xffff0000u),
                                        __uint_as_float(raw[u].y << 16), __uint_as_float(raw[u].y & 0xffff0000u));
                    }
                }
            }
        }
    };
    // The router rows are weights: their copies start before the previous kernel of the chain has finished.
    stage_rows();
    pdl_wait();
    pdl_launch_dependents();
    if (x32) {
        for (uint32_t task = tid; task < xtasks * 2; task += ROUTER_THREADS) {       // 16-byte pieces
            const uint32_t tt = task / (KC / 4), kq = task % (KC / 4), t = t0 + tt;
            float* dst = xs + tt * LD + kq * 4;
            if (t < c.T) cp_async16(dst, static_cast<const float*>(c.x) + size_t(t) * H + k0 + kq * 4);
            else *reinterpret_cast<float4*>(dst) = make_float4(0, 0, 0, 0);
        }
    } else {
        for (uint32_t first = tid; first < xtasks; first += XB * ROUTER_THREADS) {
            uint4 raw[XB];
#pragma unroll
            for (int u = 0; u < XB; ++u) {
                const uint32_t task = first + u * ROUTER_THREADS;
                raw[u] = make_uint4(0, 0, 0, 0);
                if (task < xtasks) {
                    const uint32_t tt = task / (KC / 8), kb = task % (KC / 8), t = t0 + tt;
                    if (t < c.T) raw[u] = __ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(c.x) + size_t(t) * H + k0 + kb * 8));
                }
            }
#pragma unroll
            for (int u = 0; u < XB; ++u) {
                const uint32_t task = first + u * ROUTER_THREADS;
                if (task < xtasks) {
                    const uint32_t tt = task / (KC / 8), kb = task % (KC / 8);
                    const uint32_t r[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
                    float4* dst = reinterpret_cast<float4*>(xs + tt * LD + kb * 8);
                    dst[0] = make_float4(__uint_as_float(r[0] << 16), __uint_as_float(r[0] & 0xffff0000u), __uint_as_float(r[1] << 16), __uint_as_float(r[1] & 0xffff0000u));
                    dst[1] = make_float4(__uint_as_float(r[2] << 16), __uint_as_float(r[2] & 0xffff0000u), __uint_as_float(r[3] << 16), __uint_as_float(r[3] & 0xffff0000u));
                }
            }
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // ---- chains ----
    const uint32_t tx = tid % 32, ty = tid / 32;
    float acc[CLUSTER_PARTS][TPT][RPT];
#pragma unroll
    for (int pp = 0; pp < CLUSTER_PARTS; ++pp)
#pragma unroll
        for (int j = 0; j < TPT; ++j)
#pragma unroll
            for (int i = 0; i < RPT; ++i) acc[pp][j][i] = 0.0f;
    const float* wrow = ws + tx * LD;
    const float* xrow = xs + ty * TPT * LD;
#pragma unroll 2
    for (uint32_t k = 0; k < part; k += 4) {
#pragma unroll
        for (int pp = 0; pp < CLUSTER_PARTS; ++pp) {
            float4 wv[RPT], xv[TPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i) wv[i] = *reinterpret_cast<const float4*>(wrow + i * 32 * LD + pp * part + k);
#pragma unroll
            for (int j = 0; j < TPT; ++j) xv[j] = *reinterpret_cast<const float4*>(xrow + j * LD + pp * part + k);
#pragma unroll
            for (int j = 0; j < TPT; ++j)
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    float a = acc[pp][j][i];
                    a = __fmaf_rn(xv[j].x, wv[i].x, a);
                    a = __fmaf_rn(xv[j].y, wv[i].y, a);
                    a = __fmaf_rn(xv[j].z, wv[i].z, a);
                    a = __fmaf_rn(xv[j].w, wv[i].w, a);
                    acc[pp][j][i] = a;
                }
        }
    }
#pragma unroll
    for (int pp = 0; pp < CLUSTER_PARTS; ++pp)
#pragma unroll
        for (int j = 0; j < TPT; ++j)
#pragma unroll
            for (int i = 0; i < RPT; ++i) ps[(pp * TT + ty * TPT + j) * ROW_TILE + tx + 32 * i] = acc[pp][j][i];
    cluster.sync();

    // ---- ordered sum of the sixteen partials (router_accumulate, qwen.metal:529-534) for this CTA's outputs ----
    constexpr uint32_t OUT_PER_CTA = TT * ROW_TILE / CLUSTER_SIZE;
    for (uint32_t o = cr * OUT_PER_CTA + tid; o < (cr + 1) * OUT_PER_CTA; o += ROUTER_THREADS) {
        const uint32_t tt = o / ROW_TILE, el = o % ROW_TILE, t = t0 + tt, e = e0 + el;
        float v[16];
#pragma unroll
        for (uint32_t q = 0; q < 16; ++q) {
            const float* remote = cluster.map_shared_rank(ps + ((q % CLUSTER_PARTS) * TT + tt) * ROW_TILE + el, q / CLUSTER_PARTS);
            v[q] = *remote;
        }
        float sum = 0.0f;
#pragma unroll
        for (uint32_t q = 0; q < 16; ++q) sum = __fadd_rn(sum, v[q]);
        if (t < c.T && e < rows_total) {
            if (e < c.E) c.logits[size_t(t) * c.E + e] = c.router_bias ? __fadd_rn(sum, c.router_bias[e]) : sum;
            else c.gate_logit[t] = sum;
        }
    }
    cluster.sync();          // nobody leaves while a peer may still read its partials
}

template <int TT, int RPT>
int launch_router_cluster(zc_moe* m, const Call& c, cudaStream_t s) {
    constexpr int ROW_TILE = 32 * RPT;
    const uint32_t KC = CLUSTER_PARTS * (c.H / 16), LD = KC + 4;
    const size_t smem = (size_t(ROW_TILE + TT) * LD + size_t(CLUSTER_PARTS) * TT * ROW_TILE) * sizeof(float);
    const uint32_t rows_total = c.E + (c.has_shared ? 1 : 0);
    auto kernel = router_cluster_kernel<TT, RPT>;
    const dim3 grid((rows_total + ROW_TILE - 1) / ROW_TILE, CLUSTER_SIZE, (c.T + TT - 1) / TT);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = CLUSTER_SIZE; attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};           // for the occupancy query
    cfg.gridDim = grid; cfg.blockDim = dim3(ROUTER_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cfg.attrs = attr; cfg.numAttrs = 1;
    static SmemOptIn configured;        // per instantiation, per device
    static int8_t usable[MAX_DEVICES];  // per device: 0 unknown, 1 the device hosts a cluster of this shape, 2 it cannot
    if (smem > 224 * 1024 || m->device < 0 || m->device >= MAX_DEVICES) return 0;
    if (smem > configured.bytes[m->device]) {
        if (opt_in_smem(kernel, configured, m->device, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
        usable[m->device] = 0;
    }
    if (usable[m->device] == 0) {
        int clusters = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) cudaGetLastError();
        usable[m->device] = (e == cudaSuccess && clusters > 0) ? 1 : 2;
    }
    if (usable[m->device] != 1) return 0;
    int rc;
    {
        Timed t(m, s, KERNEL_ROUTER);
        // Early launch pays for short batches (the row prefetch hides behind the previous kernel); from 64 tokens on
        // the prefetch of several token tiles competes with that kernel and measured 2 % slower per layer.
        const cudaError_t e = launch_chained(m, c.T <= 32 ? int(KERNEL_ROUTER) : -1, kernel, grid, dim3(ROUTER_THREADS), smem, s, attr, 1, c);
        if (e != cudaSuccess) return fail(m, ZC_EEXEC, std::string("router (cluster) launch: ") + cudaGetErrorString(e));
        rc = check_launch(m, "router");
    }
    return rc < 0 ? rc : 1;
}

// ---------------------------------------------------------------------------------------------------------
// Register-tiled form for more than 128 tokens. A CTA of 128 threads owns 64 tokens (128 in the widest form) x 64 rows of
// the logits and `16 / ranks` consecutive partitions of K. The bound is the FP32 pipe: every logit is a pinned chain of
// fused multiply-adds, 2 T E H flops whatever the schedule. Each thread runs 8 rows x TJ tokens of chains, two rows per
// instruction: fma.rn.f32x2 is two independent IEEE fused multiply-adds on the halves of a 64-bit register, so every chain
// keeps its own k-ascending order and its bits at half the issue slots, which the shared-memory reads and the duplicated
// token operands need. Rows are stored in pairs ([row pair][k][2]: a 16-byte read is the operand of two k), tokens as FP32
// [token][k], both padded so that the lanes of a warp (8 row groups x 4 token groups) read distinct banks. A chain's next
// link comes 4 TJ instructions later (with 4 in between the FMA latency showed: 156 against 146 us at 2048 tokens). K
// arrives in double-buffered chunks of 32: the next chunk is in registers while this one is multiplied.
// ranks = 1: each finished partition is added to the tile's running total in shared memory - the additions "partials 0..15
// in order, starting from zero" of the reference. ranks = 8 (too few tiles for the SMs): the CTAs of a cluster share the
// partitions of a tile, keep every partial in shared memory, and after a cluster barrier each adds the sixteen partials of
// its part of the tile in order, reading its peers' (DSMEM).
// Measured against the forms it replaced (partials in global memory; 4 x 4 scalar chains): 513 tokens 77 -> 56 us, 256 tokens
// at hidden 4096 85 -> 58, 2048 tokens 167 -> 146, 8192 tokens 604 -> 474 (51 % of the FP32 rate; a register tile of 8 x 4
// needs 12 shared-memory wavefronts per 16 FMA instructions and would be bound by them at 66 %, 8 x 8 at 100 %; what is left
// is the duplication of the token operand and the latency of the reads at two to three CTAs per SM).
constexpr int RT_ROWS = 64, RT_THREADS = 128, RT_CHUNK = 32;
constexpr int RT_WLD = RT_CHUNK * 2 + 4, RT_PLD = RT_ROWS + 8;      // pitches in floats: row pair, token of a partial tile
// Geometry of a CTA with TJ tokens per thread.
template <int TJ> struct RouterTile {
    static constexpr int TOKENS = 16 * TJ;
    static constexpr int XLD = RT_CHUNK + 4;                         // pitch of a token in floats
    static constexpr int STAGE_FLOATS = (RT_ROWS / 2) * RT_WLD + TOKENS * XLD, PART_FLOATS = TOKENS * RT_PLD;
};

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float4 bf16x4(uint2 raw) {
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}

template <bool X32, bool W32, int TJ>
__global__ void __launch_bounds__(RT_THREADS, TJ == 8 ? 3 : 4) router_tile_kernel(Call c, uint32_t ranks) {
    using Tile = RouterTile<TJ>;
    constexpr int RT_TOKENS = Tile::TOKENS, RT_STAGE_FLOATS = Tile::STAGE_FLOATS, RT_PART_FLOATS = Tile::PART_FLOATS, XLD = Tile::XLD;
    extern __shared__ __align__(16) float smem[];
    const uint32_t H = c.H, part = H / 16, parts = 16 / ranks;
    float* ps = smem + 2 * RT_STAGE_FLOATS;          // [parts][RT_TOKENS][RT_PLD] partials (ranks > 1), else one running total
    const uint32_t cr = blockIdx.x, e0 = blockIdx.y * RT_ROWS, t0 = blockIdx.z * RT_TOKENS;
    const uint32_t rows_total = c.E + (c.has_shared ? 1u : 0u), rows_here = min(uint32_t(RT_ROWS), rows_total - e0);
    const uint32_t tid = threadIdx.x, rg = tid % 8, tg = tid / 8;
    constexpr int NARROW_ROWS = RT_THREADS / RT_TOKENS;
    const bool narrow = rows_here <= uint32_t(NARROW_ROWS);        // the shared gate's row on its own: one chain per thread
    const uint32_t k_first = cr * parts * part, k_last = k_first + parts * part;

    // Staging: a task is four k of a row pair, or eight k of a token. Two and two of them per thread and chunk.
    constexpr int WT = (RT_ROWS / 2) * (RT_CHUNK / 4) / RT_THREADS, XT = RT_TOKENS * (RT_CHUNK / 8) / RT_THREADS;
    float4 w[WT][2];
    uint4 x[XT][X32 ? 2 : 1];
    auto load_w = [&](uint32_t k, uint32_t n) {      // n: k of this chunk (a multiple of 8, at most RT_CHUNK)
#pragma unroll
        for (int u = 0; u < WT; ++u) {
            const uint32_t kq = tid % (RT_CHUNK / 4), pr = tid / (RT_CHUNK / 4) + u * (RT_THREADS / (RT_CHUNK / 4));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t e = e0 + pr * 2 + h;
                w[u][h] = make_float4(0, 0, 0, 0);
                if (e >= rows_total || kq * 4 >= n) continue;
                const void* base = e < c.E ? c.router_w : c.shared_gate_w;
                const size_t at = size_t(e < c.E ? e : 0) * H + k + kq * 4;
                if (W32) w[u][h] = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + at));
                else w[u][h] = bf16x4(__ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + at)));
            }
        }
    };
    auto load_x = [&](uint32_t k, uint32_t n) {
#pragma unroll
        for (int u = 0; u < XT; ++u) {
            const uint32_t kb = tid % (RT_CHUNK / 8), t = t0 + tid / (RT_CHUNK / 8) + u * (RT_THREADS / (RT_CHUNK / 8));
            const bool on = t < c.T && kb * 8 < n;
            const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(c.x) + (size_t(t) * H + k + kb * 8) * (X32 ? 4 : 2));
#pragma unroll
            for (int h = 0; h < (X32 ? 2 : 1); ++h) x[u][h] = on ? __ldcg(p + h) : make_uint4(0, 0, 0, 0);
        }
    };
    auto store = [&](float* stage) {
        float* ws = stage;
        float* xs = stage + (RT_ROWS / 2) * RT_WLD;
#pragma unroll
        for (int u = 0; u < WT; ++u) {
            const uint32_t kq = tid % (RT_CHUNK / 4), pr = tid / (RT_CHUNK / 4) + u * (RT_THREADS / (RT_CHUNK / 4));
            float4* to = reinterpret_cast<float4*>(ws + pr * RT_WLD + kq * 8);
            to[0] = make_float4(w[u][0].x, w[u][1].x, w[u][0].y, w[u][1].y);
            to[1] = make_float4(w[u][0].z, w[u][1].z, w[u][0].w, w[u][1].w);
        }
#pragma unroll
        for (int u = 0; u < XT; ++u) {
            const uint32_t kb = tid % (RT_CHUNK / 8), tt = tid / (RT_CHUNK / 8) + u * (RT_THREADS / (RT_CHUNK / 8));
            if constexpr (X32) {
                uint4* to = reinterpret_cast<uint4*>(xs + tt * XLD + kb * 8);
                to[0] = x[u][0]; to[1] = x[u][X32 ? 1 : 0];
            } else {
                float4* to = reinterpret_cast<float4*>(xs + tt * XLD + kb * 8);
                to[0] = bf16x4(make_uint2(x[u][0].x, x[u][0].y)); to[1] = bf16x4(make_uint2(x[u][0].z, x[u][0].w));
            }
        }
    };

    if (ranks == 1) for (uint32_t i = tid; i < RT_PART_FLOATS; i += RT_THREADS) ps[i] = 0.0f;
    load_w(k_first, min(uint32_t(RT_CHUNK), part));
    pdl_wait();
    pdl_launch_dependents();
    load_x(k_first, min(uint32_t(RT_CHUNK), part));
    uint64_t acc[4][TJ];                             // [row pair rg + 8 i][token tg + 16 j]
    float single = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) acc[i][j] = 0ull;
    uint32_t in_part = 0, p = 0;                     // k done of the current partition, partitions done
    for (uint32_t k = k_first, buf = 0; k < k_last; buf ^= 1) {
        const uint32_t n = min(uint32_t(RT_CHUNK), part - in_part);
        float* stage = smem + buf * RT_STAGE_FLOATS;
        store(stage);
        __syncthreads();                             // the chunk is in place; the other buffer's readers finished before they stored this one
        const uint32_t next = k + n, next_in = in_part + n == part ? 0 : in_part + n;
        if (next < k_last) { load_w(next, min(uint32_t(RT_CHUNK), part - next_in)); load_x(next, min(uint32_t(RT_CHUNK), part - next_in)); }
        const float* ws = stage;
        const float* xs = stage + (RT_ROWS / 2) * RT_WLD;
        if (narrow) {
            const uint32_t tt = tid % RT_TOKENS, rr = tid / RT_TOKENS;
            for (uint32_t q = 0; q < n; ++q) single = __fmaf_rn(xs[tt * XLD + q], ws[q * 2 + rr], single);
        } else {
#pragma unroll 2
            for (uint32_t q = 0; q < n; q += 4) {
                ulonglong2 wv[2][4];                 // the row pairs' operands of k = q + 2 h and the next
                float4 xv[TJ];
#pragma unroll
                for (int j = 0; j < TJ; ++j) xv[j] = *reinterpret_cast<const float4*>(xs + (tg + 16 * j) * XLD + q);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) wv[h][i] = *reinterpret_cast<const ulonglong2*>(ws + (rg + 8 * i) * RT_WLD + (q + 2 * h) * 2);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)       // a chain's next link comes 4 TJ instructions later
#pragma unroll
                    for (int j = 0; j < TJ; ++j) {
                        const float v = kk == 0 ? xv[j].x : kk == 1 ? xv[j].y : kk == 2 ? xv[j].z : xv[j].w;
                        const uint64_t xd = pack2(v, v);
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[i][j] = fma2(xd, kk % 2 ? wv[kk / 2][i].y : wv[kk / 2][i].x, acc[i][j]);
                    }
            }
        }
        k = next; in_part = next_in;
        if (next_in == 0) {                          // partition p is complete
            float* to = ps + (ranks == 1 ? 0 : p * RT_PART_FLOATS);
            if (narrow) {
                float* o = to + (tid % RT_TOKENS) * RT_PLD + tid / RT_TOKENS;
                *o = ranks == 1 ? __fadd_rn(*o, single) : single;
                single = 0.0f;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < TJ; ++j) {
                        float2* o = reinterpret_cast<float2*>(to + (tg + 16 * j) * RT_PLD + (rg + 8 * i) * 2);
                        const float2 v = unpack2(acc[i][j]);
                        if (ranks == 1) { const float2 sum = *o; *o = make_float2(__fadd_rn(sum.x, v.x), __fadd_rn(sum.y, v.y)); }
                        else *o = v;
                        acc[i][j] = 0ull;
                    }
            }
            ++p;
        }
    }
    if (ranks == 1) __syncthreads();
    else cg::this_cluster().sync();
    const uint32_t share = RT_TOKENS * RT_ROWS / ranks;
    for (uint32_t o = cr * share + tid; o < (cr + 1) * share; o += RT_THREADS) {
        const uint32_t tt = o / RT_ROWS, el = o % RT_ROWS, t = t0 + tt, e = e0 + el;
        if (t >= c.T || e >= rows_total) continue;
        float sum = 0.0f;
        if (ranks == 1) sum = ps[tt * RT_PLD + el];
        else {
            float v[16];
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) v[q] = *cg::this_cluster().map_shared_rank(ps + (q % parts) * RT_PART_FLOATS + tt * RT_PLD + el, q / parts);
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) sum = __fadd_rn(sum, v[q]);
        }
        if (e < c.E) c.logits[size_t(t) * c.E + e] = c.router_bias ? __fadd_rn(sum, c.router_bias[e]) : sum;
        else c.gate_logit[t] = sum;
    }
    if (ranks > 1) cg::this_cluster().sync();        // nobody leaves while a peer may still read its partials
}

template <bool X32, bool W32, int TJ>
int launch_router_tile_n(zc_moe* m, const Call& c, uint32_t ranks, cudaStream_t s) {
    using Tile = RouterTile<TJ>;
    constexpr int RT_TOKENS = Tile::TOKENS, RT_STAGE_FLOATS = Tile::STAGE_FLOATS, RT_PART_FLOATS = Tile::PART_FLOATS;
    const size_t smem = (2 * size_t(RT_STAGE_FLOATS) + size_t(ranks == 1 ? 1 : 16 / ranks) * RT_PART_FLOATS) * sizeof(float);
    const uint32_t rows = c.E + (c.has_shared ? 1 : 0);
    auto kernel = router_tile_kernel<X32, W32, TJ>;
    static SmemOptIn configured;        // per instantiation, per device
    if (opt_in_smem(kernel, configured, m->device, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    const dim3 grid(ranks, (rows + RT_ROWS - 1) / RT_ROWS, (c.T + RT_TOKENS - 1) / RT_TOKENS);
    static int8_t usable[MAX_DEVICES];  // per device: 0 unknown, 1 the device hosts a cluster of this shape, 2 it cannot
    if (ranks > 1 && usable[m->device] == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid; cfg.blockDim = dim3(RT_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = s; cfg.attrs = attr; cfg.numAttrs = 1;
        int clusters = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) cudaGetLastError();
        usable[m->device] = (e == cudaSuccess && clusters > 0) ? 1 : 2;
    }
    if (ranks > 1 && usable[m->device] != 1) return 0;
    int rc;
    {
        Timed t(m, s, KERNEL_ROUTER);
        // Whole-K tiles are not launched early: such a CTA lives as long as the kernel, and placed while the kernel before still
        // holds some SMs they pile up on the others (a layer of 2048 tokens: 891 us against 771). Clusters are: 602 us
        // against 616 for the layer of 256 tokens at hidden 4096.
        const cudaError_t e = launch_chained(m, ranks > 1 ? int(KERNEL_ROUTER) : -1, kernel, grid, dim3(RT_THREADS), smem, s, ranks > 1 ? attr : nullptr, ranks > 1 ? 1 : 0, c, ranks);
        if (e != cudaSuccess) return fail(m, ZC_EEXEC, std::string("router (tile) launch: ") + cudaGetErrorString(e));
        rc = check_launch(m, "router");
    }
    return rc < 0 ? rc : 1;
}

template <bool X32, bool W32>
int launch_router_tile(zc_moe* m, const Call& c, uint32_t ranks, bool wide, cudaStream_t s) {
    return wide ? launch_router_tile_n<X32, W32, 8>(m, c, ranks, s) : launch_router_tile_n<X32, W32, 4>(m, c, ranks, s);
}

}  // namespace

// How the router is cut. Up to 128 tokens small cluster tiles win on latency: at 64 tokens, 544 CTAs of 16 tokens x 32 rows
// measured 19 us against 21 us (32 x 32) and 25 us (32 x 64, whose 144 large CTAs do not all find a cluster slot in the
// first wave).
// Beyond, the register-tiled form. Splitting the partitions over eight CTAs pays unless the 64 x 64 tiles, the shared gate's
// row tile among them, fill the SMs twice and no more: whole tiles then take 141 us at hidden 2048 whatever their number, and
// 198 as soon as one SM has a third one; split ones take 0.56 us a tile, the gate's about half of that. 512 experts and a shared one
// (whole / split us): 1856 tokens, 261 tiles, 141 / 139; 1920, 270, 141 / 143; 2048, 288, 141 / 152; 2049, 297, 198 / 154; 2368, 333,
// 200 / 173. Without the shared expert 2368 tokens, 296 tiles, 141 / 163; 128 experts and a shared one 8192 tokens, 384, 199 / 176.
// From 480 tiles of experts on, tiles of twice the tokens (a third fewer shared-memory reads per product): 387 against 405 us at
// 6430 tokens.
RouterCut router_cut(uint32_t tokens, uint32_t experts, bool shared, uint32_t sms) {
    if (tokens <= ZC_ROUTER_SMALL_T) return {uint32_t(CLUSTER_SIZE), tokens <= 8 ? 8u : 16u};
    const uint64_t token_tiles = (tokens + 63) / 64, full = token_tiles * ((experts + RT_ROWS - 1) / RT_ROWS);
    const uint64_t all = token_tiles * ((experts + shared + RT_ROWS - 1) / RT_ROWS);       // all - full: tiles of the gate's row alone
    if (full >= 480) return {1, 128};
    const bool twice = all <= 2ull * sms && 10 * full + 5 * (all - full) >= 17ull * sms;
    return {twice ? 1u : uint32_t(CLUSTER_SIZE), 64};
}

int launch_router(zc_moe* m, const Call& c, cudaStream_t s) {
    const RouterCut cut = router_cut(c.T, c.E, c.has_shared, sm_count(m));
    int n = 0;
    if (cut.tokens == 8) n = launch_router_cluster<8, 1>(m, c, s);
    else if (cut.tokens == 16) n = launch_router_cluster<16, 1>(m, c, s);
    if (n != 0) return n;
    // A device that cannot host a cluster of eight takes whole tiles.
    const bool f32x = c.act_dtype == ZC_F32, f32w = c.router_dtype == ZC_F32, wide = cut.tokens == 128;
    for (uint32_t ranks = cut.ranks;; ranks = 1) {
        n = f32x ? (f32w ? launch_router_tile<true, true>(m, c, ranks, wide, s) : launch_router_tile<true, false>(m, c, ranks, wide, s))
                 : (f32w ? launch_router_tile<false, true>(m, c, ranks, wide, s) : launch_router_tile<false, false>(m, c, ranks, wide, s));
        if (n != 0) return n;
        if (ranks == 1) return fail(m, ZC_EEXEC, "router: the device does not host the kernel");
    }
}

}  // namespace zc

// ---------------------------------------------------------------------------------------------
// Router logits for callers that must not allocate device memory.
//
// Some hosts of this library run inside a region where cudaMalloc is forbidden or would deadlock: a
// plugin called while the engine's own caching allocator holds all of HBM, a callback that runs while
// another thread is capturing a CUDA graph (allocation calls are illegal then), or a real-time loop
// that may not take the allocator's lock. zc_moe_create allocates, so those callers cannot own a
// handle. This entry point needs none: the router kernel's scratch — the [16, tokens, experts]
// partition sums and the tile arrival counters — lives in a fixed array inside the library image.
// ---------------------------------------------------------------------------------------------
namespace zc {
namespace {
constexpr uint32_t NOALLOC_MAX_TOKENS = 64, NOALLOC_MAX_EXPERTS = 512, NOALLOC_MAX_HIDDEN = 3072;
constexpr size_t NOALLOC_PARTIAL_BYTES = size_t(16) * NOALLOC_MAX_TOKENS * NOALLOC_MAX_EXPERTS * sizeof(float);   // 2 MiB
constexpr size_t NOALLOC_COUNTER_BYTES = 4096;       // (experts / 32) x (tokens / 8) counters at most = 128 words
// Held by every GPU that loads the library until the process exits: 2 MiB + 4 KiB.
static __device__ __align__(256) unsigned char noalloc_scratch[NOALLOC_PARTIAL_BYTES + NOALLOC_COUNTER_BYTES];

constexpr int NOALLOC_MAX_DEVICES = 64;
unsigned char* noalloc_address[NOALLOC_MAX_DEVICES] = {};   // device address of the array, per device
}  // namespace
}  // namespace zc

extern "C" int zc_router_logits_noalloc(const void* x, int act_dtype, const void* router_w, int router_dtype,
                                        uint32_t tokens, uint32_t hidden, uint32_t experts, float* logits, void* stream) {
    using namespace zc;
    if (!x || !router_w || !logits) return fail(nullptr, ZC_EINVAL, "linear input shape");
    if (!tokens || tokens > NOALLOC_MAX_TOKENS)
        return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: tokens must be 1..64 (the built-in scratch is sized for 64)");
    if (!experts || experts % 32 || experts > NOALLOC_MAX_EXPERTS)
        return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: experts must be a multiple of 32, at most 512");
    if (!hidden || hidden % 128 || hidden > NOALLOC_MAX_HIDDEN)
        return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: hidden must be a multiple of 128, at most 3072");
    if ((act_dtype != ZC_BF16 && act_dtype != ZC_F32) || (router_dtype != ZC_BF16 && router_dtype != ZC_F32))
        return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: dtypes must be BF16 or F32");
    // The kernel reads x and router_w and writes logits with 16-byte accesses: a misaligned or aliased buffer is an
    // argument error here, not a device fault.
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(router_w) | reinterpret_cast<uintptr_t>(logits)) & 15)
        return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: x, router_w and logits must be 16-byte aligned");
    {
        const size_t xb = size_t(tokens) * hidden * (act_dtype == ZC_F32 ? 4 : 2), wb = size_t(experts) * hidden * (router_dtype == ZC_F32 ? 4 : 2);
        const size_t lb = size_t(tokens) * experts * 4;
        const char* lo = reinterpret_cast<const char*>(logits);
        const char* xa = static_cast<const char*>(x); const char* wa = static_cast<const char*>(router_w);
        if ((lo < xa + xb && xa < lo + lb) || (lo < wa + wb && wa < lo + lb))
            return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: logits overlaps an input");
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return fail(nullptr, ZC_EEXEC, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (device < 0 || device >= NOALLOC_MAX_DEVICES) return fail(nullptr, ZC_EINVAL, "zc_router_logits_noalloc: device index above 63");
    if (!noalloc_address[device]) {
        // Set-up, once per device, with that device current: in host code the array's name is only a
        // stand-in, the kernel needs the address the runtime gives for it on this device.
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, noalloc_scratch);
        if (e != cudaSuccess || !p) return fail(nullptr, ZC_EEXEC, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        noalloc_address[device] = static_cast<unsigned char*>(p);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float* partial = reinterpret_cast<float*>(noalloc_address[device]);
    uint32_t* counters = reinterpret_cast<uint32_t*>(noalloc_address[device] + NOALLOC_PARTIAL_BYTES);
    // The counters must start at zero (a call cut short by an error would leave them dirty); the partial
    // sums are fully rewritten for the (tokens, experts) of this call before they are read.
    if ((e = cudaMemsetAsync(counters, 0, NOALLOC_COUNTER_BYTES, s)) != cudaSuccess)
        return fail(nullptr, ZC_EEXEC, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    Call c{};
    c.x = x; c.router_w = router_w; c.logits = logits;
    c.T = tokens; c.H = hidden; c.E = experts; c.act_dtype = uint8_t(act_dtype); c.router_dtype = uint8_t(router_dtype); c.has_shared = 0;
    const uint32_t part = hidden / 16, rows_padded = experts;      // a multiple of the 32-row tile already
    const bool tiny = tokens <= 8;
    const uint32_t TT = tiny ? 8 : 16;
    const size_t smem = size_t(part) * (TT + 32) * sizeof(float);   // at most 36 KiB: no opt-in attribute needed
    const dim3 grid(rows_padded / 32, 16, (tokens + TT - 1) / TT);
    if (tiny) router_partial_kernel<8><<<grid, ROUTER_THREADS, smem, s>>>(c, partial, rows_padded, counters, 1);
    else router_partial_kernel<16><<<grid, ROUTER_THREADS, smem, s>>>(c, partial, rows_padded, counters, 1);
    return check_launch(nullptr, "router (no-alloc)");
}
