// The product of gemm_tcgen05.cu for few rows (a decode step, a short slice): D[M][N] (+)= A[M][K] W[N][K]^T, M <= kFewRowsMax.
//
// With M rows on the 128-row side of the MMA, half or more of a tile is padding, a CTA's share of the weights is narrow (32 - 64
// columns) and comes with the whole activation tile for every k-block, and one CTA walks over all of K.  Nothing is saturated then:
// the step is a chain of copy latencies.  Here the weights take the 128-row side: a CTA multiplies 128 weight rows with all NB rows
// of the batch, hi and lo halves side by side as the columns of one MMA (hi in [0, NB), lo in [NB, 2 NB), added in the epilogue), and a
// cluster of up to eight CTAs shares K.  A cluster's partial results travel through distributed shared memory: every CTA receives all
// partials of its share of the rows, adds them in split order (the result does not depend on timing) and finishes these rows, lanes
// along the output columns, so that residual, result and halves are read and written in whole lines.
//
// ORDERED: in the persistent kernel's order, for models whose results must not move by a bit with the kernel: hi and lo go into the same columns, one after
// the other for every k-block, K is split as it is there, and sums of squares are taken as its threads take them.
//
// What bounds it: the latency of one round of copies and of the reduction; at many weights (the head, 2048-wide layers) their stream.
// Measured on the 48-layer base model: 16 steps of 64 sequences 31.3 -> 24.5 ms.
#include "internal.h"
#include "tcgen05.cuh"

#include <algorithm>
#include <cstdlib>

namespace lumi {

int32_t gemm_tcgen05_init();
int32_t make_bf16_operand_map(CUtensorMap* map, const void* ptr, int rows, int K, int box_rows);

namespace {

constexpr int kThreads = 256;
constexpr int kWRows = 128;                  // weight rows of a tile: the M of the MMA
constexpr int kWBytes = kWRows * BK * 2;
constexpr int kTailBytes = 1024;             // barriers, row scales
constexpr int kMaxStages = 8;
constexpr int kMaxCluster = 8;

struct Tail {
    uint64_t full[kMaxStages], empty[kMaxStages], tmem_full, drain;
    uint32_t tmem_slot;
    int skip, failed;
    float rs[128];
};
static_assert(sizeof(Tail) <= kTailBytes, "tail of the shared memory");

__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

struct FewRowsShape {
    int M, N, K, ldd, accumulate, tiles_pg, stages, vec;
};

// Warp 0: copies.  Warp 1: TMEM, MMA.  Warps 2, 3: the rows' scales.  Warps 4 - 7: accumulators to the owners of the rows.  All: finish.
template <int NB, bool SPLIT, bool EXT, bool ORDERED>
__global__ void __launch_bounds__(kThreads, 2)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, const __grid_constant__ CUtensorMap map_w,
                     float* D, FewRowsShape sh, int splits, int32_t* status, uint64_t wait_ns, int skip_unit, NormFuse nf, GemmExt ex) {
    constexpr int A_BYTES = NB * BK * 2, STAGE = kWBytes + A_BYTES * (SPLIT ? 2 : 1);
    constexpr bool APART = SPLIT && !ORDERED;                           // hi and lo in columns of their own
    constexpr uint32_t COLS = APART ? 2 * NB : NB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // partial results: behind the stages, since another CTA's arrive while this one still multiplies; without a cluster they reuse the stages
    float* part = reinterpret_cast<float*>(base + (splits > 1 ? sh.stages * STAGE : 0));
    Tail& tl = *reinterpret_cast<Tail*>(base + sh.stages * STAGE + (splits > 1 ? NB * kWRows * 4 : 0));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, S = sh.stages;
    const int rank = (int)blockIdx.x % splits, tile = (int)blockIdx.x / splits, m0 = blockIdx.y * NB;
    const int group = EXT ? tile / sh.tiles_pg : 0, n_in = (EXT ? tile % sh.tiles_pg : tile) * kWRows;      // first weight row within the group
    const int n0 = EXT ? group * ex.group_rows + n_in : n_in;
    const int num_kb = sh.K / BK, kb0 = rank * num_kb / splits, nkb = (rank + 1) * num_kb / splits - kb0;
    const int kx = (EXT ? group * sh.K : 0) + kb0 * BK;                 // first element of the rows of A
    const int RB = NB / splits;                                         // rows that this CTA finishes

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&tl.full[s], 1); mbar_init(&tl.empty[s], 1); }
        mbar_init(&tl.tmem_full, 1);
        mbar_init(&tl.drain, 1);
        tl.failed = 0;
        // a wait that expired in an earlier launch: no new work, but every barrier of the cluster is still taken
        tl.skip = status != nullptr && (*reinterpret_cast<volatile int32_t*>(status) & STATUS_TIMEOUT) ? 1 : 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tl.tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // behind the allocation: a dependent that becomes resident beside this CTA may want TMEM too, and must not get it first
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (splits > 1) cluster_arrive();                                   // "this CTA runs": partials may be sent to it
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tl.tmem_slot);
    const bool skip = *reinterpret_cast<volatile int*>(&tl.skip) != 0;
    bool timed_out = false;

    // the weights depend on no predecessor: the first stages' tiles are requested ahead of the dependency wait
    const bool loads = warp == 0 && lane == 0 && !skip && (int)(blockIdx.y * gridDim.x + blockIdx.x) != skip_unit;
    const int pre = min(S, nkb);
    if (loads)
        for (int i = 0; i < pre; ++i) {
            mbar_expect_tx(&tl.full[i], (uint32_t)STAGE);
            tma_load_2d(base + i * STAGE, &map_w, &tl.full[i], (kb0 + i) * BK, n0);
        }
    asm volatile("griddepcontrol.wait;" ::: "memory");

    float4 old[4];                                                      // what the first four rows of this warp are added to
    if (warp == 0) {
        if (loads) {
            int s = 0, issued = 0;
            uint32_t ph = 0;
            for (int i = 0; i < nkb; ++i) {
                uint8_t* st = base + s * STAGE;
                if (i >= pre) {
                    if (!mbar_wait(&tl.empty[s], ph ^ 1u, wait_ns)) { timed_out = true; break; }
                    mbar_expect_tx(&tl.full[s], (uint32_t)STAGE);
                    tma_load_2d(st, &map_w, &tl.full[s], (kb0 + i) * BK, n0);
                }
                tma_load_2d(st + kWBytes, &map_hi, &tl.full[s], kx + i * BK, m0);
                if (SPLIT) tma_load_2d(st + kWBytes + A_BYTES, &map_lo, &tl.full[s], kx + i * BK, m0);
                issued = i + 1;
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (timed_out)                                              // let the copies land (bounded) that nobody may consume
                for (int i = max(0, issued - S); i < issued; ++i) mbar_wait(&tl.full[i % S], (uint32_t)(i / S) & 1u, wait_ns);
        }
    } else if (warp == 1) {
        if (lane == 0 && !skip) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COLS >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
            int s = 0;
            uint32_t ph = 0;
            for (int i = 0; i < nkb; ++i) {
                if (!mbar_wait(&tl.full[s], ph, wait_ns)) { timed_out = true; break; }
                tc_fence_after();
                const uint32_t w = smem_u32(base + s * STAGE), act = w + kWBytes;      // the lo rows follow the hi rows
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_bf16(tmem, make_smem_desc(w + k * 32), make_smem_desc(act + k * 32), idesc, (i > 0 || k > 0) ? 1u : 0u);
                if constexpr (SPLIT && ORDERED) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem, make_smem_desc(w + k * 32), make_smem_desc(act + A_BYTES + k * 32), idesc, 1u);
                }
                umma_commit(&tl.empty[s]);
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!timed_out) {
                umma_commit(&tl.tmem_full);
            } else {                                                    // let every MMA issued so far finish (bounded), then pass the word on
                umma_commit(&tl.drain);
                mbar_wait(&tl.drain, 0, wait_ns);
                *reinterpret_cast<volatile int*>(&tl.failed) = 1;
                mbar_arrive(&tl.tmem_full);
            }
        }
    } else if (warp < 4) {
        // RMSNorm folded around the product (NormFuse): scale of a row from its partial sums of squares, added in column order
        for (int r = threadIdx.x - 64; r < RB; r += 64) {
            const int row = m0 + rank * RB + r;
            float rs = 1.0f;
            if (nf.ssq_in != nullptr && row < sh.M) {
                const float* pp = nf.ssq_in + (size_t)row * nf.ssq_stride;
                float t = 0.f;
                int pz = 0;
                if ((nf.ssq_stride & 3) == 0) {
                    for (; pz + 16 <= nf.ssq_parts; pz += 16) {
                        const float4 a0 = *reinterpret_cast<const float4*>(pp + pz), a1 = *reinterpret_cast<const float4*>(pp + pz + 4);
                        const float4 a2 = *reinterpret_cast<const float4*>(pp + pz + 8), a3 = *reinterpret_cast<const float4*>(pp + pz + 12);
                        t += a0.x; t += a0.y; t += a0.z; t += a0.w; t += a1.x; t += a1.y; t += a1.z; t += a1.w;
                        t += a2.x; t += a2.y; t += a2.z; t += a2.w; t += a3.x; t += a3.y; t += a3.z; t += a3.w;
                    }
                }
                for (; pz < nf.ssq_parts; ++pz) t += pp[pz];
                rs = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(t, nf.inv_k), nf.eps)));
            }
            tl.rs[r] = rs;
        }
    }
    __syncwarp();
    // residual and bias of this warp's first rows, on their way while the tensor core still works
    const int nl = n_in + 4 * lane, n_end = EXT ? ex.group_rows : sh.N;                 // this lane's four columns within the group
    const bool quad = sh.vec && nl + 4 <= n_end;
    auto old4 = [&](int row) {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= sh.M || nl >= n_end) return o;
        const float* dp = !EXT && sh.accumulate ? D + (size_t)row * sh.ldd + nl : nullptr;
        const float* bp = nf.bias != nullptr ? nf.bias + (EXT ? (size_t)group * ex.group_rows : 0) : nullptr;
        if (quad) {
            if (dp != nullptr) o = __ldcg(reinterpret_cast<const float4*>(dp));
            if (bp != nullptr) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(bp + nl));
                o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
            }
            return o;
        }
        float* e = &o.x;
        for (int j = 0; j < 4; ++j)
            if (nl + j < n_end) e[j] = (dp != nullptr ? __ldcg(dp + j) : 0.f) + (bp != nullptr ? bp[nl + j] : 0.f);
        return o;
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) old[j] = old4(warp + 8 * j < RB && !skip ? m0 + rank * RB + warp + 8 * j : sh.M);
    if (splits > 1) cluster_wait();                                     // every CTA of the cluster runs
    if (warp >= 4 && !skip) {
        if (!mbar_wait(&tl.tmem_full, 0, wait_ns)) timed_out = true;
        timed_out = __any_sync(0xffffffffu, timed_out);                 // tcgen05.ld below is warp-collective
        if (!timed_out && *reinterpret_cast<volatile int*>(&tl.failed) == 0) {
            tc_fence_after();
            const int q = warp & 3;                                     // TMEM lane quarter this warp may read
            const uint32_t slot = smem_u32(part) + (uint32_t)((rank * RB) * kWRows + q * 32 + lane) * 4u;
#pragma unroll 1
            for (int cb = 0; cb < NB / 32; ++cb) {
                if (m0 + cb * 32 >= sh.M) break;
                uint32_t hi[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cb * 32), hi);
                if (APART) {
                    uint32_t lo[32];
                    tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(NB + cb * 32), lo);
#pragma unroll
                    for (int j = 0; j < 32; ++j) hi[j] = __float_as_uint(__uint_as_float(hi[j]) + __uint_as_float(lo[j]));
                }
                if (splits == 1) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) part[(cb * 32 + j) * kWRows + q * 32 + lane] = __uint_as_float(hi[j]);
                } else {
                    // rows cb * 32 + j belong to CTA (cb * 32 + j) / RB; RB is a power of two of at least four
#pragma unroll
                    for (int j4 = 0; j4 < 32; j4 += 4) {
                        const int b = cb * 32 + j4, to = b / RB;
                        const uint32_t at = map_to_rank(slot + (uint32_t)(b - to * RB) * (kWRows * 4u), (uint32_t)to);
#pragma unroll
                        for (int j = 0; j < 4; ++j) st_cluster(at + (uint32_t)j * (kWRows * 4u), __uint_as_float(hi[j4 + j]));
                    }
                }
            }
            tc_fence_before();
        }
    }
    __syncwarp();
    if (splits > 1) { cluster_arrive(); cluster_wait(); } else __syncthreads();
    if (warp == 1) {                                                    // every accumulator has been read
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    }
    if (timed_out && status != nullptr) atomicOr(status, STATUS_TIMEOUT);
    if (skip) return;

    // ---- this CTA's rows: one warp per row, four columns per lane
    for (int r0 = warp; r0 < RB; r0 += 32) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + 8 * j, row = m0 + rank * RB + r;
            if (r >= RB || row >= sh.M) break;                          // the same for the whole warp
            float4 acc = reinterpret_cast<const float4*>(part + (size_t)r * kWRows)[lane];
            for (int c = 1; c < splits; ++c) {
                const float4 p = reinterpret_cast<const float4*>(part + (size_t)(c * RB + r) * kWRows)[lane];
                acc.x += p.x; acc.y += p.y; acc.z += p.z; acc.w += p.w;
            }
            const float4 o = r0 == warp ? old[j] : old4(row);
            const float rs = tl.rs[r];
            float v[4] = {fmaf(acc.x, rs, o.x), fmaf(acc.y, rs, o.y), fmaf(acc.z, rs, o.z), fmaf(acc.w, rs, o.w)};
            if constexpr (ORDERED && EXT) {                             // there the scaled sum is rounded before the bias is added
                v[0] = __fadd_rn(__fmul_rn(acc.x, rs), o.x); v[1] = __fadd_rn(__fmul_rn(acc.y, rs), o.y);
                v[2] = __fadd_rn(__fmul_rn(acc.z, rs), o.z); v[3] = __fadd_rn(__fmul_rn(acc.w, rs), o.w);
            }
            if constexpr (EXT) {
                int col = nl;
                const int lim = ex.out_n;
                bool mine = nl < n_end;
                if (ex.gate != 0) {                                     // sixteen gates, then their sixteen ups: lanes 0 - 3 and 4 - 7 of eight
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float up = __shfl_down_sync(0xffffffffu, v[e], 4), g = v[e];
                        v[e] = (ex.gate == ACT_RELU_GATE ? fmaxf(g, 0.f) : g * sigmoid_f(g)) * up;
                    }
                    col = (nl >> 5 << 4) + (nl & 15);
                    mine = mine && (lane & 4) == 0;
                }
                if (!mine || col >= lim) continue;
                const int oc = group * ex.out_step + col, cnt = min(4, lim - col);
                if (ex.mul != nullptr) {
                    const float* mp = ex.mul + (size_t)row * ex.ldmul + oc;
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (e < cnt) v[e] *= sigmoid_f(mp[e]);
                }
                const bool whole = sh.vec && cnt == 4 && ((oc | sh.ldd | ex.ldo) & 3) == 0;
                if (D != nullptr) {
                    float* dp = D + (size_t)row * sh.ldd + oc;
                    if (whole) *reinterpret_cast<float4*>(dp) = make_float4(v[0], v[1], v[2], v[3]);
                    else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) if (e < cnt) dp[e] = v[e];
                    }
                }
                if (nf.out_hi != nullptr) {
                    const size_t oo = (size_t)row * ex.ldo + oc;
                    __nv_bfloat16 h[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) { h[e] = __float2bfloat16_rn(v[e]); l[e] = __float2bfloat16_rn(v[e] - __bfloat162float(h[e])); }
                    if (whole) {
                        *reinterpret_cast<uint2*>(nf.out_hi + oo) = *reinterpret_cast<const uint2*>(h);
                        if (nf.out_lo != nullptr) *reinterpret_cast<uint2*>(nf.out_lo + oo) = *reinterpret_cast<const uint2*>(l);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (e < cnt) { nf.out_hi[oo + e] = h[e]; if (nf.out_lo != nullptr) nf.out_lo[oo + e] = l[e]; }
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = epi_act(v[e], nf.act);
                if (D != nullptr) {
                    float* dp = D + (size_t)row * sh.ldd + nl;
                    if (quad) *reinterpret_cast<float4*>(dp) = make_float4(v[0], v[1], v[2], v[3]);
                    else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) if (nl + e < sh.N) dp[e] = v[e];
                    }
                }
                if (nf.out_hi != nullptr) {                             // N % 8 == 0: four columns exist or none does
                    const bool in = nl < sh.N;
                    if (in) {
                        const float4 gm = gamma4(nf.gamma_next, nl);
                        const float w[4] = {v[0] * gm.x, v[1] * gm.y, v[2] * gm.z, v[3] * gm.w};
                        __nv_bfloat16 h[4], l[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) { h[e] = __float2bfloat16_rn(w[e]); l[e] = __float2bfloat16_rn(w[e] - __bfloat162float(h[e])); }
                        const size_t oo = (size_t)row * sh.N + nl;
                        *reinterpret_cast<uint2*>(nf.out_hi + oo) = *reinterpret_cast<const uint2*>(h);
                        if (nf.out_lo != nullptr) *reinterpret_cast<uint2*>(nf.out_lo + oo) = *reinterpret_cast<const uint2*>(l);
                    }
                    if (nf.ssq_out != nullptr) {                        // sums of squares of strips of 32 columns: eight lanes
                        float q = 0.f;
                        if constexpr (ORDERED) {                        // (N % 32 == 0: whole strips) column after column, as one thread of the persistent kernel
#pragma unroll
                            for (int x = 0; x < 8; ++x) {
                                const float t = splits > 1 ? fmaf(v[2], v[2], fmaf(v[3], v[3], fmaf(v[0], v[0], fmaf(v[1], v[1], q))))
                                                           : fmaf(v[0], v[0], fmaf(v[1], v[1], fmaf(v[2], v[2], fmaf(v[3], v[3], q))));
                                q = __shfl_sync(0xffffffffu, t, (lane & ~7) | x);
                            }
                        } else {
                            q = in ? fmaf(v[0], v[0], fmaf(v[1], v[1], fmaf(v[2], v[2], v[3] * v[3]))) : 0.f;
#pragma unroll
                            for (int x = 1; x < 8; x <<= 1) q += __shfl_xor_sync(0xffffffffu, q, x);
                        }
                        if ((lane & 7) == 0 && in) nf.ssq_out[(size_t)row * nf.ssq_stride + (nl >> 5)] = q;
                    }
                }
            }
        }
    }
}

struct FewRowsPlan { int nb, splits, stages, smem, tiles, row_tiles; };

int sms() {
    static const int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        return v;
    }();
    return n;
}

// K goes to as many CTAs as one wave has room for (one CTA per SM; a second wave, or two CTAs on an SM that draw operands at once,
// cost more than the shorter walk saves), clusters of eight only where few of them are needed: 16 such clusters no longer run at once.
// Measured with cold caches, microseconds: 64 x 1024 x 2048 on 8 / 16 / 32 / 64 CTAs 17.0 / 12.2 / 9.2 / 8.0; 64 x 7360 x 1024 on 58 / 116 /
// 232 14.0 / 11.6 / 11.4; 64 x 2048 x 5632 on 64 (clusters of four) / 128 (of eight) 14.5 / 20.1; 128 x 11264 x 2048 on 88 / 176 28.6 / 44.9.
FewRowsPlan few_rows_plan(const GemmArgs& a) {
    FewRowsPlan p{};
    p.nb = a.M <= 32 ? 32 : (a.M <= 64 ? 64 : 128);
    p.row_tiles = (a.M + p.nb - 1) / p.nb;
    p.tiles = a.ext != nullptr ? (a.ext->group_rows + kWRows - 1) / kWRows * a.ext->groups : (a.N + kWRows - 1) / kWRows;
    const int num_kb = a.K / BK, stage = kWBytes + p.nb * BK * 2 * (a.a_lo != nullptr ? 2 : 1);
    const long whole = (long)p.tiles * p.row_tiles;       // CTAs with K in one piece
    p.splits = 1;
    if (a.ordered) p.splits = gemm_persistent_splits(a);
    else while (p.splits < kMaxCluster && num_kb >= 4 * p.splits && whole * 2 * p.splits <= (p.splits == 4 ? sms() / 2 : sms())) p.splits *= 2;
    const int part = p.splits > 1 ? p.nb * kWRows * 4 : 0;
    const int budget = (whole * p.splits > sms() ? 112 : 220) * 1024 - part - kTailBytes - 1024;      // more CTAs than SMs: two share one
    p.stages = std::max(2, std::min({kMaxStages, budget / stage, (num_kb + p.splits - 1) / p.splits}));
    p.smem = p.stages * stage + part + kTailBytes + 1024;
    return p;
}

template <int NB, bool SPLIT, bool EXT, bool ORDERED>
int32_t launch_t(const GemmArgs& a, const FewRowsPlan& p, cudaStream_t st) {
    CUtensorMap mh, ml, mw;
    const int lda = EXT ? a.ext->lda : a.K;
    LUMI_TRY(make_bf16_operand_map(&mh, a.a_hi, a.M, lda, NB));
    LUMI_TRY(make_bf16_operand_map(&ml, SPLIT ? a.a_lo : a.a_hi, a.M, lda, NB));
    LUMI_TRY(make_bf16_operand_map(&mw, a.w, a.N, a.K, kWRows));
    auto kern = gemm_few_rows_kernel<NB, SPLIT, EXT, ORDERED>;
    LUMI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.tiles * p.splits, p.row_tiles);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = launch_pdl_gemm_on() ? 2 : 1;
    const bool vec = (a.ldd & 3) == 0 && (reinterpret_cast<uintptr_t>(a.d) & 15) == 0;
    const FewRowsShape sh{a.M, a.N, a.K, a.ldd, a.accumulate, EXT ? (a.ext->group_rows + kWRows - 1) / kWRows : 0, p.stages, vec ? 1 : 0};
    LUMI_CUDA(cudaLaunchKernelEx(&cfg, kern, mh, ml, mw, a.d, sh, p.splits, a.status_word, a.wait_limit_ns ? a.wait_limit_ns : kWaitLimitNs, a.debug_skip_unit,
                                 a.nf, EXT ? *a.ext : GemmExt()));
    return LUMI_OK;
}

}  // namespace

// Where it is the better kernel (otherwise the persistent one): up to 64 rows always; above, where K is shared.  With K in one piece the
// walk is as long as the persistent kernel's, whose tiles then carry less of the activations.  Measured, this kernel against the persistent
// one, microseconds: 64 rows 7360 x 1024 11.6 / 12.9, 1024 x 2048 7.8 / 12.4, 32000 x 1024 22.1 / 25.3, 2048 x 5632 14.6 / 21.5; 128 rows 1024 x
// 2048 10.4 / 14.5, 2048 x 5632 19.3 / 25.9, 8192 x 2048 19.8 / 20.6, but in one piece 32000 x 2048 40.3 / 36.6, 11264 x 2048 28.6 / 25.4; 256
// rows 1024 x 2048 12.3 / 18.7, 2048 x 5632 21.0 / 43.6, but in one piece 8192 x 2048 23.9 / 22.8; 512 rows 1024 x 2048 13.2 / 19.1.
// In the persistent kernel's order (measured on a model of width 2048 with 128 rows and of width 1024 with 23): up to 64 rows always, up to 128 where K
// is shared there.
bool gemm_few_rows_takes(const GemmArgs& a) {
    if (a.ordered) {
        // a strip cut by a tile's end adds a bias differently (width_counts in gemm_tcgen05.cu), and takes its sum of squares by single elements
        if (a.M > 128 || (a.ext == nullptr && (a.N % 32 != 0 || (a.nf.ssq_in != nullptr && a.nf.bias != nullptr) || (a.ldd & 3) != 0))) return false;
        return a.M <= 64 || gemm_persistent_splits(a) > 1;
    }
    return a.M <= 64 || (a.M <= kFewRowsMax && few_rows_plan(a).splits > 1);
}

// Arguments have been checked by launch_gemm_tcgen05.
int32_t launch_gemm_few_rows(const GemmArgs& a, cudaStream_t st) {
    const FewRowsPlan p = few_rows_plan(a);
    const bool split = a.a_lo != nullptr;
#define LUMI_FEW(NB_) \
    if (p.nb == NB_) { \
        if (a.ordered && a.ext != nullptr) return split ? launch_t<NB_, true, true, true>(a, p, st) : launch_t<NB_, false, true, true>(a, p, st); \
        if (a.ordered) return split ? launch_t<NB_, true, false, true>(a, p, st) : launch_t<NB_, false, false, true>(a, p, st); \
        if (a.ext != nullptr) return split ? launch_t<NB_, true, true, false>(a, p, st) : launch_t<NB_, false, true, false>(a, p, st); \
        return split ? launch_t<NB_, true, false, false>(a, p, st) : launch_t<NB_, false, false, false>(a, p, st); \
    }
    LUMI_FEW(32) LUMI_FEW(64) LUMI_FEW(128)
#undef LUMI_FEW
    return LUMI_OK;
}

}  // namespace lumi
