// The product of prompt rows with fp32 activations on the 5th-generation tensor cores: D[M][N] (+)= A[M][K] W[N][K]^T, W in fp32 or bf16, results as
// close to 64 bits as fp32 multiply-adds give them.
//
// Every fp32 operand is the exact sum of three bf16 numbers (8 bits each, together the 24 of fp32); bf16 weights are one such number.  Of the nine
// products of planes the six that reach fp32's last bit are taken (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi: what is left out is 2^-24 of a
// product).  Products of bf16 numbers are exact; what the tensor core loses is in its sums, which it cuts off instead of rounding: 1e-6 over K =
// 1024 in one accumulator, 4e-8 over 32.  So the hi hi products go 32 of K at a time into an empty accumulator, which eight warps take out and add up in
// fp32; the other five, 2^-8 of the size and with them their error, stay in two accumulators for 256 of K.  What was cut off has the sign of the sum, so
// it adds up where operands have one sign; its average is put back (with_cut).
// The order of a sum is fixed by K alone: two accumulators to a k-block of 64, four k-blocks and the small products to a group of 256, two groups to a
// pair, the pairs in order, wherever K is split and however many rows there are; a row's results are the same bits alone and among others.  Error
// against 64 bits (root mean square, of the results'), K = 128 / 1024 / 2048 / 2816, beside the fp32 multiply-adds that did this before: operands of both signs
// 5.6 / 7.3 / 7.9 / 8.4e-8 (8.8 / 10.1 / 10.6 / 11.0), of one sign 4.8 / 4.7 / 4.8 / 5.2e-8 (4.8 / 4.7 / 4.7 / 5.1), with a mean of two deviations 3.9 / 3.7 / 4.3 / 5.2e-8
// (4.2 / 3.9 / 4.2 / 5.1).  (Groups of 256 one by one and nothing put back: 6.4 / 8.0 / 8.9 / 9.5, 6.3 / 6.2 / 6.4 / 6.9, 4.5 / 4.3 / 5.0 / 5.7e-8.)
//
// The weights take the 128-row side of the MMA, NB rows of the prompt the other; products with two planes of the same weights go as one MMA of twice the
// width.  Warps 0 - 6: a k-block, copied densely to shared memory ahead of time, to registers and split into planes as the MMA reads them (K-major, 128-byte
// swizzle; bf16 weights are copied straight to their plane).  Warp 7: TMEM, MMA.  Warps 8 - 15: accumulators, sums, results.
// What bounds it: the splitting (15 pieces of four elements per thread and k-block of 64, 1600 of 2700 cycles), then the MMAs (16 per k-block of 100 cycles,
// operand reads).  At the cap of 128 registers the 64-row tiles load 76 bytes of spills a thread, the held group above all.  Launches back to back, weights
// from memory, against packed fp32 multiply-adds on the CUDA cores, microseconds: fp32 weights 384 x 7360 x 1024 177 -> 84, 384 x 1024 x 2048 129 -> 31, 384 x
// 32000 x 1024 692 -> 309, 960 x 7360 x 1024 401 -> 167, 32 x 7360 x 1024 30 -> 21, 32 x 1024 x 2048 15 -> 16; bf16 weights 384 x 7360 x 1024 175 -> 60, 32 x
// 7360 x 1024 27 -> 16.  Scores of 4 x 96 tokens, 48 layers in fp32: 16.6 -> 10.1 ms; a bf16 prompt of 100 tokens 10.0 -> 6.1 ms.
#include "internal.h"
#include "tcgen05.cuh"

#include <algorithm>

namespace lumi {

int32_t make_f32_map_2d(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_cols, uint32_t box_rows);
int32_t make_bf16_operand_map(CUtensorMap* map, const void* ptr, int rows, int K, int box_rows);

namespace {

constexpr int kLoadWarps = 7, kSumWarps = 8, kFirstSum = kLoadWarps + 1, kThreads = 32 * (kFirstSum + kSumWarps);      // 128 registers each
constexpr int kWRows = 128;                  // weight rows of a tile
constexpr int kGroupBlocks = 4;              // k-blocks of 64 to a group
constexpr int kAccs = 4;
constexpr int kAccK = 32;                    // K that goes into an accumulator before it is taken out

template <int NB, typename WT>
struct RowsTile {
    static constexpr int PW = sizeof(WT) == 4 ? 3 : 1;                    // planes of W
    static constexpr int W_PLANE = kWRows * BK * 2, A_PLANE = NB * BK * 2;
    static constexpr int STAGE = PW * W_PLANE + 3 * A_PLANE, STAGES = PW == 3 ? 2 : 3;
    static constexpr int RAW_W = PW == 3 ? kWRows * BK * 4 : 0, RAW = RAW_W + NB * BK * 4;      // a k-block as it lies in memory (bf16 weights: straight to their plane)
    static constexpr int RAWS = STAGES * STAGE, TOTALS = RAWS + RAW;      // sums of the groups before: [column][thread]
    static constexpr int BARS = TOTALS + kWRows * NB * 4;
    static constexpr int SMEM = BARS + 256 + 1024;
    static constexpr uint32_t COLS = NB == 64 ? 512 : 256;                // TMEM: kAccs accumulators, two times two of the small products
    static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
};

// pairs of fp32 numbers
__device__ __forceinline__ uint64_t pair2(uint32_t a, uint32_t b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
// a - b as one multiply-add by -1 (as a + (-b) the halves of b needed their signs turned first)
__device__ __forceinline__ uint64_t minus2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return d;
}
__device__ __forceinline__ float first_of(uint64_t d) { return __uint_as_float((uint32_t)d); }
__device__ __forceinline__ float second_of(uint64_t d) { return __uint_as_float((uint32_t)(d >> 32)); }

// What joins a group's sum h of hi hi products, with what the tensor core cut off of them: half a last place of every sum of 32 on the average, always toward
// zero, which in a group of such sums is about half a last place of h.  0.4 of one is put back (0.5 serves sums near a power of two, 0.3 those with a
// mantissa near 1.6).  Sums whose last three bits are zero have lost nothing as a rule (whole numbers, rows with a single entry) and stay exact.
__device__ __forceinline__ uint32_t with_cut(float h, float small) {
    const uint32_t b = __float_as_uint(h);
    return __float_as_uint(fmaf(__uint_as_float(b & 0xff800000u), (b & 7u) != 0 ? 0.4f * 1.1920929e-7f : 0.f, small));
}

// CW columns of this warp's 32 lanes of TMEM, in pairs
template <int CW>
__device__ __forceinline__ void tmem_pairs(uint32_t taddr, uint64_t (&v)[CW / 2]) {
    if constexpr (CW == 32) {
        uint32_t r[32];
        tmem_ld32(taddr, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = pair2(r[2 * j], r[2 * j + 1]);
    } else {
        static_assert(CW == 16, "half of a tile's columns");
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = pair2(r[2 * j], r[2 * j + 1]);
    }
}

// Four consecutive elements into their planes.  x = hi + mid + lo exactly: hi the nearest bf16, mid the upper eight bits of what is left, lo the eight behind
// them.  (Nearest for the first, so that mid has either sign and the products left out do not all have the sign of theirs.)  What is infinite, or
// above bf16's largest number (3.39e38), has planes that are no numbers: such sums are taken again (plain_result).
__device__ __forceinline__ void store_planes(const float4& a, uint8_t* at, int plane) {
    uint64_t r[2] = {pair2(__float_as_uint(a.x), __float_as_uint(a.y)), pair2(__float_as_uint(a.z), __float_as_uint(a.w))};
    uint32_t w[3][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(first_of(r[e]), second_of(r[e]));
        w[0][e] = *reinterpret_cast<const uint32_t*>(&h);
        r[e] = minus2(r[e], pair2(w[0][e] << 16, w[0][e] & 0xffff0000u));                  // the two halves, widened
        const uint32_t m0 = (uint32_t)r[e], m1 = (uint32_t)(r[e] >> 32);
        w[1][e] = __byte_perm(m0, m1, 0x7632);
        r[e] = minus2(r[e], pair2(m0 & 0xffff0000u, m1 & 0xffff0000u));
        w[2][e] = __byte_perm((uint32_t)r[e], (uint32_t)(r[e] >> 32), 0x7632);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * plane) = make_uint2(w[p][0], w[p][1]);
}
// One operand's ROWS rows of a k-block, from the dense copy of it into planes (K-major, 128-byte swizzle): sixteen threads take a row's pieces of four.  The
// threads do not divide the rows evenly; those left over in the last turn take the last row once more, the same bytes to the same place, so that
// there is no branch between the pieces and their chains of operations overlap.
template <int ROWS>
struct Pieces {
    static constexpr int STEP = 2 * kLoadWarps, UNITS = (ROWS + STEP - 1) / STEP;
    float4 v[UNITS];
    __device__ __forceinline__ int row(int i, int tid) const { return min((tid >> 4) + STEP * i, ROWS - 1); }
    __device__ __forceinline__ void load(const uint8_t* raw, int tid) {
#pragma unroll
        for (int i = 0; i < UNITS; ++i) v[i] = *reinterpret_cast<const float4*>(raw + row(i, tid) * 256 + (tid & 15) * 16);
    }
    __device__ __forceinline__ void store(uint8_t* st, int plane, int tid) const {
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
            const int r = row(i, tid);
            store_planes(v[i], st + r * 128 + ((((tid & 15) >> 1) ^ (r & 7)) << 4) + (tid & 1) * 8, plane);
        }
    }
};

// One result by fp32 multiply-adds: chains of 16, eight to a unit, four units to a group, the groups in order.  For sums of planes that are not finite: an infinite
// operand has planes that are no numbers, one above bf16's largest number an infinite one, though the result may be infinite or finite.
template <typename WT>
__device__ __forceinline__ float plain_result(const float* a, const WT* w, int K) {
    float total = 0.f;
    for (int k0 = 0; k0 < K; k0 += 512) {
        float group = 0.f;
        for (int k1 = k0; k1 < min(K, k0 + 512); k1 += 128) {
            float unit = 0.f;
            for (int k = k1; k < min(K, k1 + 128); k += 16) {
                float chain = 0.f;
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(a + k + e);
                    float4 y;
                    if constexpr (sizeof(WT) == 4) {
                        y = *reinterpret_cast<const float4*>(w + k + e);
                    } else {
                        const uint2 v = *reinterpret_cast<const uint2*>(w + k + e);
                        y = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
                    }
                    chain = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, chain))));
                }
                if (chain != chain) return chain;                       // no number stays none: rows without numbers cost little
                unit += chain;
            }
            group += unit;
        }
        total += group;
    }
    return total;
}

template <int NB, typename WT>
__global__ void __launch_bounds__(kThreads, 1) row_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, RowGemmArgs g, int groups_per_split) {
    using T = RowsTile<NB, WT>;
    constexpr int CW = NB / 2, kStages = T::STAGES;                       // CW: columns of a sum warp
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + T::BARS);
    uint64_t *empty = full + kStages, *acc_full = empty + kStages, *acc_empty = acc_full + kAccs, *small_full = acc_empty + kAccs, *small_empty = small_full + 2;
    uint64_t *drain = small_empty + 2, *raw_full = drain + 1, *raw_empty = raw_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + 1);
    int* last = reinterpret_cast<int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * kWRows, m0 = blockIdx.y * NB;
    const int blocks = (g.K + BK - 1) / BK, groups = (blocks + kGroupBlocks - 1) / kGroupBlocks;
    const int g0 = blockIdx.z * groups_per_split, g1 = min(groups, g0 + groups_per_split);
    const int kb0 = g0 * kGroupBlocks, kb1 = min(blocks, g1 * kGroupBlocks);

    const bool split = gridDim.z > 1;
    const int tile = blockIdx.y * gridDim.x + blockIdx.x;
    // K split: every CTA of a tile arrives at its counter, also one that has nothing to add, and the last one leaves it at zero for the next product
    auto arrive = [&]() {
        const bool is_last = atomicAdd(g.counters + tile, 1) == (int)gridDim.z - 1;
        if (is_last) g.counters[tile] = 0;
        return is_last;
    };
    // a wait that expired in an earlier launch, or in an earlier CTA of this one: no new work
    if (__syncthreads_or(g.status != nullptr && (*reinterpret_cast<volatile int32_t*>(g.status) & STATUS_TIMEOUT))) {
        if (split && threadIdx.x == 0) arrive();
        return;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], kLoadWarps + (T::PW == 1 ? 1 : 0)); mbar_init(&empty[i], 1); }
        for (int i = 0; i < kAccs; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], kSumWarps); }
        for (int i = 0; i < 2; ++i) { mbar_init(&small_full[i], 1); mbar_init(&small_empty[i], kSumWarps); }
        mbar_init(drain, 1);
        mbar_init(raw_full, 1);
        mbar_init(raw_empty, kLoadWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kLoadWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    bool timed_out = false;

    if (warp < kLoadWarps) {
        // a k-block arrives in one piece (rows and K past the end as zeros); once it is in registers the next one is on its way
        uint8_t* const raw = base + T::RAWS;
        const bool issues = threadIdx.x == 0;
        int requested = 0;
        auto request = [&](int kb) {
            ++requested;
            mbar_expect_tx(raw_full, (uint32_t)T::RAW);
            if constexpr (T::PW == 3) tma_load_2d(raw, &map_w, raw_full, kb * BK, n0);
            tma_load_2d(raw + T::RAW_W, &map_a, raw_full, kb * BK, m0);
        };
        auto request_w = [&](int kb) {                                    // bf16 weights need no splitting
            const int it = kb - kb0, s = it % kStages;
            if (!mbar_wait(&empty[s], (uint32_t)((it / kStages) & 1) ^ 1u)) return false;
            mbar_expect_tx(&full[s], (uint32_t)T::W_PLANE);
            tma_load_2d(base + s * T::STAGE, &map_w, &full[s], kb * BK, n0);
            return true;
        };
        int w_next = kb0;                                                 // (this thread) the next block of bf16 weights to be requested
        if (issues && tile + (int)(blockIdx.z * gridDim.x * gridDim.y) >= g.skip_units) {      // (test hook: nothing is asked for, and every wait runs out)
            request(kb0);
            if constexpr (T::PW == 1) for (; w_next < min(kb1, kb0 + kStages); ++w_next) request_w(w_next);
        }
        for (int kb = kb0; kb < kb1; ++kb) {
            const int it = kb - kb0, s = it % kStages;
            if (!mbar_wait(raw_full, (uint32_t)(it & 1))) timed_out = true;
            if (__any_sync(0xffffffffu, timed_out)) { timed_out = true; break; }
            Pieces<T::PW == 3 ? kWRows : 16> w;
            Pieces<NB> a;
            if constexpr (T::PW == 3) w.load(raw, threadIdx.x);
            a.load(raw + T::RAW_W, threadIdx.x);
            __syncwarp();
            if (lane == 0) mbar_arrive(raw_empty);
            if (issues && kb + 1 < kb1) {
                if (mbar_wait(raw_empty, (uint32_t)(it & 1))) request(kb + 1);
                else timed_out = true;
            }
            if (!mbar_wait(&empty[s], (uint32_t)((it / kStages) & 1) ^ 1u)) timed_out = true;
            if (__any_sync(0xffffffffu, timed_out)) { timed_out = true; break; }
            uint8_t* const st = base + s * T::STAGE;
            if constexpr (T::PW == 3) w.store(st, T::W_PLANE, threadIdx.x);
            a.store(st + T::PW * T::W_PLANE, T::A_PLANE, threadIdx.x);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if constexpr (T::PW == 1) {
                // the stage that the block before this one used: the MMA is done with it soon
                if (issues && it > 0 && w_next < kb1) {
                    if (request_w(w_next)) ++w_next;
                    else timed_out = true;
                }
            }
        }
        if (timed_out && issues) {                                        // let the copies land (bounded) that nobody may wait for
            mbar_wait(raw_full, (uint32_t)((requested - 1) & 1));
            if constexpr (T::PW == 1)
                for (int k = max(kb0, w_next - kStages); k < w_next; ++k) mbar_wait(&full[(k - kb0) % kStages], (uint32_t)(((k - kb0) / kStages) & 1));
        }
    } else if (warp == kLoadWarps) {
        if (lane == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
            constexpr uint32_t idesc2 = idesc + ((uint32_t)(NB >> 3) << 17);      // two planes of the activations, one behind the other in shared memory
            int step = 0;                                                 // kAccK of K each
            for (int kb = kb0; kb < kb1 && !timed_out; ++kb) {
                const int it = kb - kb0, s = it % kStages, grp = it / kGroupBlocks, first = it % kGroupBlocks == 0;
                if (!mbar_wait(&full[s], (uint32_t)((it / kStages) & 1))) { timed_out = true; break; }
                const uint32_t small = tmem + (uint32_t)((kAccs + 2 * (grp & 1)) * NB);
                if (first && !mbar_wait(&small_empty[grp & 1], (uint32_t)((grp / 2) & 1) ^ 1u)) { timed_out = true; break; }
                tc_fence_after();
                const uint32_t w = smem_u32(base + s * T::STAGE), a = w + T::PW * T::W_PLANE;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) {
                    const int acc = step % kAccs;
                    const bool fresh = k % (kAccK / 16) == 0, done = (k + 1) % (kAccK / 16) == 0;
                    if (fresh) {
                        if (!mbar_wait(&acc_empty[acc], (uint32_t)((step / kAccs) & 1) ^ 1u)) { timed_out = true; break; }
                        tc_fence_after();
                    }
                    auto wd = [&](int p) { return make_smem_desc(w + p * T::W_PLANE + k * 32); };
                    auto ad = [&](int p) { return make_smem_desc(a + p * T::A_PLANE + k * 32); };
                    umma_bf16(tmem + (uint32_t)(acc * NB), wd(0), ad(0), idesc, fresh ? 0u : 1u);
                    if (done) { umma_commit(&acc_full[acc]); ++step; }
                    // the small ones two planes of the activations at a time: [hi mid | hi lo] + [mid hi | mid mid], then lo hi onto the first
                    umma_bf16(small, wd(0), ad(1), idesc2, first && k == 0 ? 0u : 1u);
                    if (T::PW > 1) {
                        umma_bf16(small, wd(T::PW / 2), ad(0), idesc2, 1u);
                        umma_bf16(small, wd(T::PW - 1), ad(0), idesc, 1u);
                    }
                }
                if (timed_out) break;
                umma_commit(&empty[s]);
                if (it % kGroupBlocks == kGroupBlocks - 1 || kb + 1 == kb1) umma_commit(&small_full[grp & 1]);
            }
            if (timed_out) {                                              // let every MMA issued so far finish (bounded) before TMEM is freed
                umma_commit(drain);
                mbar_wait(drain, 0);
            }
        }
    } else {
        const int q = warp & 3, half = (warp - kFirstSum) >> 2;          // TMEM lane quarter, half of the columns
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * CW);
        const int n = n0 + q * 32 + lane, mc = m0 + half * CW, tid = threadIdx.x - 32 * kFirstSum;
        float* const total = reinterpret_cast<float*>(base + T::TOTALS) + tid;             // 256 apart
        float* const parts = g.scratch + (size_t)tile * groups * kWRows * NB + tid;        // K split: the groups' sums
        const int cols = n < g.N ? max(0, min(CW, g.M - mc)) : 0;                          // of this thread that exist
        float* const out = g.D + (size_t)mc * g.ldd + n;
        uint32_t again = 0;                                                                // columns whose sums are not finite: taken again below
        auto put8 = [&](int c, const float (&v)[8]) {                                      // columns c .. c + 7
            float old[8];
            if (cols >= c + 8) {
#pragma unroll
                for (int j = 0; j < 8; ++j) old[j] = g.accumulate ? out[(size_t)(c + j) * g.ldd] : 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const bool finite = v[j] - v[j] == 0.f;
                    if (!finite) again |= 1u << (c + j);
                    out[(size_t)(c + j) * g.ldd] = !finite ? old[j] : g.accumulate ? old[j] + v[j] : v[j];
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (c + j < cols) {
                        const float o = g.accumulate ? out[(size_t)(c + j) * g.ldd] : 0.f;
                        const bool finite = v[j] - v[j] == 0.f;
                        if (!finite) again |= 1u << (c + j);
                        out[(size_t)(c + j) * g.ldd] = !finite ? o : g.accumulate ? o + v[j] : v[j];
                    }
            }
        };
        float held[CW];                                                                    // an even group's sum, until its neighbour's is there
        int step = 0;
        for (int gr = g0; gr < g1 && !timed_out; ++gr) {
            const int gi = gr - g0, kbe = min(blocks, (gr + 1) * kGroupBlocks);
            uint64_t sum[CW / 2], unit[CW / 2];                                            // unit: the last k-block's, not yet in sum
#pragma unroll
            for (int j = 0; j < CW / 2; ++j) sum[j] = unit[j] = 0;
#pragma unroll 1
            for (int kb = gr * kGroupBlocks; kb < kbe && !timed_out; ++kb) {
#pragma unroll
                for (int j = 0; j < CW / 2; ++j) sum[j] = add2(sum[j], unit[j]);
#pragma unroll
                for (int t = 0; t < BK / kAccK; ++t, ++step) {
                    const int acc = step % kAccs;
                    if (!mbar_wait(&acc_full[acc], (uint32_t)((step / kAccs) & 1))) timed_out = true;
                    timed_out = __any_sync(0xffffffffu, timed_out);
                    if (timed_out) break;
                    tc_fence_after();
                    uint64_t v[CW / 2];
                    tmem_pairs<CW>(lanes + (uint32_t)(acc * NB), v);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[acc]);
#pragma unroll
                    for (int j = 0; j < CW / 2; ++j) unit[j] = t == 0 ? v[j] : add2(unit[j], v[j]);
                }
            }
            if (timed_out) break;
            if (!mbar_wait(&small_full[gi & 1], (uint32_t)((gi / 2) & 1))) timed_out = true;
            timed_out = __any_sync(0xffffffffu, timed_out);
            if (timed_out) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < CW / 2; c += 8) {                                          // sixteen columns at a time
                uint64_t v[8], u[8];
                tmem_pairs<16>(lanes + (uint32_t)((kAccs + 2 * (gi & 1)) * NB + 2 * c), v);
                tmem_pairs<16>(lanes + (uint32_t)((kAccs + 2 * (gi & 1) + 1) * NB + 2 * c), u);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint64_t s = add2(v[j], u[j]), h = add2(sum[c + j], unit[c + j]);
                    sum[c + j] = add2(sum[c + j], add2(unit[c + j], pair2(with_cut(first_of(h), first_of(s)), with_cut(second_of(h), second_of(s)))));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&small_empty[gi & 1]);
            float grp[CW];
#pragma unroll
            for (int j = 0; j < CW / 2; ++j) { grp[2 * j] = first_of(sum[j]); grp[2 * j + 1] = second_of(sum[j]); }
            if (split) {
#pragma unroll
                for (int j = 0; j < CW; ++j) parts[(size_t)gr * kWRows * NB + j * 256] = grp[j];
            } else if (gr % 2 == 0 && gr + 1 < g1) {
#pragma unroll
                for (int j = 0; j < CW; ++j) held[j] = grp[j];
            } else {
#pragma unroll
                for (int j = 0; j < CW; ++j) {
                    const float two = gr % 2 == 0 ? grp[j] : held[j] + grp[j];
                    total[j * 256] = gr < 2 ? two : total[j * 256] + two;
                }
            }
        }
        // a wait ran out: what is missing is no number, so that plain multiply-adds put it right where the last CTA of the tile still comes to it
        if (timed_out)
#pragma unroll 1
            for (int j = 0; j < CW; ++j) {
                if (!split) total[j * 256] = __int_as_float(0x7fffffff);
                else
                    for (int gr = g0; gr < g1; ++gr) parts[(size_t)gr * kWRows * NB + j * 256] = __int_as_float(0x7fffffff);
            }
        bool puts = true;
        if (split) {
            // the last CTA of the tile to arrive adds the groups as above
            __threadfence();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (tid == 0) *last = arrive();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            puts = *last;
            __threadfence();
        }
        if (puts)                                                                          // (in a loop: unrolled it was a third of the kernel's code, run once)
#pragma unroll 1
            for (int c = 0; c < CW; c += 8) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) if (!split) v[j] = total[(c + j) * 256];
                for (int z = 0; split && z < groups; z += 4) {                             // four groups' loads in flight
                    float u[4][8];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) u[i][j] = z + i < groups ? __ldcg(parts + (size_t)(z + i) * kWRows * NB + (c + j) * 256) : 0.f;
#pragma unroll
                    for (int i = 0; i < 4; i += 2)
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = z + i == 0 ? u[i][j] + u[i + 1][j] : v[j] + (u[i][j] + u[i + 1][j]);
                }
                put8(c, v);
            }
        for (; again != 0; again &= again - 1) {
            const int c = __ffs(again) - 1;
            float* const at = out + (size_t)c * g.ldd;
            const float x = plain_result(g.A + (size_t)(mc + c) * g.lda, static_cast<const WT*>(g.W) + (size_t)n * g.K, g.K);
            *at = g.accumulate ? *at + x : x;
        }
    }
    if (timed_out && g.status != nullptr) atomicOr(g.status, STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == kLoadWarps) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::COLS) : "memory");
    }
}

int sms() {
    static const int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        return v;
    }();
    return n;
}

template <int NB, typename WT>
cudaError_t launch_t(const RowGemmArgs& g, dim3 grid, int per, cudaStream_t st) {
    using T = RowsTile<NB, WT>;
    CUtensorMap ma, mw;
    if (make_f32_map_2d(&ma, g.A, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda * 4, BK, NB) != LUMI_OK) return cudaErrorInvalidValue;
    if ((sizeof(WT) == 4 ? make_f32_map_2d(&mw, g.W, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.K * 4, BK, kWRows)
                         : make_bf16_operand_map(&mw, g.W, g.N, g.K, kWRows)) != LUMI_OK) return cudaErrorInvalidValue;
    const cudaError_t e = cudaFuncSetAttribute(row_gemm_kernel<NB, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (e != cudaSuccess) return e;
    row_gemm_kernel<NB, WT><<<grid, kThreads, T::SMEM, st>>>(ma, mw, g, per);
    return cudaGetLastError();
}

}  // namespace

bool row_gemm_supported(int K) { return K >= 16 && K % 16 == 0; }

cudaError_t launch_row_gemm(const RowGemmArgs& g, cudaStream_t st) {
    if (!row_gemm_supported(g.K) || g.lda % 4 != 0) return cudaErrorInvalidValue;
    // Tile height and split of K with the least rounds of one CTA per SM times a CTA's walk (a k-block of the 32-row tile takes 0.7 of the 64-row one's
    // time, the rest of a CTA about as long as three blocks)
    const int blocks = (g.K + BK - 1) / BK, groups = (blocks + kGroupBlocks - 1) / kGroupBlocks;
    int best_nb = 64, best_per = groups;
    double best = -1.0;
    for (int nb : {64, 32})
        for (int per = groups; per >= 1; --per) {
            const int splits = (groups + per - 1) / per;
            const long tiles = (long)((g.M + nb - 1) / nb) * ((g.N + kWRows - 1) / kWRows);
            if (splits > 1 && (tiles > g.n_counters || (size_t)tiles * groups * kWRows * nb > g.scratch_floats)) continue;
            const double cost = (double)((tiles * splits + sms() - 1) / sms()) * ((nb == 64 ? 1.0 : 0.7) * std::min(blocks, per * kGroupBlocks) + (splits > 1 ? 4.0 : 3.0));
            if (best < 0 || cost < 0.97 * best) { best = cost; best_nb = nb; best_per = per; }
        }
    const dim3 grid((g.N + kWRows - 1) / kWRows, (g.M + best_nb - 1) / best_nb, (groups + best_per - 1) / best_per);
    if (g.w_dtype == LUMI_DTYPE_BF16) return best_nb == 64 ? launch_t<64, __nv_bfloat16>(g, grid, best_per, st) : launch_t<32, __nv_bfloat16>(g, grid, best_per, st);
    return best_nb == 64 ? launch_t<64, float>(g, grid, best_per, st) : launch_t<32, float>(g, grid, best_per, st);
}

}  // namespace lumi
