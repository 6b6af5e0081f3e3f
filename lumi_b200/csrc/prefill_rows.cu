// Prompts a layer at a time where the chunked scan does not apply: fp32 weights, short prompts, other head shapes.
//
// Fed token by token (inference/src/main.rs:121-125), a prompt of T tokens reads every weight T times.  Taken a layer at a
// time it reads them once: the projections become products over all rows (`launch_row_gemm` for fp32 activations, the tensor-core
// product for bf16 halves), and only the recurrence runs in token order (`ssm_rows_kernel`, the decode step's arithmetic with
// the state in registers).
//
// Measured on the 48-layer base model: scoring 4 x 96 tokens in fp32 125.5 -> 16.7 ms, a 32-token prompt of one sequence
// with the step behind it 4.8 ms in fp32 (token by token 16.7 without the step) and 20.9 -> 4.6 ms in bf16; twelve bf16 sequences of 100 tokens
// (halves) 10.4 ms.
#include "internal.h"

namespace lumi {
namespace {

// ---- product over rows with fp32 activations ---------------------------------------------------------------
// D[M][N] (+)= A[M][K] W[N][K]^T on the CUDA cores, fp32 throughout (bf16 weights are widened).  A CTA of 128 threads owns BM x 64 results and, with K split
// over blockIdx.z, part of the sum; a thread owns TM x 8 of them, rows sixteen and columns eight apart, so that the eight columns that a
// quarter warp reads lie in eight different bank groups (rows of 32 + 4 padding floats).  Even and odd k are summed apart in
// the two halves of packed multiply-adds (fma.rn.f32x2): operands come as 16-byte loads along K as they are stored, with no
// transposition, and one instruction does two multiply-adds.
// The order of a sum is fixed by K alone: chains of 16 products (32 of K, even and odd apart), four of them added up to a unit of 128 of K,
// four units to a group, the groups in order, wherever K is split and however many rows there are; a row's results are the same bits alone
// and among others.  With one running sum per half for 128 of K at a time prompts were further from 64 bits than token by token (48-layer base
// model, logits of a 9-token prompt 2.2e-6 against 1.6e-6, scores of 8 x 120 tokens 1.0e-7 against 0.86e-7); this order comes to 1.6e-6 and 0.82e-7.
// What bounds it: shared-memory reads at many rows (a 16-byte load for five packed multiply-adds), the stream of the weights at few.  Measured: 384 x
// 32000 x 1024 in 697 us (half of the FMA pipe's 36 T/s), 384 x 7360 x 1024 in 178 us, 384 x 1024 x 2048 in 71 us.  A thread's tile of 8 x 8 with the unit's
// sums in registers spills (225 us for the second), with them in shared memory its copies cost as much (220 us).
constexpr int kBK = 32, kPad = kBK + 4, kBN = 64, kUnit = 4, kGroup = 4, kStages = 2;      // kUnit: blocks of kBK; kGroup: units

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float halves_sum(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {      // bytes 0: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// four consecutive weights of a staged row as two packed pairs
__device__ __forceinline__ ulonglong2 weights4(const float* w) { return *reinterpret_cast<const ulonglong2*>(w); }
__device__ __forceinline__ ulonglong2 weights4(const __nv_bfloat16* w) {
    const uint2 v = *reinterpret_cast<const uint2*>(w);
    auto pair = [](uint32_t two) { return (uint64_t)(two & 0xffff0000u) << 32 | (uint64_t)(two << 16); };
    return make_ulonglong2(pair(v.x), pair(v.y));
}

template <int TM, typename WT>
struct RowTile {
    static constexpr int BM = 16 * TM, E = 16 / (int)sizeof(WT), W_PITCH = kBK + E;      // rows of weights: 32 and one 16-byte piece
    static constexpr int A_BYTES = BM * kPad * 4, STAGE = A_BYTES + kBN * W_PITCH * (int)sizeof(WT);
    static constexpr int SMEM = kStages * STAGE + 2 * BM * kBN * 4;        // TM 4: 68 KiB, with bf16 weights 60: three CTAs per SM
};

template <int TM, typename WT>
__global__ void __launch_bounds__(128, TM == 4 ? 3 : 4) row_gemm_kernel(RowGemmArgs g, int units_per_split) {
    using T = RowTile<TM, WT>;
    constexpr int BM = T::BM, E = T::E, TILE4 = BM * kBN / 4;
    extern __shared__ __align__(16) unsigned char sm[];                    // [stage][A rows, then W rows], the group's sums, the sums of the groups before
    const int tid = threadIdx.x, tn = tid & 7, tm = tid >> 3;
    const int n0 = blockIdx.x * kBN, m0 = blockIdx.y * BM;
    const int blocks = (g.K + kBK - 1) / kBK, units = (blocks + kUnit - 1) / kUnit;
    const int kb0 = blockIdx.z * units_per_split * kUnit, kb1 = min(blocks, kb0 + units_per_split * kUnit);
    const bool split = gridDim.z > 1;
    // this thread copies 16 bytes at column cq of every sixteenth row; rows past the end read the last one: never stored
    const int cq = 4 * (tid & 7), crow = tid >> 3, a_end = g.M - 1 - m0, w_end = g.N - 1 - n0;
    constexpr int WQ = kBK / E, WSTEP = 128 / WQ;                          // the same for the weights: pieces per row, rows per turn
    const int wq = E * (tid % WQ), wrow = tid / WQ;
    const float* const a0 = g.A + (size_t)m0 * g.lda + cq;
    const WT* const w0 = static_cast<const WT*>(g.W) + (size_t)n0 * g.K + wq;
    auto stage = [&](int kb) {
        if (kb < kb1) {
            unsigned char* s = sm + (kb & 1) * T::STAGE;
            float* sa = reinterpret_cast<float*>(s) + crow * kPad + cq;
            WT* sw = reinterpret_cast<WT*>(s + T::A_BYTES) + wrow * T::W_PITCH + wq;
            const bool ain = kb * kBK + cq < g.K, win = kb * kBK + wq < g.K;      // K is a multiple of 16: the last block may be half zeros
#pragma unroll
            for (int c = 0; c < BM / 16; ++c) copy16(sa + 16 * c * kPad, a0 + min(crow + 16 * c, a_end) * g.lda + (ain ? kb * kBK : 0), ain ? 16 : 0);
#pragma unroll
            for (int c = 0; c < kBN / WSTEP; ++c)
                copy16(sw + WSTEP * c * T::W_PITCH, w0 + min(wrow + WSTEP * c, w_end) * g.K + (win ? kb * kBK : 0), win ? 16 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint64_t mid[TM][8];                                                   // the unit's chains so far
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) mid[i][j] = 0ull;
    float4* const group_sum = reinterpret_cast<float4*>(sm + kStages * T::STAGE) + tid;      // this thread's results four by four, 128 apart
    float4* const total = group_sum + TILE4;
    const int tile = blockIdx.y * gridDim.x + blockIdx.x;
    float4* const parts = reinterpret_cast<float4*>(g.scratch) + (size_t)tile * units * TILE4 + tid;      // K split: the units' sums
    stage(kb0);
    for (int kb = kb0; kb < kb1; ++kb) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                                   // the block has landed, and the one before it is no longer read
        stage(kb + 1);
        const float* sa = reinterpret_cast<const float*>(sm + (kb & 1) * T::STAGE) + tm * kPad;
        const WT* sw = reinterpret_cast<const WT*>(sm + (kb & 1) * T::STAGE + T::A_BYTES) + tn * T::W_PITCH;
        uint64_t acc[TM][8];
#pragma unroll
        for (int q = 0; q < kBK / 4; ++q) {
            ulonglong2 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(sa + 16 * i * kPad + 4 * q);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 w = weights4(sw + 8 * j * T::W_PITCH + 4 * q);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fma2(a[i].y, w.y, q == 0 ? mul2(a[i].x, w.x) : fma2(a[i].x, w.x, acc[i][j]));
            }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) mid[i][j] = add2(mid[i][j], acc[i][j]);
        if (kb % kUnit != kUnit - 1 && kb + 1 != blocks) continue;
        const int u = kb / kUnit;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int at = (2 * i + q) * 128;
                float4 v = make_float4(halves_sum(mid[i][4 * q]), halves_sum(mid[i][4 * q + 1]), halves_sum(mid[i][4 * q + 2]), halves_sum(mid[i][4 * q + 3]));
#pragma unroll
                for (int j = 0; j < 4; ++j) mid[i][4 * q + j] = 0ull;
                if (split) { parts[(size_t)u * TILE4 + at] = v; continue; }
                if (u % kGroup != 0) v = add4(group_sum[at], v);
                if (u % kGroup != kGroup - 1 && u + 1 != units) group_sum[at] = v;
                else total[at] = u < kGroup ? v : add4(total[at], v);
            }
    }
    auto put4 = [&](int i, int q, float4 v) {
        const float* e = &v.x;
        const int m = m0 + tm + 16 * i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tn + 8 * (4 * q + j);
            if (m < g.M && n < g.N) {
                float* d = g.D + (size_t)m * g.ldd + n;
                *d = g.accumulate ? *d + e[j] : e[j];
            }
        }
    };
    if (!split) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) put4(i, q, total[(2 * i + q) * 128]);
        return;
    }
    // the last CTA of the tile to arrive adds the units as above
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        last = atomicAdd(g.counters + tile, 1) == (int)gridDim.z - 1;
        if (last) g.counters[tile] = 0;                                    // ready for the next product
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    float4 sum[TM][2];
    for (int u0 = 0; u0 < units; u0 += kGroup) {
        float4 grp[TM][2];
#pragma unroll
        for (int z = 0; z < kGroup; ++z) {
            if (u0 + z >= units) break;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float4 v = __ldcg(parts + (size_t)(u0 + z) * TILE4 + (2 * i + q) * 128);
                    grp[i][q] = z == 0 ? v : add4(grp[i][q], v);
                }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) sum[i][q] = u0 == 0 ? grp[i][q] : add4(sum[i][q], grp[i][q]);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) put4(i, q, sum[i][q]);
}

// ---- the recurrence over prompt rows --------------------------------------------------------------------------
// The decode step's forms (inference/src/model.rs:307-317, 338-370).
__device__ __forceinline__ float sigmoid_ref(float x) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x))); }
__device__ __forceinline__ float softplus_ref(float x) { return logf(__fadd_rn(expf(x), 1.0f)); }
__device__ __forceinline__ float silu_ref(float x) { return __fdiv_rn(x, __fadd_rn(1.0f, expf(-x))); }

constexpr int kTok = 16;             // tokens taken through the pointwise part at a time
template <int P, int N>
struct alignas(16) RowsSmem {          // B~ and C~ are read sixteen bytes at a time
    float bt[kTok][N], ct[kTok][N], xa[kTok][P], gate[kTok][P], yo[kTok][P], ang[kTok][N / 2];
    float dtp[kTok], abar[kTok], lam[kTok], c2[kTok], rb[kTok], rc[kTok];
};

// One CTA of 128 threads per (head, sequence).  Only the angle sum and the state are sequential; everything else of 16 tokens is
// computed side by side by all threads first (transcendentals are most of a step's instructions), then the 16 state updates follow
// with the head's tile in registers (P N / 128 values per thread) and B~, C~, x in shared memory.  Operation order and rounding of
// each step are ssm_step_kernel's; only the BCNorm sums run in another order.  Bound by the latency of that chain: a token costs
// one round of loads, four multiply-adds per value and a reduction over N / 4 lanes.  Measured (64 heads of 32 x 64): 0.6 us a token, 20 us for
// 32 tokens of one sequence, 62 us for 4 x 96; the step kernel takes 5 to 10 us for each token.
template <int P, int N>
__global__ void __launch_bounds__(128) ssm_rows_kernel(PrefillArgs a, float* y32) {
    constexpr int HN = N / 2, CG = N / 4, F = P * N / 512, RSTEP = 128 / CG;
    static_assert(P * N % 512 == 0 && CG <= 32, "whole 16-byte quads per thread, a row within a warp");
    __shared__ RowsSmem<P, N> sm;
    const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    const int H = a.H, DI = H * P, BC = a.G * N, g = h / (H / a.G);
    const int ts = a.lens != nullptr ? max(0, min(a.ts, a.lens[a.b0 + b] - a.t_abs0)) : a.ts;
    if (ts == 0) return;
    const size_t bh = (size_t)(a.b0 + b) * H + h, row0 = (size_t)b * a.ts;
    const int c = tid % CG, r0 = tid / CG;
    const float PI_F = 3.14159265358979323846f, TWO_PI = __fmul_rn(2.0f, PI_F);
    const float dskip = a.dskip[h], dtb = a.dtb[h];
    float4* h4 = reinterpret_cast<float4*>(a.h + bh * (size_t)(P * N));
    float4 st[F];
    float xp[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
        st[f] = h4[tid + 128 * f];
        xp[f] = a.xprev[bh * P + r0 + f * RSTEP];
    }
    float4 bp = reinterpret_cast<const float4*>(a.bprev + bh * N)[c];
    float cu = tid < HN ? a.cum[bh * HN + tid] : 0.f;

    for (int t0 = 0; t0 < ts; t0 += kTok) {
        const int nv = min(kTok, ts - t0);
        const float* pr0 = a.proj + (row0 + t0) * (size_t)a.ldp;
        if (tid < nv) {
            const float* dt = pr0 + (size_t)tid * a.ldp + 2 * DI + 2 * BC + h;
            const float dtp = softplus_ref(__fadd_rn(dt[0], dtb));
            const float av = fminf(fmaxf(-softplus_ref(dt[2 * H]), -1e6f), -1e-4f);
            const float abar = expf(__fmul_rn(av, dtp)), lam = sigmoid_ref(dt[H]);
            sm.dtp[tid] = dtp;
            sm.abar[tid] = abar;
            sm.lam[tid] = lam;
            sm.c2[tid] = __fmul_rn(abar, __fadd_rn(__fmul_rn(lam, -1.0f), 1.0f));
            sm.rb[tid] = a.rb[row0 + t0 + tid];
            sm.rc[tid] = a.rc[row0 + t0 + tid];
        }
        for (int e = tid; e < nv * P; e += 128) {
            const int i = e / P, p = e % P;
            const float* pr = pr0 + (size_t)i * a.ldp + h * P + p;
            sm.xa[i][p] = silu_ref(pr[0]);
            sm.gate[i][p] = silu_ref(pr[DI]);
        }
        __syncthreads();
        for (int e = tid; e < nv * HN; e += 128) {
            const int i = e / HN, k = e % HN;
            sm.ang[i][k] = __fmul_rn(sm.dtp[i], __fmul_rn(tanhf(pr0[(size_t)i * a.ldp + 2 * DI + 2 * BC + 3 * H + h * HN + k]), PI_F));
        }
        __syncthreads();
        if (tid < HN)                                      // the angles of one pair, token after token (model.rs:343)
            for (int i = 0; i < nv; ++i) {
                cu = __fadd_rn(cu, sm.ang[i][tid]);
                // fmod(cu, 2 pi): below 4 pi in magnitude it is the value itself or one exact subtraction
                if (fabsf(cu) >= TWO_PI) cu = fabsf(cu) < 2.f * TWO_PI ? (cu > 0.f ? __fsub_rn(cu, TWO_PI) : __fadd_rn(cu, TWO_PI)) : fmodf(cu, TWO_PI);
                sm.ang[i][tid] = cu;
            }
        __syncthreads();
        for (int e = tid; e < nv * HN; e += 128) {         // DD-RoPE (model.rs:346-350) of the normalised B and C
            const int i = e / HN, k = e % HN, q = g * N + 2 * k;
            const float* Bp = pr0 + (size_t)i * a.ldp + 2 * DI + q;
            const float rb = sm.rb[i], rc = sm.rc[i];
            const float b0 = __fadd_rn(__fmul_rn(__fmul_rn(Bp[0], rb), a.bg[q]), a.bb[q]);
            const float b1 = __fadd_rn(__fmul_rn(__fmul_rn(Bp[1], rb), a.bg[q + 1]), a.bb[q + 1]);
            const float c0 = __fadd_rn(__fmul_rn(__fmul_rn(Bp[BC], rc), a.cg[q]), a.cb[q]);
            const float c1 = __fadd_rn(__fmul_rn(__fmul_rn(Bp[BC + 1], rc), a.cg[q + 1]), a.cb[q + 1]);
            float sa, ca;
            sincosf(sm.ang[i][k], &sa, &ca);
            sm.bt[i][2 * k] = __fsub_rn(__fmul_rn(ca, b0), __fmul_rn(sa, b1));
            sm.bt[i][2 * k + 1] = __fadd_rn(__fmul_rn(sa, b0), __fmul_rn(ca, b1));
            sm.ct[i][2 * k] = __fsub_rn(__fmul_rn(ca, c0), __fmul_rn(sa, c1));
            sm.ct[i][2 * k + 1] = __fadd_rn(__fmul_rn(sa, c0), __fmul_rn(ca, c1));
        }
        __syncthreads();
#pragma unroll 2
        for (int i = 0; i < nv; ++i) {                     // model.rs:354-366
            const float4 bq = reinterpret_cast<const float4*>(sm.bt[i])[c], cq = reinterpret_cast<const float4*>(sm.ct[i])[c];
            const float abar = sm.abar[i], lam = sm.lam[i], c2 = sm.c2[i];
            float part[F];
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const float xv = sm.xa[i][r0 + f * RSTEP], xpv = xp[f];
                auto next = [&](float hv, float bpv, float bv) {
                    return __fadd_rn(__fadd_rn(__fmul_rn(abar, hv), __fmul_rn(c2, __fmul_rn(xpv, bpv))), __fmul_rn(lam, __fmul_rn(xv, bv)));
                };
                st[f].x = next(st[f].x, bp.x, bq.x);
                st[f].y = next(st[f].y, bp.y, bq.y);
                st[f].z = next(st[f].z, bp.z, bq.z);
                st[f].w = next(st[f].w, bp.w, bq.w);
                part[f] = fmaf(cq.w, st[f].w, fmaf(cq.z, st[f].z, fmaf(cq.y, st[f].y, __fmul_rn(cq.x, st[f].x))));
                xp[f] = xv;
            }
            bp = bq;
#pragma unroll
            for (int o = CG / 2; o > 0; o >>= 1)
#pragma unroll
                for (int f = 0; f < F; ++f) part[f] += __shfl_xor_sync(0xffffffffu, part[f], o);
            if (c == 0)
#pragma unroll
                for (int f = 0; f < F; ++f) sm.yo[i][r0 + f * RSTEP] = part[f];
        }
        __syncthreads();
        for (int e = tid; e < nv * P; e += 128) {
            const int i = e / P, p = e % P;
            const float v = __fmul_rn(__fadd_rn(sm.yo[i][p], __fmul_rn(dskip, sm.xa[i][p])), sm.gate[i][p]);      // model.rs:367-370
            const size_t o = (row0 + t0 + i) * (size_t)DI + h * P + p;
            if (y32 != nullptr) y32[o] = v;
            if (a.yhi != nullptr) {
                const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                a.yhi[o] = hi;
                if (a.ylo != nullptr) a.ylo[o] = __float2bfloat16_rn(v - __bfloat162float(hi));
            }
        }
        if (t0 + nv == ts) {                               // hand-over to the decode step
            if (tid < P) a.xprev[bh * P + tid] = sm.xa[nv - 1][tid];
            for (int n = tid; n < N; n += 128) a.bprev[bh * N + n] = sm.bt[nv - 1][n];
        }
        __syncthreads();                                   // the tables are rebuilt for the next tokens
    }
#pragma unroll
    for (int f = 0; f < F; ++f) h4[tid + 128 * f] = st[f];
    if (tid < HN) a.cum[bh * HN + tid] = cu;
}

template <int TM, typename WT>
cudaError_t row_gemm_launch(const RowGemmArgs& g, int splits, cudaStream_t st) {
    using T = RowTile<TM, WT>;
    const cudaError_t e = cudaFuncSetAttribute(row_gemm_kernel<TM, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (e != cudaSuccess) return e;
    const int units = (g.K + kBK * kUnit - 1) / (kBK * kUnit), per = (units + splits - 1) / splits;
    dim3 grid((g.N + kBN - 1) / kBN, (g.M + 16 * TM - 1) / (16 * TM), (units + per - 1) / per);
    row_gemm_kernel<TM, WT><<<grid, 128, T::SMEM, st>>>(g, per);
    return cudaGetLastError();
}

}  // namespace

bool row_gemm_supported(int K) { return K >= 16 && K % 16 == 0; }

cudaError_t launch_row_gemm(const RowGemmArgs& g, cudaStream_t st) {
    if (!row_gemm_supported(g.K) || g.lda % 4 != 0) return cudaErrorInvalidValue;
    // 32-row tiles while they waste less than 64-row ones; K split, unit by unit, until every SM has as many CTAs as fit it
    const bool narrow = g.M <= 32 || (g.M > 64 && g.M <= 96);
    const int bm = narrow ? 32 : 64;
    const long tiles = (long)((g.M + bm - 1) / bm) * ((g.N + kBN - 1) / kBN), units = (g.K + kBK * kUnit - 1) / (kBK * kUnit);
    long splits = std::max<long>(1, std::min<long>(units, (narrow ? 4 : 3) * 148 / tiles));
    if (tiles > g.n_counters || (size_t)(tiles * units) * bm * kBN > g.scratch_floats) splits = 1;
    if (g.w_dtype == LUMI_DTYPE_BF16) return narrow ? row_gemm_launch<2, __nv_bfloat16>(g, (int)splits, st) : row_gemm_launch<4, __nv_bfloat16>(g, (int)splits, st);
    return narrow ? row_gemm_launch<2, float>(g, (int)splits, st) : row_gemm_launch<4, float>(g, (int)splits, st);
}

#define LUMI_ROWS_SHAPES(X) X(32, 64) X(32, 16) X(32, 32) X(32, 128) X(16, 32) X(16, 64) X(16, 128) X(64, 16) X(64, 32) X(64, 64) X(64, 128)

bool ssm_rows_supported(int P, int N) {
#define LUMI_ROWS_CASE(PP, NN) if (P == PP && N == NN) return true;
    LUMI_ROWS_SHAPES(LUMI_ROWS_CASE)
#undef LUMI_ROWS_CASE
    return false;
}

cudaError_t launch_ssm_rows(const PrefillArgs& a, int P, int N, float* y32, cudaStream_t st) {
    cudaError_t e = launch_bc_stats(a, P, N, st);
    if (e != cudaSuccess) return e;
#define LUMI_ROWS_CASE(PP, NN) if (P == PP && N == NN) { ssm_rows_kernel<PP, NN><<<dim3(a.H, a.nb), 128, 0, st>>>(a, y32); return cudaGetLastError(); }
    LUMI_ROWS_SHAPES(LUMI_ROWS_CASE)
#undef LUMI_ROWS_CASE
    return cudaErrorInvalidValue;
}

}  // namespace lumi
