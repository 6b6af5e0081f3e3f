// Prompts a layer at a time where the chunked scan does not apply: fp32 weights, short prompts, other head shapes.
//
// Fed token by token (inference/src/main.rs:121-125), a prompt of T tokens reads every weight T times.  Taken a layer at a
// time it reads them once: the projections become products over all rows (`launch_row_gemm` for fp32 activations, the tensor-core
// product for bf16 halves), and only the recurrence runs in token order (`ssm_rows_kernel`, the decode step's arithmetic with
// the state in registers).
//
// Measured on the 48-layer base model: scoring 4 x 96 tokens in fp32 125.5 -> 10.1 ms, a 32-token prompt of one sequence
// with the step behind it 4.2 ms in fp32 (token by token 16.7 without the step) and 20.9 -> 3.9 ms in bf16; twelve bf16 sequences of 100 tokens
// (halves) 10.4 ms.
#include "internal.h"

namespace lumi {
namespace {

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

}  // namespace

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
