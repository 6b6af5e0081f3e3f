// Chunked (SSD-style) prefill of the Mamba-3 trapezoidal recurrence, chunk length 64, with the chunk's
// projection rows staged by TMA and the chunk products on tensor cores.
//
// The reference prefills token by token (inference/src/main.rs:121-125) and its only NVIDIA scan
// is sequential in time (training/csrc/ssm_scan.cu:137-227; SSD_FWD_CHUNK there is dead code).
// This kernel evaluates the same recurrence (inference/src/model.rs:354-368)
//     S_t = a_t S_{t-1} + (1 - lam_t) a_t U_{t-1} + lam_t U_t ,   U_t = x_t (x) B~_t ,   y_t = S_t C~_t + D x_t
// a chunk at a time.  With the augmented state  S^_t = S_t + (1 - lam_{t+1}) U_t  it becomes
//     S^_t = a_t S^_{t-1} + kap_t U_t ,   kap_t = lam_t + 1 - lam_{t+1} ,   S_t = a_t S^_{t-1} + lam_t U_t ,
// an ordinary decayed linear recurrence, so inside a chunk starting at t0 (l_i = sum of log a up to i)
//     y_i = e^{l_i} (S^_in C~_i) + sum_{j<i} e^{l_i - l_j} kap_j (C~_i . B~_j) x_j + lam_i (C~_i . B~_i) x_i + D x_i
//     S^_out = e^{l_last} S^_in + sum_j e^{l_last - l_j} kap_j x_j (x) B~_j
// — four small matrix products per (sequence, head, chunk):
//     G = C~ B~^T (64x64x64),  Y1 = W X with W = mask/decay(G) (64x64x32),  Y2 = C~ S^_in^T (64x64x32),
//     S^_out += (w x)^T B~ (32x64x64).
// The last token of a launch uses kap = lam, which makes S^ equal the true S: every launch ends with exactly
// the state the decode kernel expects (h, x_prev, B~_prev, cum_angle), and the next launch rebuilds S^ from it.
// DD-RoPE angles are a prefix sum over the chunk taken mod 2 pi (the reference reduces mod 2 pi every step:
// same angle, rounding-level differences; the stored angle may differ from the sequential one by a multiple
// of 2 pi).
//
// One CTA of four warps per (head, sequence), four CTAs per SM (54 KiB of shared memory, 128 registers, 24 bytes of spills).
//   * Staging: the chunk's x, theta (64 x 32 fp32 each) and the group's raw B, C (64 x 64 fp32 each) arrive by four
//     cp.async.bulk.tensor copies on one mbarrier (bounded wait).  The operand tiles are built IN PLACE over the
//     raw rows, so the copies for chunk c+1 are issued when chunk c's products are done; their flight time is covered
//     by the three other CTAs of the SM.  z and the next chunk's per-token scalars (dt, lambda, A, BCNorm scales) come by small
//     asynchronous copies into places that are free by then.
//   * Segments of 16 tokens, one per warp: decays are taken from segment to segment.  What later segments and the state take of token j is
//     x_j kap_j times its decay to the end of its segment, one tile for both; Y = C~ S^_in^T walks over the segments ahead of the warp's own, each time
//     a decay, then + G X; the segment's own block, which needs the warp's rows only, is the one place with a decay per pair of tokens.  A logarithm counts as
//     -88 at least, where the decay is 0 in fp32: behind the -1e6 of a clamped decay a sum would have nothing left of the -0.02 of the tokens that follow. So sums
//     stay above 16 x -88: a factor behind one such token is right to 2^-16 of itself, as the split of operands below, behind fifteen to 2^-11, and at most
//     1 but for that.
//   * Arithmetic: every operand is an fp32 value split into bf16 hi + lo; a product is three
//     mma.sync.m16n8k16 (hi*hi + hi*lo + lo*hi, fp32 accumulate), which keeps ~16 mantissa bits per factor.
//     Warp w owns tokens 16w..16w+15: its C~ rows stay in registers as A fragments, G's accumulators are
//     re-used in place as the A fragments of G X (no trip through shared memory), and the state S^
//     lives in accumulator registers across the chunks of a launch (warp w: 16 rows of P x 32 columns of N).
//     Independent accumulators are interleaved so that no multiply-add waits for the one issued just before it.
//   * The pointwise part (softplus / sigmoid / tanh / SiLU / sin / cos) uses the fast hardware forms here: their
//     error (~1e-6) is far below the operand split's (1.5e-5) — the decode step keeps the exact forms.
// What bounds it: instruction issue (half of the slots) and shared memory (half of its cycles) together; memory is at a fifth of its rate.  64 sequences x 2048
// tokens, 64 heads: 4.00 ms with decays per pair of tokens throughout and three CTAs per SM, 2.85 ms by segments with four, 2.39 ms with one address per
// tile and lane and the scalars copied ahead (15.0, 11.6 and fewer thousand warp instructions per chunk and head).
#include "internal.h"
#include "embed_post.cuh"

#include <cuda.h>

#include <type_traits>

namespace lumi {

// defined in gemm_tcgen05.cu: cuTensorMapEncodeTiled for a row-major fp32 matrix [rows][cols], no swizzle
int32_t make_f32_map_2d(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_cols,
                        uint32_t box_rows);

namespace {

constexpr int LCH = 64;          // chunk length
constexpr uint64_t kScanWaitLimitNs = 500ull * 1000 * 1000;

__device__ __forceinline__ float sigmoid_ref(float x) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x))); }
__device__ __forceinline__ float softplus_ref(float x) { return logf(__fadd_rn(expf(x), 1.0f)); }
// The hardware forms without the steps around them that keep results below 2^-126 alive: a term that small is gone behind the next addition.
__device__ __forceinline__ float ex2_ftz(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcp_ftz(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
constexpr float kLog2E = 1.44269504088896340736f;
__device__ __forceinline__ float silu_fast(float x) { return x * rcp_ftz(1.0f + ex2_ftz(-kLog2E * x)); }
// 1 - 2 / (e^{2x} + 1): absolute error ~1e-7; e^{2x} may be 0 or infinite
__device__ __forceinline__ float tanh_fast(float x) { return fmaf(-2.0f, rcp_ftz(ex2_ftz(2.0f * kLog2E * x) + 1.0f), 1.0f); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit expired.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (globaltimer_ns() - t0 > limit_ns) return false;
    }
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// D (16x8, fp32) += A (16x16, bf16, row) * B (16x8, bf16, col)
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (a_hi + a_lo)(b_hi + b_lo) without the lo*lo term, for the two 8-column tiles whose B fragments one ldmatrix.x4
// delivers (bh / bl: {b0, b1} of the first tile, {b0, b1} of the second).  The six multiply-adds alternate between
// the two accumulators so that no instruction waits for the one just before it.
__device__ __forceinline__ void mma3x2(float (&d0)[4], float (&d1)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4],
                                       const uint32_t (&bh)[4], const uint32_t (&bl)[4]) {
    mma_bf16(d0, ah, bh[0], bh[1]);
    mma_bf16(d1, ah, bh[2], bh[3]);
    mma_bf16(d0, ah, bl[0], bl[1]);
    mma_bf16(d1, ah, bl[2], bl[3]);
    mma_bf16(d0, al, bh[0], bh[1]);
    mma_bf16(d1, al, bh[2], bh[3]);
}
// the same for four tiles (two ldmatrix.x4 per plane): twelve multiply-adds round-robin over four accumulators
__device__ __forceinline__ void mma3x4(float (&d0)[4], float (&d1)[4], float (&d2)[4], float (&d3)[4], const uint32_t (&ah)[4],
                                       const uint32_t (&al)[4], const uint32_t (&bh0)[4], const uint32_t (&bl0)[4],
                                       const uint32_t (&bh1)[4], const uint32_t (&bl1)[4]) {
    mma_bf16(d0, ah, bh0[0], bh0[1]); mma_bf16(d1, ah, bh0[2], bh0[3]); mma_bf16(d2, ah, bh1[0], bh1[1]); mma_bf16(d3, ah, bh1[2], bh1[3]);
    mma_bf16(d0, ah, bl0[0], bl0[1]); mma_bf16(d1, ah, bl0[2], bl0[3]); mma_bf16(d2, ah, bl1[0], bl1[1]); mma_bf16(d3, ah, bl1[2], bl1[3]);
    mma_bf16(d0, al, bh0[0], bh0[1]); mma_bf16(d1, al, bh0[2], bh0[3]); mma_bf16(d2, al, bh1[0], bh1[1]); mma_bf16(d3, al, bh1[2], bh1[3]);
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t at, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
__device__ __forceinline__ void sts128(uint32_t at, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// (a0, a1) * s then * g + b, two fp32 at a time
__device__ __forceinline__ float2 norm2(float2 v, float s, float2 g, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tmul.rn.f32x2 x, x, y;\n\t"
        "mov.b64 y, {%5, %6};\n\tmov.b64 z, {%7, %8};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(v.x), "f"(v.y), "f"(s), "f"(g.x), "f"(g.y), "f"(b.x), "f"(b.y));
    return r;
}
// two fp32 values -> bf16x2 hi word and bf16x2 lo word (first value in the low half)
__device__ __forceinline__ void split2(float v0, float v1, uint32_t& hi, uint32_t& lo) {
    __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
    const float2 hf = __bfloat1622float2(h);
    __nv_bfloat162 l = __floats2bfloat162_rn(v0 - hf.x, v1 - hf.y);
    hi = *reinterpret_cast<uint32_t*>(&h);
    lo = *reinterpret_cast<uint32_t*>(&l);
}
__device__ __forceinline__ void split_bf16(float v, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// Shared memory of a CTA (54 KiB: four CTAs per SM).  The four bulk tensor copies of a chunk land in rx, rth, rB, rC (dense boxes).  The
// operand tiles of the tensor-core products are then written IN PLACE over raw rows that nobody reads any more: token i's raw B row
// (256 bytes) becomes B~ hi (first 128 bytes) and B~ lo (last 128 bytes) of token i, the same for C; silu(x) transposed replaces the raw x
// rows and the state S^ the raw theta rows.  A warp's rows of C~ move on into its registers, and its rows of z are copied over them.
// Inside a 128-byte row the eight 16-byte chunks are XOR-ed with a key of the row, so that ldmatrix and the stores stay free of bank
// conflicts without padding.
struct PfSmem {
    float rx[LCH][32];                 // raw x            -> X^T: [plane hi | lo][p = 32 rows][token, 128 bytes]
    float rth[LCH][32];                // raw theta        -> S^: [plane hi | lo][p = 32 rows][n, 128 bytes]
    float rB[LCH][64];                 // raw B (group)    -> B~: row = token, [hi 128 bytes | lo 128 bytes]
    float rC[LCH][64];                 // raw C (group)    -> C~: same layout -> z of the warp's tokens
    struct Scalars {                   // per token; the next chunk's are prepared under this one
        float dtp[LCH], rbs[LCH], rcs[LCH];      // dt pi, BCNorm scales
        float ell[LCH], eli[LCH];      // log2 of the decay from the start of the token's segment of 16 to the token itself, and the decay
        float lam[LCH], kap[LCH];
        float xw[LCH];                 // kap times the decay from the token to the end of its segment
        float seg[4];                  // decay over each segment
        float after, pad[3];           // raw lambda of the token behind the chunk
    } sc[2];
    float seg[4][32];                  // angle sums of the four 16-token segments
    float gam[4][64];                  // this group's BCNorm weights: b gamma, b bias, c gamma, c bias
    unsigned long long bar;
};

// Element (row, col) of the B~ / C~ tiles lies at row * 256 + (((col / 8) ^ (row % 8)) << 4) + col % 8 * 2, lo plane 128 bytes on; of the X^T / S^
// tiles (row = p) at p * 128 + (((col / 8) ^ key_of(p)) << 4) + col % 8 * 2, lo plane 4096 bytes on.  The key differs within every eight
// consecutive rows and within every eight rows {8 a + 2 n + e : a = 0 .. 3, e = 0, 1} that pcol() makes one matrix.  Columns in steps of 16
// (two chunks) then only flip bits of a lane's address: address ^ (step << 5).
__device__ __forceinline__ int key_of(int p) { return (((p >> 3) ^ (p >> 1)) & 3) << 1 | (p & 1); }
// Column c of tile nt of a product whose columns are head dims: with this order a lane's results of the four tiles are the eight head dims
// 8 t4 .. 8 t4 + 7, one 16-byte store.
__device__ __forceinline__ int pcol(int nt, int c) { return 8 * (c >> 1) + 2 * nt + (c & 1); }

// fmodf(x, y) for y > 0 in a few instructions: the remainder of the nearest smaller multiple is exact in one fused multiply-add, and a
// quotient that rounding carried over a multiple is put back and the multiply-add repeated.
__host__ __device__ __forceinline__ float fmod_near(float x, float y, float inv_y) {
    if (!(fabsf(x) < 1e6f)) return fmodf(x, y);
    const float q = truncf(x * inv_y);
    float r = fmaf(-q, y, x);
    if (r != 0.f && (r < 0.f) != (x < 0.f)) r = fmaf(-(q - copysignf(1.f, x)), y, x);
    else if (fabsf(r) >= y) r = fmaf(-(q + copysignf(1.f, x)), y, x);
    return r;
}

constexpr uint32_t kChunkTxBytes = 2 * LCH * 32 * 4 + 2 * LCH * 64 * 4;

// row r = b * ts + t  of the super-chunk; token ids come from prompt[(t_abs) * batch_total + b_abs]
template <typename WT>
__global__ void embed_rows_kernel(const WT* __restrict__ emb, const uint32_t* __restrict__ prompt, float* __restrict__ x, int D,
                                  int vocab, int ts, int t_abs0, int b_abs0, int batch_total, StepCtl* ctl, const int32_t* __restrict__ lens,
                                  EmbedPost post) {
    const int r = blockIdx.x, b = r / ts, t = r - b * ts;
    if (lens != nullptr && t_abs0 + t >= lens[b_abs0 + b]) {      // padding behind a shorter prompt: never looked at, the row is zero
        for (int k = threadIdx.x; k < D; k += blockDim.x) {
            x[(size_t)r * D + k] = 0.f;
            if (post.hi != nullptr) post.hi[(size_t)r * D + k] = __float2bfloat16_rn(0.f);
            if (post.lo != nullptr) post.lo[(size_t)r * D + k] = __float2bfloat16_rn(0.f);
        }
        return;
    }
    uint32_t tok = prompt[(size_t)(t_abs0 + t) * batch_total + b_abs0 + b];
    if (tok >= (uint32_t)vocab) { if (threadIdx.x == 0) atomicOr(&ctl->status, STATUS_BAD_TOKEN); tok = 0; }
    const WT* row = emb + (size_t)tok * D;
    for (int k = threadIdx.x; k < D; k += blockDim.x) {
        float v;
        if (sizeof(WT) == 4) v = reinterpret_cast<const float*>(row)[k];
        else v = __uint_as_float((uint32_t)reinterpret_cast<const uint16_t*>(row)[k] << 16);
        float one[1] = {v};
        embed_post<1>(post, one, k, post.pos != nullptr ? post.pos[b] + t : 0);
        x[(size_t)r * D + k] = one[0];
        if (post.hi != nullptr) {
            const __nv_bfloat16 hh = __float2bfloat16_rn(one[0]);
            post.hi[(size_t)r * D + k] = hh;
            if (post.lo != nullptr) post.lo[(size_t)r * D + k] = __float2bfloat16_rn(one[0] - __bfloat162float(hh));
        }
    }
}

// BCNorm scales of every token row: r_b, r_c = 1 / sqrt(mean(B^2) + eps) over all n_groups * d_state (model.rs:311-312)
__global__ void bc_stats_kernel(const float* __restrict__ proj, int ldp, int off_b, int BC, float eps, float* __restrict__ rb,
                                float* __restrict__ rc, int rows) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows) return;
    const float* Bp = proj + (size_t)warp * ldp + off_b;
    const float* Cp = Bp + BC;
    float sb = 0.f, sc = 0.f;
    for (int i = lane; i < BC; i += 32) { sb = fmaf(Bp[i], Bp[i], sb); sc = fmaf(Cp[i], Cp[i], sc); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { sb += __shfl_xor_sync(0xffffffffu, sb, o); sc += __shfl_xor_sync(0xffffffffu, sc, o); }
    if (lane == 0) {
        rb[warp] = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(sb, (float)(1.0 / (double)BC)), eps)));
        rc[warp] = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(sc, (float)(1.0 / (double)BC)), eps)));
    }
}

// last token's residual row of every sequence -> x[b][D] (for the lm_head after the prompt)
__global__ void gather_last_kernel(const float* __restrict__ xr, float* __restrict__ x, int D, int ts, int b0, const int32_t* __restrict__ lens,
                                   int t_abs0) {
    const int b = blockIdx.x;
    const int idx = lens != nullptr ? lens[b0 + b] - 1 - t_abs0 : ts - 1;      // the sequence's last prompt token, if this slice holds it
    if (idx < 0 || idx >= ts) return;
    for (int k = threadIdx.x; k < D; k += blockDim.x) x[(size_t)(b0 + b) * D + k] = xr[((size_t)b * ts + idx) * D + k];
}

__global__ void __launch_bounds__(128, 4)
ssd_prefill_kernel(const __grid_constant__ CUtensorMap map32, const __grid_constant__ CUtensorMap map64, PrefillArgs a) {
    constexpr int P = 32, N = 64, HN = 32;
    extern __shared__ __align__(1024) uint8_t pf_raw[];
    PfSmem& sm = *reinterpret_cast<PfSmem*>(pf_raw);
    const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g4 = lane >> 2, t4 = lane & 3;               // mma fragment coordinates: row group, column pair
    const int lm = lane >> 3, lr = lane & 7;               // ldmatrix: matrix and row that this lane addresses
    const int H = a.H, DI = H * P, BC = a.G * N, R = a.ldp;
    const int tsl = a.ts;                                   // rows per sequence in the projection / output arrays
    // tokens this sequence takes from the launch (prompts of different lengths end early; none: the state stays as it is)
    const int ts = a.lens != nullptr ? max(0, min(tsl, a.lens[a.b0 + b] - a.t_abs0)) : tsl;
    if (ts == 0) return;
    const int grp = h / (H / a.G);
    const size_t bh = (size_t)(a.b0 + b) * H + h;
    const int off_b = 2 * DI, off_c = off_b + BC, off_dt = off_c + BC;
    const float PI_F = 3.14159265358979323846f;
    const float TWO_PI = 6.28318530717958647692f;
    const float INV_TWO_PI = 0.15915494309189533577f;
    const float dskip = a.dskip[h], dtb = a.dtb[h];
    uint64_t* bar = reinterpret_cast<uint64_t*>(&sm.bar);

    // a wait that expired in an earlier CTA of this launch: do not start new work (one verdict for all threads: the word may change while they look)
    if (__syncthreads_or(a.status != nullptr && (*reinterpret_cast<volatile int32_t*>(a.status) & STATUS_TIMEOUT))) return;

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    float cum = a.cum[bh * HN + lane];                     // running angle of pair `lane`, kept by every warp
    if (tid < 64) {
        const int c = grp * N + tid;
        sm.gam[0][tid] = a.bg[c]; sm.gam[1][tid] = a.bb[c]; sm.gam[2][tid] = a.cg[c]; sm.gam[3][tid] = a.cb[c];
    }
    __syncthreads();

    auto issue_chunk = [&](int t0) {               // one thread: the four box copies of the chunk starting at token t0
        const int row0 = b * tsl + t0;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(kChunkTxBytes) : "memory");
        tma_load_2d(&sm.rth[0][0], &map32, bar, off_dt + 3 * H + h * HN, row0);
        tma_load_2d(&sm.rx[0][0], &map32, bar, h * P, row0);
        tma_load_2d(&sm.rB[0][0], &map64, bar, off_b + grp * N, row0);
        tma_load_2d(&sm.rC[0][0], &map64, bar, off_c + grp * N, row0);
    };
    // this lane's addresses in the operand tiles (ldmatrix reads and stores), the parts that change with the loops left out
    const uint32_t tB = smem_u32(&sm.rB[0][0]), tC = smem_u32(&sm.rC[0][0]), tX = smem_u32(&sm.rx[0][0]), tS = smem_u32(&sm.rth[0][0]);
    const int i0 = 16 * warp;                              // first token of this warp's segment
    const uint32_t own = (uint32_t)(i0 * 256 + ((lane >> 2) << 4) + ((lane & 3) << 2));                        // B~ / C~ stores: columns 2 lane, 2 lane + 1
    const uint32_t aC = tC + (uint32_t)((i0 + 8 * (lm & 1) + lr) * 256 + (((lm >> 1) ^ lr) << 4));           // C~ rows as A fragments
    const uint32_t aB = tB + (uint32_t)((8 * (lm >> 1) + lr) * 256 + (((lm & 1) ^ lr) << 4));                 // B~ rows of a segment as B fragments
    const int pn = pcol(lm >> 1, lr);                       // head dim of this lane's row in the two tiles 0 and 1; tiles 2 and 3: + 4, whose key differs by 4
    const uint32_t aP = (uint32_t)(pn * 128 + (((lm & 1) ^ key_of(pn)) << 4)), aP2 = (aP + 4u * 128u) ^ 64u;
    // Per-token scalars of a chunk (model.rs:307, 314-317), by warp 0 alone: lane l takes tokens 2 l and 2 l + 1, the last lane also lambda
    // of the token behind the chunk.  Done for the next chunk while the other warps, which have more of the causal products, are still at theirs.
    // Their raw values are copied (asynchronously, by the same lanes) into the places that take the results.
    auto fetch_scalars = [&](int t0, PfSmem::Scalars& q) {
        const int nv = min(LCH, ts - t0);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * lane + e;
            if (i < nv) {
                const size_t row = (size_t)b * tsl + t0 + i;
                const float* pr = a.proj + row * R + off_dt + h;
                cp_async4(&q.dtp[i], pr); cp_async4(&q.lam[i], pr + H); cp_async4(&q.ell[i], pr + 2 * H);
                cp_async4(&q.rbs[i], a.rb + row); cp_async4(&q.rcs[i], a.rc + row);
            }
        }
        if (lane == 31 && t0 + LCH < ts) cp_async4(&q.after, a.proj + ((size_t)b * tsl + t0 + LCH) * R + off_dt + H + h);
    };
    auto prepare_scalars = [&](int t0, PfSmem::Scalars& q) {      // (this lane's copies have landed)
        const int nv = min(LCH, ts - t0);
        float dtpv[2] = {0.f, 0.f}, gl[2] = {0.f, 0.f}, lv[2] = {0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * lane + e;
            if (i < nv) {
                dtpv[e] = softplus_ref(__fadd_rn(q.dtp[i], dtb));
                float av = -softplus_ref(q.ell[i]);
                av = fminf(fmaxf(av, -1e6f), -1e-4f);
                gl[e] = fmaxf(__fmul_rn(av, dtpv[e]), -88.f);      // log a_t; e^-88 < 2^-126 is 0 below
                lv[e] = sigmoid_ref(q.lam[i]);
            } else {
                q.rbs[i] = 0.f; q.rcs[i] = 0.f;
            }
        }
        const float after = lane == 31 && t0 + LCH < ts ? sigmoid_ref(q.after) : -1.0f;      // < 0: no next token in this launch
        float incl = gl[0] + gl[1];                        // inclusive prefix of log a over the segment of 16 tokens: eight lanes
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) { const float n = __shfl_up_sync(0xffffffffu, incl, o, 8); if ((lane & 7) >= o) incl += n; }
        float excl = __shfl_up_sync(0xffffffffu, incl, 1, 8);
        if ((lane & 7) == 0) excl = 0.f;
        const float l[2] = {excl + gl[0], incl};
        const float tot = __shfl_sync(0xffffffffu, incl, lane | 7), down = __shfl_down_sync(0xffffffffu, lv[0], 1);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * lane + e;
            float k = 0.f;
            if (i < nv) {
                // lambda of the next token: this lane's second one, the next lane's first, or the one behind the chunk
                float ln = -1.0f;
                if (i + 1 < nv) ln = e == 0 ? lv[1] : down;
                else if (nv == LCH) ln = after;                  // lane 31's last token only
                k = ln < 0.f ? lv[e] : __fadd_rn(lv[e], __fsub_rn(1.0f, ln));
            }
            q.dtp[i] = dtpv[e] * PI_F;
            q.ell[i] = l[e] * kLog2E; q.eli[i] = ex2_ftz(l[e] * kLog2E);
            q.lam[i] = lv[e]; q.kap[i] = k;
            q.xw[i] = ex2_ftz((tot - l[e]) * kLog2E) * k;
        }
        if ((lane & 7) == 0) q.seg[lane >> 3] = ex2_ftz(tot * kLog2E);
    };
    if (tid == 0) issue_chunk(0);
    if (warp == 0) {
        fetch_scalars(0, sm.sc[0]);
        asm volatile("cp.async.wait_all;" ::: "memory");
        prepare_scalars(0, sm.sc[0]);
    }

    // state S^ of this warp: rows p0 + {g4, g4 + 8}, columns n0 + 8 nt + 2 t4 + {0, 1}
    const int p0 = 16 * (warp & 1), n0 = 32 * (warp >> 1);
    float S[4][4];
    {
        const float* hp = a.h + bh * (size_t)(P * N);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const float2 v0 = *reinterpret_cast<const float2*>(hp + (p0 + g4) * N + n0 + 8 * nt + 2 * t4);
            const float2 v1 = *reinterpret_cast<const float2*>(hp + (p0 + g4 + 8) * N + n0 + 8 * nt + 2 * t4);
            S[nt][0] = v0.x; S[nt][1] = v0.y; S[nt][2] = v1.x; S[nt][3] = v1.y;
        }
    }

    __syncthreads();                                       // the first chunk's scalars are there

    // S^_in = S + (1 - lam_first) x_prev (x) B~_prev   (prev_bx of the decode state, model.rs:359)
    {
        const float oml = __fadd_rn(__fmul_rn(sm.sc[0].lam[0], -1.0f), 1.0f);
        const float xp0 = a.xprev[bh * P + p0 + g4] * oml, xp1 = a.xprev[bh * P + p0 + g4 + 8] * oml;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const float2 bp = *reinterpret_cast<const float2*>(a.bprev + bh * N + n0 + 8 * nt + 2 * t4);
            S[nt][0] = fmaf(xp0, bp.x, S[nt][0]); S[nt][1] = fmaf(xp0, bp.y, S[nt][1]);
            S[nt][2] = fmaf(xp1, bp.x, S[nt][2]); S[nt][3] = fmaf(xp1, bp.y, S[nt][3]);
        }
    }

    const int ia = i0 + g4, ib = ia + 8;                   // the tokens whose results this lane holds
    uint32_t phase = 0;
    // One chunk.  FULL: all 64 tokens are valid, so every "past the end of the sequence" test folds away.
    auto do_chunk = [&](auto full_c, const int t0, const int chunk) -> bool {
        constexpr bool FULL = decltype(full_c)::value;
        const int nv = FULL ? LCH : min(LCH, ts - t0);     // valid tokens in this chunk
        auto valid = [&](int i) { return FULL || i < nv; };
        const bool last_chunk = t0 + LCH >= ts;
        PfSmem::Scalars& sc = sm.sc[chunk & 1];
        // ---- 1. the chunk's raw rows have landed (every thread waits, bounded; the next barrier makes one verdict of it)
        const bool landed = mbar_wait(bar, phase, kScanWaitLimitNs);
        phase ^= 1;
        // ---- 2. thread (lane, warp) takes column `lane` (angle pair k, head dim p) of the warp's 16 tokens: angles, rotated
        //         B~ and C~ (one sin / cos for both), silu(x) transposed.  Every raw row of B and C is read only by the warp that owns
        //         its token, so a row can be overwritten by its operand tile after a warp-level barrier.
        const int k = lane, p = lane;
        float loc[16], xs[16], run = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
            const float4 dp = *reinterpret_cast<const float4*>(&sc.dtp[i0 + i4]);
            const float d4[4] = {dp.x, dp.y, dp.z, dp.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + i4 + q;
                const float d = d4[q] * tanh_fast(sm.rth[i][k]);             // model.rs:341-342
                run += valid(i) ? d : 0.f;                                   // the rows behind the sequence are another one's
                loc[i4 + q] = run;
                xs[i4 + q] = valid(i) ? silu_fast(sm.rx[i][p]) : 0.f;        // model.rs:310
            }
        }
        sm.seg[warp][k] = run;
        if (!__syncthreads_and(landed)) return false;
        // every warp has read its raw x and theta.  S^ over theta: this warp's block as bf16 hi + lo (B operand of C~ S^T)
        {
            // columns n0 + 8 nt + 2 t4: chunk n0 / 8 + nt; rows g4 and g4 + 8 of the block, whose keys differ by 2
            const uint32_t at = tS + (uint32_t)((p0 + g4) * 128 + (((n0 >> 3) ^ key_of(p0 + g4)) << 4) + 4 * t4);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                uint32_t hi, lo;
                const uint32_t a0 = at ^ (uint32_t)(nt << 4), a1 = (a0 ^ 32u) + 1024u;
                split2(S[nt][0], S[nt][1], hi, lo);
                sts32(a0, hi);
                sts32(a0 + 4096, lo);
                split2(S[nt][2], S[nt][3], hi, lo);
                sts32(a1, hi);
                sts32(a1 + 4096, lo);
            }
        }
        if (warp == 0 && !last_chunk) fetch_scalars(t0 + LCH, sm.sc[(chunk + 1) & 1]);
        // reduced mod 2 pi at every segment boundary, so sums stay small and keep their low bits
        float base = cum;
#pragma unroll
        for (int s2 = 0; s2 < 4; ++s2) {
            if (s2 == warp) base = cum;
            cum = fmod_near(cum + sm.seg[s2][k], TWO_PI, INV_TWO_PI);
        }
        if (last_chunk) {                                  // hand-over: x of the launch's last token (every warp has read the old one)
#pragma unroll
            for (int ii = 0; ii < 16; ++ii) if (i0 + ii == nv - 1) a.xprev[bh * P + p] = xs[ii];
        }
        // X^T tile over the raw x rows: row p, tokens i0 .. i0 + 15, eight to a 16-byte chunk
        auto store_x = [&]() {
            const uint32_t at = tX + (uint32_t)(p * 128 + (((i0 >> 3) ^ key_of(p)) << 4));
#pragma unroll
            for (int i8 = 0; i8 < 16; i8 += 8) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split2(xs[i8 + 2 * e], xs[i8 + 2 * e + 1], hi[e], lo[e]);
                sts128(at ^ (uint32_t)(i8 << 1), hi);
                sts128((at ^ (uint32_t)(i8 << 1)) + 4096, lo);
            }
        };
        store_x();
        {
            const float2 bgm = *reinterpret_cast<const float2*>(&sm.gam[0][2 * k]), bbs = *reinterpret_cast<const float2*>(&sm.gam[1][2 * k]);
            const float2 cgm = *reinterpret_cast<const float2*>(&sm.gam[2][2 * k]), cbs = *reinterpret_cast<const float2*>(&sm.gam[3][2 * k]);
#pragma unroll
            for (int i4 = 0; i4 < 16; i4 += 4) {           // four tokens at a time: all lanes read the raw rows, then overwrite them
                float2 rawb[4], rawc[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    rawb[q] = *reinterpret_cast<const float2*>(&sm.rB[i0 + i4 + q][2 * k]);
                    rawc[q] = *reinterpret_cast<const float2*>(&sm.rC[i0 + i4 + q][2 * k]);
                }
                const float4 rb4 = *reinterpret_cast<const float4*>(&sc.rbs[i0 + i4]), rc4 = *reinterpret_cast<const float4*>(&sc.rcs[i0 + i4]);
                const float rbv[4] = {rb4.x, rb4.y, rb4.z, rb4.w}, rcv[4] = {rc4.x, rc4.y, rc4.z, rc4.w};
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int i = i0 + i4 + q;
                    float ang = base + loc[i4 + q];
                    // into [-pi, pi] for the fast sin / cos; the sum with 1.5 * 2^23 rounds to a whole number
                    ang = fmaf(-TWO_PI, fmaf(ang, INV_TWO_PI, 12582912.f) - 12582912.f, ang);
                    float b0 = 0.f, b1 = 0.f, c0 = 0.f, c1 = 0.f;
                    if (valid(i)) {
                        const float2 nb = norm2(rawb[q], rbv[q], bgm, bbs), nc = norm2(rawc[q], rcv[q], cgm, cbs);                  // model.rs:311-313
                        float sa, ca;
                        __sincosf(ang, &sa, &ca);
                        b0 = ca * nb.x - sa * nb.y;                          // model.rs:345-348
                        b1 = sa * nb.x + ca * nb.y;
                        c0 = ca * nc.x - sa * nc.y;
                        c1 = sa * nc.x + ca * nc.y;
                        if (last_chunk && i == nv - 1) {                     // hand-over: B~ of the launch's last token, in fp32
                            a.bprev[bh * N + 2 * k] = b0;
                            a.bprev[bh * N + 2 * k + 1] = b1;
                        }
                    }
                    uint32_t hi, lo;
                    const uint32_t at = tB + (own ^ (uint32_t)(((i4 + q) & 7) << 4)) + (uint32_t)((i4 + q) * 256);      // C~ lies behind B~
                    split2(b0, b1, hi, lo);
                    sts32(at, hi);
                    sts32(at + 128, lo);
                    split2(c0, c1, hi, lo);
                    sts32(at + sizeof(sm.rB), hi);
                    sts32(at + sizeof(sm.rB) + 128, lo);
                }
            }
        }
        __syncwarp();
        // ---- 3. this warp's C~ rows as A fragments (hi, lo) from its own rows of the tile; then z of its tokens over them, token i's
        //         32 values at row i, their 16-byte chunks XOR-ed by i % 2
        uint32_t Ch[4][4], Cl[4][4];
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            ldsm_x4(Ch[ks], aC ^ (uint32_t)(ks << 5));
            ldsm_x4(Cl[ks], (aC ^ (uint32_t)(ks << 5)) + 128);
        }
        __syncwarp();
        {
            const float* zp = a.proj + ((size_t)b * tsl + t0 + i0 + lm) * R + DI + h * P + 4 * lr;
            const uint32_t dst = tC + (uint32_t)((i0 + lm) * 256 + ((lr ^ (lm & 1)) << 4));
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (valid(i0 + lm + 4 * r))
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * 1024u), "l"(zp + (size_t)(4 * r) * R) : "memory");
        }
        // G = C~ B~^T against the 16 tokens of segment jp, as accumulators of two 8-column tiles.
        // Four independent accumulation chains (hi*hi, and hi*lo with lo*hi, of the two tiles), added at the end
        auto causal_product = [&](int jp, float (&g0)[4], float (&g1)[4]) {
            float g0b[4], g1b[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) { g0[e] = 0.f; g1[e] = 0.f; g0b[e] = 0.f; g1b[e] = 0.f; }
            const uint32_t at = aB + (uint32_t)(jp * 4096);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t bh4[4], bl4[4];
                ldsm_x4(bh4, at ^ (uint32_t)(ks << 5));
                ldsm_x4(bl4, (at ^ (uint32_t)(ks << 5)) + 128);
                mma_bf16(g0, Ch[ks], bh4[0], bh4[1]);
                mma_bf16(g1, Ch[ks], bh4[2], bh4[3]);
                mma_bf16(g0b, Ch[ks], bl4[0], bl4[1]);
                mma_bf16(g1b, Ch[ks], bl4[2], bl4[3]);
                mma_bf16(g0b, Cl[ks], bh4[0], bh4[1]);
                mma_bf16(g1b, Cl[ks], bh4[2], bh4[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) { g0[e] += g0b[e]; g1[e] += g1b[e]; }
        };
        // d += W X over the 16 tokens of segment jp
        auto add_wx = [&](float (&d)[4][4], const float (&w0)[4], const float (&w1)[4], int jp) {
            uint32_t wh[4], wl[4], xh0[4], xl0[4], xh1[4], xl1[4];
            split2(w0[0], w0[1], wh[0], wl[0]);
            split2(w0[2], w0[3], wh[1], wl[1]);
            split2(w1[0], w1[1], wh[2], wl[2]);
            split2(w1[2], w1[3], wh[3], wl[3]);
            const uint32_t x01 = tX + (aP ^ (uint32_t)(jp << 5)), x23 = tX + (aP2 ^ (uint32_t)(jp << 5));
            ldsm_x4(xh0, x01);
            ldsm_x4(xl0, x01 + 4096);
            ldsm_x4(xh1, x23);
            ldsm_x4(xl1, x23 + 4096);
            mma3x4(d[0], d[1], d[2], d[3], wh, wl, xh0, xl0, xh1, xl1);
        };
        // ---- 4. the segment's own block, which needs this warp's rows only: W = mask / decay (G), lam_i (C~_i . B~_i) + D on the diagonal
        float y[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) y[nt][e] = 0.f;
        {
            float g0[4], g1[4];
            causal_product(warp, g0, g1);
            const float la = sc.ell[ia], lb = sc.ell[ib], ma = sc.lam[ia], mb = sc.lam[ib];
            // element e of tile q: row (e < 2 ? g4 : g4 + 8), column 8 q + 2 t4 + (e & 1) of the segment
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float2 lj = *reinterpret_cast<const float2*>(&sc.ell[i0 + 8 * q + 2 * t4]), kj = *reinterpret_cast<const float2*>(&sc.kap[i0 + 8 * q + 2 * t4]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = (e < 2) ? g4 : g4 + 8, j = 8 * q + 2 * t4 + (e & 1);
                    float& g = q == 0 ? g0[e] : g1[e];
                    const float below = g * (ex2_ftz((e < 2 ? la : lb) - ((e & 1) ? lj.y : lj.x)) * ((e & 1) ? kj.y : kj.x));
                    g = j < i ? below : j == i ? fmaf(g, e < 2 ? ma : mb, dskip) : 0.f;
                }
            }
            add_wx(y, g0, g1, warp);
        }
        // X^T again, now each token times kap and its decay to the end of its segment: what later segments and the state take of it
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(&sc.xw[i0 + i4]);
            xs[i4] *= w4.x; xs[i4 + 1] *= w4.y; xs[i4 + 2] *= w4.z; xs[i4 + 3] *= w4.w;
        }
        __syncwarp();
        store_x();
        __syncthreads();
        // ---- 5. Y2 = C~ S^_in^T, then the earlier segments one by one: decay over the segment, + G X of its tokens; at the end the decay
        //         from the start of the own segment to the token.  Every factor is at most 1.
        {
            float acc[4][4];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[nt][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t sh0[4], sl0[4], sh1[4], sl1[4];   // p tiles 0, 1 and 2, 3
                const uint32_t s01 = tS + (aP ^ (uint32_t)(ks << 5)), s23 = tS + (aP2 ^ (uint32_t)(ks << 5));
                ldsm_x4(sh0, s01);
                ldsm_x4(sl0, s01 + 4096);
                ldsm_x4(sh1, s23);
                ldsm_x4(sl1, s23 + 4096);
                mma3x4(acc[0], acc[1], acc[2], acc[3], Ch[ks], Cl[ks], sh0, sl0, sh1, sl1);
            }
            for (int jp = 0; jp < warp; ++jp) {            // tokens 16 jp .. 16 jp + 15
                float g0[4], g1[4];
                causal_product(jp, g0, g1);
                const float f = sc.seg[jp];
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[nt][e] *= f;
                add_wx(acc, g0, g1, jp);
            }
            const float ela = sc.eli[ia], elb = sc.eli[ib];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                y[nt][0] = fmaf(ela, acc[nt][0], y[nt][0]); y[nt][1] = fmaf(ela, acc[nt][1], y[nt][1]);
                y[nt][2] = fmaf(elb, acc[nt][2], y[nt][2]); y[nt][3] = fmaf(elb, acc[nt][3], y[nt][3]);
            }
        }
        // gated by silu(z) (model.rs:370); a lane has head dims 8 t4 .. 8 t4 + 7 of its two tokens
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int i = rr == 0 ? ia : ib;
            const float* const zr = &sm.rC[i][0];
            const float4 z0 = *reinterpret_cast<const float4*>(zr + ((2 * t4) ^ (i & 1)) * 4), z1 = *reinterpret_cast<const float4*>(zr + ((2 * t4 + 1) ^ (i & 1)) * 4);
            uint32_t vh[4], vl[4];
            split2(y[0][2 * rr] * silu_fast(z0.x), y[0][2 * rr + 1] * silu_fast(z0.y), vh[0], vl[0]);
            split2(y[1][2 * rr] * silu_fast(z0.z), y[1][2 * rr + 1] * silu_fast(z0.w), vh[1], vl[1]);
            split2(y[2][2 * rr] * silu_fast(z1.x), y[2][2 * rr + 1] * silu_fast(z1.y), vh[2], vl[2]);
            split2(y[3][2 * rr] * silu_fast(z1.z), y[3][2 * rr + 1] * silu_fast(z1.w), vh[3], vl[3]);
            if (valid(i)) {
                const size_t o = ((size_t)b * tsl + t0 + i) * DI + h * P + 8 * t4;
                *reinterpret_cast<uint4*>(a.yhi + o) = make_uint4(vh[0], vh[1], vh[2], vh[3]);
                if (a.ylo) *reinterpret_cast<uint4*>(a.ylo + o) = make_uint4(vl[0], vl[1], vl[2], vl[3]);
            }
        }
        if (warp == 0 && !last_chunk) prepare_scalars(t0 + LCH, sm.sc[(chunk + 1) & 1]);
        // ---- 6. S^ segment by segment: decay over the segment, + X^T B~ of its tokens, for this warp's 16 x 32 block
        const int pa = p0 + 8 * (lm & 1) + lr;
        const uint32_t aXA = tX + (uint32_t)(pa * 128 + (((lm >> 1) ^ key_of(pa)) << 4));                          // X^T rows as A fragments
        const uint32_t aBT = tB + (uint32_t)((8 * (lm & 1) + lr) * 256 + ((((n0 >> 3) + (lm >> 1)) ^ lr) << 4));  // B~ columns n0 .. as B fragments
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {                   // tokens 16 ks .. 16 ks + 15
            const float f = sc.seg[ks];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[nt][e] *= f;
            uint32_t ah[4], al[4], bh0[4], bl0[4], bh1[4], bl1[4];   // state columns n0 .. n0 + 15 and n0 + 16 .. n0 + 31
            const uint32_t xa = aXA ^ (uint32_t)(ks << 5), bt = aBT + (uint32_t)(ks * 4096);
            ldsm_x4(ah, xa);
            ldsm_x4(al, xa + 4096);
            ldsm_x4_trans(bh0, bt);
            ldsm_x4_trans(bl0, bt + 128);
            ldsm_x4_trans(bh1, bt ^ 32u);
            ldsm_x4_trans(bl1, (bt ^ 32u) + 128);
            mma3x4(S[0], S[1], S[2], S[3], ah, al, bh0, bl0, bh1, bl1);
        }
        // every operand tile and raw row of this chunk has been consumed: order these generic-proxy accesses before the copies
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (!last_chunk && tid == 0) issue_chunk(t0 + LCH);
        return true;
    };
    bool failed = false;
    {
        int chunk = 0;
        for (int t0 = 0; t0 < ts && !failed; t0 += LCH, ++chunk) {
            const bool okc = (t0 + LCH <= ts) ? do_chunk(std::true_type{}, t0, chunk) : do_chunk(std::false_type{}, t0, chunk);
            failed = !okc;
        }
    }
    if (failed) {
        // the wait gave up: report, let this CTA's copies land (bounded) so nothing writes into shared memory after exit
        if (tid == 0) {
            if (a.status != nullptr) atomicOr(a.status, STATUS_TIMEOUT);
            mbar_wait(bar, phase ^ 1, kScanWaitLimitNs);      // the chunk that did not land: its phase has been turned already
        }
        __syncthreads();
        return;
    }
    // ---- hand-over: the exact decode state after the last token of this launch (kap = lam on it, so S^ = S)
    {
        float* hp = a.h + bh * (size_t)(P * N);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            *reinterpret_cast<float2*>(hp + (p0 + g4) * N + n0 + 8 * nt + 2 * t4) = make_float2(S[nt][0], S[nt][1]);
            *reinterpret_cast<float2*>(hp + (p0 + g4 + 8) * N + n0 + 8 * nt + 2 * t4) = make_float2(S[nt][2], S[nt][3]);
        }
    }
    if (warp == 0) a.cum[bh * HN + lane] = cum;
}

}  // namespace

// head_dim 32 and d_state 64 are what the fragments are laid out for; n_heads % 4 keeps every box of the staged
// projection rows on a 16-byte boundary (row pitch and the offsets of the theta columns)
bool prefill_ssd_supported(const Config& c) {
    return c.head_dim() == 32 && c.d_state == 64 && c.n_groups > 0 && c.n_heads % c.n_groups == 0 && c.n_heads % 4 == 0;
}

cudaError_t launch_prefill_embed(const void* emb, int dtype, const uint32_t* prompt, float* x, int D, int vocab, int rows, int ts,
                                 int t_abs0, int b_abs0, int batch_total, StepCtl* ctl, cudaStream_t st, const int32_t* lens, const EmbedPost& post) {
    if (dtype == LUMI_DTYPE_BF16)
        embed_rows_kernel<__nv_bfloat16><<<rows, 128, 0, st>>>((const __nv_bfloat16*)emb, prompt, x, D, vocab, ts, t_abs0, b_abs0, batch_total, ctl, lens, post);
    else
        embed_rows_kernel<float><<<rows, 128, 0, st>>>((const float*)emb, prompt, x, D, vocab, ts, t_abs0, b_abs0, batch_total, ctl, lens, post);
    return cudaGetLastError();
}

cudaError_t launch_bc_stats(const PrefillArgs& a, int P, int N, cudaStream_t st) {
    const int rows = a.nb * a.ts;
    bc_stats_kernel<<<(rows + 7) / 8, 256, 0, st>>>(a.proj, a.ldp, 2 * a.H * P, a.G * N, a.eps, a.rb, a.rc, rows);
    return cudaGetLastError();
}

cudaError_t launch_prefill_scan(const PrefillArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(PfSmem);
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(ssd_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        set = true;
    }
    const int rows = a.nb * a.ts;
    // the projection rows as a 2-D fp32 tensor [rows][ldp]; boxes of 64 tokens x 32 columns (x, theta) and x 64 (B, C)
    CUtensorMap m32, m64;
    if (make_f32_map_2d(&m32, a.proj, (uint64_t)rows, (uint64_t)a.ldp, (uint64_t)a.ldp * 4, 32, LCH) != LUMI_OK ||
        make_f32_map_2d(&m64, a.proj, (uint64_t)rows, (uint64_t)a.ldp, (uint64_t)a.ldp * 4, 64, LCH) != LUMI_OK)
        return cudaErrorInvalidValue;
    cudaError_t e = launch_bc_stats(a, 32, 64, st);
    if (e != cudaSuccess) return e;
    ssd_prefill_kernel<<<dim3(a.H, a.nb), 128, smem, st>>>(m32, m64, a);
    return cudaGetLastError();
}

cudaError_t launch_gather_last(const float* xr, float* x, int D, int ts, int nb, int b0, cudaStream_t st, const int32_t* lens, int t_abs0) {
    gather_last_kernel<<<nb, 256, 0, st>>>(xr, x, D, ts, b0, lens, t_abs0);
    return cudaGetLastError();
}

}  // namespace lumi

extern "C" int32_t lumi_debug_fmod_near(const float* x, int64_t n, float* out) {
    if (!x || !out || n < 0) return lumi::fail(LUMI_E_INVALID, "null argument");
    const float two_pi = 6.28318530717958647692f, inv = 0.15915494309189533577f;      // as the scan has them
    for (int64_t i = 0; i < n; ++i) out[i] = lumi::fmod_near(x[i], two_pi, inv);
    return LUMI_OK;
}
