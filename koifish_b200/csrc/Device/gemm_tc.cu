// gemm_tc.cu -- dequant-fused tensor-core GEMM on the 5th-generation tensor cores (tcgen05 / TMEM / TMA), persistent:
//   Y[M][N] = X[M][K] . deq(W[N][K])^T       tcgen05.mma kind::f16 (bf16 x bf16 -> fp32), accumulators in TMEM
//
// Replaces the same reference pair as gemv.cu: GTensor::GetDataX (whole-matrix dequant to a bf16 scratch,
// src/Device/CUDA/kernel/quantizer.cu:249-392) + CU_mm_blasLt (src/Device/CUDA/kernel/gemm.cu:93-214) behind SLP::Forw
// (src/Device/CUDA/NeuronFuse.cu:305-381).  The packed weights cross HBM once per token panel and are expanded on chip.
//
// Work item = [128 weight rows] x [BN tokens] x [one K range (split-K)].  The weights are the A operand (UMMA_M = 128), the tokens
// the B operand (UMMA_N = BN), BK = 64.  One CTA per SM walks the items round-robin; its 15 warps are specialised:
//   * warp 9  (1 thread): TMA of the PACKED weight bytes, up to 128 B per row per stage, into a raw ring (swizzled over the row, conflict-free reads);
//   * warp 10 (1 thread): TMA of the activation tile (already permuted, see below) into the B ring (SWIZZLE_128B, K-major);
//   * warps 0-7 (producers, thread = weight row; two teams take the raw stages in turn): raw bytes -> the reference's bit-exact bf16 weights (one rounding or two, as
//     gemv.cu; times a power of two that the sums get back) -> tcgen05.st into the A ring that lives in TENSOR MEMORY (lane = row, 2 weights / column);
//     the expanded weights never touch shared memory, which stays free for the B operand;
//   * warp 8  (1 thread): tcgen05.mma [D], [A in TMEM], B-descriptor; tcgen05.commit frees the stage / publishes the accumulator;
//   * warps 11-14 (epilogue): tcgen05.ld the accumulator into shared memory (it then goes back to the MMA warp), then the final store (bf16 / +residual /
//     SwiGLU / fp32) under the next item's main loop; the producers help with a CTA's last item (from 64 tokens).  With split-K the parts of a tile are the CTAs of a
//     cluster, which add up through distributed shared memory, or, where these do not fit on the GPU at once, fp32 partials in global memory + an
//     arrival counter; either way in the order of the parts (deterministic).
// bf16 weights need no expansion: warp 9 TMA-loads them straight into a swizzled A tile in shared memory (classic SS MMA).
// The k order inside every 32-wide slot is the extraction-friendly permutation of gemv.cu; kf_tc_prepare_x permutes the activations
// identically, so the contraction is unchanged.  Every barrier wait is bounded and traps instead of hanging the GPU.
#include <string.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <tuple>
#include <type_traits>

#include "kf_common.cuh"
#include "kf_tc.cuh"

// tuning experiments (bit 0: no expansion, 1: no TMEM store, 3: no weight copies, 4: no activation copies): debug builds only
// (KF_NVCC_DEFS="-DKF_DEBUG_KNOBS -DKF_TC_EXP=n"); a release build compiles them out
#if !defined(KF_DEBUG_KNOBS) || !defined(KF_TC_EXP)
#undef KF_TC_EXP
#define KF_TC_EXP 0
#endif

namespace {

enum { TF_BF16 = 0, TF_F8 = 1, TF_Q4 = 2, TF_Q2 = 3, TF_Q1 = 4 };
enum { TM_PLAIN = 0, TM_AFFINE = 1, TM_SCALE = 3, TM_AFFINE_FMA = 4 };  // _FMA: one bf16 rounding (ctx deq_fma, default), see kf_common.cuh

constexpr int BM = 128;    // weight rows per item (UMMA M)
constexpr int BK = 64;     // k per stage: 64 bf16 = one 128-byte swizzle row of the B tile
// packed bytes per weight row per raw stage: four k-blocks of the 4-, 2- and 1-bit formats (the swizzle spans a row), two of the 8-bit one.  A K split ends on a raw-stage
// boundary, and more than 256 weights are too coarse to balance 148 SMs (1-bit 25600x5120 at 32 tokens with 128 bytes: 71 us, 38 us with 64)
template <int FMT>
__host__ __device__ constexpr int raw_bytes() { return FMT == 4 ? 32 : FMT == 3 ? 64 : 128; }  // TF_Q1, TF_Q2
constexpr int kProducerWarps = 8, kMmaWarp = 8, kRawWarp = 9, kXWarp = 10, kEpiWarp0 = 11;
constexpr int kThreadsTC = 15 * 32;
constexpr int kTeams = 2;  // of four producer warps
constexpr int kNaturalBN = 128;  // token tiles from which activations may come in their own order

constexpr int kEpiGlu = 2;  // epilogue: y = silu(w0 x) * (w1 x); an item takes 64 rows of either weight
constexpr int kMaxW = 3;  // weights of one launch (Q/K/V, gate/up): same type, same K, their row tiles share one item space
struct GemmParams {
    const uint16_t* zero[kMaxW];
    const uint16_t* step[kMaxW];
    void* y[kMaxW];            // bf16 [M][N_w] (or float when epilogue == 4)
    int Nw[kMaxW];             // rows of each weight
    int tile0[kMaxW + 1];      // first row tile of each weight in the launch's tile space (unused entries: INT_MAX)
    const uint16_t* residual;  // bf16 [M][N] or nullptr (single weight)
    float* ws;                 // split-K partials
    unsigned* cnt;             // split-K arrival counters (self-resetting)
    int M, N, K;
    int gshift, epilogue;
    int n_tiles, m_tiles, splits, n_items;
    int staged;                // outputs (and residual) may be accessed 16 bytes at a time
    int cluster;               // the parts of a split are the CTAs of a cluster, one item each
    int item_lo, item_hi;      // item = (row tile * item_hi + hi) * item_lo + lo: token tile and part, the latter innermost in clusters
    int part_raw, part_rem;    // raw stages of a part; the first part_rem have one more
    uint32_t fold2;            // qbias as bf16x2 (types without a zero)
    int bias;                  // qbias does not fold into the zero: it is taken off the codes
    int natural;               // the activations are in their own order: the expanded weights are put into it
    uint32_t qsub[8];          // qbias as a number of each code field, bf16x2
};

template <int FMT>
struct Fmt {
    static constexpr int BITS  = FMT == TF_BF16 ? 16 : FMT == TF_F8 ? 8 : FMT == TF_Q4 ? 4 : FMT == TF_Q2 ? 2 : 1;
    static constexpr int SLOTB = 4 * BITS;                             // packed bytes of one 32-weight slot
    static constexpr int RAWB  = raw_bytes<FMT>();
    static constexpr int KBR   = FMT == TF_BF16 ? 2 : RAWB / (2 * SLOTB);  // k-blocks per raw stage (bf16: granularity of a K split)
};

// ---- k permutation inside a 32-wide slot (identical to gemv.cu's xperm) ------------------------------------------------------------
template <int FMT>
__host__ __device__ constexpr int tperm(int o) {
    const int u = o >> 3, e = o & 7;
    if (FMT == TF_Q4) return 8 * u + ((e & 1) ? 3 : 7) - (e >> 1);
    if (FMT == TF_Q2) return 16 * (u >> 1) + ((e & 1) ? 7 : 15) - (e >> 1) - 4 * (u & 1);
    if (FMT == TF_Q1) return ((e & 1) ? 15 : 31) - (e >> 1) - 4 * u;
    return o;
}
// 8 consecutive elements of a 32-wide slot in the permuted order.  The lanes of a quad hold the slot's four pieces of 8 (v: this lane's, natural order); the
// 4-bit order stays within a piece, the 2- and 1-bit orders take elements from the quad.  All lanes of the warp take part.
template <int FMT>
__device__ __forceinline__ uint4 permute_piece(const uint32_t (&v)[4], int lane) {
    auto pick = [](uint32_t a, int e0, uint32_t b, int e1) {  // elements e0 & 1 of a and e1 & 1 of b
        return __byte_perm(a, b, ((e0 & 1) ? 0x32u : 0x10u) | ((e1 & 1) ? 0x7600u : 0x5400u));
    };
    uint32_t o[4];
    if constexpr (FMT == TF_Q4) {
#pragma unroll
        for (int p = 0; p < 4; p++) o[p] = pick(v[tperm<FMT>(2 * p) >> 1], tperm<FMT>(2 * p), v[tperm<FMT>(2 * p + 1) >> 1], tperm<FMT>(2 * p + 1));
    } else {
        uint32_t s[16];
#pragma unroll
        for (int d = 0; d < 4; d++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[4 * d + j] = __shfl_sync(0xffffffffu, v[j], (lane & ~3) + d);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if ((lane & 3) == u) {
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const int e0 = tperm<FMT>(8 * u + 2 * p), e1 = tperm<FMT>(8 * u + 2 * p + 1);
                    o[p] = pick(s[e0 >> 1], e0, s[e1 >> 1], e1);
                }
            }
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
// A thread permutes pieces of 8 elements, kPermPieces of them in flight; a thread per slot of 32 read and wrote its 64 bytes in four strided accesses (1999 x 4096:
// 8.6 -> 6.3 us, 700 x 2048 4.3 -> 3.4)
constexpr int kPermPieces = 4;
template <int FMT>
__global__ void __launch_bounds__(256) kf_permute_x_kernel(uint16_t* __restrict__ xp, const uint16_t* __restrict__ x, size_t n_pieces) {
    const int lane = threadIdx.x & 31;
    const size_t i0 = (size_t)blockIdx.x * (256 * kPermPieces) + threadIdx.x;
    kf_grid_dependency_wait();    // x comes from the kernel before us ...
    x = behind_wait(x);
    kf_grid_launch_dependents();  // ... and only behind it may the matmul start to stream its weights (they might have been written there as well)
    uint4 v[kPermPieces];
#pragma unroll
    for (int c = 0; c < kPermPieces; c++) v[c] = i0 + c * 256 < n_pieces ? __ldg(reinterpret_cast<const uint4*>(x) + i0 + c * 256) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int c = 0; c < kPermPieces; c++) {
        const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
        const uint4 o       = permute_piece<FMT>(w, lane);
        if (i0 + c * 256 < n_pieces) reinterpret_cast<uint4*>(xp)[i0 + c * 256] = o;
    }
}

// RMSNorm (the arithmetic and summation order of kf_rmsnorm_kernel, ops.cu: bit-identical output) written directly in the permuted
// k order: one launch instead of norm + permute in front of the Q/K/V and gate/up launches.  Latency-bound, a block per row: NC > 0 pieces of 8 per thread stay in
// registers from the sum of squares to the result (dim <= 2048 NC), with the weights fetched beside them (1999 x 4096: 15 -> 9.7 us); NC = 0 reads
// the row again.
template <int FMT, int NC>
__global__ void __launch_bounds__(256) kf_rmsnorm_permute_kernel(uint16_t* __restrict__ xp, const uint16_t* __restrict__ x, const uint16_t* __restrict__ w,
                                                                  int dim, float eps) {
    __shared__ float red[32];
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    constexpr int NV = NC > 0 ? NC : 1;
    uint4 v[NV], g[NV];
    kf_grid_dependency_wait();  // as above
    x = behind_wait(x);
    kf_grid_launch_dependents();
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)blockIdx.x * dim);
    uint4* orow     = reinterpret_cast<uint4*>(xp + (size_t)blockIdx.x * dim);
    float ss = 0.f;
    auto add = [&](const uint4& p) {
        const uint32_t q[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float a = bf16lo(q[j]), b = bf16hi(q[j]);
            ss = fmaf(a, a, ss), ss = fmaf(b, b, ss);
        }
    };
    if (NC > 0) {
#pragma unroll
        for (int c = 0; c < NV; c++) v[c] = (tid + c * 256) * 8 < dim ? xr[tid + c * 256] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int c = 0; c < NV; c++) g[c] = (tid + c * 256) * 8 < dim ? __ldg(reinterpret_cast<const uint4*>(w) + tid + c * 256) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int c = 0; c < NV; c++)
            if ((tid + c * 256) * 8 < dim) add(v[c]);
    } else {
        for (int i = tid; i * 8 < dim; i += 256) add(xr[i]);
    }
    ss = block_sum(ss, red);
    const float s = 1.0f / sqrtf(fmaf(ss, 1.0f / (float)dim, eps));
    auto put = [&](int i, const uint4& p, const uint4& gg) {  // all lanes of a warp: dim is a multiple of 32 elements, a quad is in or out as a whole
        const uint32_t q[4] = {p.x, p.y, p.z, p.w}, gw[4] = {gg.x, gg.y, gg.z, gg.w};
        uint32_t n[4];
#pragma unroll
        for (int j = 0; j < 4; j++) n[j] = pack_bf16x2((bf16lo(q[j]) * s) * bf16lo(gw[j]), (bf16hi(q[j]) * s) * bf16hi(gw[j]));
        const uint4 o = permute_piece<FMT>(n, lane);
        if (i * 8 < dim) orow[i] = o;
    };
    if (NC > 0) {
#pragma unroll
        for (int c = 0; c < NV; c++) put(tid + c * 256, v[c], g[c]);
    } else {
        for (int i0 = 0; i0 * 8 < dim; i0 += 256) {
            const int i = i0 + tid;
            const bool in = i * 8 < dim;
            put(i, in ? xr[i] : make_uint4(0, 0, 0, 0), in ? __ldg(reinterpret_cast<const uint4*>(w) + i) : make_uint4(0, 0, 0, 0));
        }
    }
}
template <int FMT>
cudaError_t launch_norm_permute(kf_ctx* ctx, void* xp, const void* x, const void* w, int M, int K, float eps) {
    auto go = [&](auto kern) { return kf_launch_pdl(ctx, kern, dim3(M), dim3(256), 0, (uint16_t*)xp, (const uint16_t*)x, (const uint16_t*)w, K, eps); };
    if (K <= 2048) return go(kf_rmsnorm_permute_kernel<FMT, 1>);
    if (K <= 4096) return go(kf_rmsnorm_permute_kernel<FMT, 2>);
    if (K <= 8192) return go(kf_rmsnorm_permute_kernel<FMT, 4>);
    return go(kf_rmsnorm_permute_kernel<FMT, 0>);
}

// the warps that finish an item: the four of the epilogue, or these and the eight producers
__device__ __forceinline__ void epi_bar_sync(int nthr) {
    if (nthr == 128) asm volatile("bar.sync 1, 128;" ::: "memory");
    else asm volatile("bar.sync 2, 384;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local, int cta_rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(cta_rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

// Codes -> bf16 weights without a shift or a conversion: a code field that lies in the low byte of a 16-bit half IS the bf16 number code * 2^(bit - 133) (exponents 0 and
// 1 share their scale, so all 256 patterns are linear), so one AND picks a pair of codes out of a register (of the register >> 8 for the upper bytes) and one bf16 fma
// with step * 2^(133 - bit - 7) and -zero * 2^-7 rounds exactly as RN(step * code - zero) does, 2^7 smaller; the sums get the factor back (kUnscale, exact) on
// their way out of tensor memory.  Two instructions a pair instead of four and a shift, which run at half rate on two pipes.  (4-bit SwiGLU 51200 x 5120 at 45 tokens, with the leaner
// producer loop below and its larger stages: 65.5 -> 40.8 us, at 16 tokens 64 -> 38.4; ternary 24576 x 4096 at 45 36 -> 24.4.  The question for larger steps: 41.0 -> 41.8, 38.6 ->
// 38.9 and nothing.)
// With 2^-7 a step has to stay below four; stages with one of two or more (or that is no number) take the long way below, which holds every step.  A smaller factor would leave more of
// them to it, a larger one takes bits from the smallest weights: now all of 2^-119 and above keep theirs, and what is lost below is less than 2^-126.
constexpr int kWShift       = 7;
constexpr float kUnscale    = 128.f;
constexpr uint32_t kFarStep = 0x4000u;  // the bit of the exponent that says so
template <int BITS>
__host__ __device__ constexpr int n_fields() { return BITS <= 4 ? 8 / BITS : 1; }  // code fields of a byte
// per group: the multiplier of each field and -zero (one fma) or zero (two roundings), scaled
template <int FMT, int MODE>
struct Gama {
    static constexpr int BITS = FMT == TF_Q4 ? 4 : FMT == TF_Q2 ? 2 : FMT == TF_Q1 ? 1 : 8, NF = n_fields<BITS>();
    uint32_t s[NF], z;
    // fold: qbias as a bf16x2 power of two or zero, whose product with the step is exact (types without a zero of their own)
    __device__ __forceinline__ void set(uint32_t zero, uint32_t step, uint32_t fold2) {
        const uint32_t st2   = __byte_perm(step, 0u, 0x1010), z2 = __byte_perm(zero, 0u, 0x1010);
        const auto down      = [](uint32_t v, int e) {  // v * 2^e
            const uint32_t p = (uint32_t)(127 + e) << 7;
            return bf162_as_u32(__hmul2_rn(u32_as_bf162(v), u32_as_bf162(p | p << 16)));
        };
        s[0] = down(st2, 133 - kWShift);
#pragma unroll
        for (int f = 1; f < NF; f++) s[f] = down(s[0], -f * BITS);
        if (MODE == TM_SCALE) z = down(bf162_as_u32(__hmul2_rn(u32_as_bf162(st2), u32_as_bf162(fold2))), -kWShift) ^ 0x80008000u;
        else z = down(z2, -kWShift) ^ (MODE == TM_AFFINE_FMA ? 0x80008000u : 0u);
    }
};
// the codes at field f of both halves of `reg` -> bf16x2 weights * 2^-7.  BIAS: qbias (as a number of that field, qf) comes off the codes first
template <int FMT, int MODE, bool BIAS>
__device__ __forceinline__ uint32_t tdeq(uint32_t reg, int f, const Gama<FMT, MODE>& g, uint32_t qf) {
    constexpr int BITS = Gama<FMT, MODE>::BITS;
    uint32_t v         = reg & (((1u << BITS) - 1u) * 0x00010001u << (f * BITS));
    if (BIAS) v = bf162_as_u32(__hsub2_rn(u32_as_bf162(v), u32_as_bf162(qf)));  // a small integer of the field: exact
    if (MODE == TM_AFFINE_FMA || (MODE == TM_SCALE && !BIAS)) return bf162_as_u32(__hfma2(u32_as_bf162(v), u32_as_bf162(g.s[f]), u32_as_bf162(g.z)));
    const __nv_bfloat162 q = __hmul2_rn(u32_as_bf162(v), u32_as_bf162(g.s[f]));  // RN(step * k)
    if (MODE == TM_SCALE) return bf162_as_u32(q);
    return bf162_as_u32(__hsub2_rn(q, u32_as_bf162(g.z)));  // RN(that - zero)
}
__device__ __forceinline__ uint32_t tf8_pair(uint32_t reg, uint32_t sel) {
    uint32_t h2 = __byte_perm(reg, 0u, sel);
    uint32_t t  = ((h2 >> 3) & 0x0FE00FE0u) | (h2 & 0x80008000u);
    return bf162_as_u32(__hmul2_rn(u32_as_bf162(t), u32_as_bf162(0x77807780u)));
}

// Any step: the codes as numbers, qbias (q2) off them, the arithmetic at its own scale, then 2^-7 -> the same 16 registers as below
template <int FMT, int MODE>
__device__ __forceinline__ void expand_slot_far(uint32_t* o, const uint32_t* w, uint32_t zero, uint32_t step, uint32_t q2) {
    constexpr int BITS = Gama<FMT, MODE>::BITS, PR = 16 / BITS;
    const uint32_t st2 = __byte_perm(step, 0u, 0x1010), z2 = __byte_perm(zero, 0u, 0x1010) ^ (MODE == TM_AFFINE_FMA ? 0x80008000u : 0u);
    constexpr uint32_t down2 = (uint32_t)(127 - kWShift) * 0x00800080u;
#pragma unroll
    for (int p = 0; p < 16; p++) {
        const uint32_t v = w[16 / PR - 1 - p / PR] >> (p % PR * BITS) & ((1u << BITS) - 1u) * 0x00010001u;
        const __nv_bfloat162 k = __hsub2_rn(__hsub2_rn(u32_as_bf162(v | 0x43004300u), u32_as_bf162(0x43004300u)), u32_as_bf162(q2));
        __nv_bfloat162 x;
        if (MODE == TM_AFFINE_FMA) x = __hfma2(k, u32_as_bf162(st2), u32_as_bf162(z2));
        else x = __hmul2_rn(k, u32_as_bf162(st2));
        if (MODE == TM_AFFINE) x = __hsub2_rn(x, u32_as_bf162(z2));
        o[p] = bf162_as_u32(__hmul2_rn(x, u32_as_bf162(down2)));
    }
}

// Expand the 32 weights of one slot (codes in `w`, memory order) into 16 bf16x2 registers in the permuted k order.  qsub: qbias as a number of each field
template <int FMT, int MODE, bool BIAS>
__device__ __forceinline__ void expand_slot(uint32_t* o, const uint32_t* w, const Gama<FMT, MODE>& g, const uint32_t* qsub) {
    if constexpr (FMT == TF_F8) {  // 8 registers, natural order
#pragma unroll
        for (int r = 0; r < 8; r++) o[2 * r] = tf8_pair(w[r], 0x1404u), o[2 * r + 1] = tf8_pair(w[r], 0x3424u);
    } else {  // 4 / 2 / 1 registers, first codes in the LAST; o[p] takes the fields at bits b = p * BITS .. of both halves of its register
        constexpr int BITS = Gama<FMT, MODE>::BITS, PR = 16 / BITS, NF = Gama<FMT, MODE>::NF;
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const uint32_t r = w[16 / PR - 1 - p / PR];
            const int i      = p % PR;
            o[p] = tdeq<FMT, MODE, BIAS>(i < NF ? r : __byte_perm(r, 0u, 0x4321), i % NF, g, BIAS ? qsub[i % NF] : 0u);
        }
    }
}

// The same 32 weights from the permuted into their own order, in place: one byte permute a pair.  Register p of a word's P holds elements 2 P - 1 - p and P - 1 - p.
template <int FMT>
__device__ __forceinline__ void natural_order(uint32_t* o) {
    constexpr int P = 16 / Gama<FMT, TM_AFFINE>::BITS;
    if constexpr (FMT != TF_F8) {
#pragma unroll
        for (int b = 0; b < 16; b += P) {
            uint32_t n[P];
#pragma unroll
            for (int j = 0; j < P; j++) {
                const int p = (j < P / 2 ? P : 2 * P) - 1 - 2 * j;
                n[j] = __byte_perm(o[b + p], o[b + p - 1], j < P / 2 ? 0x7632 : 0x5410);
            }
#pragma unroll
            for (int j = 0; j < P; j++) o[b + j] = n[j];
        }
    }
}

// Ring depths.  The three rings are decoupled because their latencies differ: the raw ring hides DRAM latency (bytes in flight per SM
// = RS x 8 or 16 KB must cover ~2 us x 44 GB/s; at 256 tokens a stage lasts a microsecond and two do), the B ring hides the L2 round trip of the (small, L2-resident)
// activation tiles (a fourth one at 256 tokens: 4-bit SwiGLU 51200 x 5120 at 200 96.3 -> 94.4 us), the A ring only the on-chip producer -> MMA hand-off.  Sized so that
// shared memory, the epilogue's output buffer included, stays below 226 KB and tensor memory within 512 columns.
template <int FMT, int BN>
struct Rings {
    static constexpr bool A_TMEM = FMT != TF_BF16;
    // k-blocks per stage of the A and B rings: a poll and two commits cost the MMA warp as much as eight small matrix instructions
    static constexpr int U       = BN == 256 ? 1 : BN == 128 || FMT == TF_BF16 || FMT == TF_F8 ? 2 : 4;
    // threads that finish a CTA's last item, and its part of a cluster's sums: the producers help from 64 and from 128 tokens on.  Below that their way there takes
    // longer than their share (4-bit 4096 x 1024 at 20 tokens, whole: tile of 16 8.3 us with them, 7.8 without, of 32 8.05 and 7.8; tile of 64 at 40 tokens 8.5 and
    // 8.8; 3072 x 6144 in clusters, at 12 tokens 13.1 and 12.65, at 40 14.1 and 13.3)
    static constexpr int NFIN    = BN >= 64 ? 384 : 128;
    static constexpr int NSUM    = BN >= 128 ? 384 : 128;
    static constexpr int NACC    = (A_TMEM && BN == 256) ? 1 : 2;
    static constexpr int A_BYTES = A_TMEM ? 0 : BM * 128;
    static constexpr int SUB     = A_BYTES + BN * 128;  // one k-block of a stage: [A tile (bf16 weights only)][B tile]
    static constexpr int STAGE   = U * SUB;
    static constexpr int SA      = !A_TMEM ? 0 : (BN <= 64 ? 12 : 8) / U;
    static constexpr int SB      = (A_TMEM ? (BN == 16 ? 32 : BN == 32 ? 20 : BN == 64 ? 12 : BN == 128 ? 6 : FMT == TF_F8 ? 3 : 4)
                                           : (BN == 16 ? 10 : BN == 32 ? 10 : BN == 64 ? 8 : BN == 128 ? 6 : 4)) / U;
    static constexpr int RAWB    = raw_bytes<FMT>();
    static constexpr int RS      = !A_TMEM ? 0 : (BN <= 128 ? 96 : FMT == TF_F8 ? 64 : 32) * 1024 / (BM * 128) * (RAWB < 128 ? 2 : 1);

    // output buffer: the item's whole accumulator in bf16 where there is only one in tensor memory, which then goes back to the MMA warp after ~1.5 us of draining
    static constexpr int OUT     = BN == 16 ? 8 * 1024 : A_TMEM && BN > 64 ? BN * 256 : 16 * 1024;  // at least one read of tensor memory in fp32
    static constexpr size_t SMEM = (size_t)SB * STAGE + (size_t)RS * BM * RAWB + OUT + 1024;
    static_assert((size_t)SB * STAGE + (size_t)RS * BM * RAWB >= (size_t)BN * BM * 4, "the rings take the partial sums of a split over a cluster");
    static_assert(SMEM <= 226 * 1024, "shared memory budget");
    // A barrier's phase is one bit: a producer that waits for a stage must know that the use before the one it waits for is over.  Raw stages: the slots belong to the
    // teams, so that use was its own.  A stages: it has waited, at its last one, for a stage at most SA later
    static_assert(RS % kTeams == 0, "every team has raw stages of its own");
    static_assert(!A_TMEM || (kTeams - 1) * (Fmt<FMT>::KBR / U) + 1 <= SA, "a team is never two rounds of the A ring ahead");
};

struct Item {
    int n0, m0, z, tile;  // tile = tn * m_tiles + mt
    int wi;               // weight of the launch
    int kb0, kb1;         // k-block range
};
// In front of every role's first and last step: two divisions (five, with the ranges of the parts taken apart here, cost 0.5 us: 4-bit 4096 x 1024 at 20 tokens 8.6 -> 7.8
// with the help above, 4096 x 2048 in clusters at 12 8.9 -> 8.0)
template <int KBR>
__device__ __forceinline__ Item decode_item(const GemmParams& p, int item) {
    Item it;
    const int t = item / p.item_lo, lo = item % p.item_lo, tn = t / p.item_hi, hi = t % p.item_hi;
    const int mt = p.cluster ? hi : lo;
    it.z         = p.cluster ? lo : hi;
    it.wi = p.epilogue == kEpiGlu ? 0 : (tn >= p.tile0[1] ? 1 : 0) + (tn >= p.tile0[2] ? 1 : 0);
    it.n0 = p.epilogue == kEpiGlu ? tn * (BM / 2) : (tn - p.tile0[it.wi]) * BM, it.m0 = mt, it.tile = tn * p.m_tiles + mt;  // m0 = token-tile index (the caller scales it by BN)
    const int r0 = it.z * p.part_raw + min(it.z, p.part_rem), r1 = r0 + p.part_raw + (it.z < p.part_rem ? 1 : 0);
    it.kb0 = r0 * KBR, it.kb1 = min(r1 * KBR, p.K / BK);
    return it;
}

// Store NC consecutive tokens (the first `valid` of them exist) of weight row `grow`: bf16, bf16 + residual, or fp32.  The residual
// values are all fetched before the first store (y may alias the residual, element for element).
template <int NC>
__device__ __forceinline__ void store_cols(const GemmParams& p, void* y, int N, const float (&acc)[NC], int m_first, int valid, int grow) {
    const size_t idx0 = (size_t)m_first * N + grow;
    if (p.epilogue == 4) {
#pragma unroll
        for (int j = 0; j < NC; j++)
            if (j < valid) reinterpret_cast<float*>(y)[idx0 + (size_t)j * N] = acc[j];
        return;
    }
    uint16_t res[NC];
    if (p.epilogue == 1) {
#pragma unroll
        for (int j = 0; j < NC; j++) res[j] = j < valid ? p.residual[idx0 + (size_t)j * N] : (uint16_t)0;
    }
#pragma unroll
    for (int j = 0; j < NC; j++) {
        if (j < valid) {
            uint16_t b = f32_to_bf16_bits(acc[j]);  // the reference's GEMM output is bf16 (gemm.cu:124-126)
            if (p.epilogue == 1) b = f32_to_bf16_bits(bf16_bits_to_f32(res[j]) + bf16_bits_to_f32(b));
            reinterpret_cast<uint16_t*>(y)[idx0 + (size_t)j * N] = b;
        }
    }
}

template <int FMT, int MODE, int BN>
__global__ void __launch_bounds__(kThreadsTC, 1)
    kf_gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_w2,
                      const __grid_constant__ CUtensorMap tm_x, const GemmParams p) {
    using F                  = Fmt<FMT>;
    using C                  = Rings<FMT, BN>;
    constexpr bool A_TMEM    = C::A_TMEM;
    constexpr int KBR        = F::KBR;
    constexpr int SA         = C::SA;    // A ring (expanded weights, tensor memory, 32 columns per stage)
    constexpr int SB         = C::SB;    // B ring (activation tiles, shared memory; for bf16 weights the stage also holds the A tile)
    constexpr int RS         = C::RS;    // raw ring (packed weight bytes, shared memory)
    constexpr int NACC       = C::NACC;  // accumulator buffers in tensor memory
    constexpr int A_BYTES    = C::A_BYTES;
    constexpr int B_BYTES    = BN * 128;
    constexpr int STAGE      = C::STAGE;
    constexpr int SUB        = C::SUB;
    constexpr int U          = C::U;     // k-blocks per stage of the A and B rings
    constexpr int RAWB       = F::RAWB;
    constexpr int RAW_BYTES  = BM * RAWB;
    constexpr int A_COL0     = NACC * BN;  // TMEM: accumulators first, then the A ring
    constexpr int TMEM_NEED  = A_COL0 + SA * U * 32;
    constexpr int TMEM_COLS  = TMEM_NEED <= 32 ? 32 : TMEM_NEED <= 64 ? 64 : TMEM_NEED <= 128 ? 128 : TMEM_NEED <= 256 ? 256 : 512;
    static_assert(TMEM_NEED <= 512, "tensor memory has 512 columns");
    constexpr int SA1 = SA > 0 ? SA : 1, RS1 = RS > 0 ? RS : 1;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* raws  = tiles + (size_t)SB * STAGE;
    uint8_t* outs  = raws + (size_t)RS * RAW_BYTES;
    const bool glu = p.epilogue == kEpiGlu;
    __shared__ uint64_t a_full[SA1], a_empty[SA1], b_full[SB], b_empty[SB], raw_full[RS1], raw_empty[RS1], tmem_full[NACC], tmem_empty[NACC];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int last_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // weight stage `it` of the CTA (k-block kb of item w): packed bytes or, for bf16 weights, the A tiles themselves
    auto load_w = [&](const Item& w, int kb, uint32_t it) {
        const CUtensorMap* tm_w = w.wi == 0 ? &tm_w0 : w.wi == 1 ? &tm_w1 : &tm_w2;
        if constexpr (A_TMEM) {
            const int rs = it % RS1, r = kb / KBR;
#if KF_TC_EXP & 8
            mbar_arrive(&raw_full[rs]);
#else
            mbar_arrive_expect_tx(&raw_full[rs], RAW_BYTES);
            tma_load_2d(raws + (size_t)rs * RAW_BYTES, tm_w, r * RAWB, w.n0, &raw_full[rs]);
            if (glu) tma_load_2d(raws + (size_t)rs * RAW_BYTES + RAW_BYTES / 2, &tm_w1, r * RAWB, w.n0, &raw_full[rs]);
#endif
        } else {
            const int s = it % SB;
            mbar_arrive_expect_tx(&b_full[s], U * A_BYTES);
#pragma unroll
            for (int u = 0; u < U; u++) {
                tma_load_2d(tiles + (size_t)s * STAGE + u * SUB, tm_w, (kb + u) * BK, w.n0, &b_full[s]);
                if (glu) tma_load_2d(tiles + (size_t)s * STAGE + u * SUB + A_BYTES / 2, &tm_w1, (kb + u) * BK, w.n0, &b_full[s]);
            }
        }
    };
    constexpr int WKB = A_TMEM ? KBR : U, WRING = A_TMEM ? RS1 : SB;  // k-blocks of a weight stage, stages of its ring
    if (warp == kRawWarp && lane == 0) {
        for (int s = 0; s < SA; s++) mbar_init(&a_full[s], 4), mbar_init(&a_empty[s], 1);  // one arrival per producer WARP of a team
        for (int s = 0; s < SB; s++) mbar_init(&b_full[s], A_TMEM ? 1 : 2), mbar_init(&b_empty[s], 1);
        for (int s = 0; s < RS; s++) mbar_init(&raw_full[s], 1), mbar_init(&raw_empty[s], 4);
        for (int s = 0; s < NACC; s++) mbar_init(&tmem_full[s], 1), mbar_init(&tmem_empty[s], 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // all 512 columns start at address 0: a constant keeps the MMA warp's operands in uniform registers, a value out of shared memory would be moved there for each instruction
    const uint32_t tmem_base = TMEM_COLS == 512 ? 0u : tmem_base_smem;
    kf_grid_launch_dependents();

    // ============ the end of an item: TMEM -> registers -> output buffer in shared memory -> Y in 16-byte accesses, or partial sums of a split.  Runs on the
    // four epilogue warps while the other roles work on the next item, and from 64 tokens on these and the eight producer warps (three to a quarter of the lanes) for
    // the CTA's last item, where nothing else is left to do.  Four warps took 4 us for the 256 tokens of an item and 10 with SwiGLU, in front of which the matrix
    // instructions of the next item waited: there is no second accumulator beside 256 columns and the A ring (4-bit SwiGLU 51200 x 5120 at 2048 tokens 836 -> 736 us,
    // 6144 x 1024 at 700, one item per CTA, 22.1 -> 16.5) ============
    const int fin_t     = warp < kProducerWarps ? 128 + tid : tid - kEpiWarp0 * 32;  // 0 .. 127: epilogue warps
    const bool f32out   = p.epilogue == 4;
    auto sum_of         = [](uint32_t v) { return __uint_as_float(v) * (MODE == TM_PLAIN ? 1.0f : kUnscale); };
    constexpr int kRes  = 4;  // residual pieces in flight per thread
    // the residual of pieces j0 .. j0 + kRes - 1 of this thread: piece i = token t0 + i / 16, rows 8 (i % 16) ..
    auto fetch_res = [&](uint4 (&res)[kRes], const Item& w, int m0, int N, int t0, int t1, int j0, int nthr) {
#pragma unroll
        for (int j = 0; j < kRes; j++) {
            const int i = fin_t + (j0 + j) * nthr, t = t0 + (i >> 4), n = w.n0 + (i & 15) * 8;
            res[j]      = t < t1 && n < N ? *reinterpret_cast<const uint4*>(p.residual + (size_t)(m0 + t) * N + n) : make_uint4(0, 0, 0, 0);
        }
    };
    // output buffer (tokens t0 .. t1 of the item) -> Y ; res: the first kRes pieces of the residual
    auto copy_out = [&](uint4 (&res)[kRes], const Item& w, int m0, int N, int t0, int t1, int nthr) {
        void* const y = p.y[w.wi];
        if (glu) {
            for (int i = fin_t; i < (t1 - t0) * 8; i += nthr) {
                const int t = i >> 3, n = w.n0 + (i & 7) * 8;
                if (n >= N) continue;
                const uint4 g4 = *reinterpret_cast<const uint4*>(outs + t * 256 + (i & 7) * 16), u4 = *reinterpret_cast<const uint4*>(outs + t * 256 + 128 + (i & 7) * 16);
                const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {  // CU_swiglu_v0 on the bf16 gate / up (Activation.cu:86-93), as kf_swiglu computes it
                    const float g0 = bf16lo(g[j]), g1 = bf16hi(g[j]), u0 = bf16lo(u[j]), u1 = bf16hi(u[j]);
                    v[j] = pack_bf16x2((g0 * u0) / (1.0f + expf(-g0)), (g1 * u1) / (1.0f + expf(-g1)));
                }
                *reinterpret_cast<uint4*>((uint16_t*)y + (size_t)(m0 + t0 + t) * N + n) = make_uint4(v[0], v[1], v[2], v[3]);
            }
        } else if (f32out) {
            for (int i = fin_t; i < (t1 - t0) * 32; i += nthr) {
                const int t = i >> 5, n = w.n0 + (i & 31) * 4;
                if (n < N) *reinterpret_cast<uint4*>((float*)y + (size_t)(m0 + t0 + t) * N + n) = *reinterpret_cast<const uint4*>(outs + i * 16);
            }
        } else {
            for (int j0 = 0; j0 * nthr < (t1 - t0) * 16; j0 += kRes) {
                if (p.epilogue == 1 && j0 > 0) fetch_res(res, w, m0, N, t0, t1, j0, nthr);
#pragma unroll
                for (int j = 0; j < kRes; j++) {
                    const int i = fin_t + (j0 + j) * nthr, t = t0 + (i >> 4), n = w.n0 + (i & 15) * 8;
                    if (t >= t1 || n >= N) continue;
                    uint4 v4 = *reinterpret_cast<const uint4*>(outs + i * 16);
                    if (p.epilogue == 1) {
                        const uint32_t r[4] = {res[j].x, res[j].y, res[j].z, res[j].w};
                        uint32_t v[4]       = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                        for (int q = 0; q < 4; q++) v[q] = pack_bf16x2(bf16lo(r[q]) + bf16lo(v[q]), bf16hi(r[q]) + bf16hi(v[q]));
                        v4 = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                    *reinterpret_cast<uint4*>((uint16_t*)y + (size_t)(m0 + t) * N + n) = v4;
                }
            }
        }
    };
    // the sums of rows 4 lane .. 4 lane + 3 of token t -> output buffer that starts at token t0, or Y
    auto put4 = [&](const Item& w, int m0, int N, int t0, int t, const float4& f) {
        if (p.staged) {
            if (f32out) *reinterpret_cast<float4*>(outs + (t - t0) * 512 + lane * 16) = f;
            else *reinterpret_cast<uint2*>(outs + (t - t0) * 256 + lane * 8) = make_uint2(pack_bf16x2(f.x, f.y), pack_bf16x2(f.z, f.w));
            return;
        }
        const float v[4] = {f.x, f.y, f.z, f.w};
        for (int j = 0; j < 4; j++) {
            const float one[1] = {v[j]};
            if (w.n0 + lane * 4 + j < N) store_cols<1>(p, p.y[w.wi], N, one, m0 + t, 1, w.n0 + lane * 4 + j);
        }
    };
    auto finish = [&](const Item& w, uint32_t ait, int et, int nthr) {
        constexpr int TC = BN < 32 ? 16 : 32;  // tokens of one read of tensor memory
        const int quad = warp & 3, row = quad * 32 + lane, part = et >> 7, nparts = nthr >> 7;
        const int buf = ait % NACC, m0 = w.m0 * BN, cnt = min(BN, p.M - m0), N = p.Nw[w.wi];
        const int round = C::OUT / (f32out ? 512 : 256);  // tokens that the output buffer takes
        const uint32_t tbase = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
        const bool direct = p.splits == 1 && p.staged;
        uint4 res[kRes];
        if (direct && p.epilogue == 1) fetch_res(res, w, m0, N, 0, min(cnt, round), 0, nthr);
        epi_bar_sync(nthr);  // the output buffer is free
        if (nthr == 128) mbar_wait_sleepy(&tmem_full[buf], (ait / NACC) & 1, NACC == 2 ? 200 : 20);  // a main loop away: poll politely
        else mbar_wait(&tmem_full[buf], (ait / NACC) & 1);
        tc_fence_after();
        auto release = [&]() {  // the accumulator buffer may be overwritten by the next item
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && warp >= kEpiWarp0) mbar_arrive(&tmem_empty[buf]);
        };
        if (direct) {
            for (int r0 = 0; r0 < cnt; r0 += round) {
                const int r1 = min(cnt, r0 + round);
                if (r0 > 0) {
                    epi_bar_sync(nthr);
                    if (p.epilogue == 1) fetch_res(res, w, m0, N, r0, r1, 0, nthr);
                }
                for (int c0 = r0 + part * TC; c0 < r1; c0 += nparts * TC) {
                    uint32_t v[TC];
                    if constexpr (TC == 16) tmem_ld16(tbase + (uint32_t)c0, v);
                    else tmem_ld32(tbase + (uint32_t)c0, v);
#pragma unroll
                    for (int j = 0; j < TC; j++) {
                        const float sum = sum_of(v[j]);
                        if (f32out) *reinterpret_cast<float*>(outs + (c0 - r0 + j) * 512 + row * 4) = sum;
                        else *reinterpret_cast<uint16_t*>(outs + (c0 - r0 + j) * 256 + row * 2) = f32_to_bf16_bits(sum);  // the reference's GEMM output is bf16 (gemm.cu:124-126)
                    }
                }
                if (r1 == cnt) release();
                epi_bar_sync(nthr);
                copy_out(res, w, m0, N, r0, r1, nthr);
            }
            return;
        }
        float* wsp = p.ws + ((size_t)w.tile * p.splits + w.z) * (size_t)(BN * BM);
        for (int c0 = part * 16; c0 < cnt; c0 += nparts * 16) {
            uint32_t v[16];
            tmem_ld16(tbase + (uint32_t)c0, v);
            if (p.splits > 1) {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (c0 + j < cnt) wsp[(size_t)(c0 + j) * BM + row] = sum_of(v[j]);
            } else if (w.n0 + row < N) {
                float acc[16];
#pragma unroll
                for (int j = 0; j < 16; j++) acc[j] = sum_of(v[j]);
                store_cols<16>(p, p.y[w.wi], N, acc, m0 + c0, cnt - c0, w.n0 + row);
            }
        }
        release();
        if (p.splits == 1) return;
        __threadfence();
        epi_bar_sync(nthr);
        if (et == 0) {
            const unsigned old = atomicAdd(&p.cnt[w.tile], 1u);
            last_flag          = (old == (unsigned)(p.splits - 1));
            if (last_flag) p.cnt[w.tile] = 0;  // self-reset for the next launch
        }
        epi_bar_sync(nthr);
        if (!last_flag) return;
        __threadfence();
        const float* base = p.ws + (size_t)w.tile * p.splits * (size_t)(BN * BM);
        // a thread sums four rows of one token (16-byte loads), two tokens and four partials in flight; the partials are added in split order
        for (int r0 = 0; r0 < cnt; r0 += round) {
            const int r1 = min(cnt, r0 + round), nw = nthr >> 5;
            if (r0 > 0) epi_bar_sync(nthr);
            if (p.epilogue == 1 && p.staged) fetch_res(res, w, m0, N, r0, r1, 0, nthr);
            for (int t = r0 + (et >> 5); t < r1; t += 2 * nw) {
                const bool two  = t + nw < r1;
                const float* b0 = base + (size_t)t * BM + lane * 4;
                float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
#pragma unroll 4
                for (int z = 0; z < p.splits; z++) {
                    const float4 a = __ldcg(reinterpret_cast<const float4*>(b0 + (size_t)z * (BN * BM)));
                    const float4 c = two ? __ldcg(reinterpret_cast<const float4*>(b0 + (size_t)z * (BN * BM) + nw * BM)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    s0.x += a.x, s0.y += a.y, s0.z += a.z, s0.w += a.w;
                    s1.x += c.x, s1.y += c.y, s1.z += c.z, s1.w += c.w;
                }
                put4(w, m0, N, r0, t, s0);
                if (two) put4(w, m0, N, r0, t + nw, s1);
            }
            if (p.staged) {
                epi_bar_sync(nthr);
                copy_out(res, w, m0, N, r0, r1, nthr);
            }
        }
        epi_bar_sync(nthr);  // last_flag is rewritten by the next item
    };

    if (warp < kProducerWarps) {
        if constexpr (A_TMEM) {
            // ============ producers: raw bytes -> bf16 -> TMEM.  Teams of four warps take the raw stages in turn; a warp expands all of a stage for 32 weight rows
            // (thread = row).  What bounds them is the number of instructions: with the two slots of 32 weights on two warps, a poll of the free A stage and a wait for the
            // stores per two k-blocks, and zero / step fetched by both warps, 440 clk a k-block were spent where the bytes take 187; now 250.  A second set of eight warps
            // gained nothing once the loop was lean (41.4 us against 40.9) ============
            constexpr int NW = F::SLOTB / 4;                           // registers of one packed slot of 32 weights
            constexpr int SPR = KBR / U, TEAMS = kTeams;  // A stages of a raw stage
            const int quad = warp & 3, team = warp >> 2;
            const int row = quad * 32 + lane, gpr = (p.K >> 7) >> p.gshift;
            // the row's first byte in a raw stage.  TMA swizzle: the 16-byte chunk index is XORed with address bits [7,8) (32-byte rows) / [7,9) (64) / [7,10) (128)
            const uint32_t rsw     = RAWB == 32 ? (uint32_t)((row >> 2) & 1) : RAWB == 64 ? (uint32_t)((row >> 1) & 3) : (uint32_t)(row & 7);
            const uint32_t raw_row = smem_u32(raws) + (uint32_t)(row * RAWB) + (rsw << 4);
            const uint32_t a_row   = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)A_COL0;
            const uint32_t full0 = smem_u32(&a_full[0]), empty0 = smem_u32(&a_empty[0]);
            const uint32_t rfull0 = smem_u32(&raw_full[0]), rempty0 = smem_u32(&raw_empty[0]);
            // zero / step of the groups in a raw stage; fetched a round ahead (the first beside the first weights, which are as long on their way)
            constexpr int GN = KBR / 2;
            uint32_t zn[GN] = {}, sn[GN] = {};
            const uint16_t *zrow = nullptr, *srow = nullptr;
            auto rows_of = [&](const Item& w) {
                if constexpr (MODE != TM_PLAIN) {
                    const int seg  = glu ? row >> 6 : w.wi;
                    const int grow = min(w.n0 + (glu ? row & 63 : row), p.Nw[seg] - 1);
                    zrow = p.zero[seg] + (size_t)grow * gpr, srow = p.step[seg] + (size_t)grow * gpr;
                }
            };
            auto fetch_gama = [&](int r) {
                if constexpr (MODE != TM_PLAIN) {
#pragma unroll
                    for (int j = 0; j < GN; j++) {
                        const int g = min((r * (KBR / 2) + j) >> p.gshift, gpr - 1);
                        zn[j] = __ldg(zrow + g), sn[j] = __ldg(srow + g);
                    }
                }
            };
            enum { kPlainWay, kBias, kFar };
            uint32_t a0 = 0, raw0 = 0;  // A and raw stages of the items so far
            int item = blockIdx.x, r = 0, re = 0, kend = 0;  // the item to open next, the raw stage of the one at hand, its end and that of its k-blocks
            uint32_t s = 0, eph = 0, rs = 0, rph = 0;
            Item w = decode_item<KBR>(p, item);
            auto first = [&]() { return w.kb0 / KBR + (int)(((uint32_t)team + raw0) % (uint32_t)TEAMS); };  // the team's first raw stage of an item
            auto next_item = [&]() {  // and its first zero / step
                item += gridDim.x;
                if (item < p.n_items) w = decode_item<KBR>(p, item), rows_of(w), fetch_gama(first());
            };
            rows_of(w), fetch_gama(first());
            // the stages from the one at hand: to the end, or (not kFar) up to one with a step that the quick expansion does not hold
            auto produce = [&](auto way) {
                constexpr int WAY = decltype(way)::value;
                for (;;) {
                    while (r < re) {
                        const int nk = kend - r * KBR;  // k-blocks from here to the end of the part: an even number
                        mbar_wait_a(rfull0 + rs * 8, rph);
                        if constexpr (MODE != TM_PLAIN && WAY != kFar) {  // in any row of the warp
                            uint32_t top = 0;
#pragma unroll
                            for (int j = 0; j < GN; j++) top |= sn[j];
                            if (__any_sync(0xffffffffu, top & kFarStep)) return;
                        }
                        const uint32_t src = raw_row + rs * RAW_BYTES;
                        uint32_t zc[GN], sc[GN];
#pragma unroll
                        for (int j = 0; j < GN; j++) zc[j] = zn[j], sc[j] = sn[j];
                        r += TEAMS;
                        if (r < re) fetch_gama(r);
                        else next_item();
                        Gama<FMT, MODE> gm;
#pragma unroll
                        for (int k = 0; k < KBR; k++) {
                            if (KBR > 2 && (k & 1) == 0 && k >= nk) break;
                            uint32_t v[2 * NW];  // both slots of the k-block, the first codes in the last register of each
                            if constexpr (F::SLOTB >= 16) {
#pragma unroll
                                for (int c = 0; c < NW / 2; c++) lds128(src ^ (uint32_t)((k * (NW / 2) + c) << 4), &v[4 * c]);
                            } else if constexpr (F::SLOTB == 8) {  // 16 bytes a k-block, the first slot in their upper half
                                uint32_t q[4];
                                lds128(src ^ (uint32_t)(k << 4), q);
                                v[0] = q[2], v[1] = q[3], v[2] = q[0], v[3] = q[1];
                            } else {  // 8 bytes a k-block, likewise in 16
                                uint32_t q[2];
                                lds64((src ^ (uint32_t)(k >> 1 << 4)) + ((k & 1) ? 0 : 8), q);
                                v[0] = q[1], v[1] = q[0];
                            }
                            if (WAY != kFar && MODE != TM_PLAIN && (k & 1) == 0) gm.set(zc[k / 2], sc[k / 2], p.fold2);
                            uint32_t o[32];
#if KF_TC_EXP & 1
                            for (int i = 0; i < 32; i++) o[i] = v[i % (2 * NW)] ^ gm.z;
#else
                            if constexpr (WAY == kFar) {
                                expand_slot_far<FMT, MODE>(o, &v[0], zc[k / 2], sc[k / 2], p.fold2);
                                expand_slot_far<FMT, MODE>(o + 16, &v[NW], zc[k / 2], sc[k / 2], p.fold2);
                            } else {
                                expand_slot<FMT, MODE, WAY == kBias>(o, &v[0], gm, p.qsub);
                                expand_slot<FMT, MODE, WAY == kBias>(o + 16, &v[NW], gm, p.qsub);
                            }
                            if constexpr (BN >= kNaturalBN) {  // below, the branch alone costs the producers 4 % (51200 x 5120 at 45 tokens 49.3 -> 51.2 us)
                                if (p.natural) natural_order<FMT>(o), natural_order<FMT>(o + 16);
                            }
#endif
                            if (k % U == 0) {
                                mbar_wait_a(empty0 + s * 8, eph);
                                tc_fence_after();
                            }
#if KF_TC_EXP & 2
                            asm volatile("" ::"r"(o[0] ^ o[5] ^ o[10] ^ o[15] ^ o[17] ^ o[22] ^ o[27] ^ o[31]));
#else
                            tmem_st32(a_row + s * (32 * U) + (k % U) * 32, o);
#endif
                            // The raw stage goes back to the loader with its last A stage: tcgen05.wait::st cannot complete before the weights it stores have been
                            // computed, so every byte of the stage has reached its register.  An arrival right behind the shared-memory loads is no such proof: it
                            // overtakes loads that still queue in the load / store unit (behind a burst of zero / step fetches at the start of an item), the loader
                            // refills the stage and lanes expand the bytes of the stage RS further on (4-bit 8192 x 5120 at 2048 tokens: every call wrong).  One
                            // arrival per warp: per-thread arrivals on one barrier word serialise in the shared-memory atomic unit.
                            if (k % U == U - 1 || (k & 1 && k + 1 >= nk)) {
                                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) {
                                    mbar_arrive_a(full0 + s * 8);
                                    if (k == KBR - 1 || (k & 1 && k + 1 >= nk)) mbar_arrive_a(rempty0 + rs * 8);
                                }
                                if (++s == SA) s = 0, eph ^= 1;
                            }
                        }
                        rs += TEAMS;
                        if (rs >= RS) rs -= RS, rph ^= 1;
                        // over the other teams' stages
                        constexpr int OVER = (TEAMS - 1) * SPR;
                        s += OVER % SA;
                        if (s >= SA) s -= SA, eph ^= 1;
                        if (OVER / SA & 1) eph ^= 1;
                    }
                    if (item >= p.n_items) return;
                    const int rb = w.kb0 / KBR;
                    re = (w.kb1 + KBR - 1) / KBR, kend = w.kb1, r = first();
                    const uint32_t a1 = a0 + (uint32_t)((r - rb) * SPR), raw1 = raw0 + (uint32_t)(r - rb);
                    s = a1 % SA, eph = (a1 / SA & 1u) ^ 1u, rs = raw1 % RS, rph = raw1 / RS & 1u;
                    a0 += (uint32_t)(w.kb1 - w.kb0 + U - 1) / U, raw0 += (uint32_t)(re - rb);
                    if (r >= re) next_item();
                }
            };
            if (MODE != TM_PLAIN && p.bias) produce(std::integral_constant<int, kBias>());
            else produce(std::integral_constant<int, kPlainWay>());
            // a loop of its own: within the one above, on its branch, the same code costs 4 % where the branch is never taken (51200 x 5120 at 45 tokens 41.1 -> 42.8 us)
            if constexpr (MODE != TM_PLAIN) produce(std::integral_constant<int, kFar>());
        }
    } else if (warp == kRawWarp) {
        if (lane == 0) {
            // ============ weight loader: packed bytes (or, for bf16, the A tile itself) by TMA ============
            uint32_t it = 0;
            for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
                const Item w = decode_item<KBR>(p, item);
                for (int kb = w.kb0; kb < w.kb1; kb += WKB, it++) {
                    mbar_wait(A_TMEM ? &raw_empty[it % RS1] : &b_empty[it % SB], ((it / WRING) & 1) ^ 1);
                    load_w(w, kb, it);
                }
            }
        }
    } else if (warp == kXWarp) {
        if (lane == 0) {
            // ============ activation loader: B tile by TMA (reads what the previous kernel wrote -> dependency wait first) ============
            kf_grid_dependency_wait();
            uint32_t it = 0;
            for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
                const Item w = decode_item<KBR>(p, item);
                for (int kb = w.kb0; kb < w.kb1; kb += U) {
                    const int s = it % SB;
                    mbar_wait(&b_empty[s], ((it / SB) & 1) ^ 1);
#if KF_TC_EXP & 16
                    mbar_arrive(&b_full[s]);
#else
                    mbar_arrive_expect_tx(&b_full[s], min(U, w.kb1 - kb) * B_BYTES);
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (u < 2 || kb + u < w.kb1) tma_load_2d(tiles + (size_t)s * STAGE + u * SUB + A_BYTES, &tm_x, (kb + u) * BK, w.m0 * BN, &b_full[s]);
#endif
                    it++;
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ============ MMA issuer.  The whole warp walks the loop converged (ring state and descriptors stay in uniform registers);
        // one elected lane -- always the same one -- issues the MMAs and the commits (elect.sync inside the asm) ============
        constexpr uint32_t idesc = make_idesc_bf16(BN);
        uint32_t ait = 0;
        uint32_t sa = 0, aph = 0, sb = 0, bph = 0;  // ring positions and the parities to wait for
        uint32_t okb = 0, oka = A_TMEM ? 0 : 1;
        const uint32_t bfull0 = smem_u32(&b_full[0]), bempty0 = smem_u32(&b_empty[0]);
        const uint32_t afull0 = smem_u32(&a_full[0]), aempty0 = smem_u32(&a_empty[0]);
        const uint32_t tiles0 = smem_u32(tiles);
        for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
            const Item w  = decode_item<KBR>(p, item);
            const int buf = ait % NACC;
            mbar_wait(&tmem_empty[buf], ((ait / NACC) & 1) ^ 1);
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
            uint32_t acc = 0;
            auto stage = [&](auto blocks) {
                if (!okb) mbar_wait_a(bfull0 + sb * 8, bph);
                if (!oka) mbar_wait_a(afull0 + sa * 8, aph);
                tc_fence_after();
#pragma unroll
                for (int u = 0; u < decltype(blocks)::value; u++) {
                    const uint32_t st_addr = tiles0 + sb * STAGE + u * SUB;
                    const uint64_t bdesc   = make_desc_sw128(st_addr + A_BYTES);
                    if constexpr (A_TMEM) {
                        const uint32_t ta = tmem_base + (uint32_t)(A_COL0 + sa * (32 * U) + u * 32);
                        umma_ts_x4(tmem_d, ta, bdesc, idesc, u > 0 ? 1u : acc);
                    } else {
                        const uint64_t adesc = make_desc_sw128(st_addr);
#pragma unroll
                        for (int k = 0; k < BK / 16; k++)
                            umma_ss(tmem_d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (k > 0 || u > 0) ? 1u : acc);
                    }
                }
                acc = 1;
                // the commits arrive when the MMAs above have finished reading the stages
                umma_commit_a(bempty0 + sb * 8);
                if (++sb == SB) sb = 0, bph ^= 1;
                if constexpr (A_TMEM) {
                    umma_commit_a(aempty0 + sa * 8);
                    if (++sa == SA) sa = 0, aph ^= 1;
                    oka = mbar_test(afull0 + sa * 8, aph);
                }
                okb = mbar_test(bfull0 + sb * 8, bph);  // the next stage's state, asked for ahead of the loop's bookkeeping (a poll takes ~90 cycles)
            };
            int kb = w.kb0;
            for (; kb + U <= w.kb1; kb += U) stage(std::integral_constant<int, U>());
            if (U > 2 && kb < w.kb1) stage(std::integral_constant<int, 2>());  // K is a multiple of 128
            umma_commit_a(smem_u32(&tmem_full[buf]));
            ait++;
        }
    } else {
        kf_grid_dependency_wait();  // residual / workspace / counters may still be in use by the previous kernel
        uint32_t ait = 0;
        const int last_item = blockIdx.x + (p.n_items - 1 - (int)blockIdx.x) / (int)gridDim.x * gridDim.x;
        for (int item = blockIdx.x; item < last_item; item += gridDim.x, ait++) {
            const Item w = decode_item<KBR>(p, item);
            finish(w, ait, (warp - kEpiWarp0) * 32 + lane, 128);
        }
    }
    constexpr int NFIN  = C::NFIN, NSUM = C::NSUM;
    const bool finisher = warp >= kEpiWarp0 || ((p.cluster ? NSUM : NFIN) == 384 && warp < kProducerWarps);
    if (finisher) {  // the last item
        if (warp < kProducerWarps) kf_grid_dependency_wait();
        if (!p.cluster) {
            const int last_ait = (p.n_items - 1 - (int)blockIdx.x) / (int)gridDim.x;
            finish(decode_item<KBR>(p, blockIdx.x + last_ait * gridDim.x), last_ait, fin_t, NFIN);
        } else {
            if (NACC == 2 && NSUM == 128) mbar_wait_sleepy(&tmem_full[0], 0, 200);
            else mbar_wait(&tmem_full[0], 0);
            tc_fence_after();
            const int quad = warp & 3, cnt = min(BN, p.M - decode_item<KBR>(p, blockIdx.x).m0 * BN);
            float* sums    = reinterpret_cast<float*>(tiles) + quad * 32 + lane;  // the rings are idle: this is the CTA's only item and its MMAs have completed
            for (int c0 = (fin_t >> 7) * 16; c0 < cnt; c0 += NSUM / 8) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int j = 0; j < 16; j++) sums[(c0 + j) * BM] = sum_of(v[j]);
            }
        }
    }
    // ============ split over a cluster: every CTA has its partial sums in shared memory and adds up its share of the tokens, in the order of the parts.  Takes
    // 3 us, of which the reads from the other CTAs are half; through global memory, where the last CTA to arrive did it all, 4-bit 4096 x 12288 at 300 tokens
    // took 75.5 us (now 46.4), 4096 x 4096 at 64 16.0 (11.6), 3072 x 6144 at 120 26.0 (14.7) ============
    if (p.cluster) {
        __syncwarp();
        cluster_arrive(), cluster_wait();
        if (finisher) {
            const Item w  = decode_item<KBR>(p, blockIdx.x);
            const int m0 = w.m0 * BN, cnt = min(BN, p.M - m0), N = p.Nw[w.wi];
            const int t0 = cnt * w.z / p.splits, t1 = cnt * (w.z + 1) / p.splits;
            const int round = C::OUT / (f32out ? 512 : 256);  // tokens that the output buffer takes
            const uint32_t part = smem_u32(tiles);
            uint4 res[kRes];
            for (int r0 = t0; r0 < t1; r0 += round) {
                const int r1 = min(t1, r0 + round);
                if (r0 > t0) epi_bar_sync(NSUM);
                if (p.epilogue == 1 && p.staged) fetch_res(res, w, m0, N, r0, r1, 0, NSUM);
                for (int t = r0 + (fin_t >> 5); t < r1; t += NSUM / 16) {  // a warp adds up two tokens at a time
                    const bool two = t + NSUM / 32 < r1;
                    float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
#pragma unroll 4
                    for (int z = 0; z < p.splits; z++) {
                        const float4 a = ld_cluster_f4(part + (uint32_t)(t * BM + lane * 4) * 4, z);
                        const float4 c = ld_cluster_f4(part + (uint32_t)((two ? t + NSUM / 32 : t) * BM + lane * 4) * 4, z);
                        s0.x += a.x, s0.y += a.y, s0.z += a.z, s0.w += a.w;
                        s1.x += c.x, s1.y += c.y, s1.z += c.z, s1.w += c.w;
                    }
                    put4(w, m0, N, r0, t, s0);
                    if (two) put4(w, m0, N, r0, t + NSUM / 32, s1);
                }
                if (p.staged) {
                    epi_bar_sync(NSUM);
                    copy_out(res, w, m0, N, r0, r1, NSUM);
                }
            }
        }
        __syncwarp();
        cluster_arrive(), cluster_wait();  // nobody leaves while others still read its sums
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
struct TmapKey {
    const void* base;
    uint64_t inner, outer;
    uint32_t box_inner, box_outer, dt, sw, esize;
    uint64_t planes, plane_stride;  // third dimension (1: a matrix)
    bool operator<(const TmapKey& o) const {
        return std::tie(base, inner, outer, box_inner, box_outer, dt, sw, esize, planes, plane_stride) <
               std::tie(o.base, o.inner, o.outer, o.box_inner, o.box_outer, o.dt, o.sw, o.esize, o.planes, o.plane_stride);
    }
};
// Maps of weights apart from those of what changes from call to call (activations and queries by their number of tokens, the cache by the number of sequences): a
// 64-layer model in steps of varying size makes 128 of the latter for every size, which must not cost the weights theirs.  Each is dropped when it is full.
struct TmapCache {
    std::map<TmapKey, CUtensorMap> maps[2];  // [0] weights: models hold a few hundred; [1] the others
};
constexpr size_t kTmapMost[2] = {4096, 16384};
EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return (EncodeTiledFn)f;
    }();
    return fn;
}
}  // namespace
static int tmap_encode(kf_ctx* ctx, CUtensorMap* tm, CUtensorMapDataType dt, int esize, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                       uint32_t box_outer, CUtensorMapSwizzle sw, uint64_t planes, uint64_t plane_stride, bool weight) {
    // a tensor map depends only on (address, geometry, box, swizzle): encode each once per context and reuse it (weights and the context's
    // activation scratch keep their addresses from token to token)
    TmapKey key = {base, inner, outer, box_inner, box_outer, (uint32_t)dt, (uint32_t)sw, (uint32_t)esize, planes, plane_stride};
    if (!ctx->tmap_cache) ctx->tmap_cache = new TmapCache();
    auto& cache = reinterpret_cast<TmapCache*>(ctx->tmap_cache)->maps[weight ? 0 : 1];
    auto hit    = cache.find(key);
    if (hit != cache.end()) {
        *tm = hit->second;
        return KF_OK;
    }
    EncodeTiledFn fn = encode_fn();
    KF_REQUIRE(ctx, fn != nullptr, "cuTensorMapEncodeTiled not available from the driver");
    KF_REQUIRE(ctx, ((uintptr_t)base & 15) == 0 && (inner * esize) % 16 == 0, "TMA needs 16-byte aligned rows");
    cuuint64_t dims[3]    = {inner, outer, planes};
    cuuint64_t strides[2] = {inner * (uint64_t)esize, plane_stride};
    cuuint32_t box[3]     = {box_inner, box_outer, 1};
    cuuint32_t estr[3]    = {1, 1, 1};
    CUresult r = fn(tm, dt, plane_stride ? 3 : 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char b[128];
        snprintf(b, sizeof(b), "cuTensorMapEncodeTiled failed (%d)", (int)r);
        ctx->last_error = b;
        return KF_ERR_CUDA;
    }
    if (cache.size() >= kTmapMost[weight ? 0 : 1]) cache.clear();
    cache[key] = *tm;
    return KF_OK;
}
int kf_tmap_2d(kf_ctx* ctx, CUtensorMap* tm, CUtensorMapDataType dt, int esize, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
               uint32_t box_outer, CUtensorMapSwizzle sw, bool weight) {
    return tmap_encode(ctx, tm, dt, esize, base, inner, outer, box_inner, box_outer, sw, 1, 0, weight);
}
int kf_tmap_count(const kf_ctx* ctx, bool weights) {
    return ctx->tmap_cache ? (int)reinterpret_cast<const TmapCache*>(ctx->tmap_cache)->maps[weights ? 0 : 1].size() : 0;
}
int kf_tmap_rows(kf_ctx* ctx, CUtensorMap* tm, const void* base, uint64_t inner, uint64_t rows, uint64_t planes, uint64_t plane_stride, uint32_t box_inner,
                 uint32_t box_rows) {
    return tmap_encode(ctx, tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, inner, rows, box_inner, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, planes, plane_stride,
                       false);
}
namespace {

// Row tiles of a launch: 128 rows of one weight each, or (SwiGLU) 64 rows of gate and the same 64 of up
int row_tiles(const GemmParams& p, int nw) {
    if (p.epilogue == kEpiGlu) return (p.Nw[0] + BM / 2 - 1) / (BM / 2);
    int n = 0;
    for (int i = 0; i < nw; i++) n += (p.Nw[i] + BM - 1) / BM;
    return n;
}
struct TcPlan {
    int bn, splits;
    bool cluster;
};
// CTAs of the kernel that can be resident in clusters of s (2 .. 8); 0 where the driver cannot say.  A property of the device, asked until it has answered; contexts of
// several threads may ask at once.
template <int FMT, int MODE, int BN>
int cluster_ctas(const kf_ctx* ctx, int s) {
    static std::atomic<int> known[kf_ctx::kMaxDevices][9];  // + 1
    std::atomic<int>& k = known[ctx->device][s];
    if (const int had = k.load(std::memory_order_relaxed)) return had - 1;
    auto kern = kf_gemm_tc_kernel<FMT, MODE, BN>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id               = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(ctx->sm_count / s * s)), cfg.blockDim = dim3(kThreadsTC), cfg.dynamicSmemBytes = Rings<FMT, BN>::SMEM;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Rings<FMT, BN>::SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    k.store(n * s + 1, std::memory_order_relaxed);
    return n * s;
}
template <int FMT, int MODE>
int cluster_ctas(const kf_ctx* ctx, int bn, int s) {
    switch (bn) {
        case 256: return cluster_ctas<FMT, MODE, 256>(ctx, s);
        case 128: return cluster_ctas<FMT, MODE, 128>(ctx, s);
        case 64: return cluster_ctas<FMT, MODE, 64>(ctx, s);
        case 32: return cluster_ctas<FMT, MODE, 32>(ctx, s);
        default: return cluster_ctas<FMT, MODE, 16>(ctx, s);
    }
}
template <int FMT, int MODE, int BN>
int launch_tc(kf_ctx* ctx, GemmParams& p, const void* const* wdata, int nw, const void* xp, const TcPlan& plan) {
    using F              = Fmt<FMT>;
    constexpr bool A_TMEM = FMT != TF_BF16;
    const size_t smem    = Rings<FMT, BN>::SMEM;
    auto kern            = kf_gemm_tc_kernel<FMT, MODE, BN>;
    static bool attr_set[kf_ctx::kMaxDevices] = {};  // function attributes are per device (one flag per instantiation and device)
    if (!attr_set[ctx->device]) {
        KF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[ctx->device] = true;
    }
    // ---- decomposition: row tiles x token tiles x split-K, walked round-robin by one CTA per SM ----
    const bool glu = p.epilogue == kEpiGlu;
    for (int i = 0, n = 0; i <= kMaxW; i++) {
        p.tile0[i] = i < nw && !(glu && i) ? n : 0x7fffffff;
        if (i < nw) n += (p.Nw[i] + BM - 1) / BM;
    }
    p.n_tiles = row_tiles(p, nw);
    p.m_tiles = (p.M + BN - 1) / BN;
    const int base_items = p.n_tiles * p.m_tiles;
    p.splits = plan.splits, p.n_items = base_items * plan.splits, p.cluster = plan.cluster;
    p.item_lo = plan.cluster ? plan.splits : p.m_tiles, p.item_hi = plan.cluster ? p.m_tiles : plan.splits;
    const int nraw = (p.K / BK + F::KBR - 1) / F::KBR;
    p.part_raw = nraw / plan.splits, p.part_rem = nraw % plan.splits;
    ctx->tc_last = BN | plan.splits << 12 | (plan.cluster ? 1 << 30 : 0);
    if (plan.splits > 1 && !plan.cluster) {
        int rc = kf_ensure_gemv_ws(ctx, (size_t)p.n_items * BN * BM * sizeof(float), base_items);
        if (rc) return rc;
        p.ws = ctx->gemv_ws, p.cnt = ctx->gemv_cnt;
    }
    CUtensorMap tm_w[kMaxW], tm_x;
    int rc = KF_OK;
    for (int i = 0; i < kMaxW && !rc; i++) {
        const int j = i < nw ? i : 0;  // unused slots repeat the first weight (never dereferenced)
        if (A_TMEM)
            rc = kf_tmap_2d(ctx, &tm_w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wdata[j], (uint64_t)p.K * F::BITS / 8, (uint64_t)p.Nw[j], F::RAWB, glu ? BM / 2 : BM,
                            F::RAWB == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : F::RAWB == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, true);
        else
            rc = kf_tmap_2d(ctx, &tm_w[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, wdata[j], (uint64_t)p.K, (uint64_t)p.Nw[j], BK, glu ? BM / 2 : BM,
                            CU_TENSOR_MAP_SWIZZLE_128B, true);
    }
    if (!rc) rc = kf_tmap_2d(ctx, &tm_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xp, (uint64_t)p.K, (uint64_t)p.M, BK, BN, CU_TENSOR_MAP_SWIZZLE_128B, false);
    if (rc) return rc;
    const int grid = std::min(p.n_items, ctx->sm_count);
    if (plan.cluster) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        attr[0].id               = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)plan.splits, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        attr[1].id               = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3(p.n_items), cfg.blockDim = dim3(kThreadsTC), cfg.dynamicSmemBytes = smem, cfg.stream = ctx->stream;
        cfg.attrs = attr, cfg.numAttrs = ctx->pdl ? 2 : 1;
        KF_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, tm_w[0], tm_w[1], tm_w[2], tm_x, p));
    } else {
        KF_CUDA(ctx, kf_launch_pdl(ctx, kern, dim3(grid), dim3(kThreadsTC), smem, tm_w[0], tm_w[1], tm_w[2], tm_x, p));
    }
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
// Token tile and k-split by their modelled time: waves x (k-blocks x time per k-block + epilogue) + the fix-up of split sums.  The times per k-block of 64 are
// measured ones (us; the 4-, 2- and 1-bit types share theirs; below 64 tokens the weights' bytes or their expansion, above the matrix
// instructions).  Splitting pays for few row tiles and a handful of tokens only: 1024 x 3072 at 16 tokens 9.9 us in 8 parts against 15.7 whole, at 256 tokens 34 against
// 17.  (The rule before it charged BN / 16 k-blocks for the fix-up: 1024 x 3072 at 256 tokens went into 12 parts and took 91 us.)  Parts that fit on the GPU as clusters
// cost no second pass, but the placement of the clusters, two barriers and the sum: 2.5 to 7 us, less for bf16 weights (the same for SwiGLU in the
// epilogue, so that it has the bits of gate and up written out first); a
// split through the workspace has a fixed cost of its own, which shows where it is one wave; so does the fetching of the same weights by several small token tiles.  Swept
// over 124 shapes, five types and 8 to 1000 tokens, every tile and up to 12 parts: the choice is 1.5 % behind the best in the mean, more than 5 % in 45 of 372 cases;
// with clusters at 1 us + 0.006 BN it was 2.0 % and 58 (1-bit SwiGLU 7680 x 1536 at 40 tokens went into two parts of 64, 12.2 us; whole 10.5).  The packed types were swept
// again with their lighter expansion, 90 shapes: 0.7 % behind the best, 5 cases above 5 %, with the earlier prices 2.8 % and 17.  The reference-exact
// arithmetic keeps the earlier rule and the order of sums it was compared in.
template <int FMT, int MODE>
int launch_tc_bn(kf_ctx* ctx, GemmParams& p, const void* const* wdata, int nw, const void* xp) {
    constexpr int KBR = Fmt<FMT>::KBR;
    const int nkb = p.K / BK, nraw = (nkb + KBR - 1) / KBR, tiles = row_tiles(p, nw);
    TcPlan plan = {256, 1, false};
    double best = 1e30;
    for (int b = 16, i = 0; b <= 256; b *= 2, i++) {
        const int by_m = p.M > 128 ? 256 : p.M > 64 ? 128 : p.M > 32 ? 64 : p.M > 16 ? 32 : 16;  // one token tile where the panel fits one
        if (ctx->tc_bn > 0 ? b != ctx->tc_bn : ctx->gemv_exact ? b != by_m : ((b < 256 && p.M > 8 * b) || (b > 16 && p.M <= b / 2))) continue;
        if (p.natural && b < kNaturalBN) continue;
        static const double kb_packed[5] = {0.154, 0.154, 0.15, 0.219, 0.361}, kb_f8[5] = {0.235, 0.235, 0.24, 0.26, 0.42}, kb_bf16[5] = {0.09, 0.10, 0.16, 0.24, 0.39};
        constexpr bool PACKED = FMT != TF_BF16 && FMT != TF_F8;
        const int m_tiles = (p.M + b - 1) / b, items = tiles * m_tiles;
        const double t_kb0 = FMT == TF_BF16 ? kb_bf16[i] : FMT == TF_F8 ? kb_f8[i] : kb_packed[i] * (p.natural && b == 128 ? 1.25 : 1.0);
        const int given = std::min(ctx->gemv_splitk, nraw);  // > 0: the split asked for
        for (int s = given > 0 ? given : 1; s <= (given > 0 ? given : std::min(16, nraw)); s++) {
            const int waves = (items * s + ctx->sm_count - 1) / ctx->sm_count, len = (nraw + s - 1) / s * KBR;
            if (ctx->gemv_exact) {
                const double c = waves * (len + 2.0 + (s > 1 ? b / 16.0 : 0.0));
                if (c < best * 0.95) best = c, plan = {b, s, false};
                continue;
            }
            const bool cluster = s > 1 && s <= 8 && items * s <= ctx->sm_count && items * s <= cluster_ctas<FMT, MODE>(ctx, b, s);
            // a workspace cannot grow inside a graph capture: a split that was not asked for is not chosen there before an eager call has sized it
            if (s > 1 && !cluster && given <= 0 && ctx->capturing && ((size_t)items * s * b * BM * sizeof(float) > ctx->gemv_ws_bytes || items > ctx->gemv_cnt_n)) continue;
            const double t_kb = t_kb0 * (waves == 1 && b <= 64 ? 1.0 + (PACKED ? 0.045 : 0.033) * (m_tiles - 1) : 1.0);
            const double t = cluster ? len * t_kb + (PACKED ? 2.9 : 2.5) + 0.017 * b + 0.03 * (s - 2) - (FMT == TF_BF16 ? 0.2 + 0.0025 * b : 0.0)
                                     : waves * (len * t_kb + (PACKED ? 0.6 : 0.5) + 0.006 * b + (s > 1 ? 0.5 + 0.02 * b : 0.0)) + (s > 1 ? b * (0.03 + 0.008 * s) + (waves == 1 ? 1.5 : 0.0) : 0.0);
            if (t < best * 0.98) best = t, plan = {b, s, cluster};
        }
    }
    switch (plan.bn) {
        case 256: return launch_tc<FMT, MODE, 256>(ctx, p, wdata, nw, xp, plan);
        case 128: return launch_tc<FMT, MODE, 128>(ctx, p, wdata, nw, xp, plan);
        case 64: return launch_tc<FMT, MODE, 64>(ctx, p, wdata, nw, xp, plan);
        case 32: return launch_tc<FMT, MODE, 32>(ctx, p, wdata, nw, xp, plan);
        default: return launch_tc<FMT, MODE, 16>(ctx, p, wdata, nw, xp, plan);
    }
}

int tc_format(const kf_tensor_desc* w, int* fmt, int* mode, int deq_fma) {
    switch (w->type) {
        case KF_T_BF16: *fmt = TF_BF16, *mode = TM_PLAIN; return KF_OK;
        case KF_T_F8E5M2: *fmt = TF_F8, *mode = TM_PLAIN; return KF_OK;
        case KF_T_Q4: *fmt = TF_Q4, *mode = deq_fma ? TM_AFFINE_FMA : TM_AFFINE; return KF_OK;
        case KF_T_Q2: *fmt = TF_Q2, *mode = deq_fma ? TM_AFFINE_FMA : TM_AFFINE; return KF_OK;
        case KF_T_SIGN: *fmt = TF_Q2, *mode = TM_SCALE; return KF_OK;
        case KF_T_BINARY: *fmt = TF_Q1, *mode = TM_SCALE; return KF_OK;
    }
    return KF_ERR_UNSUPPORTED;
}

// the bf16 number q * 2^(bit - 133), |q| < 256
uint32_t field_bf16(int q, int bit) {
    const float v = std::ldexp((float)q, bit - 133);  // exact, also below the normal range
    uint32_t u;
    memcpy(&u, &v, 4);
    return u >> 16;
}

}  // namespace
void kf_tmap_cache_destroy(kf_ctx* ctx) {
    delete reinterpret_cast<TmapCache*>(ctx->tmap_cache);
    ctx->tmap_cache = nullptr;
}

// The k order the tensor-core kernel expects for weights of w's type: identity for bf16 / f8, the extraction-friendly permutation
// inside every 32-wide slot for the packed types.  Returns x itself or the context's scratch holding the permuted copy.
int kf_tc_prepare_x(kf_ctx* ctx, const kf_tensor_desc* w, const void* x, int M, const void** xp_out) {
    int fmt, mode;
    if (tc_format(w, &fmt, &mode, 1)) return KF_ERR_UNSUPPORTED;
    if (fmt == TF_BF16 || fmt == TF_F8) {
        *xp_out = x;
        return KF_OK;
    }
    const int K         = w->cols;
    const size_t xbytes = (size_t)M * K * 2;
    int rc = kf_ensure_buf(ctx, &ctx->xperm, &ctx->xperm_bytes, xbytes);
    if (rc) return rc;
    const size_t n_pieces = (size_t)M * K / 8;
    const unsigned blocks = (unsigned)((n_pieces + 256 * kPermPieces - 1) / (256 * kPermPieces));
    auto go = [&](auto kern) { return kf_launch_pdl(ctx, kern, dim3(blocks), dim3(256), 0, (uint16_t*)ctx->xperm, (const uint16_t*)x, n_pieces); };
    KF_CUDA(ctx, fmt == TF_Q4 ? go(kf_permute_x_kernel<TF_Q4>) : fmt == TF_Q2 ? go(kf_permute_x_kernel<TF_Q2>) : go(kf_permute_x_kernel<TF_Q1>));
    KF_LAUNCH_CHECK(ctx);
    *xp_out = ctx->xperm;
    return KF_OK;
}
// RMSNorm + kf_tc_prepare_x in one launch (packed types); bf16 / f8 weights get the plain RMSNorm into the context's xnorm scratch
int kf_tc_prepare_x_norm(kf_ctx* ctx, const kf_tensor_desc* w, const void* x, const void* norm_w, float eps, int M, const void** xp_out) {
    int fmt, mode;
    if (tc_format(w, &fmt, &mode, 1)) return KF_ERR_UNSUPPORTED;
    const int K = w->cols;
    KF_REQUIRE(ctx, K % 32 == 0, "K");
    if (fmt == TF_BF16 || fmt == TF_F8) {
        int rc = kf_ensure_buf(ctx, &ctx->xnorm, &ctx->xnorm_bytes, (size_t)M * K * 2);
        if (!rc) rc = kf_rmsnorm(ctx, ctx->xnorm, x, norm_w, M, K, eps);
        *xp_out = ctx->xnorm;
        return rc;
    }
    int rc = kf_ensure_buf(ctx, &ctx->xperm, &ctx->xperm_bytes, (size_t)M * K * 2);
    if (rc) return rc;
    KF_CUDA(ctx, fmt == TF_Q4   ? launch_norm_permute<TF_Q4>(ctx, ctx->xperm, x, norm_w, M, K, eps)
                 : fmt == TF_Q2 ? launch_norm_permute<TF_Q2>(ctx, ctx->xperm, x, norm_w, M, K, eps)
                                : launch_norm_permute<TF_Q1>(ctx, ctx->xperm, x, norm_w, M, K, eps));
    KF_LAUNCH_CHECK(ctx);
    *xp_out = ctx->xperm;
    return KF_OK;
}
// 0 when both weights want the same activation order (one prepared copy serves both)
int kf_tc_same_order(const kf_tensor_desc* a, const kf_tensor_desc* b) {
    int fa, fb, ma, mb;
    if (tc_format(a, &fa, &ma, 1) || tc_format(b, &fb, &mb, 1)) return 1;
    const bool pa = !(fa == TF_BF16 || fa == TF_F8), pb = !(fb == TF_BF16 || fb == TF_F8);
    if (!pa && !pb) return 0;
    return fa == fb ? 0 : 1;
}

// xp: activations as returned by kf_tc_prepare_x for weights of this type, or in their own order anywhere but in its scratch (packed types: more work in the producers).  n <= 3 weights of the SAME storage type, K and group share
// one launch (their row tiles form one item space): Q/K/V and gate/up cost one kernel each instead of three / two.
int kf_gemm_tc_multi(kf_ctx* ctx, int n, void* const* y, const kf_tensor_desc* w, const void* xp, int M, int epilogue, const void* residual) {
    KF_REQUIRE(ctx, n >= 1 && n <= kMaxW && y && w && xp && M >= 1, "args");
    const int K = w[0].cols;
    int fmt, mode;
    if (tc_format(&w[0], &fmt, &mode, ctx->deq_fma)) return KF_ERR_UNSUPPORTED;
    GemmParams p;
    memset(&p, 0, sizeof(p));
    const void* wdata[kMaxW] = {};
    p.residual = (const uint16_t*)residual, p.M = M, p.K = K;
    p.epilogue = epilogue;
    if (mode != TM_PLAIN) {
        const int q = w[0].qbias, bits = fmt == TF_Q4 ? 4 : fmt == TF_Q2 ? 2 : 1;
        p.bias = mode == TM_SCALE ? (q & (q - 1)) != 0 : q != 0;
        for (int f = 0; f < 8 / bits; f++) p.qsub[f] = field_bf16(q, f * bits) * 0x00010001u;
        p.fold2 = field_bf16(q, 133) * 0x00010001u;
    }
    for (int i = 0; i < n; i++) {
        int f2, m2;
        KF_REQUIRE(ctx, y[i] && !tc_format(&w[i], &f2, &m2, ctx->deq_fma) && f2 == fmt && m2 == mode && w[i].cols == K && w[i].group == w[0].group &&
                            w[i].qbias == w[0].qbias,
                   "weights of one launch must share type, K, group");
        KF_REQUIRE(ctx, K % 128 == 0 && w[i].rows % 16 == 0, "K must be a multiple of 128, rows of 16");
        p.y[i] = y[i], p.Nw[i] = w[i].rows, wdata[i] = w[i].data_dev;
        if (mode != TM_PLAIN) {
            KF_REQUIRE(ctx, kf_has_gama(w[i]) && w[i].group >= 128 && (w[i].group & (w[i].group - 1)) == 0 && K % w[i].group == 0,
                       "group = 128 * 2^n dividing K");
            p.zero[i] = kf_gama_zero(w[i]), p.step[i] = kf_gama_step(w[i]);
        }
    }
    if (mode != TM_PLAIN) {
        int gs = 0;
        while ((128 << gs) < w[0].group) gs++;
        p.gshift = gs;
    }
    if (epilogue == 1) KF_REQUIRE(ctx, residual && n == 1, "residual: single weight");
    p.natural = fmt != TF_BF16 && fmt != TF_F8 && xp != ctx->xperm;
    p.staged  = ((uintptr_t)residual & 15) == 0;
    for (int i = 0; i < n; i++) p.staged = p.staged && ((uintptr_t)y[i] & 15) == 0;
    if (epilogue == kEpiGlu) KF_REQUIRE(ctx, n == 2 && w[0].rows == w[1].rows && y[0] == y[1] && p.staged, "SwiGLU: gate and up of equal shape, one 16-byte aligned output");
#define KF_TC_CASE(F, MD) \
    if (fmt == F && mode == MD) return launch_tc_bn<F, MD>(ctx, p, wdata, n, xp);
    KF_TC_CASE(TF_Q4, TM_AFFINE_FMA)
    KF_TC_CASE(TF_Q2, TM_AFFINE_FMA)
    KF_TC_CASE(TF_Q4, TM_AFFINE)
    KF_TC_CASE(TF_Q2, TM_AFFINE)
    KF_TC_CASE(TF_Q2, TM_SCALE)
    KF_TC_CASE(TF_Q1, TM_SCALE)
    KF_TC_CASE(TF_F8, TM_PLAIN)
    KF_TC_CASE(TF_BF16, TM_PLAIN)
#undef KF_TC_CASE
    return KF_ERR_UNSUPPORTED;
}
int kf_gemm_tc(kf_ctx* ctx, void* y, const kf_tensor_desc* w, const void* xp, int M, int epilogue, const void* residual) {
    void* ys[1] = {y};
    return kf_gemm_tc_multi(ctx, 1, ys, w, xp, M, epilogue, residual);
}
