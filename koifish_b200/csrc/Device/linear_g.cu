// linear_g.cu -- matmuls of ANY shape over bf16 weights with fp32 results, for the layers whose sizes the tuned kernels of gemv.cu /
// gemm_tc.cu do not take (their K must be a multiple of 128 and their N of 16): y[m][n] = sum_k x[m][k] * W[n][k].
//   * activations x are bf16 bits (act_f32 = 0: the products are exact in fp32 and accumulate in fp32, i.e. the arithmetic of a bf16
//     tensor-core matmul) or float (act_f32 = 1: a true 32-bit matmul, FMA by FMA, no reduced-precision mode);
//   * "grouped" form for mixtures of experts: every output row (a slot) names the weight matrix it uses; slots of one expert are
//     contiguous (offsets[e] .. offsets[e+1]) and may gather their input row through src_row;
//   * DUAL form: two weight tables A, B of equal shape and y = silu(A x) * (B x), the gate / up pair of a gated feed-forward, or its clamped
//     form y = g sigmoid(alpha g) (u + shift) with g = min(A x, limit), u = clamp(B x, -limit, limit);
//   * "batch" form for a handful of rows: several weights, each with an input and an output of its own, in one launch.
// A warp-per-output GEMV for a handful of rows (decode: every weight row is read once, 16-byte loads when the row length allows) and shared-memory tile kernels for
// panels: a cp.async ring with tcgen05 for bf16 activations (128 weight rows x 64 slots; mma.sync on 64 x 64 where that leaves most SMs idle), 64 x 64 tiles with
// FFMA for float ones (mma.sync for bf16 rows of odd lengths).
// No reference equivalent: the reference's SLP::Forw hands every shape to cuBLASLt (src/Device/CUDA/NeuronFuse.cu:305-381).
#include <algorithm>

#include "kf_common.cuh"
#include "kf_tc.cuh"

namespace {

struct LinArgs {
    const uint16_t* W0;          // single weight (dense) -- or
    const uint16_t* const* Wt0;  // table of per-expert weights (grouped)
    const uint16_t* W1;          // DUAL: second weight
    const uint16_t* const* Wt1;
    const void* x;               // [rows][ldx] bf16 bits or float
    void* y;                     // [slots][ldy] float (or, DUAL with out_act, the activation type)
    const int32_t* offsets;      // grouped: [E + 1] slot ranges; nullptr: one group [0, M)
    const int32_t* src_row;      // slot -> row of x; nullptr: slot
    const int32_t* slot_group;   // GEMV form: slot -> expert; nullptr: 0
    int M, N, K, ldx, ldy;
    int out_act;                 // DUAL or act != 0: 0 = float out, 1 = bf16 out, (float activations: float out)
    int act;                     // single-weight form: 0 = none, 1 = gelu (tanh form), 2 = relu squared, 3 = tanh, applied to the result
    int glu;                     // DUAL: 0 = silu(a) * b, 1 = the clamped form
    float limit, alpha, shift;   // ... its constants (limit <= 0: not clamped)
};
__device__ __forceinline__ float lin_act(float v, int act) {
    if (act == 1) return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    if (act == 2) return v > 0.f ? v * v : 0.f;
    if (act == 3) return tanhf(v);
    return v;
}

template <typename TA>
__device__ __forceinline__ float ld_act(const TA* p);
template <>
__device__ __forceinline__ float ld_act<uint16_t>(const uint16_t* p) { return bf16_bits_to_f32(*p); }
template <>
__device__ __forceinline__ float ld_act<float>(const float* p) { return *p; }

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float lin_pair(const LinArgs& a, float g, float u) {
    if (!a.glu) return silu_f(g) * u;
    if (a.limit > 0.f) g = fminf(g, a.limit), u = fminf(fmaxf(u, -a.limit), a.limit);
    return g / (1.f + expf(-a.alpha * g)) * (u + a.shift);
}

// ------------------------------------------------------------------------------------------------------------------ GEMV (few slots)
// one warp per (slot, output n): lanes stride over k, fixed butterfly reduction -> deterministic.
template <typename TA, bool DUAL>
__global__ void __launch_bounds__(256) kf_lin_gemv_kernel(LinArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n    = blockIdx.x * 8 + warp;
    const int slot = blockIdx.y;
    if (n >= a.N) return;
    const int g   = a.slot_group ? a.slot_group[slot] : 0;
    if (g < 0) return;  // a slot that no token uses
    const int row = a.src_row ? a.src_row[slot] : slot;
    const uint16_t* w0 = (a.Wt0 ? a.Wt0[g] : a.W0) + (size_t)n * a.K;
    const uint16_t* w1 = DUAL ? (a.Wt1 ? a.Wt1[g] : a.W1) + (size_t)n * a.K : nullptr;
    const TA* x = (const TA*)a.x + (size_t)row * a.ldx;
    float s0 = 0.f, s1 = 0.f;
    const bool vec = (a.K % 8 == 0) && (a.ldx % 8 == 0) && (((uintptr_t)w0 & 15) == 0) && (((uintptr_t)x & 15) == 0) && (!DUAL || ((uintptr_t)w1 & 15) == 0);
    if (vec) {
#pragma unroll DUAL ? 2 : 4
        for (int k = lane * 8; k < a.K; k += 256) {
            const uint4 wv = *reinterpret_cast<const uint4*>(w0 + k);
            const uint32_t wq[4] = {wv.x, wv.y, wv.z, wv.w};
            float xv[8];
            if (sizeof(TA) == 2) {
                const uint4 xq4 = *reinterpret_cast<const uint4*>((const uint16_t*)x + k);
                const uint32_t xq[4] = {xq4.x, xq4.y, xq4.z, xq4.w};
#pragma unroll
                for (int j = 0; j < 4; j++) xv[2 * j] = bf16lo(xq[j]), xv[2 * j + 1] = bf16hi(xq[j]);
            } else {
                const float4 f0 = *reinterpret_cast<const float4*>((const float*)x + k), f1 = *reinterpret_cast<const float4*>((const float*)x + k + 4);
                xv[0] = f0.x, xv[1] = f0.y, xv[2] = f0.z, xv[3] = f0.w, xv[4] = f1.x, xv[5] = f1.y, xv[6] = f1.z, xv[7] = f1.w;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) s0 = fmaf(bf16lo(wq[j]), xv[2 * j], s0), s0 = fmaf(bf16hi(wq[j]), xv[2 * j + 1], s0);
            if (DUAL) {
                const uint4 uv = *reinterpret_cast<const uint4*>(w1 + k);
                const uint32_t uq[4] = {uv.x, uv.y, uv.z, uv.w};
#pragma unroll
                for (int j = 0; j < 4; j++) s1 = fmaf(bf16lo(uq[j]), xv[2 * j], s1), s1 = fmaf(bf16hi(uq[j]), xv[2 * j + 1], s1);
            }
        }
    } else {
        for (int k = lane; k < a.K; k += 32) {
            const float xv = ld_act<TA>(x + k);
            s0 = fmaf(bf16_bits_to_f32(w0[k]), xv, s0);
            if (DUAL) s1 = fmaf(bf16_bits_to_f32(w1[k]), xv, s1);
        }
    }
    s0 = warp_sum(s0);
    if (DUAL) s1 = warp_sum(s1);
    if (lane == 0) {
        const float r = DUAL ? lin_pair(a, s0, s1) : lin_act(s0, a.act);
        if ((DUAL || a.act) && a.out_act == 1)
            ((uint16_t*)a.y)[(size_t)slot * a.ldy + n] = f32_to_bf16_bits(r);
        else
            ((float*)a.y)[(size_t)slot * a.ldy + n] = r;
    }
}

// Several independent products of one reduction length, each with its own weight, input and output, for a handful of rows: a warp per
// (row, output) as above; blockIdx.x walks the outputs of all of them one after the other.
constexpr int kBatchMax = 8;
struct BatchArgs {
    const uint16_t* W[kBatchMax];
    const void* x[kBatchMax];
    float* y[kBatchMax];
    int N[kBatchMax], ldy[kBatchMax], act[kBatchMax], first[kBatchMax + 1];  // first: the block at which a product starts
    int n, K, ldx;
};
template <typename TA>
__global__ void __launch_bounds__(256) kf_lin_gemv_batch_kernel(BatchArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.y;
    int j = 0;
#pragma unroll
    for (int i = 1; i < kBatchMax; i++)
        if (i < a.n && (int)blockIdx.x >= a.first[i]) j = i;
    const int n = ((int)blockIdx.x - a.first[j]) * 8 + warp;
    if (n >= a.N[j]) return;
    const uint16_t* w = a.W[j] + (size_t)n * a.K;
    const TA* x = (const TA*)a.x[j] + (size_t)row * a.ldx;
    float s = 0.f;
    if ((a.K % 8 == 0) && (a.ldx % 8 == 0) && (((uintptr_t)w & 15) == 0) && (((uintptr_t)x & 15) == 0)) {
#pragma unroll 4
        for (int k = lane * 8; k < a.K; k += 256) {
            const uint4 wv = *reinterpret_cast<const uint4*>(w + k);
            const uint32_t wq[4] = {wv.x, wv.y, wv.z, wv.w};
            float xv[8];
            if (sizeof(TA) == 2) {
                const uint4 xq4 = *reinterpret_cast<const uint4*>((const uint16_t*)x + k);
                const uint32_t xq[4] = {xq4.x, xq4.y, xq4.z, xq4.w};
#pragma unroll
                for (int i = 0; i < 4; i++) xv[2 * i] = bf16lo(xq[i]), xv[2 * i + 1] = bf16hi(xq[i]);
            } else {
                const float4 f0 = *reinterpret_cast<const float4*>((const float*)x + k), f1 = *reinterpret_cast<const float4*>((const float*)x + k + 4);
                xv[0] = f0.x, xv[1] = f0.y, xv[2] = f0.z, xv[3] = f0.w, xv[4] = f1.x, xv[5] = f1.y, xv[6] = f1.z, xv[7] = f1.w;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) s = fmaf(bf16lo(wq[i]), xv[2 * i], s), s = fmaf(bf16hi(wq[i]), xv[2 * i + 1], s);
        }
    } else {
        for (int k = lane; k < a.K; k += 32) s = fmaf(bf16_bits_to_f32(w[k]), ld_act<TA>(x + k), s);
    }
    s = warp_sum(s);
    if (lane == 0) a.y[j][(size_t)row * a.ldy[j] + n] = lin_act(s, a.act[j]);
}

// Few outputs over a long reduction for a panel of rows (a router, a low-rank projection): a warp takes kSkC outputs of kSkR rows, so a weight
// fragment serves kSkR rows and a row fragment kSkC outputs.  Row lengths are multiples of 8 and everything is 16-byte aligned.
constexpr int kSkR = 4, kSkC = 2;
template <typename TA>
__global__ void __launch_bounds__(256) kf_lin_skinny_kernel(LinArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (blockIdx.x * 8 + warp) * kSkC, m0 = blockIdx.y * kSkR;
    if (n0 >= a.N) return;
    const uint16_t* w[kSkC];
    const TA* x[kSkR];
#pragma unroll
    for (int j = 0; j < kSkC; j++) w[j] = a.W0 + (size_t)min(n0 + j, a.N - 1) * a.K;
#pragma unroll
    for (int i = 0; i < kSkR; i++) x[i] = (const TA*)a.x + (size_t)min(m0 + i, a.M - 1) * a.ldx;
    float s[kSkR][kSkC];
#pragma unroll
    for (int i = 0; i < kSkR; i++)
#pragma unroll
        for (int j = 0; j < kSkC; j++) s[i][j] = 0.f;
#pragma unroll 2
    for (int k = lane * 8; k < a.K; k += 256) {
        float wv[kSkC][8];
#pragma unroll
        for (int j = 0; j < kSkC; j++) {
            const uint4 q = *reinterpret_cast<const uint4*>(w[j] + k);
            const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; e++) wv[j][2 * e] = bf16lo(u[e]), wv[j][2 * e + 1] = bf16hi(u[e]);
        }
#pragma unroll
        for (int i = 0; i < kSkR; i++) {
            float xv[8];
            if (sizeof(TA) == 2) {
                const uint4 q = *reinterpret_cast<const uint4*>((const uint16_t*)x[i] + k);
                const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int e = 0; e < 4; e++) xv[2 * e] = bf16lo(u[e]), xv[2 * e + 1] = bf16hi(u[e]);
            } else {
                const float4 f0 = *reinterpret_cast<const float4*>((const float*)x[i] + k), f1 = *reinterpret_cast<const float4*>((const float*)x[i] + k + 4);
                xv[0] = f0.x, xv[1] = f0.y, xv[2] = f0.z, xv[3] = f0.w, xv[4] = f1.x, xv[5] = f1.y, xv[6] = f1.z, xv[7] = f1.w;
            }
#pragma unroll
            for (int j = 0; j < kSkC; j++)
#pragma unroll
                for (int e = 0; e < 8; e++) s[i][j] = fmaf(wv[j][e], xv[e], s[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < kSkR; i++)
#pragma unroll
        for (int j = 0; j < kSkC; j++) {
            const float t = warp_sum(s[i][j]);
            if (lane == 0 && m0 + i < a.M && n0 + j < a.N) {
                const float r = lin_act(t, a.act);
                if (a.act && a.out_act == 1) ((uint16_t*)a.y)[(size_t)(m0 + i) * a.ldy + n0 + j] = f32_to_bf16_bits(r);
                else ((float*)a.y)[(size_t)(m0 + i) * a.ldy + n0 + j] = r;
            }
        }
}

// ------------------------------------------------------------------------------------------------------------------ tile kernel
// 64 slots x 64 outputs per CTA, k in steps of 64 (bf16) or 32 (float); 256 threads.  Float activations: each thread a 4 x 4 block of FFMA accumulators.
// bf16 activations: 8 warps as 4 (m) x 2 (n), each warp 16 x 32 through mma.sync.m16n8k16; operands come from the same shared tiles.
// The next k step's operands are fetched into registers (16-byte loads when the row length and alignment allow, else element by
// element) while the current one is multiplied.  Every load is bounds-checked, so M, N and K are free.
constexpr int BM = 64, BN = 64;  // k step: 64 for bf16 activations (two 16-byte fetches per operand and thread in flight), 32 for float

__device__ __forceinline__ void mma_bf16_16816(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm_x4(uint32_t* r, const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// 8 consecutive k of one row: thread t fetches row t / 4, k offset (t % 4) * 8
template <typename T>
struct __align__(16) Frag8 {
    T v[8];
};
template <typename T>
__device__ __forceinline__ void fetch8(Frag8<T>& f, const T* base, size_t row_off, int k, int K, bool row_ok, bool vec) {
    if (row_ok && vec && k + 8 <= K) {
        if (sizeof(T) == 2) {
            *reinterpret_cast<uint4*>(f.v) = *reinterpret_cast<const uint4*>(base + row_off + k);
        } else {
            *reinterpret_cast<float4*>(f.v)     = *reinterpret_cast<const float4*>(base + row_off + k);
            *reinterpret_cast<float4*>(f.v + 4) = *reinterpret_cast<const float4*>(base + row_off + k + 4);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) f.v[j] = (row_ok && k + j < K) ? base[row_off + k + j] : T(0);
}

// The same shapes with bf16 activations on the tensor cores: a CTA takes 16 rows and all outputs (up to 8 * NT), its 8 warps deal the k chunks of
// 32 among themselves and their sums meet in shared memory, always in the same order.  Fragments come straight from memory: a product over k
// does not mind how k is numbered, so lane (g, t) of an operand's row g loads the 8 consecutive k 8t .. 8t + 7 of a chunk in one access and
// hands them out as the k places that two m16n8k16 steps expect of it; both operands use the same numbering.
template <int NT>
__global__ void __launch_bounds__(256) kf_lin_skinny_mma_kernel(LinArgs a) {
    __shared__ __align__(16) float part[4][16][NT * 8 + 2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, m0 = blockIdx.x * 16;
    const uint16_t* xa = (const uint16_t*)a.x + (size_t)min(m0 + g, a.M - 1) * a.ldx + 8 * t;
    const uint16_t* xb = (const uint16_t*)a.x + (size_t)min(m0 + g + 8, a.M - 1) * a.ldx + 8 * t;
    const uint16_t* w[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) w[j] = a.W0 + (size_t)min(j * 8 + g, a.N - 1) * a.K + 8 * t;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    for (int k = warp * 32; k < a.K; k += 256) {
        const uint4 pa = *reinterpret_cast<const uint4*>(xa + k), pb = *reinterpret_cast<const uint4*>(xb + k);
        uint4 q[NT];
#pragma unroll
        for (int j = 0; j < NT; j++) q[j] = *reinterpret_cast<const uint4*>(w[j] + k);
        const uint32_t a0[4] = {pa.x, pb.x, pa.y, pb.y}, a1[4] = {pa.z, pb.z, pa.w, pb.w};
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const uint32_t b0[2] = {q[j].x, q[j].y}, b1[2] = {q[j].z, q[j].w};
            mma_bf16_16816(acc[j], a0, b0);
            mma_bf16_16816(acc[j], a1, b1);
        }
    }
    auto put = [&](int slot) {
#pragma unroll
        for (int j = 0; j < NT; j++) {
            part[slot][g][j * 8 + 2 * t] = acc[j][0], part[slot][g][j * 8 + 2 * t + 1] = acc[j][1];
            part[slot][g + 8][j * 8 + 2 * t] = acc[j][2], part[slot][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
        }
    };
    if (warp >= 4) put(warp - 4);
    __syncthreads();
    if (warp < 4) {
#pragma unroll
        for (int j = 0; j < NT; j++) {
            acc[j][0] += part[warp][g][j * 8 + 2 * t], acc[j][1] += part[warp][g][j * 8 + 2 * t + 1];
            acc[j][2] += part[warp][g + 8][j * 8 + 2 * t], acc[j][3] += part[warp][g + 8][j * 8 + 2 * t + 1];
        }
        put(warp);  // the places this thread has just read
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * a.N; i += blockDim.x) {
        const int r = i / a.N, n = i - r * a.N;
        if (m0 + r >= a.M) break;
        const float v = lin_act((part[0][r][n] + part[1][r][n]) + (part[2][r][n] + part[3][r][n]), a.act);
        if (a.act && a.out_act == 1) ((uint16_t*)a.y)[(size_t)(m0 + r) * a.ldy + n] = f32_to_bf16_bits(v);
        else ((float*)a.y)[(size_t)(m0 + r) * a.ldy + n] = v;
    }
}

template <typename TA, bool DUAL>
__global__ void __launch_bounds__(256) kf_lin_tile_any_kernel(LinArgs a) {
    const int g    = blockIdx.z;
    const int lo   = a.offsets ? a.offsets[g] : 0;
    const int hi   = a.offsets ? a.offsets[g + 1] : a.M;
    const int n0 = blockIdx.x * BN;
    // a CTA walks the slot tiles blockIdx.y, blockIdx.y + gridDim.y, ... of its group: the grid is sized for the average group, not the worst
    for (int m0 = lo + blockIdx.y * BM; m0 < hi; m0 += gridDim.y * BM) {
    const uint16_t* W0 = a.Wt0 ? a.Wt0[g] : a.W0;
    const uint16_t* W1 = DUAL ? (a.Wt1 ? a.Wt1[g] : a.W1) : nullptr;
    constexpr bool MMA = sizeof(TA) == 2;
    constexpr int BK  = MMA ? 64 : 32, NF = BK / 32;
    constexpr int LDS = BK + 8;  // row pitch in elements: 16-byte aligned rows, conflict-free fragment loads
    __shared__ __align__(16) TA sx[BM][LDS];
    __shared__ __align__(16) uint16_t sw0[BN][LDS];
    __shared__ __align__(16) uint16_t sw1[DUAL ? BN : 1][LDS];
    const int tid = threadIdx.x;
    const int lr = tid >> 2, lk = (tid & 3) * 8;  // this thread's load: row lr, k offset lk
    int xrow = -1;
    {
        const int s = m0 + lr;
        if (s < hi) xrow = a.src_row ? a.src_row[s] : s;
    }
    const bool wok = n0 + lr < a.N;
    const size_t xoff = (size_t)(xrow < 0 ? 0 : xrow) * a.ldx, woff = (size_t)(n0 + lr) * a.K;
    const bool xvec = (a.ldx % 8 == 0) && (((uintptr_t)a.x & 15) == 0) && (a.K % 8 == 0);
    const bool wvec = (a.K % 8 == 0) && (((uintptr_t)W0 & 15) == 0) && (!DUAL || ((uintptr_t)W1 & 15) == 0);
    float acc0[16], acc1[DUAL ? 16 : 1];
#pragma unroll
    for (int i = 0; i < 16; i++) acc0[i] = 0.f;
    if (DUAL)
#pragma unroll
        for (int i = 0; i < 16; i++) acc1[i] = 0.f;
    const int warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 3, wn = warp >> 2;      // MMA: warp tile rows wm*16, cols wn*32
    const int tr = tid >> 4, tc = tid & 15;        // FFMA: thread rows tr*4.., cols tc*4..
    Frag8<TA> fx[NF];
    Frag8<uint16_t> fw0[NF], fw1[NF];
    auto fetch = [&](int kb) {  // fragment f covers k = kb + f * 32 + lk .. + 7
#pragma unroll
        for (int f = 0; f < NF; f++) {
            fetch8<TA>(fx[f], (const TA*)a.x, xoff, kb + f * 32 + lk, a.K, xrow >= 0, xvec);
            fetch8<uint16_t>(fw0[f], W0, woff, kb + f * 32 + lk, a.K, wok, wvec);
            if (DUAL) fetch8<uint16_t>(fw1[f], W1, woff, kb + f * 32 + lk, a.K, wok, wvec);
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < a.K; k0 += BK) {
        __syncthreads();  // the previous step's fragments have been read
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const int kc = f * 32 + lk;
            if (MMA) {
                *reinterpret_cast<uint4*>(&sx[lr][kc]) = *reinterpret_cast<const uint4*>(fx[f].v);
            } else {
                *reinterpret_cast<float4*>(&sx[lr][kc])     = *reinterpret_cast<const float4*>(fx[f].v);
                *reinterpret_cast<float4*>(&sx[lr][kc + 4]) = *reinterpret_cast<const float4*>(fx[f].v + 4);
            }
            *reinterpret_cast<uint4*>(&sw0[lr][kc]) = *reinterpret_cast<const uint4*>(fw0[f].v);
            if (DUAL) *reinterpret_cast<uint4*>(&sw1[lr][kc]) = *reinterpret_cast<const uint4*>(fw1[f].v);
        }
        __syncthreads();
        if (k0 + BK < a.K) fetch(k0 + BK);  // next step's operands travel while this one is multiplied
        if (MMA) {
            // fragments through ldmatrix: A = 16 rows x 16 k of this warp's slots; B = two 8-output tiles per instruction
            const uint16_t* xa = (const uint16_t*)&sx[wm * 16][0];
#pragma unroll
            for (int kk = 0; kk < BK; kk += 16) {
                uint32_t af[4];
                ldsm_x4(af, xa + (lane & 15) * LDS + kk + (lane >> 4) * 8);
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const int nr = wn * 32 + j * 8 + (lane & 7) + (lane >> 4) * 8, kc = kk + ((lane >> 3) & 1) * 8;
                    uint32_t bf[4];
                    ldsm_x4(bf, &sw0[nr][kc]);
                    mma_bf16_16816(&acc0[j * 4], af, bf);
                    mma_bf16_16816(&acc0[(j + 1) * 4], af, bf + 2);
                    if (DUAL) {
                        ldsm_x4(bf, &sw1[nr][kc]);
                        mma_bf16_16816(&acc1[j * 4], af, bf);
                        mma_bf16_16816(&acc1[(j + 1) * 4], af, bf + 2);
                    }
                }
            }
        } else {
            // a step's products are summed on their own and then added: the rounding error grows with K / BK + BK terms, not with K
            float p0[16], p1[DUAL ? 16 : 1];
#pragma unroll
            for (int i = 0; i < 16; i++) p0[i] = 0.f;
            if (DUAL)
#pragma unroll
                for (int i = 0; i < 16; i++) p1[DUAL ? i : 0] = 0.f;
#pragma unroll 8
            for (int k = 0; k < BK; k++) {
                float xv[4], wv[4], uv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) xv[i] = ld_act<TA>(&sx[tr * 4 + i][k]);
#pragma unroll
                for (int j = 0; j < 4; j++) wv[j] = bf16_bits_to_f32(sw0[tc * 4 + j][k]);
                if (DUAL)
#pragma unroll
                    for (int j = 0; j < 4; j++) uv[j] = bf16_bits_to_f32(sw1[tc * 4 + j][k]);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        p0[i * 4 + j] = fmaf(xv[i], wv[j], p0[i * 4 + j]);
                        if (DUAL) p1[DUAL ? i * 4 + j : 0] = fmaf(xv[i], uv[j], p1[DUAL ? i * 4 + j : 0]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 16; i++) acc0[i] += p0[i];
            if (DUAL)
#pragma unroll
                for (int i = 0; i < 16; i++) acc1[DUAL ? i : 0] += p1[DUAL ? i : 0];
        }
    }
    auto store = [&](int r, int n, float v0, float v1) {
        const int s = m0 + r;
        if (s >= hi || n >= a.N) return;
        const float v = DUAL ? lin_pair(a, v0, v1) : lin_act(v0, a.act);
        if ((DUAL || a.act) && a.out_act == 1)
            ((uint16_t*)a.y)[(size_t)s * a.ldy + n] = f32_to_bf16_bits(v);
        else
            ((float*)a.y)[(size_t)s * a.ldy + n] = v;
    };
    if (MMA) {
        const int gr = lane >> 2, tg = lane & 3;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + wn * 32 + j * 8 + tg * 2, r = wm * 16 + gr;
            store(r, n, acc0[j * 4 + 0], DUAL ? acc1[j * 4 + 0] : 0.f);
            store(r, n + 1, acc0[j * 4 + 1], DUAL ? acc1[j * 4 + 1] : 0.f);
            store(r + 8, n, acc0[j * 4 + 2], DUAL ? acc1[j * 4 + 2] : 0.f);
            store(r + 8, n + 1, acc0[j * 4 + 3], DUAL ? acc1[j * 4 + 3] : 0.f);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) store(tr * 4 + i, n0 + tc * 4 + j, acc0[i * 4 + j], DUAL ? acc1[i * 4 + j] : 0.f);
    }
    __syncthreads();  // the shared tiles are free for the next slot tile
    }
}

// bf16 activations: 128 weight rows (DUAL: 64 of either weight) x 64 slots per CTA on tcgen05, k in steps of 64.  The weights of a routed panel are the traffic (64
// experts of 2 x 1408 x 2048: 738 MB), 48 slots each, so the CTA is built to keep bytes on their way: two CTAs per SM with four 24 KB stages each, filled by
// cp.async (the table of weights is on the device, the rows of x are gathered: no tensor map), two to three of them in flight, 96 KB or more an SM; nothing
// but the copies and one thread's matrix instructions in the loop.  On mma.sync, whose fragments went through ldmatrix, shared memory was as busy as DRAM (8
// warps of 16 x 32 read 82 KB a step of 24 KB): 177 us for those and 113 for the down projections, 130 (0.86 of the copy rate) and 75 (0.77) here.
// Rows lie as 128 bytes, 16-byte chunk c of row r at c ^ (r & 7): the K-major SWIZZLE_128B layout of the matrix descriptors.  A weight that is not 16-byte
// aligned (only the kernel sees it) is fetched element by element into the same places.
constexpr int kTileRows = 128, kTileStages = 4, kTileStage = (kTileRows + BM) * 128;  // weight rows, then slots, 128 bytes each
constexpr size_t kTileSmem = (size_t)kTileStages * kTileStage + 1024;
static_assert(kTileStages * kTileStage >= BM * kTileRows * 4, "the ring takes the fp32 results");
// two neighbouring outputs, of which `left` exist
__device__ __forceinline__ void store_pair(uint16_t* y, float v0, float v1, int left, bool pairs) {
    if (pairs && left > 1) *reinterpret_cast<uint32_t*>(y) = pack_bf16x2(v0, v1);
    else {
        if (left > 0) y[0] = f32_to_bf16_bits(v0);
        if (left > 1) y[1] = f32_to_bf16_bits(v1);
    }
}
__device__ __forceinline__ void store_pair(float* y, float v0, float v1, int left, bool pairs) {
    if (pairs && left > 1) *reinterpret_cast<float2*>(y) = make_float2(v0, v1);
    else {
        if (left > 0) y[0] = v0;
        if (left > 1) y[1] = v1;
    }
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
template <bool DUAL>
__global__ void __launch_bounds__(256, 2) kf_lin_tile_kernel(LinArgs a) {
    constexpr int BK = 64, NS = kTileStages, OUTS = DUAL ? 64 : 128;  // outputs of a CTA
    extern __shared__ uint8_t tile_raw[];
    __shared__ uint64_t done[NS];  // the matrix instructions that read a stage have finished
    __shared__ uint32_t tmem_smem;
    uint8_t* const tile_smem = tile_raw + ((1024u - smem_u32(tile_raw)) & 1023u);
    const uint32_t ring = smem_u32(tile_smem);
    const int g  = blockIdx.z;
    const int lo = a.offsets ? a.offsets[g] : 0, hi = a.offsets ? a.offsets[g + 1] : a.M;
    const int n0 = blockIdx.x * OUTS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (lo + (int)blockIdx.y * BM >= hi) return;  // the whole CTA: nothing to do
    if (tid == 0) {
        for (int i = 0; i < NS; i++) mbar_init(&done[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(smem_u32(&tmem_smem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_smem;
    const int lr = tid >> 3, lc = tid & 7;  // this thread's loads: rows lr, lr + 32, ... of either operand, chunk lc
    const int steps = (a.K + BK - 1) / BK;
    const uint16_t* W[2] = {a.Wt0 ? a.Wt0[g] : a.W0, DUAL ? (a.Wt1 ? a.Wt1[g] : a.W1) : nullptr};
    const bool wvec = ((uintptr_t)W[0] & 15) == 0 && (!DUAL || ((uintptr_t)W[1] & 15) == 0);
    uint32_t it = 0;  // k-steps of the CTA so far: stage it % NS
    // a CTA walks the slot tiles blockIdx.y, blockIdx.y + gridDim.y, ... of its group: the grid is sized for the average group, not the worst
    for (int m0 = lo + blockIdx.y * BM; m0 < hi; m0 += gridDim.y * BM) {
        const uint16_t *xr[2], *wr[4];
        bool xok[2], wok[4];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int s = m0 + lr + 32 * i;
            xok[i] = s < hi;
            xr[i]  = (const uint16_t*)a.x + (size_t)(xok[i] ? (a.src_row ? a.src_row[s] : s) : 0) * a.ldx + lc * 8;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {  // rows 0 .. 127 of the tile: DUAL 64 of W[0], then the same 64 of W[1]
            const int n = n0 + (DUAL ? (lr + 32 * i) & 63 : lr + 32 * i);
            wok[i] = n < a.N;
            wr[i]  = W[DUAL ? i >> 1 : 0] + (size_t)(wok[i] ? n : 0) * a.K + lc * 8;
        }
        auto load = [&](int step, uint32_t stage) {
            const uint32_t st = ring + stage * kTileStage;
            const bool kok    = step * BK + lc * 8 < a.K;  // K is a multiple of 8
            const size_t kof  = (size_t)(kok ? step * BK : 0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = lr + 32 * i;
                const uint32_t dst = st + (uint32_t)(r * 128 + ((lc ^ (r & 7)) << 4));
                const bool ok = wok[i] && kok;
                if (wvec) {
                    cp16(dst, ok ? wr[i] + kof : W[0], ok);
                } else {
                    uint16_t* d = reinterpret_cast<uint16_t*>(tile_smem + (dst - ring));
                    for (int e = 0; e < 8; e++) d[e] = ok ? wr[i][kof + e] : (uint16_t)0;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int r = lr + 32 * i;
                cp16(st + (uint32_t)(kTileRows * 128 + r * 128 + ((lc ^ (r & 7)) << 4)), xok[i] && kok ? xr[i] + kof : (const uint16_t*)a.x, xok[i] && kok);
            }
        };
        const uint32_t it0 = it;
#pragma unroll
        for (int i = 0; i < NS - 1; i++) {  // the stages are free: the slot tile before this one ended behind its last matrix instruction
            if (i < steps) load(i, (it0 + i) % NS);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const int cols = min(BM, (hi - m0 + 15) & ~15);  // slots that the matrix instructions see
        const uint32_t idesc = make_idesc_bf16(cols);
        for (int step = 0; step < steps; step++, it++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // what this thread has copied or stored is for the tensor cores to read
            __syncthreads();
            if (warp == 0) {
                const uint32_t st = ring + (it % NS) * kTileStage;
                const uint64_t ad = make_desc_sw128(st), bd = make_desc_sw128(st + kTileRows * 128);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < BK / 16; k++) umma_ss(tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc, (step > 0 || k > 0) ? 1u : 0u);
                umma_commit_a(smem_u32(&done[it % NS]));
            }
            if (step + NS - 1 < steps) {  // into the stage of the step before this one
                if (step > 0) mbar_wait(&done[(it - 1) % NS], ((it - 1) / NS) & 1);
                load(step + NS - 1, (it + NS - 1) % NS);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        mbar_wait(&done[(it - 1) % NS], ((it - 1) / NS) & 1);  // all of them: they finish in order
        tc_fence_after();
        // ---- accumulator -> shared memory [slot][row] -> y, the outputs of a slot side by side ----
        float* res = reinterpret_cast<float*>(tile_smem);
        const int row = (warp & 3) * 32 + lane;
        for (int c0 = (warp >> 2) * 16; c0 < cols; c0 += 32) {
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
            for (int j = 0; j < 16; j++) res[(c0 + j) * kTileRows + row] = __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncthreads();
        const bool quads = a.ldy % 4 == 0 && ((uintptr_t)a.y & 15) == 0, pairs = a.ldy % 2 == 0 && ((uintptr_t)a.y & 7) == 0;
        for (int i = tid; i < (min(hi, m0 + BM) - m0) * (OUTS / 4); i += 256) {
            const int t = i / (OUTS / 4), c = (i % (OUTS / 4)) * 4, n = n0 + c;
            if (n >= a.N) continue;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float r0 = res[t * kTileRows + c + e];
                v[e] = DUAL ? lin_pair(a, r0, res[t * kTileRows + (DUAL ? 64 : 0) + c + e]) : lin_act(r0, a.act);
            }
            const size_t at = (size_t)(m0 + t) * a.ldy + n;
            const bool four = quads && n + 3 < a.N;
            if ((DUAL || a.act) && a.out_act == 1) {
                uint16_t* y = (uint16_t*)a.y + at;
                if (four) *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
                else store_pair(y, v[0], v[1], a.N - n, pairs), store_pair(y + 2, v[2], v[3], a.N - n - 2, pairs);
            } else {
                float* y = (float*)a.y + at;
                if (four) *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]);
                else store_pair(y, v[0], v[1], a.N - n, pairs), store_pair(y + 2, v[2], v[3], a.N - n - 2, pairs);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the ring and the accumulator are free for the next slot tile
    }
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(tmem) : "memory");
    }
}

// One weight and few CTAs: 64 slots x 64 outputs per CTA, k in steps of 64 through a ring of six stages filled by cp.async, 8 warps as 4 (m) x 2 (n) on mma.sync
// m16n8k16.  Twice as many CTAs as the kernel above and no tensor memory to set up (1 us); shared memory, which bounds this form where all warps multiply, has
// little to do while a warp whose 16 slots lie past the group's end only helps to load.
constexpr int kFewStages = 6, kFewTile = 64 * 128, kFewStage = 2 * kFewTile;
constexpr size_t kFewSmem = (size_t)kFewStages * kFewStage;
__global__ void __launch_bounds__(256, 2) kf_lin_tile_few_kernel(LinArgs a) {
    constexpr int BK = 64, NS = kFewStages;
    extern __shared__ __align__(128) uint8_t tile_smem[];
    const uint32_t ring = smem_u32(tile_smem);
    const int g  = blockIdx.z;
    const int lo = a.offsets ? a.offsets[g] : 0, hi = a.offsets ? a.offsets[g + 1] : a.M;
    const int n0 = blockIdx.x * BN, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 3, wn = warp >> 2;             // warp tile: rows wm * 16, columns wn * 32
    const int lr = tid >> 3, lc = tid & 7;                // this thread's loads: rows lr and lr + 32 of either operand, chunk lc
    const int steps = (a.K + BK - 1) / BK;
    for (int m0 = lo + blockIdx.y * BM; m0 < hi; m0 += gridDim.y * BM) {
        const uint16_t* W = a.Wt0 ? a.Wt0[g] : a.W0;
        const bool wvec = ((uintptr_t)W & 15) == 0;
        const uint16_t* xr[2];
        bool xok[2], wok[2];
        size_t woff[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int s = m0 + lr + 32 * i, n = n0 + lr + 32 * i;
            xok[i]  = s < hi, wok[i] = n < a.N;
            xr[i]   = (const uint16_t*)a.x + (size_t)(xok[i] ? (a.src_row ? a.src_row[s] : s) : 0) * a.ldx + lc * 8;
            woff[i] = (size_t)(wok[i] ? n : 0) * a.K + lc * 8;
        }
        auto load = [&](int step) {
            const uint32_t st = ring + (uint32_t)(step % NS) * kFewStage;
            const int k       = step * BK + lc * 8;
            const bool kok    = k < a.K;  // K is a multiple of 8
            const size_t kof  = (size_t)(kok ? step * BK : 0);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int r        = lr + 32 * i;
                const uint32_t dst = st + (uint32_t)(r * 128 + ((lc ^ (r & 7)) << 4));
                cp16(dst, xok[i] && kok ? xr[i] + kof : (const uint16_t*)a.x, xok[i] && kok);
                const bool ok = wok[i] && kok;
                if (wvec) {
                    cp16(dst + kFewTile, ok ? W + woff[i] + kof : W, ok);
                } else {
                    uint16_t* d = reinterpret_cast<uint16_t*>(tile_smem + (dst - ring) + kFewTile);
                    for (int e = 0; e < 8; e++) d[e] = ok ? W[woff[i] + kof + e] : (uint16_t)0;
                }
            }
        };
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = 0.f;
#pragma unroll
        for (int i = 0; i < NS - 1; i++) {
            if (i < steps) load(i);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const bool busy = m0 + wm * 16 < hi;
        for (int step = 0; step < steps; step++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
            __syncthreads();  // this step's bytes are there for everybody, and everybody has left the stage that is filled next
            if (step + NS - 1 < steps) load(step + NS - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (!busy) continue;
            const uint8_t* xs = tile_smem + (size_t)(step % NS) * kFewStage;
            auto at = [](const uint8_t* base, int row, int c) { return base + row * 128 + ((c ^ (row & 7)) << 4); };
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
                uint32_t af[4];
                ldsm_x4(af, at(xs, wm * 16 + (lane & 15), kk * 2 + (lane >> 4)));
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const int nr = wn * 32 + j * 8 + (lane & 7) + (lane >> 4) * 8, c = kk * 2 + ((lane >> 3) & 1);
                    uint32_t bf[4];
                    ldsm_x4(bf, at(xs + kFewTile, nr, c));
                    mma_bf16_16816(&acc[j * 4], af, bf);
                    mma_bf16_16816(&acc[(j + 1) * 4], af, bf + 2);
                }
            }
        }
        const int gr = lane >> 2, tg = lane & 3;
        const bool pairs = a.ldy % 2 == 0 && ((uintptr_t)a.y & 7) == 0;
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int s = m0 + wm * 16 + gr + 8 * h, n = n0 + wn * 32 + j * 8 + tg * 2;
                if (s >= hi || n >= a.N) continue;
                float v[2];
#pragma unroll
                for (int e = 0; e < 2; e++) v[e] = lin_act(acc[j * 4 + 2 * h + e], a.act);
                const size_t at = (size_t)s * a.ldy + n;
                const bool two  = n + 1 < a.N;
                if (a.act && a.out_act == 1) {
                    uint16_t* y = (uint16_t*)a.y + at;
                    if (two && pairs) *reinterpret_cast<uint32_t*>(y) = pack_bf16x2(v[0], v[1]);
                    else {
                        y[0] = f32_to_bf16_bits(v[0]);
                        if (two) y[1] = f32_to_bf16_bits(v[1]);
                    }
                } else {
                    float* y = (float*)a.y + at;
                    if (two && pairs) *reinterpret_cast<float2*>(y) = make_float2(v[0], v[1]);
                    else {
                        y[0] = v[0];
                        if (two) y[1] = v[1];
                    }
                }
            }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the ring is free for the next slot tile
    }
}

template <typename TA, bool DUAL>
int launch(kf_ctx* ctx, const LinArgs& a, int slots, int groups, bool gemv) {
    if (gemv) {
        dim3 grid((a.N + 7) / 8, slots);
        kf_lin_gemv_kernel<TA, DUAL><<<grid, 256, 0, ctx->stream>>>(a);
    } else {
        const int tiles = (slots + BM - 1) / BM;
        const int gy    = groups > 1 ? std::min(tiles, std::max(1, (2 * slots / groups + BM - 1) / BM)) : tiles;
        dim3 grid((a.N + BN - 1) / BN, gy, groups);
        if (sizeof(TA) == 2 && a.K % 8 == 0 && a.ldx % 8 == 0 && ((uintptr_t)a.x & 15) == 0) {  // rows that can be fetched 16 bytes at a time
            static bool set[kf_ctx::kMaxDevices] = {};  // function attributes are per device (one flag per instantiation and device)
            if (!set[ctx->device]) {
                KF_CUDA(ctx, cudaFuncSetAttribute(kf_lin_tile_kernel<DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem));
                if (!DUAL) KF_CUDA(ctx, cudaFuncSetAttribute(kf_lin_tile_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewSmem));
                set[ctx->device] = true;
            }
            // 64 x 64 tiles while they do not outnumber the SMs (8 groups of 18 slots, 512 outputs over 1792: 13.7 us, 17.0 in 128 x 64; 16 groups of 60 slots, 256
            // outputs: 15.5, 17.0), or the two places of every SM where most groups hold up to 16 slots, one row of warps (16 groups of 8 slots, 1024 outputs over 1024:
            // 11.4, 12.0; with 20 slots each 13.1, 12.5; three times as many tiles as SMs, 9 slots: 13.1, 10.3)
            const long long ctas = (long long)grid.x * gy * groups;
            if (!DUAL && (ctas <= ctx->sm_count || (ctas <= 2 * ctx->sm_count && slots <= 8ll * groups))) {
                kf_lin_tile_few_kernel<<<grid, 256, kFewSmem, ctx->stream>>>(a);
                KF_LAUNCH_CHECK(ctx);
                return KF_OK;
            }
            const int outs = DUAL ? kTileRows / 2 : kTileRows;
            kf_lin_tile_kernel<DUAL><<<dim3((a.N + outs - 1) / outs, gy, groups), 256, kTileSmem, ctx->stream>>>(a);
        } else {
            kf_lin_tile_any_kernel<TA, DUAL><<<grid, 256, 0, ctx->stream>>>(a);
        }
    }
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
int dispatch(kf_ctx* ctx, const LinArgs& a, int slots, int groups, bool gemv, bool dual, int act_f32) {
    if (act_f32) return dual ? launch<float, true>(ctx, a, slots, groups, gemv) : launch<float, false>(ctx, a, slots, groups, gemv);
    return dual ? launch<uint16_t, true>(ctx, a, slots, groups, gemv) : launch<uint16_t, false>(ctx, a, slots, groups, gemv);
}
constexpr int kGemvMaxSlots = 16;
// one weight, a panel of rows, few outputs and a long reduction: tiles would leave all but a handful of SMs idle
bool skinny_shape(const LinArgs& a) { return a.N <= 128 && a.K >= 512 && a.M > kGemvMaxSlots; }
int dispatch_one(kf_ctx* ctx, const LinArgs& a, int act_f32) {
    const bool skinny = skinny_shape(a);
    if (skinny && a.K % 8 == 0 && a.ldx % 8 == 0 && (((uintptr_t)a.W0 | (uintptr_t)a.x) & 15) == 0 && (a.M + kSkR - 1) / kSkR <= 65535) {
        if (!act_f32 && a.K % 32 == 0) {
            const int nt = (a.N + 7) / 8, blocks = (a.M + 15) / 16;
            if (nt <= 4) kf_lin_skinny_mma_kernel<4><<<blocks, 256, 0, ctx->stream>>>(a);
            else if (nt <= 8) kf_lin_skinny_mma_kernel<8><<<blocks, 256, 0, ctx->stream>>>(a);
            else if (nt <= 10) kf_lin_skinny_mma_kernel<10><<<blocks, 256, 0, ctx->stream>>>(a);
            else kf_lin_skinny_mma_kernel<16><<<blocks, 256, 0, ctx->stream>>>(a);
            KF_LAUNCH_CHECK(ctx);
            return KF_OK;
        }
        const dim3 grid((a.N + 8 * kSkC - 1) / (8 * kSkC), (a.M + kSkR - 1) / kSkR);
        if (act_f32) kf_lin_skinny_kernel<float><<<grid, 256, 0, ctx->stream>>>(a);
        else kf_lin_skinny_kernel<uint16_t><<<grid, 256, 0, ctx->stream>>>(a);
        KF_LAUNCH_CHECK(ctx);
        return KF_OK;
    }
    return dispatch(ctx, a, a.M, 1, a.M <= kGemvMaxSlots || (skinny && a.N <= 64), false, act_f32);
}
}  // namespace

extern "C" int kf_linear_g(kf_ctx* ctx, float* y, int ldy, const kf_tensor_desc* w, const void* x, int act_f32, int ldx, int M) {
    if (!ctx || !y || !w || !x) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, w->type == KF_T_BF16 && M >= 1 && w->rows >= 1 && w->cols >= 1 && ldx >= w->cols && ldy >= w->rows, "bf16 weight, ld >= extent");
    LinArgs a = {};
    a.W0 = (const uint16_t*)w->data_dev, a.x = x, a.y = y, a.M = M, a.N = w->rows, a.K = w->cols, a.ldx = ldx, a.ldy = ldy;
    // a few rows over a small weight: the warp-per-output kernel is through before the tuned ones have filled their pipelines (measured: 2.9 against
    // 5.3 us at 1024 x 1024, 4.5 against 6.0 at 2048 x 2048, even at 34 MB of weight x rows)
    const bool few = M <= kGemvMaxSlots && w->cols <= 4096 && (size_t)M * w->rows * w->cols * 2 <= ((size_t)34 << 20);
    // shapes the tuned kernels take go there (tcgen05 / TMEM panels, the HBM-rate GEMV); fp32 result through their fp32 epilogue
    if (!few && !skinny_shape(a) && !act_f32 && ldx == w->cols && ldy == w->rows && w->cols % 128 == 0 && w->rows % 16 == 0 && w->rows >= 16 && ctx->tc_min_m != 0 &&
        (((uintptr_t)w->data_dev | (uintptr_t)x | (uintptr_t)y) & 15) == 0)
        return kf_linear(ctx, y, w, x, M, KF_EPI_F32, nullptr);
    return dispatch_one(ctx, a, act_f32);
}
// y = silu(Wg x) * (Wu x), written in the activation type (bf16 bits, or float when act_f32)
extern "C" int kf_linear_g_swiglu(kf_ctx* ctx, void* y, int ldy, const kf_tensor_desc* wg, const kf_tensor_desc* wu, const void* x, int act_f32,
                                  int ldx, int M) {
    if (!ctx || !y || !wg || !wu || !x) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, wg->type == KF_T_BF16 && wu->type == KF_T_BF16 && wg->rows == wu->rows && wg->cols == wu->cols && M >= 1 && ldx >= wg->cols &&
                        ldy >= wg->rows, "gate / up: bf16, equal shapes");
    LinArgs a = {};
    a.W0 = (const uint16_t*)wg->data_dev, a.W1 = (const uint16_t*)wu->data_dev, a.x = x, a.y = y, a.M = M, a.N = wg->rows, a.K = wg->cols;
    a.ldx = ldx, a.ldy = ldy, a.out_act = act_f32 ? 0 : 1;
    return dispatch(ctx, a, M, 1, M <= kGemvMaxSlots, true, act_f32);
}
// Grouped matmul over expert-sorted slots.  w_table / w2_table: device arrays of n_groups bf16 weight pointers ([N][K] each);
// offsets: device int32 [n_groups + 1]; slot_group: device int32 [slots] (the expert of each slot); src_row: device int32 [slots] or
// NULL.  w2_table != NULL: y = silu(W x) * (W2 x) in the activation type; else y is float.  `slots` is the launch bound (tokens x top).
extern "C" int kf_linear_grouped(kf_ctx* ctx, void* y, int ldy, const void* const* w_table, const void* const* w2_table, int n_groups, int N, int K,
                                 const void* x, int act_f32, int ldx, const int32_t* offsets, const int32_t* slot_group, const int32_t* src_row,
                                 int slots) {
    if (!ctx || !y || !w_table || !x || !offsets || !slot_group) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, n_groups >= 1 && N >= 1 && K >= 1 && slots >= 1 && ldx >= K && ldy >= N, "shape");
    LinArgs a = {};
    a.Wt0 = (const uint16_t* const*)w_table, a.Wt1 = (const uint16_t* const*)w2_table, a.x = x, a.y = y, a.M = slots, a.N = N, a.K = K;
    a.ldx = ldx, a.ldy = ldy, a.offsets = offsets, a.slot_group = slot_group, a.src_row = src_row, a.out_act = act_f32 ? 0 : 1;
    return dispatch(ctx, a, slots, n_groups, slots <= kGemvMaxSlots, w2_table != nullptr, act_f32);
}

// The single-weight grouped form with an activation on the result (1: gelu, tanh form; 2: relu squared), written in the activation type
// (bf16 bits, or float when act_f32): the up projection of experts that have no gate.  act 0 = kf_linear_grouped without a second table.
extern "C" int kf_linear_grouped_act(kf_ctx* ctx, void* y, int ldy, const void* const* w_table, int n_groups, int N, int K, const void* x, int act_f32, int ldx,
                                     const int32_t* offsets, const int32_t* slot_group, const int32_t* src_row, int slots, int act) {
    if (!ctx || !y || !w_table || !x || !offsets || !slot_group) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, n_groups >= 1 && N >= 1 && K >= 1 && slots >= 1 && ldx >= K && ldy >= N && act >= 0 && act <= 2, "shape / act");
    LinArgs a = {};
    a.Wt0 = (const uint16_t* const*)w_table, a.x = x, a.y = y, a.M = slots, a.N = N, a.K = K;
    a.ldx = ldx, a.ldy = ldy, a.offsets = offsets, a.slot_group = slot_group, a.src_row = src_row, a.out_act = act_f32 ? 0 : 1, a.act = act;
    return dispatch(ctx, a, slots, n_groups, slots <= kGemvMaxSlots, false, act_f32);
}
// kf_linear_grouped's two-weight form with the clamped gate: y = g sigmoid(alpha g) (u + shift), g = min(W x, limit), u = clamp(W2 x, -limit,
// limit) (limit <= 0: not clamped), written in the activation type.  A slot whose slot_group is -1 is left out.
extern "C" int kf_linear_grouped_glu(kf_ctx* ctx, void* y, int ldy, const void* const* w_table, const void* const* w2_table, int n_groups, int N, int K,
                                     const void* x, int act_f32, int ldx, const int32_t* offsets, const int32_t* slot_group, const int32_t* src_row, int slots,
                                     float limit, float alpha, float shift) {
    if (!ctx || !y || !w_table || !w2_table || !x || !offsets || !slot_group) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, n_groups >= 1 && N >= 1 && K >= 1 && slots >= 1 && ldx >= K && ldy >= N, "shape");
    LinArgs a = {};
    a.Wt0 = (const uint16_t* const*)w_table, a.Wt1 = (const uint16_t* const*)w2_table, a.x = x, a.y = y, a.M = slots, a.N = N, a.K = K;
    a.ldx = ldx, a.ldy = ldy, a.offsets = offsets, a.slot_group = slot_group, a.src_row = src_row, a.out_act = act_f32 ? 0 : 1;
    a.glu = 1, a.limit = limit, a.alpha = alpha, a.shift = shift;
    return dispatch(ctx, a, slots, n_groups, slots <= kGemvMaxSlots, true, act_f32);
}
// y[i][m] = act_i(W_i x[i][m]) for n <= 8 bf16 weights with the same number of columns, each with an input [M][ldx] and a float output [M][rows of
// W_i] of its own; act: 0 none, 3 tanh (host array, NULL: none).  A handful of rows: one launch; panels: one matmul per weight.
extern "C" int kf_linear_batch(kf_ctx* ctx, int n, float* const* y, const kf_tensor_desc* w, const void* const* x, const int* act, int act_f32, int ldx, int M) {
    if (!ctx || !y || !w || !x) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, n >= 1 && n <= kBatchMax && M >= 1, "1 .. 8 weights");
    for (int i = 0; i < n; i++) {
        KF_REQUIRE(ctx, y[i] && x[i] && w[i].type == KF_T_BF16 && w[i].rows >= 1 && w[i].cols == w[0].cols && ldx >= w[i].cols, "bf16 weights, equal columns");
        KF_REQUIRE(ctx, !act || act[i] == 0 || act[i] == 3, "act");
    }
    if (M > kGemvMaxSlots) {
        for (int i = 0; i < n; i++) {
            int rc;
            if (act && act[i]) {
                LinArgs a = {};
                a.W0 = (const uint16_t*)w[i].data_dev, a.x = x[i], a.y = y[i], a.M = M, a.N = w[i].rows, a.K = w[i].cols, a.ldx = ldx, a.ldy = w[i].rows, a.act = act[i];
                rc = dispatch_one(ctx, a, act_f32);
            } else {
                rc = kf_linear_g(ctx, y[i], w[i].rows, &w[i], x[i], act_f32, ldx, M);
            }
            if (rc) return rc;
        }
        return KF_OK;
    }
    BatchArgs a = {};
    a.n = n, a.K = w[0].cols, a.ldx = ldx;
    for (int i = 0; i < n; i++) {
        a.W[i] = (const uint16_t*)w[i].data_dev, a.x[i] = x[i], a.y[i] = y[i], a.N[i] = a.ldy[i] = w[i].rows, a.act[i] = act ? act[i] : 0;
        a.first[i + 1] = a.first[i] + (w[i].rows + 7) / 8;
    }
    const dim3 grid(a.first[n], M);
    if (act_f32) kf_lin_gemv_batch_kernel<float><<<grid, 256, 0, ctx->stream>>>(a);
    else kf_lin_gemv_batch_kernel<uint16_t><<<grid, 256, 0, ctx->stream>>>(a);
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
