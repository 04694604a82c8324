// gemv_i8.cu -- dequant-GEMV for one or two tokens over 4-, 2- and 1-bit weights on the integer tensor cores:  y[M][N] = x[M][K] . deq(W[N][K])^T
//
// The same operation, reference and epilogues as gemv.cu (GTensor::GetDataX, src/Device/CUDA/kernel/quantizer.cu:249-392, T.cu:245-294 + CU_mm_blasLt,
// kernel/gemm.cu:93-214, behind SLP::Forw, NeuronFuse.cu:305-381), in the decode arithmetic only: codes times activations in full, the group's step and zero applied
// to the group's sums.
//
// What bounds such a matmul on paper is the bytes of the weights.  gemv.cu feeds codes to mma.sync as fp16 numbers, one register per two weights whatever their width: 40
// half-rate integer instructions and 8 matrix instructions a tile of 16 rows x 128 k, so 2- and 1-bit weights take as long as 4-bit ones; and its CTAs normalise and stage
// the activations with three k-steps of weights in flight.  Here
//   * a register holds FOUR codes: the bytes of `word & mask` are unsigned 8-bit operands of mma.sync.m16n8k32 (u8 x s8 -> s32), code * 2^bit where the field lies bit bits up in its
//     byte, and the activation that meets it is staged 2^-bit smaller: 16 ANDs and 4 matrix instructions a tile for every width;
//   * an activation is a whole number below 2^31 in units of its group of 128 k, in four signed 8-bit limbs, which are four of the eight columns of the matrix
//     instruction (two tokens fit).  All products and the sums of a group are exact integers; what is rounded is the fp32 sum over the groups;
//   * the 8 bits of a bf16 number are whole down to 2^-23 of the group's largest under the lowest field of a byte, down to 2^-19, 2^-17 and 2^-16 under the highest of 4-, 2- and
//     1-bit codes.  A k-step with a number that is not (of a SwiGLU's outputs one group in 190, 90 and 57, of normal ones hardly any), with infinities or NaN, or with numbers
//     that together leave the range, keeps its activations as they are, as bf16 pairs in the room of two limbs, and goes through mma.sync.m16n8k16 on codes as bf16 numbers: no
//     activation loses a bit that it has above 2^-180 of the largest.  The loop that asks for such steps runs in the CTAs that hold one, and their staging lies out of line.  (5120 x
//     25600: 18.6 us, 18.9 with the question everywhere, 18.2 without such steps; ternary 4096 x 12288 at two tokens behind a SwiGLU 10.3 without, 10.8; 32B decode 209.4 tokens/s without,
//     204 with both loops in the other order and nothing out of line, 206.4 so.  Where a quarter of the k-steps are such, 4-bit matmuls take as long as gemv.cu (51200 x 5120 31.2 and 31.8
//     us, 5120 x 25600 20.0 and 21.6), the others 3 to 7 % longer; where all are, 1.3 to 1.7 times as long: 50.9 and 30.9.)  Against 64 bits the fp32 sums are off by 1e-7, whatever the activations (gemv.cu: 3e-7 for normal ones,
//     2e-6 for a SwiGLU's, 1e-5 with outliers of 2^14);
//   * zero and code bias, which multiply the group's plain sum of activations, take one fma per row, group and token on the lanes that fetched them;
//   * a CTA takes a run of 16-row tiles, and its eight warps equal shares of the run's k-steps: no barrier between the first copy and the last sum.  Every lane streams its own
//     words through a ring in shared memory (cp.async), started before the kernel waits for its predecessor.  A k-step costs a warp 45 instructions beside 18 for its share of the
//     copies and the loop; two CTAs an SM hide their latency, one leaves the issue slots 70 % idle;
//   * a warp's sums of a tile go to shared memory and are added in the order of the warps; K is cut in halves over a cluster of two CTAs where tiles are few or the staged activations
//     too many, and the leader adds them in order: bit-reproducible.
// Measured against gemv.cu, us a launch in a chain of its own kind: 4-bit SwiGLU 51200 x 5120 at one token 31.9 -> 29.3 (4.75 TB/s), 5120 x 25600 21.2 -> 18.6, 10240 x 5120 11.5 -> 9.9,
// 5120 x 8192 9.2 -> 7.5; ternary SwiGLU 24576 x 4096 at two tokens 16.2 -> 14.0, 4096 x 12288 12.1 -> 9.9; binary 24576 x 4096 at one token 14.3 -> 11.4; Qwen3-32B decode in 4 bits
// 185 -> 206 tokens/s.
#include <string.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kf_common.cuh"

namespace {

enum { IF_Q4 = 0, IF_Q2 = 1, IF_Q1 = 2 };
enum { EPI_NONE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2, EPI_F32 = 4 };

constexpr int kWarps   = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kCh      = 2;  // k-steps of a chunk: copied, waited for and computed together
// ring of a lane's zeros or steps: blocks of eight, and one block more between lanes for the banks
constexpr int kGB = 4, kGLane = (kGB + 1) * 16, kGRing = 32 * kGLane;

template <int FMT>
struct Fmt {
    static constexpr int BITS = FMT == IF_Q4 ? 4 : FMT == IF_Q2 ? 2 : 1;
    static constexpr int CPB  = 4 * BITS;           // bytes of a lane's 32 codes of one row
    static constexpr int NW   = CPB / 4;            // their registers
    static constexpr int SLOT = kCh * 32 * 2 * CPB;  // bytes of a chunk in the ring: two rows a lane
};

struct ISeg {
    const uint8_t* data;
    const uint16_t* zero;
    const uint16_t* step;
    uint16_t* y;
    int rows;
    int tile0;  // its first tile of 16 rows in the launch's tiles
};
struct IParams {
    ISeg seg[3];
    int nseg;
    const uint16_t* x;
    const uint16_t* residual;
    const uint16_t* norm_w;  // RMSNorm of x first (nullptr: x as it is)
    float norm_eps;
    int M, K;
    int ksteps;             // K / 128
    int tiles, S, clusters;  // 16-row tiles of the launch, k-slices (CTAs of a cluster), clusters
    int unit;               // tiles that stay together (SwiGLU: a tile of gate rows and the same of up)
    int qbias, epilogue;
    int off_sx, off_part, off_red, off_gama, off_ring;  // byte offsets in dynamic shared memory (staged activations at 0)
};

__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void lds(uint32_t (&r)[N], uint32_t a) {
    if constexpr (N == 4) asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    else if constexpr (N == 2) asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
    else asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r[0]) : "r"(a) : "memory");
}

// Matrix instruction i of a k-step takes, for its k 0..15 (q = 0) and 16..31 (q = 1), the codes under `field << (8 * byte)` of one register: word(i, q) and bit(i, q).
template <int FMT>
__host__ __device__ constexpr int mma_word(int i, int q) { return FMT == IF_Q4 ? 2 * (i >> 1) + q : FMT == IF_Q2 ? q : 0; }
template <int FMT>
__host__ __device__ constexpr int mma_bit(int i, int q) { return FMT == IF_Q4 ? 4 * (i & 1) : FMT == IF_Q2 ? 2 * i : i + 4 * q; }
// index, in the lane's 32 codes, of the code in byte e of that operand (the storage words keep the first code in their most significant bits, PackedQ.hpp:160-211)
template <int FMT>
__host__ __device__ constexpr int mma_elem(int i, int q, int e) {
    const int per = 32 / Fmt<FMT>::BITS;  // codes of a register
    return per * (Fmt<FMT>::NW - 1 - mma_word<FMT>(i, q)) + (per - 1) - (8 * e + mma_bit<FMT>(i, q)) / Fmt<FMT>::BITS;
}

// A step in bf16: register p of 16 holds codes pair_elem(p) (its lower half) and pair_elem(p) - 16 / BITS
template <int FMT>
__host__ __device__ constexpr int pair_elem(int p) {
    const int per = 32 / Fmt<FMT>::BITS;
    return per * (Fmt<FMT>::NW - 1 - p / (per / 2)) + per - 1 - p % (per / 2);
}
template <int FMT>
__device__ __forceinline__ uint32_t pair_codes(const uint32_t (&w)[Fmt<FMT>::NW], int p) {
    constexpr int half = 16 / Fmt<FMT>::BITS;
    constexpr uint32_t mask = ((1u << Fmt<FMT>::BITS) - 1u) * 0x00010001u;
    const uint32_t v = ((w[p / half] >> (p % half * Fmt<FMT>::BITS)) & mask) | 0x43004300u;  // 128 + code
    return bf162_as_u32(__hsub2_rn(u32_as_bf162(v), u32_as_bf162(0x43004300u)));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A group as bf16 pairs at their places, times 2^up so that the largest lies in [2^63, 2^64) -> {sum of its numbers, -2^-up}
template <int FMT, int MX>
__device__ __noinline__ float2 stage_wide(uint4 v0, uint4 v1, uint4 v2, uint4 v3, uint4* at, int e) {
    constexpr int BITS = Fmt<FMT>::BITS;
    uint32_t v[16] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w, v3.x, v3.y, v3.z, v3.w};
    const int up      = min(100, 190 - e);  // 190 = 127 + 63
    const uint32_t by = (uint32_t)(127 + up) * 0x00800080u;
    const unsigned quad = 0xFu << (threadIdx.x & 28);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = bf162_as_u32(__hmul2_rn(u32_as_bf162(v[i]), u32_as_bf162(by)));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint32_t w[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int lo = pair_elem<FMT>(4 * i + c), hi = lo - 16 / BITS;
            w[c] = __byte_perm(v[lo >> 1], v[hi >> 1], ((lo & 1) ? 0x32 : 0x10) | ((hi & 1) ? 0x7600 : 0x5400));
        }
        at[((i >> 1) * 4 * MX + (i & 1)) * 4] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i++) sum += bf16lo(v[i]), sum += bf16hi(v[i]);
    sum += __shfl_xor_sync(quad, sum, 1), sum += __shfl_xor_sync(quad, sum, 2);
    return make_float2(sum, -__uint_as_float((uint32_t)(127 - up) << 23));
}

// MX: tokens (1, 2) ; D: chunks in flight per warp
template <int FMT, int MX, int D>
__global__ void __launch_bounds__(kThreads, 2) kf_gemv_i8_kernel(const __grid_constant__ IParams p) {
    using F             = Fmt<FMT>;
    constexpr int NC    = 4 * MX;                   // columns staged: token * 4 + limb
    constexpr int NF    = 8 / F::BITS;              // code fields of a byte
    constexpr int STEPB = 16 * F::BITS, CH = kCh;      // bytes of a row's k-step, k-steps of a chunk
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float s_red[MX * 8], s_scale[MX];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    kf_grid_launch_dependents();  // the next kernel's CTAs may come up beside this one and start their own copies
    const int S = p.S, q = blockIdx.x / (unsigned)S, slice = blockIdx.x - q * S;
    if (S > 1) cluster_arrive();  // matched in front of the first store to another CTA: by then every CTA of the cluster runs
    const bool glu = p.epilogue == EPI_SWIGLU;

    // ---- this CTA: tiles [t0, t0 + nt) x k-steps [s0, s0 + n), nc chunks a tile ; this warp: chunks [p0, p1) of the run, tile after tile ----
    const int units = p.tiles / p.unit;
    // (32-bit divisions, few of them: with 64 bits they cost 1 us in front of the first copy and more behind the last sum)
    const unsigned ub = (unsigned)units / p.clusters, ur = (unsigned)units % p.clusters;  // the first ur clusters have one unit more
    const int t0 = (int)(q * ub + min((unsigned)q, ur)) * p.unit, nt = (int)(ub + ((unsigned)q < ur ? 1u : 0u)) * p.unit;
    const int s0 = (int)((unsigned)(slice * p.ksteps) / (unsigned)S), n = (int)((unsigned)((slice + 1) * p.ksteps) / (unsigned)S) - s0;
    const int nc = (n + CH - 1) / CH, run = nt * nc;
    auto share = [&](int w) { return (int)((unsigned)(run * w) / kWarps); };
    const int p0 = share(warp), p1 = share(warp + 1);
    const size_t row_bytes = (size_t)p.K * F::BITS / 8;

    // ---- the copies: a lane's words of rows g and g + 8 of the tile.  Beside them its own stream of zeros (t even) or steps (t odd) of row g (t < 2) or g + 8, in blocks of
    //      16 bytes, which rows start anywhere in: 4-byte copies of one entry each missed the small L1 that the rings leave, 32 lines a step (5120 x 25600: 49.5 us) ----
    const uint32_t ring  = (uint32_t)__cvta_generic_to_shared(smem + p.off_ring) + (uint32_t)(warp * D * F::SLOT);
    const uint32_t gring = (uint32_t)__cvta_generic_to_shared(smem + p.off_gama) + (uint32_t)(warp * kGRing + lane * kGLane);
    const int toff = FMT == IF_Q4 ? 16 * t : FMT == IF_Q2 ? 16 * (t >> 1) + 8 * (1 - (t & 1)) : 12 - 4 * t;  // first codes in word.high (PackedQ.hpp:185-211)
    const uint32_t goff = (uint32_t)(((g + (t & 2) * 4) * p.ksteps + s0) * 2) & 15u;  // of the lane's first entry of a tile in its block: tiles are 16 rows, whole blocks
    const uint32_t glen = (goff + 2 * (uint32_t)n + 14) & ~15u;                       // bytes of a tile's blocks
    const uint8_t *src = nullptr, *gsrc = nullptr;  // the tile's words at k-step 0 of the slice, its first block of zeros or steps
    uint32_t gbase = 0, gend = 0;                   // the tile's first block in the ring, end of what has been copied of it (from its start)
    int itile = p0 / nc, ik = (p0 - itile * nc) * CH, left = p1 - p0;
    auto open = [&](int tile) {
        int seg = 0, row;
        if (glu) {
            seg = tile & 1, row = (tile >> 1) * 16;
        } else {
            if (p.nseg > 1 && tile >= p.seg[1].tile0) seg = 1;
            if (p.nseg > 2 && tile >= p.seg[2].tile0) seg = 2;
            row = (tile - p.seg[seg].tile0) * 16;
        }
        const ISeg& sg = p.seg[seg];
        src  = sg.data + (size_t)(row + g) * row_bytes + (size_t)s0 * STEPB + toff;
        gsrc = reinterpret_cast<const uint8_t*>(((t & 1) ? sg.step : sg.zero) + (size_t)(row + g + (t & 2) * 4) * p.ksteps + s0) - goff;
        gend = (goff + 2 * (uint32_t)ik) & ~15u;
    };
    auto copy = [&](int slot) {  // the next chunk into a slot of the ring
        if (left > 0) {
            const uint32_t dst  = ring + (uint32_t)(slot * F::SLOT);
            const uint8_t* from = src + (size_t)ik * STEPB;
#pragma unroll
            for (int j = 0; j < CH; j++) {
                if (j > 0 && ik + j >= n) break;  // past the slice's end: the activations there are zeros
                cp_async<F::CPB>(dst + (64 * j + lane) * F::CPB, from + j * STEPB);
                cp_async<F::CPB>(dst + (64 * j + 32 + lane) * F::CPB, from + j * STEPB + 8 * row_bytes);
            }
            const uint32_t need = goff + 2 * (uint32_t)min(ik + CH, n);
#pragma unroll
            for (int b = 0; b < 2; b++)
                if (gend < need) cp_async<16>(gring + ((gbase + gend) & (kGB * 16 - 1)), gsrc + gend), gend += 16;
            left--, ik += CH;
            if (ik >= n) {
                ik = 0, itile++, gbase += glen;
                if (left > 0) open(t0 + itile);
            }
        }
        cp_async_commit();  // one group per chunk, empty at the tail, so that the wait count stays uniform
    };
    if (left > 0) open(t0 + itile);
#pragma unroll
    for (int i = 0; i < D; i++) copy(i);

    // ---- everything above touched only the weights; x, the residual and y belong to the predecessor until here ----
    kf_grid_dependency_wait();
    const uint16_t* const px = behind_wait(p.x);

    // ---- activations.  Item = 32 consecutive values of a token (what one lane's codes of a k-step meet); the four lanes of a quad hold a group of 128 ----
    uint4* xs  = reinterpret_cast<uint4*>(smem);                       // [step][h][column][t]: operands of matrix instructions 2 h, 2 h + 1
    float2* sx = reinterpret_cast<float2*>(smem + p.off_sx);           // [step][token] {sum of the group, 2^-scale} ; in bf16: {sum * 2^scale, -2^-scale}
    const int items = MX * nc * CH * 4;
    uint4 xv[4];
    auto load_x = [&](int it) {
        const int m = (it >> 2) % MX, s = it / (4 * MX);
        const uint4* gp = reinterpret_cast<const uint4*>(px + (size_t)m * p.K + (size_t)(s0 + s) * 128 + (it & 3) * 32);
#pragma unroll
        for (int i = 0; i < 4; i++) xv[i] = s < n ? __ldg(gp + i) : make_uint4(0, 0, 0, 0);
    };
    if (tid < items) load_x(tid);  // beside the sums below
    int any_wide = 0;
    if (p.norm_w) {  // the scale of each token, in the order of kf_rmsnorm_kernel (ops.cu): 256 threads
        float ss[MX];
#pragma unroll
        for (int m = 0; m < MX; m++) ss[m] = 0.f;
        for (int i = tid * 8; i < p.K; i += kThreads * 8) {
            uint4 v[MX];
#pragma unroll
            for (int m = 0; m < MX; m++) v[m] = __ldg(reinterpret_cast<const uint4*>(px + (size_t)m * p.K + i));
#pragma unroll
            for (int m = 0; m < MX; m++) {
                const uint32_t w[4] = {v[m].x, v[m].y, v[m].z, v[m].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float a = bf16lo(w[j]), b = bf16hi(w[j]);
                    ss[m] = fmaf(a, a, ss[m]), ss[m] = fmaf(b, b, ss[m]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MX; m++) {
            ss[m] = warp_sum(ss[m]);
            if (lane == 0) s_red[m * 8 + warp] = ss[m];
        }
        __syncthreads();
        if (tid < MX) {
            float tot = 0.f;
            for (int w = 0; w < 8; w++) tot += s_red[tid * 8 + w];
            s_scale[tid] = 1.0f / sqrtf(fmaf(tot, 1.0f / (float)p.K, p.norm_eps));
        }
        __syncthreads();
    }
    for (int it = tid; it < items; it += kThreads) {
        const int tt = it & 3, m = (it >> 2) % MX, s = it / (4 * MX);
        if (it != tid) load_x(it);
        uint32_t v[16];
#pragma unroll
        for (int i = 0; i < 4; i++) v[4 * i] = xv[i].x, v[4 * i + 1] = xv[i].y, v[4 * i + 2] = xv[i].z, v[4 * i + 3] = xv[i].w;
        if (p.norm_w && s < n) {  // (x * s) * w, rounded to bf16 like the stand-alone kernel's output
            const float sc  = s_scale[m];
            const uint4* wp = reinterpret_cast<const uint4*>(p.norm_w + (size_t)(s0 + s) * 128 + tt * 32);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 wv = __ldg(wp + i);
                const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                for (int j = 0; j < 4; j++) v[4 * i + j] = pack_bf16x2((bf16lo(v[4 * i + j]) * sc) * bf16lo(ww[j]), (bf16hi(v[4 * i + j]) * sc) * bf16hi(ww[j]));
            }
        }
        // the power of two that puts the group's largest magnitude into [2^30, 2^31), one lower where that is 255 * 2^23, which the digits below cannot hold.  Beside it the least
        // exponent of its numbers less the place that each meets in a byte (elements 2 i and 2 i + 1 always the same two; a zero less one is the largest there is)
        const unsigned quad = 0xFu << (lane & ~3);
        uint32_t amax = 0, low[NF / 2];
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < NF / 2; c++) low[c] = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            amax = __vmaxu2(amax, v[i] & 0x7fff7fffu);
            low[i % (NF / 2)] = __viaddmin_u16x2(v[i] & 0x7fff7fffu, 0xffffffffu, low[i % (NF / 2)]);
            sum += bf16lo(v[i]), sum += bf16hi(v[i]);
        }
        int least = 512;
#pragma unroll
        for (int c = 0; c < NF / 2; c++) {
            const int hi = F::BITS * (NF - 1 - 2 * c), lo = hi - F::BITS;  // the first codes are the highest
            least = min(least, min((int)(low[c] >> 7 & 0x1ffu) - hi, (int)(low[c] >> 23) - lo));
        }
        amax = max(amax & 0xffffu, amax >> 16) | (uint32_t)(1023 - least) << 16;
        amax = __vmaxu2(amax, __shfl_xor_sync(quad, amax, 1)), amax = __vmaxu2(amax, __shfl_xor_sync(quad, amax, 2));
        least = 1023 - (int)(amax >> 16), amax &= 0xffffu;
        const int e = (int)(amax >> 7);                        // biased exponent of the largest
        const int scale = min(100, 157 - (int)((amax + 1) >> 7));  // 157 = 127 + 30 ; so that a step times 2^-scale stays a normal number
        float f[NF];                                               // 2^scale for each place a field may lie at
#pragma unroll
        for (int b = 0; b < NF; b++) f[b] = __uint_as_float((uint32_t)(127 + scale - b * F::BITS) << 23);
        sum += __shfl_xor_sync(quad, sum, 1), sum += __shfl_xor_sync(quad, sum, 2);
        // Does every number come out whole?  Those with all their 8 bits above one do; infinities, NaN and numbers whose sum is none do not.  (Asking the others one by one spares half of
        // these steps and takes longer.)  One token's group decides for the step
        int wide = e >= 246 || least < 134 - scale;
        if (MX == 2) wide |= __shfl_xor_sync(0xFFu << (lane & ~7), wide, 4);
        any_wide |= wide;
        // a step that does not fit: bf16 pairs as the code pairs meet them, in the place of limbs 0 and 1 ; marked by the sign
        float inv = __uint_as_float((uint32_t)(127 - scale) << 23);
        if (__builtin_expect(wide, 0)) {
            const float2 r = stage_wide<FMT, MX>(make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]), make_uint4(v[8], v[9], v[10], v[11]), make_uint4(v[12], v[13], v[14], v[15]),
                                                 xs + (s * 2 * NC + 4 * m) * 4 + tt, e);
            sum = r.x, inv = r.y;
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t o[4][4];  // [limb][instruction, k half]
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int i = 2 * h + (c >> 1), qq = c & 1;
                    uint32_t w[4];
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        const int el = mma_elem<FMT>(i, qq, b);
                        const float a = (el & 1) ? bf16hi(v[el >> 1]) : bf16lo(v[el >> 1]);
                        // signed digits in base 256: adding 128 to the lower three makes them bytes without borrow, flipping their top bits takes it off again
                        w[b] = ((uint32_t)__float2int_rn(a * f[mma_bit<FMT>(i, qq) / F::BITS]) + 0x00808080u) ^ 0x00808080u;
                    }
                    const uint32_t l01 = __byte_perm(w[0], w[1], 0x5140), h01 = __byte_perm(w[2], w[3], 0x5140);
                    const uint32_t l23 = __byte_perm(w[0], w[1], 0x7362), h23 = __byte_perm(w[2], w[3], 0x7362);
                    o[0][c] = __byte_perm(l01, h01, 0x5410), o[1][c] = __byte_perm(l01, h01, 0x7632);
                    o[2][c] = __byte_perm(l23, h23, 0x5410), o[3][c] = __byte_perm(l23, h23, 0x7632);
                }
#pragma unroll
                for (int l = 0; l < 4; l++) xs[((s * 2 + h) * NC + 4 * m + l) * 4 + tt] = make_uint4(o[l][0], o[l][1], o[l][2], o[l][3]);
            }
        }
        if (tt == 0) sx[s * MX + m] = make_float2(sum, inv);
    }
    any_wide = __syncthreads_or(any_wide);

    // ---- the stream: k-steps of this warp, each lane's words as it copied them ----
    float* part = reinterpret_cast<float*>(smem + p.off_part);  // [tile + warp][token][16 rows]: a warp's sums of a tile (the pairs lie on a path, so the index is their own)
    auto stream = [&](auto with_bf16) {
        float acc[4], z[MX];
        auto clear = [&]() {
#pragma unroll
            for (int c = 0; c < 4; c++) acc[c] = 0.f;
#pragma unroll
            for (int m = 0; m < MX; m++) z[m] = 0.f;
        };
        clear();
        int tile = p0 / nc, k = (p0 - tile * nc) * CH, slot = 0;
        uint32_t gnext = 0, gat = goff + 2 * (uint32_t)k;  // the tile's blocks in the ring, the chunk's first entry
        const uint32_t xbase = (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)(((MX == 1 ? g & 3 : g) * 4 + t) * 16);
        const float fq = (float)p.qbias;
#pragma unroll 1
        for (int pos = p0; pos < p1; pos++) {
            cp_async_wait<D - 1>();
            const uint32_t at = ring + (uint32_t)(slot * F::SLOT) + lane * F::CPB;
            uint32_t wa[CH][F::NW], wb[CH][F::NW], gv[CH];
#pragma unroll
            for (int j = 0; j < CH; j++) {
                lds(wa[j], at + 64 * j * F::CPB), lds(wb[j], at + (64 * j + 32) * F::CPB);
                asm volatile("ld.shared.u16 %0, [%1];" : "=r"(gv[j]) : "r"(gring + ((gat + 2 * j) & (kGB * 16 - 1))) : "memory");
            }
            int d[CH][4];
            float2 sv[CH][MX];
#pragma unroll
            for (int j = 0; j < CH; j++) {
#pragma unroll
                for (int c = 0; c < 4; c++) d[j][c] = 0;
#pragma unroll
                for (int m = 0; m < MX; m++) sv[j][m] = sx[(k + j) * MX + m];
            }
            const uint32_t xk = xbase + (uint32_t)(k * (2 * NC * 64));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t xb[CH][4];
#pragma unroll
                for (int j = 0; j < CH; j++) lds(xb[j], xk + (uint32_t)((2 * j + h) * NC * 64));
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int i = 2 * h + c;
                    constexpr uint32_t field = ((1u << F::BITS) - 1u) * 0x01010101u;
                    const uint32_t m0 = field << mma_bit<FMT>(i, 0), m1 = field << mma_bit<FMT>(i, 1);
#pragma unroll
                    for (int j = 0; j < CH; j++) {
                        const uint32_t a0 = wa[j][mma_word<FMT>(i, 0)] & m0, a1 = wb[j][mma_word<FMT>(i, 0)] & m0;
                        const uint32_t a2 = wa[j][mma_word<FMT>(i, 1)] & m1, a3 = wb[j][mma_word<FMT>(i, 1)] & m1;
                        mma_u8s8(d[j], a0, a1, a2, a3, xb[j][2 * c], xb[j][2 * c + 1]);
                    }
                }
            }
            if (decltype(with_bf16)::value && fminf(sv[0][0].y, sv[CH - 1][0].y) < 0.f) {  // a step in bf16 (CH is two)
#pragma unroll
                for (int j = 0; j < CH; j++) {
                    if (sv[j][0].y >= 0.f) continue;
                    const float val = bf16_bits_to_f32(gv[j]);
#pragma unroll
                    for (int m = 0; m < MX; m++) z[m] = fmaf(-val * sv[j][m].y, sv[j][m].x, z[m]), sv[j][m].x = 0.f;
                    const float gs = MX == 2 && (t & 2) ? sv[j][MX - 1].y : sv[j][0].y;
                    const float stepa = __shfl_sync(0xffffffffu, val, (lane & ~3) | 1), stepb = __shfl_sync(0xffffffffu, val, (lane & ~3) | 3);
                    float fd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        uint32_t xb[4];  // the column's token as the limbs have it: columns 0 and 4, which even lanes hold the sums of, are those of tokens 0 and 1
                        lds(xb, xk + (uint32_t)(((2 * j + (i >> 1)) * NC + (i & 1) - (g & 3)) * 64));
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            const int pr = 4 * i + 2 * c;
                            mma_bf16(fd, pair_codes<FMT>(wa[j], pr), pair_codes<FMT>(wb[j], pr), pair_codes<FMT>(wa[j], pr + 1), pair_codes<FMT>(wb[j], pr + 1), xb[2 * c], xb[2 * c + 1]);
                        }
                    }
                    if (!(t & 1)) acc[0] = fmaf(-stepa * gs, fd[0], acc[0]), acc[2] = fmaf(-stepb * gs, fd[2], acc[2]);
#pragma unroll
                    for (int c = 0; c < 4; c++) d[j][c] = 0;
                }
            }
            copy(slot);  // its words are in the matrix instructions' registers
            slot = slot + 1 == D ? 0 : slot + 1;
#pragma unroll
            for (int j = 0; j < CH; j++) {
                // past the slice's end the ring holds what was there: the sum of activations and the scale are zero, which an infinity or NaN would survive
                const float val = j > 0 && k + j >= n ? 0.f : bf16_bits_to_f32(gv[j]);
                const float stepa = __shfl_sync(0xffffffffu, val, (lane & ~3) | 1), stepb = __shfl_sync(0xffffffffu, val, (lane & ~3) | 3);
#pragma unroll
                for (int m = 0; m < MX; m++) z[m] = fmaf(val, sv[j][m].x, z[m]);
                const float gs = MX == 2 && (t & 2) ? sv[j][MX - 1].y : sv[j][0].y;  // of this lane's columns' token
                const float fa = stepa * gs, fb = stepb * gs;
                acc[0] = fmaf(fa, (float)d[j][0], acc[0]), acc[1] = fmaf(fa, (float)d[j][1], acc[1]);
                acc[2] = fmaf(fb, (float)d[j][2], acc[2]), acc[3] = fmaf(fb, (float)d[j][3], acc[3]);
            }
            gat += 2 * CH, k += CH;
            if (k >= n || pos + 1 == p1) {  // the end of the tile or of this warp's share of it
                float* out = part + (size_t)(tile + warp) * (MX * 16);
                // zero * sum and qbias * step * sum of row g in lanes t = 0, 1, of g + 8 in t = 2, 3
                float za[MX], zb[MX];
#pragma unroll
                for (int m = 0; m < MX; m++) {
                    float v = (t & 1) ? z[m] * fq : z[m];
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    za[m] = __shfl_sync(0xffffffffu, v, lane & ~3), zb[m] = __shfl_sync(0xffffffffu, v, (lane & ~3) | 2);
                }
                // limbs 0, 1 in even lanes, 2, 3 in odd ones ; token 0 in lanes t = 0, 1, token 1 in t = 2, 3
                const float up = (t & 1) ? 65536.f : 1.f;
                float va = fmaf(acc[1], 256.f, acc[0]) * up, vb = fmaf(acc[3], 256.f, acc[2]) * up;
                va += __shfl_xor_sync(0xffffffffu, va, 1), vb += __shfl_xor_sync(0xffffffffu, vb, 1);
#pragma unroll
                for (int m = 0; m < MX; m++)
                    if ((t >> 1) == m) out[m * 16 + g + 8 * (t & 1)] = (t & 1) ? vb - zb[m] : va - za[m];
                clear();
                if (k >= n) k = 0, tile++, gnext += glen, gat = gnext + goff;
            }
        }
    };
    if (!any_wide) stream(std::false_type());
    else stream(std::true_type());
    cp_async_wait<0>();
    __syncthreads();

    // ---- the warps' sums of each tile, in their order ----
    constexpr int TO = MX * 16;  // outputs of a tile: [token][row]
    const int outs   = nt * TO;
    const float inv  = (float)kWarps / (float)run;
    auto tile_sum = [&](int tile, int o) {
        const int lo = tile * nc, hi = lo + nc;
        int w = (int)((float)lo * inv);  // about the warp whose share the tile begins in
        w = min(w, kWarps - 1);
        while (share(w) > lo) w--;
        while (share(w + 1) <= lo) w++;
        float sum = 0.f;
        for (; w < kWarps && share(w) < hi; w++)
            if (share(w + 1) > share(w)) sum += part[(size_t)(tile + w) * TO + o];
        return sum;
    };
    float* red = reinterpret_cast<float*>(smem + p.off_red);  // [slice][tile][token][row]: the leader's, S > 1
    if (S > 1) {
        cluster_wait();
        for (int i = tid; i < outs; i += kThreads) st_cluster_f32(red + slice * outs + i, 0, tile_sum(i / TO, i % TO));
        cluster_arrive(), cluster_wait();
        if (slice != 0) return;
    }
    auto total = [&](int tile, int o) {
        if (S == 1) return tile_sum(tile, o);
        float sum = 0.f;
        for (int s = 0; s < S; s++) sum += red[s * outs + tile * TO + o];  // in slice order
        return sum;
    };
    if (glu) {
        const int rows = p.seg[0].rows;
        for (int i = tid; i < outs / 2; i += kThreads) {
            const int r = i & 15, m = i / 16 % MX, pair = i / TO, row = (t0 / 2 + pair) * 16 + r;
            const float gt = bf16_bits_to_f32(f32_to_bf16_bits(total(2 * pair, i % TO))), up = bf16_bits_to_f32(f32_to_bf16_bits(total(2 * pair + 1, i % TO)));
            p.seg[0].y[(size_t)m * rows + row] = f32_to_bf16_bits((gt * up) / (1.0f + expf(-gt)));  // CU_swiglu_v0, Activation.cu:86-93
        }
        return;
    }
    for (int i = tid; i < outs; i += kThreads) {
        const int r = i & 15, m = i / 16 % MX, tile = i / TO;
        int seg = 0;
        if (p.nseg > 1 && t0 + tile >= p.seg[1].tile0) seg = 1;
        if (p.nseg > 2 && t0 + tile >= p.seg[2].tile0) seg = 2;
        const ISeg& sg  = p.seg[seg];
        const size_t at = (size_t)m * sg.rows + (t0 + tile - sg.tile0) * 16 + r;
        const float v   = total(tile, i % TO);
        if (p.epilogue == EPI_F32) {  // tensor-parallel partial sums stay fp32 until the exchange
            reinterpret_cast<float*>(sg.y)[at] = v;
            continue;
        }
        uint16_t b = f32_to_bf16_bits(v);  // the reference's GEMM writes bf16 (gemm.cu:124-126)
        if (p.epilogue == EPI_RESIDUAL) b = f32_to_bf16_bits(bf16_bits_to_f32(p.residual[at]) + bf16_bits_to_f32(b));  // then CU_add3 (packedN.cuh:867-875)
        sg.y[at] = b;
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------------------
// Shared memory of a CTA: what few tiles, two CTAs an SM, and at most two CTAs an SM take (a deeper ring is worth less than the room for a successor's CTAs: 32B feed-forward
// 47.1 us with 74 KB, 46.3 with 90, 47.7 with 112)
constexpr size_t kEarly = 74 * 1024, kTwo = 92 * 1024, kHalfSM = 112 * 1024;
constexpr size_t kMost   = 224 * 1024;

struct IPlan {
    int S, clusters, depth;
    size_t smem;
};
template <int FMT, int MX, int D>
int launch_depth(kf_ctx* ctx, const IParams& p, size_t smem) {
    auto kern = kf_gemv_i8_kernel<FMT, MX, D>;
    static std::atomic<bool> attr_set[kf_ctx::kMaxDevices];  // function attributes are per device
    if (!attr_set[ctx->device].load(std::memory_order_relaxed)) {
        KF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
        attr_set[ctx->device].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.clusters * p.S), cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = smem, cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ctx->pdl) attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization, attr[na].val.programmaticStreamSerializationAllowed = 1, na++;
    if (p.S > 1) attr[na].id = cudaLaunchAttributeClusterDimension, attr[na].val.clusterDim.x = (unsigned)p.S, attr[na].val.clusterDim.y = 1, attr[na].val.clusterDim.z = 1, na++;
    cfg.attrs = attr, cfg.numAttrs = na;
    KF_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, p));
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
// bytes in flight per CTA: warps x depth x 2, 1 or half a KB (4-, 2- and 1-bit weights)
template <int FMT, int MX>
int launch_fmt(kf_ctx* ctx, const IParams& p, const IPlan& plan) {
    switch (plan.depth) {
        case 2: return launch_depth<FMT, MX, 2>(ctx, p, plan.smem);
        case 3: return launch_depth<FMT, MX, 3>(ctx, p, plan.smem);
        default: return launch_depth<FMT, MX, 4>(ctx, p, plan.smem);
    }
}
template <int FMT>
int launch_tokens(kf_ctx* ctx, const IParams& p, const IPlan& plan) {
    if (p.M == 1) return launch_fmt<FMT, 1>(ctx, p, plan);
    return launch_fmt<FMT, 2>(ctx, p, plan);
}
}  // namespace

// KF_OK: launched, 1: not covered by this kernel (the caller goes on to gemv.cu), < 0: error
int kf_gemv_i8(kf_ctx* ctx, int n, void* const* y, const kf_tensor_desc* w, const void* x, int M, int epilogue, const void* residual, const void* norm_w,
               float norm_eps) {
    if (M > 2 || ctx->gemv_i8_max_m < M || M < 1 || n < 1 || n > 3 || !x) return 1;
    const int type = w[0].type, K = w[0].cols;
    const int fmt  = type == KF_T_Q4 ? IF_Q4 : type == KF_T_Q2 || type == KF_T_SIGN ? IF_Q2 : type == KF_T_BINARY ? IF_Q1 : -1;
    if (fmt < 0 || K % 128 || K < 128) return 1;
    if (((uintptr_t)x & 15) || ((uintptr_t)norm_w & 15)) return 1;
    const int bits = fmt == IF_Q4 ? 4 : fmt == IF_Q2 ? 2 : 1;
    IParams p;
    memset(&p, 0, sizeof(p));
    int tiles = 0;
    for (int i = 0; i < n; i++) {
        if (w[i].type != type || w[i].cols != K || w[i].qbias != w[0].qbias || w[i].group != w[0].group || w[i].rows % 16 || w[i].rows < 16 || !w[i].data_dev || !y[i]) return 1;
        if (!kf_has_gama(w[i]) || w[i].group != 128) return 1;
        const uint16_t *z = kf_gama_zero(w[i]), *s = kf_gama_step(w[i]);
        if (((uintptr_t)w[i].data_dev & 15) || ((uintptr_t)z & 15) || ((uintptr_t)s & 15)) return 1;
        p.seg[i] = ISeg{(const uint8_t*)w[i].data_dev, z, s, (uint16_t*)y[i], w[i].rows, tiles};
        tiles += w[i].rows / 16;
    }
    if (epilogue == EPI_SWIGLU && (n != 2 || w[0].rows != w[1].rows)) return 1;
    if (epilogue == EPI_RESIDUAL && (n != 1 || !residual)) return 1;
    if (epilogue != EPI_NONE && epilogue != EPI_RESIDUAL && epilogue != EPI_SWIGLU && epilogue != EPI_F32) return 1;
    p.nseg = n, p.x = (const uint16_t*)x, p.residual = (const uint16_t*)residual, p.norm_w = (const uint16_t*)norm_w, p.norm_eps = norm_eps;
    p.M = M, p.K = K, p.ksteps = K / 128, p.tiles = tiles, p.unit = epilogue == EPI_SWIGLU ? 2 : 1, p.qbias = w[0].qbias, p.epilogue = epilogue;

    // What gemv.cu answers.  Two tokens over the largest 4-bit weights: its activations take half the shared memory (51200 x 5120, 128000 steps: 34.0 us there, 35.4 here; 24576 x 4096,
    // 49152 steps: 17.3 and 16.0).  Weights of small models (a handful of tiles): 0.1 to 0.5 us are to be had here (at one token 256 x 2048 3.1 there and 2.85 here, 1024 x 896 3.2 and
    // 2.85), but a step of several sequences, which is gemv.cu's, then keeps the bits of single ones.  (Three and four tokens take two matrix instructions here and gain nothing: 3968 x
    // 3328 at four 6.3 us there and 6.8 here.)
    const long long steps = (long long)tiles * p.ksteps;
    if (steps < 512 || (M == 2 && fmt == IF_Q4 && steps > 64000)) return 1;

    // ---- plan: K whole or in halves, by modelled time ----
    const int units = tiles / p.unit;
    constexpr int ch  = kCh;
    const size_t slot = (size_t)ch * 32 * 8 * bits;
    // blocks of zeros or steps that the chunks in flight and the one in work can meet, at most: those of a run of entries, and the two ends of each tile in it (K = 128 and 256 meet too
    // many: gemv.cu).  The bound is one block above what ten entries of long rows meet, so that four chunks are in flight for slices of 7 and 8 steps alone, three or two elsewhere
    auto blocks = [&](int depth, int ns) {
        const int steps = (depth + 1) * ch, chunks = (ns + ch - 1) / ch, tiles_met = (depth + 1 - 2) / chunks + 2;
        return std::min(tiles_met * ((2 * ns + 14) / 16 + 1), (2 * steps + 15) / 16 + 2 * tiles_met - 1);
    };
    IPlan best = {};
    double best_t = 1e30;
    // us a k-step of an SM with one and with two CTAs on it, by bits (the bytes alone take 24, 13 and 7 ns), and what is fixed, measured over 46 shapes at one and two
    // tokens.  Two CTAs an SM wherever there are tiles for them, which is all that its registers take: one a SM is a little faster behind itself (10240 x 5120 9.3 against 9.7
    // us), but not behind a kernel whose SMs come free one by one, where CTAs meant for one SM each pile up on the first (a user's attention block over 30000 positions 59.2
    // against 53.7 us, 32B decode 197 against 207 tokens/s).  K whole or in halves: clusters of four and more do not fill the GPCs (5120 x 25600: S = 1, 2, 4 and 8 take 21.0,
    // 17.9, 26 and 28 us)
    static const double step_ns[2][3] = {{36.5, 31.2, 23.1}, {24.3, 18.3, 13.6}};
    for (int S = 1; S <= 2 && S <= p.ksteps; S++) {
        const int clusters = std::min(units, ctx->sm_count * 2 / S), on_sm = clusters * S > ctx->sm_count ? 2 : 1;
        const int tpc = (units + clusters - 1) / clusters * p.unit, n0 = p.ksteps / S, ns = (p.ksteps + S - 1) / S;
        const size_t sx = (size_t)(ns + ch) * M * 512, part = sx + (size_t)(ns + ch) * M * 8, red = part + (size_t)(tpc + kWarps) * M * 64;
        const size_t gama = (red + (S > 1 ? (size_t)S * tpc * M * 64 : 0) + 15) & ~(size_t)15, ring = gama + kWarps * kGRing;
        int depth = 0;
        bool late = false;
        for (size_t room : {on_sm == 2 ? kTwo : kEarly, kHalfSM, kMost}) {
            // one CTA an SM, and the next kernel starts only behind this one.  Not at two tokens where there are tiles for two CTAs an SM, whose activations then leave no room for a
            // plan (K from about 18000): gemv.cu, as fast (5120 x 25600 at two: 22.2 us in 4 bits there, 21.2 in 2, 20.1 in 1)
            late = room == kMost;
            if (late && (on_sm == 2 || (M == 2 && fmt != IF_Q4))) break;
            for (int d : {4, 3, 2})
                if (!depth && ring + kWarps * slot * d <= room && blocks(d, ns) <= kGB && blocks(d, n0) <= kGB) depth = d;
            if (depth) break;
        }
        if (!depth) continue;
        const int rounds = (ns * 4 * M + kThreads - 1) / kThreads;
        const double t   = 4.1 + on_sm * (tpc * ns * step_ns[on_sm - 1][fmt] * 1e-3 * (1.0 + 0.13 * (M - 1)) + 0.5 * rounds + 0.046 * tpc) + (S > 1 ? 0.35 : 0.0) + (late ? 1.65 : 0.0);
        if (t < best_t) {
            best_t = t, best = IPlan{S, clusters, depth, ring + kWarps * slot * depth};
            p.off_sx = (int)sx, p.off_part = (int)part, p.off_red = (int)red, p.off_gama = (int)gama, p.off_ring = (int)ring;
        }
    }
    if (!best.S) return 1;
    p.S = best.S, p.clusters = best.clusters;
    ctx->gemv_last_s = best.S, ctx->gemv_last_kernel = 2;
    return fmt == IF_Q4 ? launch_tokens<IF_Q4>(ctx, p, best) : fmt == IF_Q2 ? launch_tokens<IF_Q2>(ctx, p, best) : launch_tokens<IF_Q1>(ctx, p, best);
}
