// attn_gqa.cu -- decode attention with the query heads of a kv group processed together (one token each for many sequences, or one sequence deep into its context).
//
// Replaces the same reference kernels as attention.cu (attention_qk / softmax / attention_v, src/Device/CUDA/kernel/operator.cuh:573-668).  Every cached row is
// read once per kv head, so the bytes of the cache bound it; what matters is how many of them are on their way and that no SM runs dry.
//   * a CTA takes one (sequence, kv head, run of `chunk` positions).  Sequences have their own lengths: equal runs, as many as a sequence needs, keep the SMs
//     evenly busy where a fixed number of slices per sequence left the long ones for last (64 sequences of 500 .. 2000 positions: 108 us for 50 us of bytes);
//   * tiles of 64 positions of K and V come by TMA into a ring of three stages (96 KB a CTA, two CTAs per SM: 28 MB in flight); the four compute warps take 16
//     positions of a tile each and meet only at its barriers.  Filling a double buffer by cp.async cost them 32 copies a tile and two block barriers;
//   * scores and P V on mma.sync with the group's heads as the 16 rows of the A operand (tensor work is a fifth of the time the bytes take);
//   * the run that arrives last at its (sequence, kv head) merges all of them in order: no second launch.
// Rows behind a sequence's last position are zeroed in shared memory before P V: their weight is zero, but they need not hold numbers.
#include <algorithm>

#include "kf_common.cuh"
#include "kf_tc.cuh"

namespace {
constexpr int kTok = 64, kRing = 3, kWarps = 4, kThreadsG = (kWarps + 1) * 32, kMaxRuns = 128;

__device__ int g_gqa_error;
__device__ __noinline__ bool gqa_wait_slow(uint32_t bar, uint32_t parity, volatile int* dead) {
    for (int it = 0; it < (1 << 20); it++) {
        if (mbar_try(bar, parity)) return true;
        if (*dead) return false;
    }
    *dead = 1;
    atomicExch(&g_gqa_error, 1);
    return false;
}
__device__ __forceinline__ bool gqa_wait(uint32_t bar, uint32_t parity, volatile int* dead) {
    return __all_sync(0xffffffffu, mbar_try(bar, parity) || gqa_wait_slow(bar, parity, dead));
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)), "l"(tm), "r"(c0),
                 "r"(c1), "r"(c2), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// partial of a run in the workspace: [sequence][kv head][run][group][HD + 2] floats: sum p v, maximum (log2 domain), sum p
template <int HD>
__global__ void __launch_bounds__(kThreadsG, 2)
    kf_attn_gqa_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, uint16_t* __restrict__ out, float* __restrict__ ws,
                       unsigned* __restrict__ cnt, const uint16_t* __restrict__ q, const int32_t* __restrict__ pos_dev, int n_head, int n_kv, int max_seq, int min_chunk,
                       float sc2 /* log2(e) / sqrt(hd) */) {
    constexpr int HALVES = HD / 64, TILE = kTok * HD * 2, HALF = kTok * 128;  // a tile lies as halves of 64 dims: 64 rows of 128 bytes (SWIZZLE_128B)
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);  // [kRing][K tile | V tile]
    __shared__ uint64_t full[kRing], empty[kRing];
    __shared__ volatile int dead;
    __shared__ int s_last;
    __shared__ float s_m[kWarps][16], s_l[kWarps][16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int kvh = blockIdx.x, m = blockIdx.y, run = blockIdx.z, group = n_head / n_kv;
    if (tid == 0) {
        for (int s = 0; s < kRing; s++) mbar_init(&full[s], 1), mbar_init(&empty[s], kWarps);
        dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    kf_grid_launch_dependents();
    kf_grid_dependency_wait();  // queries, the rows of the current position, positions, workspace
    // the launch was sized from a hint: a sequence takes all runs if it must, so any length is covered
    const int len   = min(pos_dev[m] + 1, max_seq);
    const int chunk = max(min_chunk, ((len + (int)gridDim.z - 1) / (int)gridDim.z + kTok - 1) / kTok * kTok), runs = (len + chunk - 1) / chunk;
    if (run >= runs) return;
    const int t0 = run * chunk, t1 = min(len, t0 + chunk), ntiles = (t1 - t0 + kTok - 1) / kTok;

    float o[HD / 8][4];
    float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;
    if (warp == kWarps) {
        bool live = true;
        int kt = 0;
        for (; kt < ntiles; kt++) {
            const int st = kt % kRing;
            if (!(live = gqa_wait(smem_u32(&empty[st]), ((kt / kRing) & 1) ^ 1, &dead))) break;
            if (lane == 0) {
                mbar_arrive_expect_tx(&full[st], 2 * TILE);
                uint8_t* d = ring + st * 2 * TILE;
#pragma unroll
                for (int i = 0; i < HALVES; i++) {
                    tma_load_3d(d + i * HALF, &tm_k, kvh * HD + i * 64, t0 + kt * kTok, m, &full[st]);
                    tma_load_3d(d + TILE + i * HALF, &tm_v, kvh * HD + i * 64, t0 + kt * kTok, m, &full[st]);
                }
            }
        }
        if (!live)  // copies in flight write shared memory
            for (int k = kt > kRing ? kt - kRing : 0; k < kt; k++)
                for (int it = 0; it < (1 << 14) && !mbar_try(smem_u32(&full[k % kRing]), (k / kRing) & 1); it++) {}
    } else {
        // the group's queries as A fragments: row r of 16 is head r (rows past the group are zero)
        uint32_t qa[HD / 16][4];
        const uint16_t* qb = q + ((size_t)m * n_head + (size_t)kvh * group) * HD;
#pragma unroll
        for (int kc = 0; kc < HD / 16; kc++) {
            const uint32_t* lo = reinterpret_cast<const uint32_t*>(qb + (size_t)g * HD + kc * 16 + 2 * t4);
            const uint32_t* hi = reinterpret_cast<const uint32_t*>(qb + (size_t)(g + 8) * HD + kc * 16 + 2 * t4);
            qa[kc][0] = g < group ? lo[0] : 0u, qa[kc][2] = g < group ? lo[4] : 0u;
            qa[kc][1] = g + 8 < group ? hi[0] : 0u, qa[kc][3] = g + 8 < group ? hi[4] : 0u;
        }
#pragma unroll
        for (int j = 0; j < HD / 8; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
        // 16-byte chunk c (0 .. HD / 8 - 1) of a row: half c / 8, chunk c % 8 swizzled by the row
        auto at = [](uint32_t base, int row, int c) { return base + (uint32_t)((c >> 3) * HALF + row * 128 + (((c & 7) ^ (row & 7)) << 4)); };
        for (int kt = 0; kt < ntiles; kt++) {
            const int st = kt % kRing;
            if (!gqa_wait(smem_u32(&full[st]), (kt / kRing) & 1, &dead)) break;
            const uint32_t kb = smem_u32(ring + st * 2 * TILE), vb = kb + TILE;
            const int tok0 = t0 + kt * kTok + warp * 16;  // this warp's 16 positions
            if (tok0 < t1) {
                float sc[2][4];
#pragma unroll
                for (int j = 0; j < 2; j++) sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
#pragma unroll
                for (int kc = 0; kc < HD / 16; kc++) {
                    uint32_t b[4];
                    ldsm4(b, at(kb, warp * 16 + (lane & 7) + (lane >> 4) * 8, kc * 2 + ((lane >> 3) & 1)));
                    mma16816(sc[0], qa[kc], b[0], b[1]);
                    mma16816(sc[1], qa[kc], b[2], b[3]);
                }
                if (tok0 + 16 > t1) {  // the run's last positions: no weight, and no value that might not be a number
#pragma unroll
                    for (int j = 0; j < 2; j++)
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (tok0 + j * 8 + 2 * t4 + (e & 1) >= t1) sc[j][e] = -INFINITY;
                    const int r0 = t1 - tok0;
                    for (int i = lane; i < (16 - r0) * (HD / 8); i += 32) {
                        const int row = warp * 16 + r0 + i / (HD / 8), c = i % (HD / 8);
                        *reinterpret_cast<uint4*>(ring + st * 2 * TILE + TILE + (c >> 3) * HALF + row * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    __syncwarp();
                }
                float mx_lo = fmaxf(fmaxf(sc[0][0], sc[0][1]), fmaxf(sc[1][0], sc[1][1])), mx_hi = fmaxf(fmaxf(sc[0][2], sc[0][3]), fmaxf(sc[1][2], sc[1][3]));
                mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1)), mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
                mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1)), mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
                const float mn_lo = fmaxf(m_lo, mx_lo * sc2), mn_hi = fmaxf(m_hi, mx_hi * sc2);  // finite: position tok0 is seen
                const float c_lo = exp2f(m_lo - mn_lo), c_hi = exp2f(m_hi - mn_hi);
                m_lo = mn_lo, m_hi = mn_hi;
                float rs_lo = 0.f, rs_hi = 0.f;
                uint32_t pa[4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const float p0 = exp2f(fmaf(sc[j][0], sc2, -mn_lo)), p1 = exp2f(fmaf(sc[j][1], sc2, -mn_lo));
                    const float p2 = exp2f(fmaf(sc[j][2], sc2, -mn_hi)), p3 = exp2f(fmaf(sc[j][3], sc2, -mn_hi));
                    rs_lo += p0 + p1, rs_hi += p2 + p3;
                    pa[j * 2 + 0] = pack_bf16x2(p0, p1), pa[j * 2 + 1] = pack_bf16x2(p2, p3);
                }
                l_lo = l_lo * c_lo + rs_lo, l_hi = l_hi * c_hi + rs_hi;
                if (__any_sync(0xffffffffu, c_lo != 1.f || c_hi != 1.f)) {
#pragma unroll
                    for (int j = 0; j < HD / 8; j++) o[j][0] *= c_lo, o[j][1] *= c_lo, o[j][2] *= c_hi, o[j][3] *= c_hi;
                }
#pragma unroll
                for (int jp = 0; jp < HD / 16; jp++) {
                    uint32_t b[4];
                    ldsm4_t(b, at(vb, warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, jp * 2 + (lane >> 4)));
                    mma16816(o[2 * jp], pa, b[0], b[1]);
                    mma16816(o[2 * jp + 1], pa, b[2], b[3]);
                }
            }
            // every ldmatrix above has delivered: the matrix instructions behind them were issued with its registers
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[st]);
        }
    }
    __syncthreads();
    if (dead) return;
    // ---- merge the four warps (fixed order) through shared memory: the ring is free now ----
    float* s_o = reinterpret_cast<float*>(ring);  // [4][16][HD]
    if (warp < kWarps) {
        l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1), l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
        l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1), l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
#pragma unroll
        for (int j = 0; j < HD / 8; j++) {
            float* r0 = s_o + ((size_t)warp * 16 + g) * HD + j * 8 + 2 * t4;
            *reinterpret_cast<float2*>(r0) = make_float2(o[j][0], o[j][1]), *reinterpret_cast<float2*>(r0 + 8 * HD) = make_float2(o[j][2], o[j][3]);
        }
        if (t4 == 0) s_m[warp][g] = m_lo, s_m[warp][g + 8] = m_hi, s_l[warp][g] = l_lo, s_l[warp][g + 8] = l_hi;
    }
    __syncthreads();
    float* part = ws + (((size_t)m * n_kv + kvh) * gridDim.z) * (size_t)group * (HD + 2);
    for (int idx = tid; idx < group * HD; idx += kThreadsG) {
        const int r = idx / HD, c = idx % HD;
        float M_ = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; w++) M_ = fmaxf(M_, s_m[w][r]);
        float L_ = 0.f, acc = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const float f = s_m[w][r] == -INFINITY ? 0.f : exp2f(s_m[w][r] - M_);
            L_ += s_l[w][r] * f;
            acc = fmaf(s_o[((size_t)w * 16 + r) * HD + c], f, acc);
        }
        if (runs == 1) {
            out[((size_t)m * n_head + (size_t)kvh * group + r) * HD + c] = f32_to_bf16_bits(acc / L_);
        } else {
            float* wp = part + ((size_t)run * group + r) * (HD + 2);
            __stcg(wp + c, acc);
            if (c == 0) __stcg(wp + HD, M_), __stcg(wp + HD + 1, L_);
        }
    }
    if (runs == 1) return;
    // ---- the last run of this (sequence, kv head) merges all of them in order ----
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned* c = cnt + (size_t)m * n_kv + kvh;
        s_last      = atomicAdd(c, 1u) == (unsigned)(runs - 1);
        if (s_last) *c = 0u;  // self-reset for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float* s_f = reinterpret_cast<float*>(ring);  // [group][runs] factors, then [group] inverse denominators
    float* s_i = s_f + group * kMaxRuns;
    for (int r = warp; r < group; r += kThreadsG / 32) {
        float M_ = -INFINITY;
        for (int s = lane; s < runs; s += 32) M_ = fmaxf(M_, __ldcg(part + ((size_t)s * group + r) * (HD + 2) + HD));
        M_ = warp_max(M_);
        float L_ = 0.f;
        for (int s = lane; s < runs; s += 32) {
            const float f = exp2f(__ldcg(part + ((size_t)s * group + r) * (HD + 2) + HD) - M_);
            L_ += __ldcg(part + ((size_t)s * group + r) * (HD + 2) + HD + 1) * f;
            s_f[r * kMaxRuns + s] = f;
        }
        L_ = warp_sum(L_);
        if (lane == 0) s_i[r] = 1.f / L_;
    }
    __syncthreads();
    for (int idx = tid; idx < group * (HD / 2); idx += kThreadsG) {
        const int r = idx / (HD / 2), c = (idx % (HD / 2)) * 2;
        const float* wp = part + (size_t)r * (HD + 2) + c;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
        for (int s = 0; s < runs; s++) {
            const float2 v = __ldcg(reinterpret_cast<const float2*>(wp + (size_t)s * group * (HD + 2)));
            const float f  = s_f[r * kMaxRuns + s];
            a0 = fmaf(v.x, f, a0), a1 = fmaf(v.y, f, a1);
        }
        *reinterpret_cast<uint32_t*>(out + ((size_t)m * n_head + (size_t)kvh * group + r) * HD + c) = pack_bf16x2(a0 * s_i[r], a1 * s_i[r]);
    }
}

template <int HD>
int gqa_launch(kf_ctx* ctx, void* out, const void* q, const void* kc, const void* vc, const int32_t* pos_dev, int M, int n_head, int n_kv, int max_seq, int len,
               size_t seq_stride) {
    // ---- runs.  One sequence: one wave of two CTAs per SM, all equally long.  Several: their lengths differ, so about six waves of shorter runs, of at least 256
    // positions (four tiles: a run's set-up and merge cost about one).  `attn_split` fixes the number of runs instead. ----
    const int slots = 2 * ctx->sm_count;
    int chunk = 2 * kTok, runs;
    if (ctx->attn_split > 0) chunk = kTok, runs = ctx->attn_split;
    else if (M == 1) runs = std::max(1, slots / n_kv);
    else chunk = (int)std::max<long long>(256, (long long)n_kv * M * len / (6 * slots) / kTok * kTok), runs = (len + chunk - 1) / chunk;
    runs = std::max(1, std::min(runs, std::min(kMaxRuns, (len + chunk - 1) / chunk)));
    float* ws = nullptr;
    if (runs > 1) {
        int rc = kf_ensure_attn_ws(ctx, (size_t)M * n_head * runs * (HD + 2) * sizeof(float));
        if (!rc) rc = kf_ensure_attn_cnt(ctx, M * n_kv);
        if (rc) return rc;
        ws = ctx->attn_ws;
    }
    CUtensorMap tk, tv;
    const uint64_t stride = M > 1 ? (uint64_t)seq_stride * 2 : (uint64_t)n_kv * HD * 2;
    int rc = kf_tmap_rows(ctx, &tk, kc, (uint64_t)n_kv * HD, (uint64_t)max_seq, (uint64_t)M, stride, 64, kTok);
    if (!rc) rc = kf_tmap_rows(ctx, &tv, vc, (uint64_t)n_kv * HD, (uint64_t)max_seq, (uint64_t)M, stride, 64, kTok);
    if (rc) return rc;
    const size_t smem = (size_t)kRing * 2 * kTok * HD * 2 + 1024;
    static_assert(kRing * 2 * kTok * HD * 2 >= 4 * 16 * HD * 4 && kRing * 2 * kTok * HD * 2 >= 16 * (kMaxRuns + 1) * 4, "the merges use the ring");
    static bool set[kf_ctx::kMaxDevices] = {};  // function attributes are per device
    if (!set[ctx->device]) {
        KF_CUDA(ctx, cudaFuncSetAttribute(kf_attn_gqa_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        set[ctx->device] = true;
    }
    KF_CUDA(ctx, kf_launch_pdl(ctx, kf_attn_gqa_kernel<HD>, dim3(n_kv, M, runs), dim3(kThreadsG), smem, tk, tv, (uint16_t*)out, ws, ctx->attn_cnt, (const uint16_t*)q, pos_dev,
                               n_head, n_kv, max_seq, chunk, 1.4426950408889634f / sqrtf((float)HD)));
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
}  // namespace

// Decode attention for MANY sequences per step (one token each): the query heads of a kv group share every cached row through the tensor cores.  Same contract
// as kf_attn_decode; q normalised + rotated, K / V of the current position appended.
extern "C" int kf_attn_decode_gqa(kf_ctx* ctx, void* out, const void* q, const void* kc, const void* vc, const int32_t* pos_dev, int M, int n_head,
                                  int n_kv, int hd, int max_seq, int max_pos_hint, size_t seq_stride) {
    if (!ctx || !out || !q || !kc || !vc || !pos_dev) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, (hd == 128 || hd == 64) && n_head % n_kv == 0 && n_head / n_kv <= 16 && M >= 1 && max_seq >= 1, "head_dim 64/128, group <= 16");
    KF_REQUIRE(ctx, M == 1 || seq_stride > 0, "one sequence per token");
    KF_REQUIRE(ctx, (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) & 15) == 0 && (M == 1 || seq_stride % 8 == 0), "16-byte aligned rows");
    const int len = std::max(1, std::min(max_seq, max_pos_hint + 1));
    if (hd == 128) return gqa_launch<128>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, len, seq_stride);
    return gqa_launch<64>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, len, seq_stride);
}
int kf_attn_gqa_error() {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_gqa_error, sizeof(v));
    return v;
}
