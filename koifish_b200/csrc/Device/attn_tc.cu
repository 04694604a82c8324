// attn_tc.cu -- causal attention of a prompt panel on the 5th-generation tensor cores (tcgen05 / TMEM / TMA), head size 128.
//
// Replaces the same reference chain as the mma.sync panel kernel of attention.cu (the token-by-token prompt loop, src/Manifold/GoPT.cpp:1111-1235, through
// attention_qk / softmax / attention_v, src/Device/CUDA/kernel/operator.cuh:573-668).
//
// A CTA takes 128 consecutive queries of TWO heads of one kv group, so both share every K / V tile of 128 positions, and the two chains fill each other's gaps:
// while the softmax warps of one head turn its scores into weights, the tensor cores work for the other.
//   warps 0-3 / 4-7  softmax of head 0 / 1, thread = query: scores from tensor memory, running maximum, weights as bf16 back over the scores of the second half
//   warp 8           matrix instructions: S = Q K^T (both operands in shared memory), O += P V (P from tensor memory, V as it lies: MN-major)
//   warp 9           TMA: both Q tiles once, then the K and V tiles through two stages each
// Tensor memory: S0 S1 O0 O1, 128 columns each.  What bounds it: a tile pair needs 2 x 1024 clocks of matrix instructions and 2 x 16384 exponentials, 2048 clocks
// of the special-function units.  Measured: 1999 queries of 32 heads behind 4096 positions 575 us with the mma.sync kernel (64 queries of one head per CTA,
// fragments through ldmatrix: 290 TFLOP/s), 199 us here (840 TFLOP/s; tensor pipe half busy).  A chain on its own
// (few heads and queries) advances a tile in 1.7 us.
// The output is rescaled whenever a maximum of the warp's rows grows, so the largest weight of a row is 1 and has no rounding error: waiting until it has grown by
// 2^8 is 20 us faster here, but its error against 64 bits is 3 % (flat) to 20 % (sharp scores) above the mma.sync kernel's.  The denominator adds the unrounded weights.
// Rows of V behind the last position are zeroed in shared memory: their weight is zero, but whatever the cache holds there need not be a number.
// Every wait is bounded: when one runs out, `dead` ends all roles, copies and matrix instructions in flight are awaited and tensor memory is freed.
#include "kf_common.cuh"
#include "kf_tc.cuh"

namespace {
constexpr int kQ = 128, kKV = 128, kHD = 128, kStages = 2;
constexpr int kTile = kKV * kHD * 2, kHalf = kTile / 2;  // a tile lies as two halves of 64 dims, 128 rows of 128 bytes each (SWIZZLE_128B)
constexpr int kMmaW = 8, kLoadW = 9, kThreads = 10 * 32;
constexpr size_t kSmem = 2 * kTile + 2 * kStages * kTile + 1024;

// 32 columns of this lane's row; the caller waits (tcgen05.wait::ld) before it uses them
__device__ __forceinline__ void ld32_async(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, "
        "[%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
          "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
        "%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
        "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// the maximum of scores that are all -inf so far is taken as 0, so that their weights are 0
__device__ __forceinline__ float finite_or_0(float m) { return m == -INFINITY ? 0.f : m; }
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// shared-memory descriptor of a V tile: MN-major (64 dims side by side, then the next position's 128-byte row), SWIZZLE_128B; the dims' second half lies kHalf
// behind the first (leading byte offset), eight positions 1024 bytes behind the eight before (stride byte offset)
__device__ __forceinline__ uint64_t make_desc_v(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)(kHalf >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__global__ void __launch_bounds__(kThreads, 1)
    kf_attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                              uint16_t* __restrict__ out, const int32_t* __restrict__ pos_dev, int M, int n_head, int n_kv, int max_seq, float sc2 /* log2(e) / sqrt(hd) */,
                              const __grid_constant__ KfBound bound) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sk = sq + 2 * kTile;
    uint8_t* sv = sk + kStages * kTile;
    __shared__ uint64_t q_full, k_full[kStages], k_empty[kStages], v_full[kStages], v_empty[kStages], v_land, s_full[2], p_full[2][2], o_done[2], done_bar;
    __shared__ uint32_t tmem_base_smem;
    __shared__ volatile int dead;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qt = (int)gridDim.x - 1 - (int)blockIdx.x, h0 = blockIdx.y * 2, kvh = h0 / (n_head / n_kv);  // late (long) query tiles first
    const int q0 = qt * kQ;

    if (tid == 0) {
        mbar_init(&q_full, 1), mbar_init(&v_land, 1), mbar_init(&done_bar, 1);
        for (int s = 0; s < kStages; s++) mbar_init(&k_full[s], 1), mbar_init(&k_empty[s], 1), mbar_init(&v_full[s], 1), mbar_init(&v_empty[s], 1);
        for (int t = 0; t < 2; t++) mbar_init(&s_full[t], 1), mbar_init(&p_full[t][0], 4), mbar_init(&p_full[t][1], 4), mbar_init(&o_done[t], 1);
        dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_smem;
    kf_grid_launch_dependents();
    kf_grid_dependency_wait();  // queries, cache rows and the position come from the kernels before us
    pos_dev = behind_wait(pos_dev);
    const int pos0 = pos_dev[0], kv_len = min(pos0 + min(M, q0 + kQ), max_seq), n_tiles = (kv_len + kKV - 1) / kKV;

    if (warp < 8) {
        const int t = warp >> 2, quad = warp & 3, row = quad * 32 + lane, pos = pos0 + q0 + row;
        const uint32_t s_row = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t * 128), o_row = s_row + 256;
        const uint32_t sfull = smem_u32(&s_full[t]), pfull = smem_u32(&p_full[t][0]), odone = smem_u32(&o_done[t]);
        float m = -INFINITY;           // the maximum that the weights and O refer to
        unsigned long long l2 = 0ull;  // the denominator, even and odd positions apart
        bool live = true;
        for (int kt = 0; kt < n_tiles; kt++) {
            if (!(live = mbar_wait_warp(sfull, kt & 1, &dead, bound))) break;
            tc_fence_after();
            // The scores are read twice, 64 positions at a time: 128 of them beside the weights do not fit the registers.  The second half is still there when the
            // maximum is known, so it goes first.
            const bool diag = (kt + 1) * kKV > pos0 + q0;  // tiles that reach the panel: positions behind the query are not seen
            const int lim   = pos - kt * kKV;
            uint32_t s[64];
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            auto fetch = [&](int c) {
                ld32_async(s_row + 64 * c, s), ld32_async(s_row + 64 * c + 32, s + 32);
                wait_ld();
                if (diag) {
#pragma unroll
                    for (int j = 0; j < 64; j++)
                        if (64 * c + j > lim) s[j] = 0xff800000u;
                }
            };
#pragma unroll
            for (int c = 0; c < 2; c++) {
                fetch(c);
#pragma unroll
                for (int j = 0; j < 64; j += 4)
#pragma unroll
                    for (int e = 0; e < 4; e++) mx[e] = fmaxf(mx[e], __uint_as_float(s[j + e]));
            }
            const float mn = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if (kt == 0) {
                m = mn;
            } else if (__any_sync(0xffffffffu, mn > m)) {
                const float n = fmaxf(m, mn), f = ex2((m - finite_or_0(n)) * sc2);
                if (!(live = mbar_wait_warp(odone, (kt - 1) & 1, &dead, bound))) break;  // the last O += P V is through
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    uint32_t o[32];
                    ld32_async(o_row + 32 * c, o);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                    st32(o_row + 32 * c, o);
                }
                wait_st();
                l2 = mul2(l2, pack2(f, f)), m = n;
            }
            const float base = finite_or_0(m) * sc2;
            const unsigned long long sc22 = pack2(sc2, sc2), nm2 = pack2(-base, -base);
#pragma unroll
            for (int c = 1; c >= 0; c--) {  // one half's O += P V runs while the other half's weights are formed
                if (c == 0) fetch(0);
                uint32_t p[32];
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const float2 x = unpack2(fma2(pack2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), sc22, nm2));
                    const float a = ex2(x.x), b = ex2(x.y);
                    l2   = add2(l2, pack2(a, b));
                    p[j] = pack_bf16x2(a, b);
                }
                st32(s_row + 64 + 32 * c, p);  // over scores of the second half, which are in registers
                wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_a(pfull + 8 * c);
            }
        }
        if (live) live = mbar_wait_warp(odone, (n_tiles - 1) & 1, &dead, bound);
        if (live) {
            tc_fence_after();
            const float2 l  = unpack2(l2);
            const float inv = 1.f / (l.x + l.y);
            uint16_t* op    = out + (size_t)(q0 + row) * n_head * kHD + (size_t)(h0 + t) * kHD;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t o[32];
                ld32_async(o_row + 32 * c, o);
                wait_ld();
                if (q0 + row < M) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t v[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) v[e] = pack_bf16x2(__uint_as_float(o[8 * j + 2 * e]) * inv, __uint_as_float(o[8 * j + 2 * e + 1]) * inv);
                        *reinterpret_cast<uint4*>(op + 32 * c + 8 * j) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                }
            }
        }
    } else if (warp == kMmaW) {
        constexpr uint32_t id_s = make_idesc_bf16(128), id_o = make_idesc_bf16(128) | (1u << 16);  // bit 16: B is MN-major
        const uint32_t q_addr = smem_u32(sq), k_addr = smem_u32(sk), v_addr = smem_u32(sv);
        bool live = mbar_wait_warp(smem_u32(&q_full), 0, &dead, bound);
        auto score = [&](int t, int stage) {  // S_t = Q_t K^T, 16 of the 128 dims per instruction
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t off = (uint32_t)((k >> 2) * kHalf + (k & 3) * 32);
                umma_ss(tmem + t * 128, make_desc_sw128(q_addr + t * kTile + off), make_desc_sw128(k_addr + stage * kTile + off), id_s, k > 0);
            }
            umma_commit_a(smem_u32(&s_full[t]));
        };
        if (live) live = mbar_wait_warp(smem_u32(&k_full[0]), 0, &dead, bound);
        if (live) {
            tc_fence_after();
            score(0, 0), score(1, 0);
            umma_commit_a(smem_u32(&k_empty[0]));
        }
        for (int kt = 0; live && kt < n_tiles; kt++) {
            const int st = kt % kStages, sn = (kt + 1) % kStages;
#pragma unroll
            for (int t = 0; t < 2; t++) {
                if (t == 0 && !(live = mbar_wait_warp(smem_u32(&v_full[st]), (kt / kStages) & 1, &dead, bound))) break;
#pragma unroll
                for (int i = 0; i < 8; i++) {  // O_t += P_t V, 16 positions per instruction, the second half of the positions first
                    const int k = i ^ 4;
                    if (i % 4 == 0) {
                        live = live && mbar_wait_warp(smem_u32(&p_full[t][k / 4]), kt & 1, &dead, bound);
                        tc_fence_after();
                    }
                    if (live) umma_ts(tmem + 256 + t * 128, tmem + t * 128 + 64 + k * 8, make_desc_v(v_addr + st * kTile + k * 2048), id_o, kt > 0 || i > 0);
                }
                if (!live) break;
                umma_commit_a(smem_u32(&o_done[t]));
                if (kt + 1 < n_tiles) {
                    if (t == 0) {
                        if (!(live = mbar_wait_warp(smem_u32(&k_full[sn]), ((kt + 1) / kStages) & 1, &dead, bound))) break;
                        tc_fence_after();
                    }
                    score(t, sn);  // behind the O above, which reads the weights from the same columns
                }
            }
            if (!live) break;
            umma_commit_a(smem_u32(&v_empty[st]));
            if (kt + 1 < n_tiles) umma_commit_a(smem_u32(&k_empty[sn]));
        }
        if (!live) {
            umma_commit_a(smem_u32(&done_bar));
            mbar_drain(smem_u32(&done_bar), 0, bound);
        }
    } else if (warp == kLoadW && bound.drop != (int)(blockIdx.y * gridDim.x + blockIdx.x) + 1) {
        bool live = true;
        if (lane == 0) {
            mbar_arrive_expect_tx(&q_full, 2 * kTile);
#pragma unroll
            for (int i = 0; i < 4; i++) tma_load_2d(sq + i * kHalf, &tm_q, (h0 + (i >> 1)) * kHD + (i & 1) * 64, q0, &q_full);
        }
        int kt = 0;
        for (; kt < n_tiles; kt++) {
            const int st = kt % kStages;
            const uint32_t ph = ((kt / kStages) & 1) ^ 1;
            if (!(live = mbar_wait_warp(smem_u32(&k_empty[st]), ph, &dead, bound))) break;
            if (lane == 0) {
                mbar_arrive_expect_tx(&k_full[st], kTile);
#pragma unroll
                for (int i = 0; i < 2; i++) tma_load_2d(sk + st * kTile + i * kHalf, &tm_k, kvh * kHD + i * 64, kt * kKV, &k_full[st]);
            }
            if (!(live = mbar_wait_warp(smem_u32(&v_empty[st]), ph, &dead, bound))) break;
            const bool ragged = (kt + 1) * kKV > kv_len;  // the last tile, unless it ends with a position
            uint64_t* bar = ragged ? &v_land : &v_full[st];
            if (lane == 0) {
                mbar_arrive_expect_tx(bar, kTile);
#pragma unroll
                for (int i = 0; i < 2; i++) tma_load_2d(sv + st * kTile + i * kHalf, &tm_v, kvh * kHD + i * 64, kt * kKV, bar);
            }
            if (ragged) {
                if (!(live = mbar_wait_warp(smem_u32(&v_land), 0, &dead, bound))) break;
                const int r0 = kv_len - kt * kKV;
                for (int i = lane; i < (kKV - r0) * 16; i += 32)
                    *reinterpret_cast<uint4*>(sv + st * kTile + (i & 1) * kHalf + (r0 + (i >> 4)) * 128 + ((i >> 1) & 7) * 16) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_full[st]);
            }
        }
        if (!live) {  // copies in flight write shared memory: wait for what was asked for
            mbar_drain(smem_u32(&q_full), 0, bound);
            for (int k = kt > 0 ? kt - 1 : 0; k <= kt && k < n_tiles; k++)
                mbar_drain(smem_u32(&k_full[k % kStages]), (k / kStages) & 1, bound), mbar_drain(smem_u32(&v_full[k % kStages]), (k / kStages) & 1, bound);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaW) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}
}  // namespace

// Panels the kernel takes: head size 128, an even number of query heads per kv head, 16-byte aligned rows, and more than 64 queries -- but not those of up to 512
// queries for whose blocks (64 queries of a head) the mma.sync kernel has an SM each and that cannot lie deep in their context, the cache having room for no more than
// 512 positions in front of them (where they do lie is known on the device only).  There that kernel's finer tiles win.  With norm and append in front, here / there in us:
// 16 heads, 96 queries 11.0 / 10.4, behind 300 positions 18.6 / 16.5, behind 700 24.8 / 22.7; 300 queries 16.5 / 16.5, behind 700 28.8 / 28.7; 513 behind 4000 78 / 92; 700 queries
// 24.7 / 30.8.  32 heads, 256 queries 16.5 / 14.5, 300 queries 17.4 / 18.6.  64 heads, 128 queries 13.0 / 12.4, 129 queries 14.5 / 16.5.  2 heads, 512 queries 18.6 / 17.5.
int kf_attn_prefill_tc_ok(const kf_ctx* ctx, const void* out, const void* q, const void* kc, const void* vc, int M, int n_head, int n_kv, int hd, int max_seq) {
    const bool gains = ctx->attn_tc_min_m > 0 ? M >= ctx->attn_tc_min_m : M > 512 || max_seq - M > 512 || (long long)((M + 63) / 64) * n_head > ctx->sm_count;
    return hd == kHD && M > 64 && gains && (n_head / n_kv) % 2 == 0 && n_head / 2 <= 65535 && (((uintptr_t)out | (uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) & 15) == 0;
}
int kf_attn_prefill_tc(kf_ctx* ctx, void* out, const void* q, const void* kc, const void* vc, const int32_t* pos_dev, int M, int n_head, int n_kv, int max_seq) {
    CUtensorMap tq, tk, tv;
    int rc = kf_wait_status(ctx);
    if (!rc) rc = kf_tmap_2d(ctx, &tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, (uint64_t)n_head * kHD, (uint64_t)M, 64, kQ, CU_TENSOR_MAP_SWIZZLE_128B, false);
    if (!rc) rc = kf_tmap_2d(ctx, &tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, kc, (uint64_t)n_kv * kHD, (uint64_t)max_seq, 64, kKV, CU_TENSOR_MAP_SWIZZLE_128B, false);
    if (!rc) rc = kf_tmap_2d(ctx, &tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, vc, (uint64_t)n_kv * kHD, (uint64_t)max_seq, 64, kKV, CU_TENSOR_MAP_SWIZZLE_128B, false);
    if (rc) return rc;
    static bool set[kf_ctx::kMaxDevices] = {};  // function attributes are per device
    if (!set[ctx->device]) {
        KF_CUDA(ctx, cudaFuncSetAttribute(kf_attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
        set[ctx->device] = true;
    }
    KF_CUDA(ctx, kf_launch_pdl(ctx, kf_attn_prefill_tc_kernel, dim3((M + kQ - 1) / kQ, n_head / 2), dim3(kThreads), kSmem, tq, tk, tv, (uint16_t*)out, pos_dev, M, n_head, n_kv,
                               max_seq, 1.4426950408889634f / sqrtf((float)kHD), KfBound{ctx->wait_flags, (unsigned)ctx->attn_wait_us, ctx->attn_drop}));
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
