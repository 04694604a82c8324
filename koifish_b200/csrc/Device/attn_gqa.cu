// attn_gqa.cu -- decode attention with the query heads of a kv group processed together (one token each for many sequences, or one sequence deep into its context).
//
// Replaces the same reference kernels as attention.cu (attention_qk / softmax / attention_v, src/Device/CUDA/kernel/operator.cuh:573-668).  Every cached row is
// read once per kv head, so the bytes of the cache bound it; what matters is how many of them are on their way and that no SM runs dry.
//   * persistent CTAs walk the (sequence, run of positions, kv head) items.  A step whose (sequence, kv head) pairs fill the SMs is not cut at all: the pairs are
//     dealt out longest first, there and back (64 sequences of 1250 positions: 58 us whole, 78 / 89 / 99 in 2 / 3 / 4 runs, each of which pays a fence, a
//     counter and its share of a merge).  Fewer pairs are cut into equal runs, as many as there are SMs, and only the runs that exist are dealt out;
//   * whole pairs: two CTAs per SM of four computing warps, so one's merge runs beside the other's tiles.  Runs: one CTA of eight warps per SM, half the merge
//     (30000 positions: 34 us against 42);
//   * one warp loads tiles of 64 positions of K and V by TMA into a ring of 16 KB stages and runs ahead of the computing warps, across items as well;
//   * four computing warps take a tile, 16 positions each (the other four the next).  Scores and P V on mma.sync with the group's heads as the 16 rows of the A operand (tensor work is
//     a fifth of the time the bytes take);
//   * the run that arrives last at its (sequence, kv head) merges all of them in order, with 16-byte loads: no second launch.
// Measured, whole attention block: 64 sequences of 500 .. 2000 positions and 8 kv heads (328 MB of cache) 154 us with a fixed number of slices and a cp.async double
// buffer, 111 here; one sequence at 30000 positions (123 MB) 78 us with the slices merged by a second launch, 59 here.
// Rows behind a sequence's last position are zeroed in shared memory before P V: their weight is zero, but they need not hold numbers.
#include <algorithm>

#include "kf_common.cuh"
#include "kf_tc.cuh"

namespace {
constexpr int kTok = 64, kMaxRuns = 128, kMaxSeqs = 512;

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

// Stages of the ring: what shared memory holds beside the warps' areas (SETS 1: two CTAs per SM), at most ten per set.  With two sets, whose tiles alternate, their
// number is a multiple of 4 (K and V of a tile of either), so that a stage always comes back to the set that used it last: a wait tells a phase of a barrier from
// the one before by a single bit, so the warps that wait for a use of a stage have to have waited for the use before.  With ten stages tile 5 lay where tile 0
// had, for the other set, which would have taken it for landed while the copies of tile 0 were still under way (copies may overtake each other).  Between two
// items of a CTA all its warps meet, behind every wait of the first.
constexpr int gqa_area(int hd, int sets, int group) { return 4 * sets * ((group + 1) & ~1) * hd * 4; }
constexpr int gqa_stages(int hd, int sets, int group) {
    const int fit = ((sets == 1 ? 97 : 200) * 1024 - gqa_area(hd, sets, group)) / (kTok * hd * 2), most = fit < 10 * sets ? fit : 10 * sets;
    return sets == 1 ? most : most & ~3;
}
constexpr bool gqa_rings_fit() {
    for (int hd = 64; hd <= 128; hd += 64)
        for (int sets = 1; sets <= 2; sets++)
            for (int group = 1; group <= 16; group++) {
                const int n = gqa_stages(hd, sets, group);
                if (n < 4 * sets || (sets == 2 && n % 4)) return false;
            }
    return true;
}
static_assert(gqa_rings_fit(), "two tiles of every set in flight, and a stage stays with its set");

// two results; out may start at any element
__device__ __forceinline__ void put2(uint16_t* p, float a, float b, bool pairs) {
    if (pairs) *reinterpret_cast<uint32_t*>(p) = pack_bf16x2(a, b);
    else p[0] = f32_to_bf16_bits(a), p[1] = f32_to_bf16_bits(b);
}

struct GqaItem {
    int m, run, kvh, t0, t1, runs;
};
// partials in the workspace: [sequence][kv head][run][group] rows of HD sums, then the same number of (maximum, denominator) pairs
template <int HD, int SETS>
__global__ void __launch_bounds__((4 * SETS + 1) * 32, 3 - SETS)
    kf_attn_gqa_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, uint16_t* __restrict__ out, float* __restrict__ ws,
                       float2* __restrict__ ws_ml, unsigned* __restrict__ cnt, const uint16_t* __restrict__ q, const int32_t* __restrict__ pos_dev, int M, int n_head, int n_kv,
                       int max_seq, int min_chunk, int max_runs, int stages, float sc2 /* log2(e) / sqrt(hd) */, const __grid_constant__ KfBound bound) {
    constexpr int HALVES = HD / 64, TILE = kTok * HD * 2, HALF = kTok * 128;  // a tile lies as halves of 64 dims: 64 rows of 128 bytes (SWIZZLE_128B)
    constexpr int kWarps = 4 * SETS, kComp = kWarps * 32, kMaxStages = 20;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int group = n_head / n_kv;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);  // [stages] tiles, K and V in turn
    float* s_o    = reinterpret_cast<float*>(ring + (size_t)stages * TILE);                                      // [kWarps][group][HD]
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], meet_bar;
    __shared__ volatile int dead;
    __shared__ int s_last, s_first[kMaxSeqs + 1];                // runs of the sequences before; with one run each: the sequences, longest first
    __shared__ float s_m[kWarps][16], s_l[kWarps][16], s_f[16][kMaxRuns], s_i[16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    if (tid == 0) {
        for (int s = 0; s < stages; s++) mbar_init(&full[s], 1), mbar_init(&empty[s], 4);
        mbar_init(&meet_bar, kWarps);
        dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    kf_grid_launch_dependents();
    kf_grid_dependency_wait();  // queries, the rows of the current position, positions, workspace
    q = behind_wait(q), pos_dev = behind_wait(pos_dev);
    // the launch was sized from a hint: a sequence that needs them takes longer runs, so any length is covered; one without positions has one empty run, whose
    // result is what an empty softmax gives (0 / 0)
    auto shape = [&](int m, int& chunk, int& len) {
        len   = max(0, min(pos_dev[m] + 1, max_seq));
        chunk = max(min_chunk, ((len + max_runs - 1) / max_runs + kTok - 1) / kTok * kTok);
        return max(1, (len + chunk - 1) / chunk);
    };
    const bool whole = max_runs == 1, dealt = M <= (whole ? kMaxSeqs / 2 : kMaxSeqs);
    if (dealt && whole) {
        int* s_len = s_first + kMaxSeqs / 2;
        for (int m = tid; m < M; m += blockDim.x) s_len[m] = pos_dev[m];
        __syncthreads();
        for (int m = tid; m < M; m += blockDim.x) {
            const int len = s_len[m];
            int before = 0;
            for (int j = 0; j < M; j++) before += s_len[j] > len || (s_len[j] == len && j < m);
            s_first[before] = m;
        }
    } else if (dealt && warp == 0) {
        int sum = 0;
        for (int m0 = 0; m0 < M; m0 += 32) {
            int chunk, len, n = m0 + lane < M ? shape(m0 + lane, chunk, len) : 0, inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (m0 + lane < M) s_first[m0 + lane] = sum + inc - n;
            sum += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) s_first[M] = sum;
    }
    __syncthreads();
    const int n_items = (dealt && !whole ? s_first[M] : M * max_runs) * n_kv, grid = (int)gridDim.x;
    // a CTA's k-th item: there and back, so that with the longest first the one that took the longest of a pass takes the shortest of the next
    auto nth = [&](int k) { return k * grid + ((k & 1) ? grid - 1 - (int)blockIdx.x : (int)blockIdx.x); };
    // item -> (sequence, run, kv head); kv heads of one run next to each other: their rows lie side by side in memory.  false: no such run
    auto item_of = [&](int i, GqaItem& it) {
        it.kvh = i % n_kv;
        const int j = i / n_kv;
        int chunk, len;
        if (whole) {
            it.m = dealt ? s_first[j] : j, it.run = 0;
        } else if (dealt) {
            int lo = 0, hi = M - 1;  // the last sequence that starts at or before j
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_first[mid] <= j) lo = mid;
                else hi = mid - 1;
            }
            it.m = lo, it.run = j - s_first[lo];
        } else {
            it.m = j / max_runs, it.run = j % max_runs;
        }
        it.runs = shape(it.m, chunk, len);
        it.t0 = it.run * chunk, it.t1 = min(len, it.t0 + chunk);
        return it.run < it.runs;
    };
    uint32_t st = 0, ph = 0;  // ring position and its phase
    if (warp == kWarps) {
        if (bound.drop == (int)blockIdx.x + 1) return;
        bool live = true;
        uint32_t asked = 0;
        for (int k = 0; live && k * grid < n_items; k++) {
            GqaItem it;
            if (nth(k) >= n_items || !item_of(nth(k), it)) continue;
            for (int t = it.t0; live && t < it.t1; t += kTok)
                for (int kv = 0; kv < 2; kv++) {
                    if (!(live = mbar_wait_warp(smem_u32(&empty[st]), ph ^ 1, &dead, bound))) break;
                    if (lane == 0) {
                        mbar_arrive_expect_tx(&full[st], TILE);
#pragma unroll
                        for (int hf = 0; hf < HALVES; hf++)
                            tma_load_3d(ring + (size_t)st * TILE + hf * HALF, kv ? &tm_v : &tm_k, it.kvh * HD + hf * 64, t, it.m, &full[st]);
                    }
                    asked++;
                    if (++st == (uint32_t)stages) st = 0, ph ^= 1;
                }
        }
        if (!live)  // copies in flight write shared memory
            for (uint32_t k = asked > (uint32_t)stages ? asked - stages : 0; k < asked; k++) mbar_drain(smem_u32(&full[k % stages]), (k / stages) & 1, bound);
        return;
    }
    const int set = warp >> 2, w4 = warp & 3;
    const bool pairs = ((uintptr_t)out & 3) == 0;
    uint32_t mph = 0, done = 0;  // done: tiles of this CTA before the current item
    bool live = true;
    auto meet = [&]() {  // all computing warps; bounded like every wait
        __syncwarp();
        if (lane == 0) mbar_arrive(&meet_bar);
        live = mbar_wait_warp(smem_u32(&meet_bar), mph, &dead, bound) && live;
        mph ^= 1;
    };
    // 16-byte chunk c (0 .. HD / 8 - 1) of a row: half c / 8, chunk c % 8 swizzled by the row
    auto at = [](uint32_t base, int row, int c) { return base + (uint32_t)((c >> 3) * HALF + row * 128 + (((c & 7) ^ (row & 7)) << 4)); };
    for (int k = 0; live && k * grid < n_items; k++) {
        GqaItem it;
        if (nth(k) >= n_items || !item_of(nth(k), it)) continue;
        const int ntiles = (it.t1 - it.t0 + kTok - 1) / kTok;
        // the group's queries as A fragments: row r of 16 is head r (rows past the group are zero)
        uint32_t qa[HD / 16][4];
        const uint16_t* qb = q + ((size_t)it.m * n_head + (size_t)it.kvh * group) * HD;
#pragma unroll
        for (int kc = 0; kc < HD / 16; kc++) {
            const uint32_t* lo = reinterpret_cast<const uint32_t*>(qb + (size_t)g * HD + kc * 16 + 2 * t4);
            const uint32_t* hi = reinterpret_cast<const uint32_t*>(qb + (size_t)(g + 8) * HD + kc * 16 + 2 * t4);
            qa[kc][0] = g < group ? lo[0] : 0u, qa[kc][2] = g < group ? lo[4] : 0u;
            qa[kc][1] = g + 8 < group ? hi[0] : 0u, qa[kc][3] = g + 8 < group ? hi[4] : 0u;
        }
        float o[HD / 8][4];
#pragma unroll
        for (int j = 0; j < HD / 8; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
        float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;
        for (int kt = set; kt < ntiles; kt += SETS) {
            const uint32_t n = 2 * (done + kt);
            const uint32_t sk = n % stages, pk = (n / stages) & 1, sv = (n + 1) % stages, pv = ((n + 1) / stages) & 1;
            if (!(live = mbar_wait_warp(smem_u32(&full[sk]), pk, &dead, bound))) break;
            const uint32_t kb = smem_u32(ring + (size_t)sk * TILE), vb = smem_u32(ring + (size_t)sv * TILE);
            const int tok0 = it.t0 + kt * kTok + w4 * 16;  // this warp's 16 positions
            const bool mine = tok0 < it.t1;
            float sc[2][4];
#pragma unroll
            for (int j = 0; j < 2; j++) sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
            if (mine) {
#pragma unroll
                for (int kc = 0; kc < HD / 16; kc++) {
                    uint32_t b[4];
                    ldsm4(b, at(kb, w4 * 16 + (lane & 7) + (lane >> 4) * 8, kc * 2 + ((lane >> 3) & 1)));
                    mma16816(sc[0], qa[kc], b[0], b[1]);
                    mma16816(sc[1], qa[kc], b[2], b[3]);
                }
            }
            // a stage goes back when every ldmatrix of it has delivered: the matrix instructions behind them were issued with its registers
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[sk]);
            if (!(live = mbar_wait_warp(smem_u32(&full[sv]), pv, &dead, bound))) break;
            if (mine) {
                if (tok0 + 16 > it.t1) {  // the run's last positions: no weight, and no value that might not be a number
#pragma unroll
                    for (int j = 0; j < 2; j++)
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (tok0 + j * 8 + 2 * t4 + (e & 1) >= it.t1) sc[j][e] = -INFINITY;
                    const int r0 = it.t1 - tok0;
                    for (int c = lane; c < (16 - r0) * (HD / 8); c += 32) {
                        const int row = w4 * 16 + r0 + c / (HD / 8), ch = c % (HD / 8);
                        *reinterpret_cast<uint4*>(ring + (size_t)sv * TILE + (ch >> 3) * HALF + row * 128 + (ch & 7) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    // the stage is refilled by the asynchronous proxy later: these writes come before that
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
                float mx_lo = fmaxf(fmaxf(sc[0][0], sc[0][1]), fmaxf(sc[1][0], sc[1][1])), mx_hi = fmaxf(fmaxf(sc[0][2], sc[0][3]), fmaxf(sc[1][2], sc[1][3]));
                mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1)), mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
                mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1)), mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
                const float mn_lo = fmaxf(m_lo, mx_lo * sc2), mn_hi = fmaxf(m_hi, mx_hi * sc2);
                // where all scores so far are -inf their weights are 0, whichever positions a run starts with
                const float b_lo = mn_lo == -INFINITY ? 0.f : mn_lo, b_hi = mn_hi == -INFINITY ? 0.f : mn_hi;
                const float c_lo = exp2f(m_lo - b_lo), c_hi = exp2f(m_hi - b_hi);
                m_lo = mn_lo, m_hi = mn_hi;
                float rs_lo = 0.f, rs_hi = 0.f;
                uint32_t pa[4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const float p0 = exp2f(fmaf(sc[j][0], sc2, -b_lo)), p1 = exp2f(fmaf(sc[j][1], sc2, -b_lo));
                    const float p2 = exp2f(fmaf(sc[j][2], sc2, -b_hi)), p3 = exp2f(fmaf(sc[j][3], sc2, -b_hi));
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
                    ldsm4_t(b, at(vb, w4 * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, jp * 2 + (lane >> 4)));
                    mma16816(o[2 * jp], pa, b[0], b[1]);
                    mma16816(o[2 * jp + 1], pa, b[2], b[3]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[sv]);
        }
        done += (uint32_t)ntiles;
        if (!live) break;
        // ---- merge the warps (fixed order) through shared memory ----
        l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1), l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
        l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1), l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
#pragma unroll
        for (int j = 0; j < HD / 8; j++) {
            float* r0 = s_o + ((size_t)warp * group + g) * HD + j * 8 + 2 * t4;
            if (g < group) *reinterpret_cast<float2*>(r0) = make_float2(o[j][0], o[j][1]);
            if (g + 8 < group) *reinterpret_cast<float2*>(r0 + 8 * HD) = make_float2(o[j][2], o[j][3]);
        }
        if (t4 == 0) s_m[warp][g] = m_lo, s_m[warp][g + 8] = m_hi, s_l[warp][g] = l_lo, s_l[warp][g + 8] = l_hi;
        meet();
        if (!live) break;
        const size_t head0 = ((size_t)it.m * n_kv + it.kvh), part0 = head0 * max_runs * group;
        for (int idx = tid; idx < group * (HD / 4); idx += kComp) {
            const int r = idx / (HD / 4), c = idx % (HD / 4) * 4;
            float M_ = -INFINITY, L_ = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; w++) M_ = fmaxf(M_, s_m[w][r]);
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                const float f  = s_m[w][r] == -INFINITY ? 0.f : exp2f(s_m[w][r] - M_);
                const float4 v = *reinterpret_cast<const float4*>(s_o + ((size_t)w * group + r) * HD + c);
                L_ += s_l[w][r] * f;
                a.x = fmaf(v.x, f, a.x), a.y = fmaf(v.y, f, a.y), a.z = fmaf(v.z, f, a.z), a.w = fmaf(v.w, f, a.w);
            }
            if (it.runs == 1) {
                uint16_t* op = out + (head0 * group + r) * HD + c;
                put2(op, a.x / L_, a.y / L_, pairs), put2(op + 2, a.z / L_, a.w / L_, pairs);
            } else {
                __stcg(reinterpret_cast<float4*>(ws + (part0 + (size_t)it.run * group + r) * HD + c), a);
                if (c == 0) __stcg(ws_ml + part0 + (size_t)it.run * group + r, make_float2(M_, L_));
            }
        }
        if (it.runs > 1) {
            // ---- the last run of this (sequence, kv head) merges all of them in order ----
            __threadfence();
            meet();
            if (live && tid == 0) {
                unsigned* c = cnt + head0;
                s_last      = atomicAdd(c, 1u) == (unsigned)(it.runs - 1);
                if (s_last) *c = 0u;  // self-reset for the next launch
            }
            meet();
            if (live && s_last) {
                __threadfence();
                for (int r = warp; r < group; r += kWarps) {
                    float M_ = -INFINITY, L_ = 0.f;
                    float2 ml[kMaxRuns / 32];
#pragma unroll
                    for (int j = 0; j < kMaxRuns / 32; j++) {
                        const int s = j * 32 + lane;
                        ml[j] = s < it.runs ? __ldcg(ws_ml + part0 + (size_t)s * group + r) : make_float2(-INFINITY, 0.f);
                        M_    = fmaxf(M_, ml[j].x);
                    }
                    M_ = warp_max(M_);
#pragma unroll
                    for (int j = 0; j < kMaxRuns / 32; j++) {
                        const float f = exp2f(ml[j].x - M_);
                        L_ += ml[j].y * f;
                        s_f[r][j * 32 + lane] = f;
                    }
                    L_ = warp_sum(L_);
                    if (lane == 0) s_i[r] = 1.f / L_;
                }
                meet();
                // a slice of HD / 4 threads adds every kSlices-th run of a row, then the slices are added
                constexpr int VEC = HD / 4, kSlices = kComp / VEC;
                const int slice = tid / VEC, c = tid % VEC * 4;
                static_assert(kSlices <= 2 * kWarps, "slices fit the warps' area for half the heads at a time");
                const int per = HD == 128 ? group : (group + 1) / 2;  // rows at a time
                for (int r0 = 0; live && r0 < group; r0 += per) {
#pragma unroll 4
                    for (int r = r0; r < min(group, r0 + per); r++) {
                        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                        for (int s = slice; s < it.runs; s += kSlices) {
                            const float4 v = __ldcg(reinterpret_cast<const float4*>(ws + (part0 + (size_t)s * group + r) * HD + c));
                            const float f  = s_f[r][s];
                            a.x = fmaf(v.x, f, a.x), a.y = fmaf(v.y, f, a.y), a.z = fmaf(v.z, f, a.z), a.w = fmaf(v.w, f, a.w);
                        }
                        *reinterpret_cast<float4*>(s_o + ((size_t)slice * per + (r - r0)) * HD + c) = a;
                    }
                    meet();
                    for (int idx = tid; live && idx < min(per, group - r0) * (HD / 2); idx += kComp) {
                        const int r = idx / (HD / 2), d = idx % (HD / 2) * 2;
                        float a0 = 0.f, a1 = 0.f;
#pragma unroll
                        for (int sl = 0; sl < kSlices; sl++) {
                            const float2 v = *reinterpret_cast<const float2*>(s_o + ((size_t)sl * per + r) * HD + d);
                            a0 += v.x, a1 += v.y;
                        }
                        put2(out + (head0 * group + r0 + r) * HD + d, a0 * s_i[r0 + r], a1 * s_i[r0 + r], pairs);
                    }
                    if (r0 + per < group) meet();
                }
            }
        }
        meet();  // the area and the factors belong to the next item
    }
}

template <int HD, int SETS>
int gqa_launch(kf_ctx* ctx, void* out, const void* q, const void* kc, const void* vc, const int32_t* pos_dev, int M, int n_head, int n_kv, int max_seq, size_t seq_stride,
               int chunk, int runs) {
    const int group = n_head / n_kv;
    float* ws = nullptr;
    const size_t rows = (size_t)M * n_head * runs;
    if (runs > 1) {
        int rc = kf_ensure_attn_ws(ctx, rows * (HD + 2) * sizeof(float));
        if (!rc) rc = kf_ensure_attn_cnt(ctx, M * n_kv);
        if (rc) return rc;
        ws = ctx->attn_ws;
    }
    CUtensorMap tk, tv;
    const uint64_t stride = M > 1 ? (uint64_t)seq_stride * 2 : (uint64_t)n_kv * HD * 2;
    int rc = kf_tmap_rows(ctx, &tk, kc, (uint64_t)n_kv * HD, (uint64_t)max_seq, (uint64_t)M, stride, 64, kTok);
    if (!rc) rc = kf_tmap_rows(ctx, &tv, vc, (uint64_t)n_kv * HD, (uint64_t)max_seq, (uint64_t)M, stride, 64, kTok);
    if (rc) return rc;
    const int stages  = gqa_stages(HD, SETS, group);
    const size_t smem = (size_t)stages * kTok * HD * 2 + gqa_area(HD, SETS, group) + 1024;
    auto kern         = kf_attn_gqa_kernel<HD, SETS>;
    static bool set[kf_ctx::kMaxDevices] = {};  // function attributes are per device
    if (!set[ctx->device]) {
        KF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (SETS == 1 ? 98 : 201) * 1024));
        set[ctx->device] = true;
    }
    const long long items = (long long)M * runs * n_kv, slots = (long long)(3 - SETS) * ctx->sm_count;
    KF_CUDA(ctx, kf_launch_pdl(ctx, kern, dim3((unsigned)std::min(items, slots)), dim3((4 * SETS + 1) * 32), smem, tk, tv, (uint16_t*)out, ws,
                               reinterpret_cast<float2*>(ws ? ws + rows * HD : nullptr), ctx->attn_cnt, (const uint16_t*)q, pos_dev, M, n_head, n_kv, max_seq, chunk, runs, stages,
                               1.4426950408889634f / sqrtf((float)HD), KfBound{ctx->wait_flags + 1, (unsigned)ctx->attn_wait_us, ctx->attn_drop}));
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
template <int HD>
int gqa_any(kf_ctx* ctx, void* out, const void* q, const void* kc, const void* vc, const int32_t* pos_dev, int M, int n_head, int n_kv, int max_seq, int len,
            size_t seq_stride) {
    const int pairs = n_kv * M, sms = ctx->sm_count;
    const bool few  = pairs < sms;
    int chunk = 2 * kTok, runs = few ? sms / pairs : 1;
    // between a half and two thirds as many pairs as SMs: thirds make two passes over nearly all SMs, where whole ones leave a third or more of the SMs idle (12 ragged
    // sequences of 8 kv heads and 64 heads, norm and append in front: 58 against 65 us up to 6000 positions, 107 against 145 up to 16000; 49 against
    // 47 up to 4200 and 34 against 27 up to 2000, where the merges cost more).  From there on whole ones again (16 sequences: 56 against 71 us, 146 against 156)
    if (few && 2 * pairs > sms && 3 * pairs <= 2 * sms && len >= 5120) runs = 3;
    if (ctx->attn_split > 0) chunk = kTok, runs = ctx->attn_split;
    runs = std::max(1, std::min(runs, std::min(kMaxRuns, (len + chunk - 1) / chunk)));
    if (runs == 1) chunk = std::max(chunk, (max_seq + kTok - 1) / kTok * kTok);
    return few ? gqa_launch<HD, 2>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, seq_stride, chunk, runs)
               : gqa_launch<HD, 1>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, seq_stride, chunk, runs);
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
    const int rc = kf_wait_status(ctx);
    if (rc) return rc;
    const int len = std::max(1, std::min(max_seq, max_pos_hint + 1));
    if (hd == 128) return gqa_any<128>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, len, seq_stride);
    return gqa_any<64>(ctx, out, q, kc, vc, pos_dev, M, n_head, n_kv, max_seq, len, seq_stride);
}
// Ring stages of a launch: host arithmetic for the test of the protocol, no device
extern "C" int kf_attn_gqa_stages(int hd, int sets, int group) { return gqa_stages(hd, sets, group); }
