// sampler.cu -- temperature / top-k / top-p sampling ON THE DEVICE, one cluster of CTAs (or one CTA) per sequence: the step right after the logits
// (GeneratOnPrompt::Sample, reference src/Manifold/GoPT.cpp:614-630, with LogitsInfo::TopK :632-640, UpdateLogits :751-766, TopP :729-748,
// Qu_FlipCoin :768-786 and the xorshift64* generator :594-600).  The reference copies the [vocab] logits to the host every token and samples
// there; here only the 4-byte token leaves the GPU (or nothing at all inside the device-resident decode loop).
//
//   1. candidates  selection 0: the top_k largest logits, ties to the lower index (what TOPK_heap::Select is meant to do);
//                  selection 1: what TOPK_heap::Select (GoPT.cpp:667-700) actually keeps -- its std::priority_queue<int> orders INDICES, so
//                  the running "smallest kept" is always the newest index: indices 0 .. k-2 plus the first arg-max of the rest;
//                  both sorted by (logit descending, index ascending);
//   2. p_i = expf((l_i - l_max) / T), normalised by their sum in sorted order (sequential fp32, like the host loop);
//   3. top-p: keep the shortest prefix whose cumulative probability exceeds top_p;
//   4. coin = random_f32(state) * sum(kept p); first i with coin < cdf_i (else the last kept).
// The two running sums of steps 2-4 (of the exponentials, of the probabilities) are formed by one thread in the reference's order; exponentials, quotients and the
// search for the cut and the coin by one thread per candidate.  So the CPU port (oracle kfo_sample) and the kernel agree except where expf's last ulp moves
// a cdf boundary across the coin.
#include <math.h>

#include "kf_common.cuh"

namespace {
constexpr int kSampThreads = 1024;
constexpr int kMaxTopK     = 1024;

__device__ __forceinline__ uint32_t order_key(uint16_t b) {  // bf16 bits -> 16-bit key, increasing with the value (-0 < +0 adjacent: equal as floats
    return (b & 0x8000u) ? (uint32_t)(uint16_t)~b : (uint32_t)(b | 0x8000u);  // is handled by comparing floats wherever ties matter)
}
__device__ __forceinline__ uint32_t xorshift_u32(unsigned long long* s) {  // GoPT.cpp:594-599
    *s ^= *s >> 12;
    *s ^= *s << 25;
    *s ^= *s >> 27;
    return (uint32_t)((*s * 0x2545F4914F6CDD1Dull) >> 32);
}

// block-wide exclusive scan of one int per thread (1024 threads); returns the exclusive prefix, *total = the sum
__device__ int block_exscan(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += n;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = s_warp[lane], winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += n;
        }
        s_warp[lane] = winc - w;
        if (lane == 31) s_warp[32] = winc;
    }
    __syncthreads();
    *total = s_warp[32];
    return s_warp[warp] + inc - v;
}

// The top_k candidates of one row in (value descending, index ascending) order, by one CTA of kSampThreads threads: any vocabulary, any top_k up to
// kMaxTopK, both selections.
__device__ void select_any(float* s_val, int* s_idx, const uint16_t* __restrict__ row, int vocab, int top_k, int selection) {
    __shared__ int s_hist[256];
    __shared__ int s_warp[33];
    __shared__ int s_bin, s_above;
    const int tid       = threadIdx.x;
    const int chunk     = (vocab + kSampThreads - 1) / kSampThreads;  // contiguous indices per thread: tie ranks follow the index order
    const int i0 = tid * chunk, i1 = min(vocab, i0 + chunk);
    const int k  = top_k;

    if (selection == 1) {
        // the reference's heap as it behaves: indices 0 .. k-2, plus the first maximum over [k-1, vocab)
        float best = -INFINITY;
        int bi     = 0x7fffffff;
        for (int i = max(i0, k - 1); i < i1; i++) {
            const float v = bf16_bits_to_f32(row[i]);
            if (v > best) best = v, bi = i;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi   = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) best = ov, bi = oi;
        }
        __shared__ float s_bv[32];
        __shared__ int s_bi[32];
        if ((tid & 31) == 0) s_bv[tid >> 5] = best, s_bi[tid >> 5] = bi;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < 32; w++)
                if (s_bv[w] > best || (s_bv[w] == best && s_bi[w] < bi)) best = s_bv[w], bi = s_bi[w];
            s_val[k - 1] = best, s_idx[k - 1] = bi;
        }
        if (tid < k - 1) s_val[tid] = bf16_bits_to_f32(row[tid]), s_idx[tid] = tid;
    } else {
        // ---- radix select of the k-th largest 16-bit key: high byte, then low byte inside that bin ---------------------------------
        if (tid < 256) s_hist[tid] = 0;
        __syncthreads();
        for (int i = i0; i < i1; i++) atomicAdd(&s_hist[order_key(row[i]) >> 8], 1);
        __syncthreads();
        if (tid == 0) {
            int above = 0, b = 255;
            for (; b > 0 && above + s_hist[b] < k; b--) above += s_hist[b];
            s_bin = b, s_above = above;
        }
        __syncthreads();
        const int hb = s_bin;
        int above    = s_above;
        __syncthreads();
        if (tid < 256) s_hist[tid] = 0;
        __syncthreads();
        for (int i = i0; i < i1; i++) {
            const uint32_t key = order_key(row[i]);
            if ((int)(key >> 8) == hb) atomicAdd(&s_hist[key & 255u], 1);
        }
        __syncthreads();
        if (tid == 0) {
            int a = above, b = 255;
            for (; b > 0 && a + s_hist[b] < k; b--) a += s_hist[b];
            s_bin = b, s_above = a;
        }
        __syncthreads();
        const uint32_t thr = ((uint32_t)hb << 8) | (uint32_t)s_bin;  // the k-th largest key
        const int need     = k - s_above;                            // how many of the elements AT the threshold are kept: the lowest indices
        // ---- collect: everything above the threshold, and the first `need` at it (rank by index through a block scan) ---------------
        int n_above = 0, n_tie = 0;
        for (int i = i0; i < i1; i++) {
            const uint32_t key = order_key(row[i]);
            n_above += key > thr, n_tie += key == thr;
        }
        int tot_above, tot_tie;
        int off_above = block_exscan(n_above, s_warp, &tot_above);
        int off_tie   = block_exscan(n_tie, s_warp, &tot_tie);
        for (int i = i0; i < i1; i++) {
            const uint16_t b    = row[i];
            const uint32_t key = order_key(b);
            if (key > thr) {
                s_val[off_above] = bf16_bits_to_f32(b), s_idx[off_above] = i, off_above++;
            } else if (key == thr) {
                if (off_tie < need) s_val[tot_above + off_tie] = bf16_bits_to_f32(b), s_idx[tot_above + off_tie] = i;
                off_tie++;
            }
        }
    }
    for (int i = k + tid; i < kMaxTopK; i += kSampThreads) s_val[i] = -INFINITY, s_idx[i] = 0x7fffffff;
    __syncthreads();
    // ---- bitonic sort of the 1024 slots by (value descending, index ascending) --------------------------------------------------------
    for (int size = 2; size <= kMaxTopK; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const int j = tid ^ stride;
            if (j > tid) {
                const float va = s_val[tid], vb = s_val[j];
                const int ia = s_idx[tid], ib = s_idx[j];
                const bool a_first = va > vb || (va == vb && ia < ib);  // a belongs before b in the final order
                const bool desc    = (tid & size) == 0;
                if (desc ? !a_first : a_first) s_val[tid] = vb, s_val[j] = va, s_idx[tid] = ib, s_idx[j] = ia;
            }
            __syncthreads();
        }
}

// Softmax with temperature over the candidates, top-p, coin.  The host loop's order of operations: the two running sums are formed by one thread,
// entry after entry; what is independent per entry (exponential, quotient) by one thread each.  The cumulative probabilities of the top-p cut, the
// sum under the coin and the cdf are one and the same running sum.  Called by a whole CTA; s_val is overwritten.
__device__ void draw(int32_t* out, float* s_val, const int* s_idx, int k, float temperature, float top_p, unsigned long long* rng) {
    __shared__ float s_sum;
    __shared__ int s_last;
    const int tid  = threadIdx.x;
    const float mx = s_val[0];
    __syncthreads();
    if (tid < k) s_val[tid] = expf((s_val[tid] - mx) / temperature);
    if (tid == 0) s_last = k - 1;
    __syncthreads();
    if (tid == 0) {
        float sum = 0.f;
#pragma unroll 8
        for (int i = 0; i < k; i++) sum += s_val[i];
        s_sum = sum;
    }
    __syncthreads();
    if (tid < k) s_val[tid] /= s_sum;
    __syncthreads();
    if (tid == 0) {
        float cum = 0.f;
#pragma unroll 8
        for (int i = 0; i < k; i++) cum += s_val[i], s_val[i] = cum;
    }
    __syncthreads();
    if (top_p < 1.0f && tid < k && s_val[tid] > top_p) atomicMin(&s_last, tid);
    __syncthreads();
    const int last = s_last;
    __syncthreads();
    unsigned long long st = *rng;
    const float coin      = (float)(xorshift_u32(&st) >> 8) / 16777216.0f * s_val[last];
    if (tid < last && coin < s_val[tid]) atomicMin(&s_last, tid);
    __syncthreads();
    if (tid == 0) *rng = st, *out = s_idx[s_last];
}

__global__ void __launch_bounds__(kSampThreads) kf_sample_kernel(int32_t* __restrict__ out, const uint16_t* __restrict__ logits, int vocab, float temperature,
                                                                 int top_k, float top_p, unsigned long long* __restrict__ rng, int selection) {
    __shared__ float s_val[kMaxTopK];
    __shared__ int s_idx[kMaxTopK];
    select_any(s_val, s_idx, logits + (size_t)blockIdx.x * vocab, vocab, top_k, selection);
    draw(out + blockIdx.x, s_val, s_idx, top_k, temperature, top_p, rng + blockIdx.x);
}

// ---- up to kFastTopK candidates: ONE pass over the logits, held in registers by a cluster of CTAs per row --------------------------------------------
// The single CTA above reads its row three times with 2-byte loads and sorts 1024 slots: 148 us at 8 rows of 151936 (a row is 304 KB: 0.4 us at the HBM
// rate for all eight), all latency.  Here the row is spread over up to 8 CTAs, 24 logits per thread, loaded once.  The k-th largest of a CTA's
// per-thread maxima bounds the k-th largest logit of the row from below (k threads hold one at least as large), so only what reaches the largest of
// these bounds -- a few hundred logits -- is collected, and the first CTA finds the exact k-th key among them, ranks the survivors by counting and
// draws: 152 -> 21.5 us a call.  Rows that leave too many (long runs of equal logits) or that hold NaN among the chosen take the general selection.
constexpr int kFastTopK = 256, kFastPer = 24, kFastCtas = 8, kFastLocal = 2048, kFastTotal = 4096;

// the largest t that the keys of at least k threads of the CTA reach (k <= 1024; 0: fewer than k hold a key).  Bisects between the smallest and the largest key: the
// maxima of 24 logits each lie close together, so about nine of the 17 rounds over all bits are left, each a block barrier (8 rows of 151936, with the second search
// below: 20.6 -> 18.4 us a call)
__device__ __forceinline__ uint32_t kth_bound(uint32_t key, int k, uint32_t* s_range) {
    const uint32_t mn = __reduce_min_sync(0xffffffffu, key), mx = __reduce_max_sync(0xffffffffu, key);
    if ((threadIdx.x & 31) == 0) atomicMin(&s_range[0], mn), atomicMax(&s_range[1], mx);
    __syncthreads();
    uint32_t lo = s_range[0], hi = s_range[1];
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__syncthreads_count(key >= mid) >= k) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(const void* local_ptr, int cta_rank) {
    uint32_t remote, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(local_ptr)), "r"(cta_rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
    return v;
}

template <bool VEC>
__global__ void __launch_bounds__(kSampThreads) kf_sample_cluster_kernel(int32_t* __restrict__ out, const uint16_t* __restrict__ logits, int vocab, float temperature,
                                                                         int k, float top_p, unsigned long long* __restrict__ rng, int ctas) {
    __shared__ uint32_t s_key[kFastLocal], s_at[kFastLocal];  // this CTA's candidates: key (1 .. 65536), index
    __shared__ uint32_t s_bound, s_n;
    __shared__ uint32_t g_key[kFastTotal];                    // first CTA: the candidates of all
    __shared__ float s_val[kMaxTopK];
    __shared__ int s_idx[kMaxTopK];
    __shared__ uint32_t s_cnt[20];
    __shared__ int s_above, s_ties, s_nan;
    __shared__ uint32_t s_range[3];  // smallest and largest of the threads' maxima, largest candidate
    const int tid = threadIdx.x, rank = blockIdx.x % ctas;
    const uint16_t* row = logits + (size_t)(blockIdx.x / ctas) * vocab;
    if (tid == 0) s_range[0] = 0xffffffffu, s_range[1] = s_range[2] = 0;
    __syncthreads();
    // ---- the one pass: keys in registers, one each; 0 marks what lies past the end ----
    uint32_t kk[kFastPer];
#pragma unroll
    for (int j = 0; j < kFastPer; j++) kk[j] = 0;
    if (VEC) {
#pragma unroll
        for (int j = 0; j < kFastPer / 8; j++) {
            const int i = ((j * ctas + rank) * kSampThreads + tid) * 8;
            if (i < vocab) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + i));
                const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++) kk[8 * j + 2 * e] = order_key((uint16_t)q[e]) + 1, kk[8 * j + 2 * e + 1] = order_key((uint16_t)(q[e] >> 16)) + 1;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < kFastPer; j++) {
            const int i = (j * ctas + rank) * kSampThreads + tid;
            if (i < vocab) kk[j] = order_key(__ldg(row + i)) + 1;
        }
    }
    uint32_t mx = 0;
#pragma unroll
    for (int j = 0; j < kFastPer; j++) mx = max(mx, kk[j]);
    uint32_t bound = max(kth_bound(mx, k, s_range), 1u);
    if (tid == 0) s_bound = bound, s_n = 0;
    if (tid < 20) s_cnt[tid] = 0;
    __syncthreads();
    if (ctas > 1) {
        cluster_arrive();
        cluster_wait();
        for (int c = 0; c < ctas; c++) bound = max(bound, ld_cluster_u32(&s_bound, c));
    }
    // ---- what reaches the bound ----
    if (mx >= bound) {
#pragma unroll
        for (int j = 0; j < kFastPer; j++)
            if (kk[j] >= bound) {
                const uint32_t at = atomicAdd(&s_n, 1u);
                const int i = VEC ? (((j / 8) * ctas + rank) * kSampThreads + tid) * 8 + (j & 7) : (j * ctas + rank) * kSampThreads + tid;
                if (at < (uint32_t)kFastLocal) s_key[at] = kk[j], s_at[at] = (uint32_t)i;
            }
    }
    __syncthreads();
    if (ctas > 1) {
        cluster_arrive();
        cluster_wait();
    }
    if (rank == 0) {
        // ---- gather: thread t holds candidates t, t + 1024, .. of the concatenated lists ----
        constexpr int PER = kFastTotal / kSampThreads;
        uint32_t start[kFastCtas + 1];
        start[0] = 0;
        bool fits = true;
        for (int c = 0; c < kFastCtas; c++) {
            const uint32_t n = c < ctas ? (c ? ld_cluster_u32(&s_n, c) : s_n) : 0u;
            fits = fits && n <= (uint32_t)kFastLocal;
            start[c + 1] = start[c] + n;
        }
        const uint32_t total = start[kFastCtas];
        fits = fits && total <= (uint32_t)kFastTotal;
        uint32_t ck[PER], ci[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const uint32_t t = (uint32_t)(j * kSampThreads + tid);
            ck[j] = 0, ci[j] = 0;
            if (fits && t < total) {
                int c = 0;
#pragma unroll
                for (int u = 1; u < kFastCtas; u++) c += t >= start[u];
                uint32_t o = t;
#pragma unroll
                for (int u = 1; u < kFastCtas; u++)
                    if (c == u) o = t - start[u];
                ck[j] = ld_cluster_u32(&s_key[o], c), ci[j] = ld_cluster_u32(&s_at[o], c);
            }
        }
        if (tid == 0) s_above = 0, s_ties = 0, s_nan = 0;
        __syncthreads();
        if (fits) {
            // ---- the k-th largest key: the bound, which at least k candidates reach, or above it ----
            uint32_t top = 0;
#pragma unroll
            for (int j = 0; j < PER; j++) top = max(top, ck[j]);
            top = __reduce_max_sync(0xffffffffu, top);
            if ((tid & 31) == 0) atomicMax(&s_range[2], top);
            __syncthreads();
            uint32_t thr = bound, hi = s_range[2];
            for (int b = 0; thr < hi; b++) {  // at most 17 rounds: a counter each
                const uint32_t cand = (thr + hi + 1) >> 1;
                int n = 0;
#pragma unroll
                for (int j = 0; j < PER; j++) n += ck[j] >= cand;
                n = __reduce_add_sync(0xffffffffu, n);
                if ((tid & 31) == 0 && n) atomicAdd(&s_cnt[b], (uint32_t)n);
                __syncthreads();
                if (s_cnt[b] >= (uint32_t)k) thr = cand;
                else hi = cand - 1;
            }
            // ---- everything above it (fewer than k), and the entries at it with the lowest indices ----
            uint32_t* a_key = s_key;  // the local lists have been read
            uint32_t* a_at  = s_at;
            __syncthreads();
#pragma unroll
            for (int j = 0; j < PER; j++) {
                if (ck[j] > thr) {
                    const int at = atomicAdd(&s_above, 1);
                    a_key[at] = ck[j], a_at[at] = ci[j];
                } else if (ck[j] == thr && ck[j]) {
                    g_key[atomicAdd(&s_ties, 1)] = ci[j];
                }
            }
            __syncthreads();
            const int above = s_above, ties = s_ties;
            for (int i = tid; i < ties; i += kSampThreads) {
                const uint32_t me = g_key[i];
                int before = 0;
                for (int j = 0; j < ties; j++) before += g_key[j] < me;
                if (above + before < k) a_key[above + before] = thr, a_at[above + before] = me;
            }
            __syncthreads();
            // ---- order by (value descending, index ascending): the two zeros are one value ----
            if (tid < k) {
                const uint32_t zero = 0x8001u, me = a_key[tid] == zero - 1 ? zero : a_key[tid], at = a_at[tid];
                const uint32_t raw = a_key[tid] - 1;
                int before = 0;
                for (int j = 0; j < k; j++) {
                    const uint32_t o = a_key[j] == zero - 1 ? zero : a_key[j];
                    before += o > me || (o == me && a_at[j] < at);
                }
                const float v = bf16_bits_to_f32((uint16_t)((raw & 0x8000u) ? (raw & 0x7fffu) : ~raw));
                if (v != v) s_nan = 1;
                s_val[before] = v, s_idx[before] = (int)at;
            }
            __syncthreads();
            fits = !s_nan;
        }
        if (!fits) {
            __syncthreads();
            select_any(s_val, s_idx, row, vocab, k, 0);
        }
        draw(out + blockIdx.x / ctas, s_val, s_idx, k, temperature, top_p, rng + blockIdx.x / ctas);
    }
    if (ctas > 1) {  // the lists of the other CTAs stay until the first one has read them
        cluster_arrive();
        cluster_wait();
    }
}
}  // namespace

// next[m] = a token drawn from row m of the logits; rng_state_dev: one 64-bit xorshift64* state per row (seeded by the caller, advanced here).
// temperature == 0 or top_k == 1: greedy (kf_argmax).  selection: 0 = true top-k, 1 = the reference's TOPK_heap::Select as it behaves.
extern "C" int kf_sample(kf_ctx* ctx, int32_t* next_dev, const void* logits_bf16_dev, int M, int vocab, float temperature, int top_k, float top_p,
                         uint64_t* rng_state_dev, int selection) {
    if (!ctx || !next_dev || !logits_bf16_dev) return KF_ERR_BAD_ARG;
    KF_REQUIRE(ctx, M >= 1 && vocab >= 2, "shape");
    if (temperature == 0.0f || top_k == 1) return kf_argmax(ctx, next_dev, logits_bf16_dev, M, vocab);
    KF_REQUIRE(ctx, rng_state_dev, "sampling needs the generator state");
    KF_REQUIRE(ctx, temperature > 0.0f && top_p > 0.0f && (selection == 0 || selection == 1), "temperature > 0, top_p > 0");
    if (top_k <= 0 || top_k > vocab) top_k = vocab;  // CHAT_SAMPLER: nCanTopK = min(top_k, n_vocab), GoPT.cpp:389
    KF_REQUIRE(ctx, top_k <= kMaxTopK && top_k < vocab / 2, "top_k <= 1024 candidates (and < vocab / 2, TOPK_heap::Select's own assert)");
    if (selection == 0 && top_k <= kFastTopK && vocab <= kFastCtas * kSampThreads * kFastPer) {
        // as few CTAs per row as hold 16 logits per thread: small rows in one CTA (no cluster barriers), Qwen3's 151936 in eight
        int ctas = 1;
        while (ctas < kFastCtas && vocab > ctas * kSampThreads * 16) ctas *= 2;
        const bool vec = vocab % 8 == 0 && ((uintptr_t)logits_bf16_dev & 15) == 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)M * ctas), cfg.blockDim = dim3(kSampThreads), cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id               = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ctas, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr, cfg.numAttrs = ctas > 1 ? 1 : 0;
        KF_CUDA(ctx, cudaLaunchKernelEx(&cfg, vec ? kf_sample_cluster_kernel<true> : kf_sample_cluster_kernel<false>, (int32_t*)next_dev, (const uint16_t*)logits_bf16_dev, vocab,
                                        temperature, top_k, top_p, (unsigned long long*)rng_state_dev, ctas));
        KF_LAUNCH_CHECK(ctx);
        return KF_OK;
    }
    kf_sample_kernel<<<M, kSampThreads, 0, ctx->stream>>>(next_dev, (const uint16_t*)logits_bf16_dev, vocab, temperature, top_k, top_p,
                                                          (unsigned long long*)rng_state_dev, selection);
    KF_LAUNCH_CHECK(ctx);
    return KF_OK;
}
