// Next-token sampling on the device, one thread-block cluster per row of logits.
//
// Order of operations is the reference sampler's (core/src/sampling.cpp:11-118):
//   repetition penalty on previously generated tokens (positive logit / penalty, else
//   * penalty, once per occurrence) -> temperature == 0: first maximum -> logits / T ->
//   top-k (others dropped) -> top-p (smallest set of most probable tokens whose mass
//   exceeds p) -> softmax over what is left -> the first index whose cumulative
//   probability reaches the uniform draw u.
// The reference sorts on the host.  Here nothing is sorted and nothing leaves the device.  Ties at the
// k-th value are all kept.  The uniform draw comes from the caller (a counter-based generator
// keyed by the request's seed and its count of generated tokens), which makes a request's
// tokens independent of what else is in the batch.
//
// What bounds it is the latency of a row's chain (walks, meetings of its blocks, cuts), then the instructions of a walk (a
// division and an exponential a value where they are needed).  A row is shared out over the blocks of a cluster in
// stretches of 512 or 1,024 values, a warp each.  The first walk only looks for the maximum and, where there is a
// k, for the largest few lanes' maxima of each stretch: the k-th largest of those is a value that at least k values
// reach, and seldom many more.  Those few are collected, and one block makes both cuts and the draw among them.  A cut
// by mass alone takes a histogram over the values near the maximum, linear in the distance to it, that the blocks
// add up through distributed shared memory: a value adds its part of the bucket's upper end, as a count and a whole
// number of its exponential's last places, in 32-bit (64-bit additions in shared memory are loops of compare and swap: 183 us for 128
// rows that made them for all values), and the values of the one bucket the cut falls into are picked among by counting.
// A larger k takes a histogram of counts over the whole row first; a bucket with more than kList values (rows
// whose values are all but equal, or with outliers that stretch the range) is bisected instead, on the order-preserving
// integer image of the floats, as many as 32 walks.  Few rows leave their values, divided, in shared memory for the walks
// behind the first; of many, walks after the first find the logits in L2, so that twice as many blocks fit an SM.
// 128 rows of 128,256 logits (greedy, temperature, top-k, top-p and both in turn): 1,425 us with one block a row and
// bisection throughout, 100 us with every row's slices in shared memory and a histogram for each cut, 76 us so; 8 rows
// 28 and 26 us, with top-k 20 and 12.
//
// Probabilities are exp(x - max) in 32-bit.  A lane adds its few dozen of a stretch in 32-bit, everything beyond is added in
// 64-bit in a fixed order or, where it arrives in any order, as integers (exp * 2^44, so that even a tail of values below 1e-9
// counts): the same token every time.  No sum depends on how many blocks share a row, so that how many rows are sampled
// beside it changes nothing either.
//
// `work` is scratch of the same shape as the logits, used only for rows with a penalty whose slice does not fit
// shared memory (lsb_sample_needs_work).
#include "common.cuh"

#include <cooperative_groups.h>
#include <float.h>

#include <type_traits>
#include <utility>

namespace cg = cooperative_groups;

LSB_DEFINE_STATUS()

typedef unsigned long long u64;

constexpr int kMaxBlocks = 8;                 // blocks of a row's cluster (the portable size)
constexpr int kSliceTarget = 8192;            // logits a block takes before another one joins the cluster
constexpr int kStretch = 512;                 // values a warp takes at a time: four pieces of four a lane
constexpr int kMaxStretches = 128;            // of a row (longer rows have longer ones)
constexpr int kBuckets = 1024;                // of the histogram
constexpr int kList = 1024;                   // values of one bucket that are picked among directly
constexpr int kWhole = 512;                   // values up to the k-th that are, all of them
constexpr int kFewK = 128;                    // a k whose values the stretches' maxima lead to
constexpr int kTops = 8;                      // most of a stretch's lanes' maxima that are looked at
constexpr int kPool = 2 * kFewK + kMaxStretches;              // ... of all stretches together
constexpr float kNear = 10.f;                 // how far below the maximum the histogram of masses goes at first
constexpr float kStep = kNear / (kBuckets - 1);               // ... a bucket's
constexpr float kRestScale = 16777216.f;      // 2^24, places of what a value lacks to the upper end of its bucket
constexpr double kMostRest = 0.01;            // ... more than any lacks (1 - e^(-kNear / 1023))
constexpr int kSliceBytes = 176 * 1024;       // most shared memory for a slice

__device__ __forceinline__ unsigned int ordered(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(unsigned int o) {
    return __uint_as_float((o & 0x80000000u) ? o & 0x7fffffffu : ~o);
}

// (value, index) maximum with the lowest index winning ties
__device__ __forceinline__ void argmax_merge(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

template <int THREADS>
struct Shared {
    static constexpr int kWarps = THREADS / 32;
    float mx;                                 // a block's maximum, and the first place of it
    int mi;
    double slot[2];                           // a block's count or mass, by turns
    u64 tail;                                 // ... its mass beyond the histogram
    u64 scratch[kWarps];
    double scratch_d[kWarps];
    float scratch_f[kWarps];
    int scratch_i[kWarps];
    double seg[kMaxStretches];                // kept mass of this block's stretches
    double all_seg[kMaxStretches];            // ... of the row's
    float pool[kPool], all_pool[kPool];       // largest lanes' maxima of this block's stretches, of the row's
    unsigned int cnt[kBuckets];               // this block's histogram
    union {
        u64 mass[kBuckets];
        unsigned int rest[2 * kBuckets];      // what the counted values' masses lack to the upper end of their bucket (behind those: odd lanes')
        u64 list_mass[kList];
    };
    unsigned int tot_cnt[kBuckets];           // the row's, the same in every block
    union {
        u64 tot_mass[kBuckets];
        int list_at[kList];                   // places of the list's values (the largest few of a row)
    };
    float list[kList];                        // (of the cluster's first block) values of one bucket
    unsigned int list_n;
    unsigned int thr_k, thr_p;                // the first block's work on the two cuts
    unsigned int cut, cut_mass;               // ... and what it tells the others
    int token;
    int found;                                // bucket picked by find_bucket, and what stands before it
    u64 before;
};

__device__ __forceinline__ u64 warp_sum(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int THREADS>
__device__ __forceinline__ u64 block_sum(u64 v, Shared<THREADS>& s) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s.scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    u64 t = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) t += s.scratch[w];
    return t;
}
template <int THREADS>
__device__ __forceinline__ double block_sum(double v, Shared<THREADS>& s) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s.scratch_d[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) t += s.scratch_d[w];
    return t;
}

// The first bucket at which the running sum of val(b) is ok, once total(sum of all) has been called; every thread gets it
// (kBuckets: none) together with the sum before it.
template <int THREADS, typename Val, typename Total, typename Ok>
__device__ __forceinline__ int find_bucket(Shared<THREADS>& s, u64& before, Val val, Total total, Ok ok) {
    constexpr int kPer = kBuckets / THREADS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    u64 own = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) own += val(kPer * tid + i);
    u64 run = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    __syncthreads();
    if (lane == 31) s.scratch[warp] = run;
    if (tid == 0) { s.found = kBuckets; s.before = 0; }
    __syncthreads();
    u64 base = run - own, all = 0ull;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        if (w == warp) base += all;
        all += s.scratch[w];
    }
    total(all);
    // (the condition turns true once along the buckets: exactly one thread finds the turn)
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const u64 end = base + val(kPer * tid + i);
        if (!ok(base) && ok(end)) { s.found = kPer * tid + i; s.before = base; }
        base = end;
    }
    __syncthreads();
    before = s.before;
    return s.found;
}

// params per row: {temperature, top_p, repetition_penalty, u}.  stretch: values of a stretch; slice: of a block, whole stretches.
// PARKED: the first walk leaves the row's values, penalties applied, in shared memory (`work` where a slice does not fit) for
// the walks behind it; otherwise they are read, and divided by the temperature, again.
template <int THREADS, bool PARKED, int PER_SM>
__global__ void __launch_bounds__(THREADS, PER_SM)
sample_kernel(const float* __restrict__ logits, float* __restrict__ work, int vocab, int stretch, int slice, int slice_in_smem,
              float mass_scale, int near, const float* __restrict__ params, const int* __restrict__ top_ks,
              const int* __restrict__ prev_start, const int* __restrict__ prev_tokens, int* __restrict__ out) {
    constexpr int kWarps = THREADS / 32;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ Shared<THREADS> s;
    cg::cluster_group cluster = cg::this_cluster();
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int blocks = (int)gridDim.z, rank = (int)blockIdx.z;
    const float temperature = params[row * 4 + 0], top_p = params[row * 4 + 1];
    const float penalty = params[row * 4 + 2], u = params[row * 4 + 3];
    const int top_k = top_ks[row];
    const int i0 = min(vocab, rank * slice), n = min(vocab, i0 + slice) - i0;      // this block's slice
    const float* src = logits + (size_t)row * vocab + i0;
    const bool greedy = temperature == 0.0f;
    const bool cut_k = !greedy && top_k > 0 && top_k < vocab, cut_p = !greedy && top_p < 1.0f;
    const float* xs = src;                                    // what the walks read
    float by = temperature;                                   // ... and divide by
    float* put = nullptr;
    bool park = PARKED && !greedy;                            // by the first walk
    if constexpr (PARKED) {
        put = slice_in_smem ? reinterpret_cast<float*>(dyn) : work + (size_t)row * vocab + i0;
        const int pb = prev_start ? prev_start[row] : 0, pe = prev_start ? prev_start[row + 1] : 0;
        if (penalty != 1.0f && pe > pb) {
            for (int i = tid; i < n; i += THREADS) put[i] = src[i];
            __syncthreads();
            for (int j = pb; j < pe; ++j) {                   // in order; a token is one thread's alone
                const int t = prev_tokens[j] - i0;
                if (t >= 0 && t < n && t % THREADS == tid) put[t] = put[t] > 0.f ? put[t] / penalty : put[t] * penalty;
            }
            if (!greedy)
                for (int i = tid; i < n; i += THREADS) put[i] = put[i] / temperature;
            __syncthreads();
            xs = put;
            by = 1.f;
            park = false;
        }
    }
    const int stretches = (n + stretch - 1) / stretch;        // of this block
    const int row_stretches = (vocab + stretch - 1) / stretch, per_block = slice / stretch;
    const bool fours = ((reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(put)) & 15) == 0;
    // f(first place, values, how many of the four there are) for this lane's pieces of a stretch
    auto fetch = [&](int i, int end, float (&v)[4]) {
        if (fours && i + 3 < end) {
            const float4 x = *reinterpret_cast<const float4*>(xs + i);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = i + e < end ? xs[i + e] : 0.f;
        }
    };
    auto walk = [&](int st, auto f) {
        const int end = min(n, (st + 1) * stretch);
        for (int p0 = st * stretch; p0 < end; p0 += kStretch) {
            float v[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) fetch(p0 + (k * 32 + lane) * 4, end, v[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = p0 + (k * 32 + lane) * 4;
                if (i < end) f(i, v[k], min(4, end - i));
            }
        }
    };

    // f of what lies at a place of every block's shared memory, blocks in order (all asked for at once)
    auto of_blocks = [&](const auto* at, auto f) {
        std::remove_cv_t<std::remove_reference_t<decltype(*at)>> got[kMaxBlocks];
#pragma unroll
        for (int r = 0; r < kMaxBlocks; ++r)
            if (r < blocks) got[r] = *cluster.map_shared_rank(at, r);
#pragma unroll
        for (int r = 0; r < kMaxBlocks; ++r)
            if (r < blocks) f(got[r]);
    };

    // ---- greedy: the first maximum
    if (greedy) {
        float mx = -FLT_MAX;
        int mi = 0x7fffffff;
        for (int st = warp; st < stretches; st += kWarps)
            walk(st, [&](int i, const float (&v)[4], int m) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < m) argmax_merge(mx, mi, v[e], i0 + i + e);
            });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            argmax_merge(mx, mi, __shfl_xor_sync(0xffffffffu, mx, o), __shfl_xor_sync(0xffffffffu, mi, o));
        if (lane == 0) { s.scratch_f[warp] = mx; s.scratch_i[warp] = mi; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kWarps; ++w) argmax_merge(mx, mi, s.scratch_f[w], s.scratch_i[w]);
            s.mx = mx;
            s.mi = mi;
        }
        cluster.sync();
        if (rank == 0 && tid == 0) {
            for (int r = 1; r < blocks; ++r) argmax_merge(mx, mi, *cluster.map_shared_rank(&s.mx, r), *cluster.map_shared_rank(&s.mi, r));
            out[row] = mi < vocab ? mi : 0;                   // (nothing but -infinities and NaN: the first token)
        }
        cluster.sync();                                       // (the first block may still read this block's)
        return;
    }

    // ---- the row's maximum; each stretch's `tops` largest lanes' maxima
    const bool upright = by > 0.f;                            // (division keeps the values' order)
    const int tops = cut_k && upright && top_k <= kFewK ? (2 * top_k + row_stretches - 1) / row_stretches : 0;
    const bool few = tops > 0 && tops <= kTops && by >= 1e-10f && by <= 1e10f;
    float mx = -INFINITY;
    for (int st = warp; st < stretches; st += kWarps) {
        float own = -INFINITY;
        auto see = [&](int i, const float (&w)[4], int m) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e < m) own = fmaxf(own, w[e]);
            if (!park) return;
            if (fours && m == 4) *reinterpret_cast<float4*>(put + i) = make_float4(w[0], w[1], w[2], w[3]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < m) put[i + e] = w[e];
        };
        // (what is parked is divided already, unless a bound on the values themselves is all that follows)
        if (upright && (few || !park)) walk(st, see);
        else
            walk(st, [&](int i, const float (&v)[4], int m) {
                const float w[4] = {v[0] / by, v[1] / by, v[2] / by, v[3] / by};
                see(i, w, m);
            });
        mx = fmaxf(mx, own);
        if (few) {
            unsigned int left = ordered(own);
            for (int j = 0; j < tops; ++j) {
                const unsigned int top = __reduce_max_sync(0xffffffffu, left);
                if (lane == __ffs(__ballot_sync(0xffffffffu, left == top)) - 1) left = 0u;
                if (lane == 0) s.pool[st * tops + j] = from_ordered(top);
            }
        }
    }
    mx = lsb_warp_max(mx);
    if (lane == 0) s.scratch_f[warp] = mx;
    if (tid == 0) s.list_n = 0u;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kWarps; ++w) mx = fmaxf(mx, s.scratch_f[w]);
        s.mx = mx;
    }
    cluster.sync();
    mx = -INFINITY;
    of_blocks(&s.mx, [&](float x) { mx = fmaxf(mx, x); });
    const float most_raw = mx;
    if (upright && (few || !park)) mx = mx / by;
    mx = fmaxf(mx, -FLT_MAX);                                 // (nothing but -infinities and NaN)
    if (park) {                                               // (every lane comes back to the places it has written)
        xs = put;
        if (!few) by = 1.f;
    }

    // exp(x - max), as a number and as an integer; a value that is not a number counts nothing
    auto weight_of = [&](float x) -> float {
        const float e = expf(x - mx);
        return e > 0.f ? e : 0.f;
    };
    auto mass_of = [&](float x) -> u64 { return __float2ull_rn(weight_of(x) * mass_scale); };
    // (first block) the r-th largest of the list's m values; none so large: nothing is cut
    auto pick_kth = [&](int m, u64 r) -> unsigned int {
        if (tid == 0) s.thr_k = 0u;
        __syncthreads();
        for (int i = tid; i < m; i += THREADS) {
            const unsigned int o = ordered(s.list[i]);
            int above = 0, same = 0;
            for (int j = 0; j < m; ++j) {
                const unsigned int oj = ordered(s.list[j]);
                above += oj > o;
                same += oj == o;
            }
            if ((u64)above < r && r <= (u64)(above + same)) s.thr_k = o;      // (equal values write the same)
        }
        __syncthreads();
        return s.thr_k;
    };
    // (first block) the smallest of the list's values >= least before which there is no more mass than `most`;
    // list_mass is there, `before` is the mass of larger values that are not in the list
    auto pick_mass = [&](int m, unsigned int least, u64 before, double most) -> unsigned int {
        if (tid == 0) s.thr_p = ordered(mx);
        __syncthreads();
        for (int i = tid; i < m; i += THREADS) {
            const unsigned int o = ordered(s.list[i]);
            if (o < least) continue;
            u64 above = before;
            for (int j = 0; j < m; ++j)
                if (ordered(s.list[j]) > o) above += s.list_mass[j];
            if ((double)above <= most) atomicMin(&s.thr_p, o);
        }
        __syncthreads();
        return s.thr_p;
    };

    // ---- few values up to the k-th: both cuts and the draw among those that reach a bound at least k values reach
    if (few) {
        // (for a k far below the number of stretches several of them are one: no more than some four k values are compared)
        const int join = max(1, row_stretches / (2 * top_k)), pool = join > 1 ? (row_stretches + join - 1) / join : row_stretches * tops;
        for (int i = tid; i < pool; i += THREADS) {
            float top = -INFINITY;
            for (int j = i * join; j < min((i + 1) * join, row_stretches * tops); ++j) {
                const int st = j / tops, r = st / per_block;
                top = fmaxf(top, *cluster.map_shared_rank(&s.pool[(st - r * per_block) * tops + j % tops], r));
            }
            s.all_pool[i] = top;
        }
        if (tid == 0) s.thr_k = 0u;
        __syncthreads();
        for (int i = tid; i < pool; i += THREADS) {
            const float x = s.all_pool[i];
            int above = 0, same = 0;
            for (int j = 0; j < pool; ++j) {
                above += s.all_pool[j] > x;
                same += s.all_pool[j] == x;
            }
            if (above < top_k && top_k <= above + same) s.thr_k = ordered(x);
        }
        __syncthreads();
        const float bound = from_ordered(s.thr_k);            // (-infinity: every value is taken)
        const bool none = bound == -INFINITY;
        // A quotient that equals the k-th largest one ties with it: the bound is lowered by more than the roundings of
        // a division, as long as nothing is so small or so large that they are not relative.
        if (fabsf(most_raw) <= 1e25f && (none || (fabsf(bound) >= 1e-25f && fabsf(bound) <= 1e25f))) {
            const float low = none ? -FLT_MAX : bound - fabsf(bound) * 0x1p-21f;
            unsigned int* count = cluster.map_shared_rank(&s.list_n, 0);
            float* list = cluster.map_shared_rank(&s.list[0], 0);
            int* list_at = cluster.map_shared_rank(&s.list_at[0], 0);
            for (int st = warp; st < stretches; st += kWarps)
                walk(st, [&](int i, const float (&v)[4], int m) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (e < m && v[e] >= low) {
                            const unsigned int at = atomicAdd(count, 1u);
                            if (at < (unsigned int)kList) { list[at] = v[e] / by; list_at[at] = i0 + i + e; }
                        }
                });
            cluster.sync();
            const unsigned int listed = *count;
            if (listed <= (unsigned int)kList) {
                cluster.sync();                               // (the others have read the count and are done)
                if (rank != 0) return;
                const int m = (int)listed;
                if (tid == 0) { s.token = 0x7fffffff; s.found = -1; }
                const unsigned int t = pick_kth(m, (u64)top_k);
                auto total = [&](unsigned int least) {        // masses of what is kept, and their sum
                    u64 sum = 0ull;
                    for (int i = tid; i < m; i += THREADS) {
                        s.list_mass[i] = ordered(s.list[i]) >= least ? mass_of(s.list[i]) : 0ull;
                        sum += s.list_mass[i];
                    }
                    return block_sum(sum, s);
                };
                u64 kept = total(t);
                if (cut_p) {
                    const unsigned int least = pick_mass(m, t, 0ull, (double)top_p * (double)kept);
                    kept = total(least);
                }
                __syncthreads();
                // the first place whose sum, in the order of places, reaches the target; else the last that is kept
                const double target = (double)u * (double)kept;
                for (int i = tid; i < m; i += THREADS) {
                    const u64 own = s.list_mass[i];
                    if (!own) continue;
                    const int at = s.list_at[i];
                    u64 before = 0ull;
                    for (int j = 0; j < m; ++j)
                        if (s.list_at[j] < at) before += s.list_mass[j];
                    if ((double)(before + own) >= target) atomicMin(&s.token, at);
                    atomicMax(&s.found, at);
                }
                __syncthreads();
                if (tid == 0) out[row] = s.token != 0x7fffffff ? s.token : s.found >= 0 ? s.found : 0;
                return;
            }
            cluster.sync();                                   // (every block has read the count)
            if (rank == 0 && tid == 0) s.list_n = 0u;
            cluster.sync();
        }
    }

    if constexpr (PARKED) {
        if (few && park) {                                    // (parked as they were)
            for (int st = warp; st < stretches; st += kWarps)
                walk(st, [&](int i, const float (&v)[4], int m) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (e < m) put[i + e] = v[e] / by;
                });
        }
        by = 1.f;
    }
    auto divided = [&](float raw) -> float { return PARKED ? raw : raw / by; };       // (raw: as a walk gives it)
    // f(value) for every value of the slice
    auto each = [&](auto f) {
        for (int st = warp; st < stretches; st += kWarps)
            walk(st, [&](int, const float (&v)[4], int m) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < m) f(divided(v[e]));
            });
    };
    unsigned int thr = 0u;                                    // keep x with ordered(x) >= thr
    if (cut_k || cut_p) {
        int turn = 0;
        // the row's sum of c over its blocks
        auto over_row = [&](double c) -> double {
            if (tid == 0) s.slot[turn] = c;
            cluster.sync();
            double t = 0.0;
            of_blocks(&s.slot[turn], [&](double x) { t += x; });
            turn ^= 1;
            return t;
        };
        // how many of the row's values are kept by a bisection's guess, and the mass of those, an integer a stretch
        auto row_count = [&](auto val) -> double {
            int part = 0;
            each([&](float x) { part += val(x) ? 1 : 0; });
            return over_row((double)block_sum((u64)part, s));
        };
        auto stretch_masses = [&](auto val) -> u64 {          // (of this block)
            u64 sum = 0ull;
            for (int st = warp; st < stretches; st += kWarps) {
                float part = 0.f;
                walk(st, [&](int, const float (&v)[4], int m) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (e < m) part += val(divided(v[e]));
                });
                sum += __double2ull_rn(warp_sum((double)part) * (double)mass_scale);
            }
            return block_sum(lane == 0 ? sum : 0ull, s);
        };
        auto row_mass = [&](auto val) -> double { return over_row((double)stretch_masses(val)); };
        // The histogram's buckets are linear in the distance to the maximum, as far as `span`: a larger value never has
        // a later bucket (kBuckets: none).
        float span = INFINITY, inv = 0.f;
        bool ranged = false;
        auto whole_range = [&]() {                            // ... over all that is not -infinity
            if (!ranged) {
                float mn = FLT_MAX;
                each([&](float x) { if (x > -INFINITY) mn = fminf(mn, x); });
                mn = -lsb_warp_max(-mn);
                __syncthreads();
                if (lane == 0) s.scratch_f[warp] = mn;
                __syncthreads();
                for (int w = 0; w < kWarps; ++w) mn = fminf(mn, s.scratch_f[w]);
                if (tid == 0) s.slot[turn] = (double)mn;
                cluster.sync();
                of_blocks(&s.slot[turn], [&](double x) { mn = fminf(mn, (float)x); });
                turn ^= 1;
                span = INFINITY;
                inv = mx > mn ? (float)(kBuckets - 1) / (mx - mn) : 0.f;
                ranged = true;
            }
        };
        auto bucket = [&](float x) {
            const float d = mx - x;
            return d <= span ? min(kBuckets - 1, max(0, (int)(d * inv))) : kBuckets;
        };
        // counts (and masses) of the values that are kept so far, over the whole row
        auto histogram = [&](bool masses) {
            for (int b = tid; b < kBuckets; b += THREADS) { s.cnt[b] = 0u; s.mass[b] = 0ull; }
            __syncthreads();
            each([&](float x) {
                const int b = ordered(x) >= thr ? bucket(x) : kBuckets;
                if (b < kBuckets) {
                    atomicAdd(&s.cnt[b], 1u);
                    if (masses) {
                        const u64 m = mass_of(x);
                        if (m) atomicAdd(&s.mass[b], m);
                    }
                }
            });
            cluster.sync();
            const int share = kBuckets / blocks;              // (blocks is a power of two)
            for (int j = tid; j < share; j += THREADS) {
                const int b = rank * share + j;
                unsigned int c = 0u;
                u64 m = 0ull;
                of_blocks(&s.cnt[b], [&](unsigned int x) { c += x; });
                if (masses) of_blocks(&s.mass[b], [&](u64 x) { m += x; });
                for (int r = 0; r < blocks; ++r) {
                    *cluster.map_shared_rank(&s.tot_cnt[b], r) = c;
                    if (masses) *cluster.map_shared_rank(&s.tot_mass[b], r) = m;
                }
            }
            cluster.sync();
        };
        // The same for the values down to kNear below the maximum, in one walk with the mass of those that are kept further down,
        // which is returned.  Within a bucket a mass is its upper end's, e^(-b step), times 1 - r with r below 1 %: 1 - r is an
        // exponential of 24 bits, so r is a whole number of 2^-24, which 32-bit integers add up without a loss (a value that is a
        // rounding above the upper end lacks nothing).  `near`: how many of them a bucket takes, by odd and even lanes, so that a
        // slice's values fit.
        auto near_histogram = [&]() -> u64 {
            for (int b = tid; b < kBuckets; b += THREADS) {
                s.cnt[b] = s.rest[b] = 0u;
                if (near > 1) s.rest[kBuckets + b] = 0u;
            }
            __syncthreads();
            u64 beyond = 0ull;
            const int half = near > 1 ? (lane & 1) * kBuckets : 0;
            for (int st = warp; st < stretches; st += kWarps) {
                float part = 0.f;
                walk(st, [&](int, const float (&v)[4], int m) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float x = divided(v[e]);
                        if (e < m && ordered(x) >= thr) {
                            const float d = mx - x;
                            const int b = bucket(x);
                            const float w = expf(b < kBuckets ? fmaf((float)b, kStep, -d) : -d);      // (one exponential for both)
                            if (b < kBuckets) {
                                atomicAdd(&s.cnt[b], 1u);
                                const unsigned int r = __float2uint_rn((1.f - w) * kRestScale);
                                if (r) atomicAdd(&s.rest[half + b], r);
                            } else {
                                part += w > 0.f ? w : 0.f;
                            }
                        }
                    }
                });
                beyond += __double2ull_rn(warp_sum((double)part) * (double)mass_scale);
            }
            beyond = block_sum(lane == 0 ? beyond : 0ull, s);
            if (tid == 0) s.tail = beyond;
            auto arrival = cluster.barrier_arrive();
            const int share = kBuckets / blocks;
            double ends[kBuckets / THREADS];
#pragma unroll
            for (int i = 0; i < kBuckets / THREADS; ++i) {
                const int j = tid + i * THREADS;
                ends[i] = j < share ? exp(-(double)(rank * share + j) * (double)kStep) * (double)mass_scale : 0.0;
            }
            cluster.barrier_wait(std::move(arrival));
            u64 all = 0ull;
            of_blocks(&s.tail, [&](u64 x) { all += x; });
#pragma unroll
            for (int i = 0; i < kBuckets / THREADS; ++i) {
                const int j = tid + i * THREADS, b = rank * share + j;
                if (j >= share) continue;
                unsigned int c = 0u;
                u64 lack = 0ull;
                of_blocks(&s.cnt[b], [&](unsigned int x) { c += x; });
                of_blocks(&s.rest[b], [&](unsigned int x) { lack += x; });
                if (near > 1) of_blocks(&s.rest[kBuckets + b], [&](unsigned int x) { lack += x; });
                const u64 m = __double2ull_rn(ends[i] * ((double)c - (double)lack * (1.0 / (double)kRestScale)));
                for (int r = 0; r < blocks; ++r) {
                    *cluster.map_shared_rank(&s.tot_cnt[b], r) = c;
                    *cluster.map_shared_rank(&s.tot_mass[b], r) = m;
                }
            }
            cluster.sync();
            return all;
        };
        // the values of buckets b0 .. b1 that are kept so far, in the first block's list
        auto collect = [&](int b0, int b1) {
            unsigned int* count = cluster.map_shared_rank(&s.list_n, 0);
            float* list = cluster.map_shared_rank(&s.list[0], 0);
            // (what is far from those buckets is passed by without a division)
            const float wide = 1e-5f * (fabsf(mx) + kNear);
            const bool bounded = upright && span == kNear;
            const float lo = bounded ? (mx - (float)(b1 + 1) / inv - wide) * by : -INFINITY, hi = bounded ? (mx - (float)b0 / inv + wide) * by : INFINITY;
            for (int st = warp; st < stretches; st += kWarps)
                walk(st, [&](int, const float (&v)[4], int m) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (e >= m || v[e] < lo || v[e] > hi) continue;
                        const float x = divided(v[e]);
                        const int b = bucket(x);
                        if (b >= b0 && b <= b1 && ordered(x) >= thr) {
                            const unsigned int at = atomicAdd(count, 1u);
                            if (at < (unsigned int)kList) list[at] = x;
                        }
                    }
                });
            cluster.sync();
        };
        auto share_out = [&](unsigned int* slot, unsigned int v) {     // (first block, thread 0)
            for (int r = 0; r < blocks; ++r) *cluster.map_shared_rank(slot, r) = v;
        };
        bool done = !cut_p;                                    // nothing is left to be cut behind the k-th value
        bool listed = false;                                   // the list has been used
        if (cut_k) {
            u64 before;
            const u64 k = (u64)top_k;
            whole_range();
            histogram(false);
            const int kb = find_bucket(s, before, [&](int b) { return (u64)s.tot_cnt[b]; }, [](u64) {}, [&](u64 sum) { return sum >= k; });
            if (kb < kBuckets && before + s.tot_cnt[kb] <= (u64)kWhole) {
                // a few values up to the k-th: both cuts among them
                collect(0, kb);
                if (rank == 0) {
                    const int m = (int)min(s.list_n, (unsigned int)kList);
                    unsigned int t = pick_kth(m, k);
                    if (cut_p) {
                        u64 tot = 0ull;
                        for (int i = tid; i < m; i += THREADS) {
                            s.list_mass[i] = ordered(s.list[i]) >= t ? mass_of(s.list[i]) : 0ull;
                            tot += s.list_mass[i];
                        }
                        tot = block_sum(tot, s);
                        t = pick_mass(m, t, 0ull, (double)top_p * (double)tot);
                    }
                    if (tid == 0) share_out(&s.cut, t);
                }
                cluster.sync();
                thr = s.cut;
                done = true;
            } else if (kb < kBuckets && s.tot_cnt[kb] <= (unsigned int)kList) {
                collect(kb, kb);
                listed = true;
                if (rank == 0) {
                    const unsigned int t = pick_kth((int)min(s.list_n, (unsigned int)kList), k - before);
                    if (tid == 0) share_out(&s.cut, t);
                }
                cluster.sync();
                thr = s.cut;
            } else {
                unsigned int lo = 0u, hi = 0xffffffffu;        // count(>= lo) >= k always holds
                while (lo < hi) {
                    const unsigned int mid = lo + (hi - lo) / 2u + ((hi - lo) & 1u);
                    if (row_count([&](float x) { return ordered(x) >= mid; }) >= (double)k) lo = mid;
                    else hi = mid - 1u;
                }
                thr = lo;
            }
        }
        if (!done) {
            // the smallest v with mass(x > v) <= top_p * (mass kept so far); everything >= v is kept.  Most of the mass lies
            // near the maximum and most of the values do not: the histogram goes kNear down (e^-10 of the maximum's weight)
            // first, all the way if the cut lies further.
            double tot = 0.0, most = 0.0;
            span = kNear;
            inv = (float)(kBuckets - 1) / kNear;
            ranged = false;
            u64 before = 0ull, beyond = 0ull;
            if (near > 0) beyond = near_histogram();
            else {
                tot = row_mass([&](float x) { return ordered(x) >= thr ? weight_of(x) : 0.f; });
                most = (double)top_p * tot;
                histogram(true);
            }
            auto find = [&](bool first) {
                return find_bucket(s, before, [&](int i) { return s.tot_mass[i]; },
                                   [&](u64 sum) {
                                       if (near == 0 || !first) return;
                                       tot = (double)(sum + beyond);
                                       most = (double)top_p * tot;
                                   },
                                   [&](u64 sum) { return (double)sum > most; });
            };
            int b = find(true);
            if (most < 0.0) {
                thr = ordered(mx);                             // (a negative top_p: the maximum alone)
            } else if (tot > 0.0) {
                if (b == kBuckets) {
                    whole_range();
                    histogram(true);
                    b = find(false);
                }
                if (b < kBuckets && s.tot_cnt[b] <= (unsigned int)kList) {
                    if (listed) {
                        if (rank == 0 && tid == 0) s.list_n = 0u;
                        cluster.sync();
                    }
                    collect(b, b);
                    if (rank == 0) {
                        const int m = (int)min(s.list_n, (unsigned int)kList);
                        for (int i = tid; i < m; i += THREADS) s.list_mass[i] = mass_of(s.list[i]);
                        const unsigned int t = pick_mass(m, thr, before, most);
                        if (tid == 0) share_out(&s.cut_mass, t);
                    }
                    cluster.sync();
                    thr = s.cut_mass;
                } else {
                    unsigned int lo = thr, hi = ordered(mx);
                    while (lo < hi) {
                        const unsigned int mid = lo + (hi - lo) / 2u;
                        const double above = row_mass([&](float x) { return ordered(x) > mid ? weight_of(x) : 0.f; });
                        if (above <= most) hi = mid; else lo = mid + 1u;
                    }
                    thr = lo;
                }
            }
        }
    }

    // ---- inverse CDF in index order: the stretches' kept masses meet, one warp finds the place in its own
    // (values well below the cut are passed by without a division)
    float below = -INFINITY;
    if (thr && upright) {
        const float cut = from_ordered(thr);
        below = (cut - 1e-5f * fabsf(cut) - 1e-37f) * by;
    }
    auto kept_of = [&](float raw) -> float {
        if (raw < below) return 0.f;
        const float x = divided(raw);
        return ordered(x) >= thr ? weight_of(x) : 0.f;
    };
    for (int st = warp; st < stretches; st += kWarps) {
        float mine = 0.f;
        walk(st, [&](int, const float (&v)[4], int m) {
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = e < m ? kept_of(v[e]) : 0.f;
            mine += (w[0] + w[1]) + (w[2] + w[3]);
        });
        const double sum = warp_sum((double)mine);
        if (lane == 0) s.seg[st] = sum;
    }
    cluster.sync();
    for (int i = tid; i < row_stretches; i += THREADS) s.all_seg[i] = *cluster.map_shared_rank(&s.seg[i % per_block], i / per_block);
    __syncthreads();
    // (no block reads another's sums beyond this point; the wait for that is at the end)
    auto arrival = cluster.barrier_arrive();
    // (every warp works the answer out for itself; the one whose stretch holds it writes it)
    const int per = (row_stretches + 31) / 32;
    double sum = 0.0;
    for (int j = 0; j < per; ++j) sum += lane * per + j < row_stretches ? s.all_seg[lane * per + j] : 0.0;
    double run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    const double target = (double)u * __shfl_sync(0xffffffffu, run, 31);
    // the first stretch with mass at whose end the sum reaches the target; if none does (a draw of
    // one or more), the last stretch with mass, and in it the last kept value (the reference's
    // fallback, sampling.cpp:113-116)
    int first = 0x7fffffff, last = -1;
    double first_before = 0.0, at_end = run - sum;
    for (int j = 0; j < per; ++j) {
        const double part = lane * per + j < row_stretches ? s.all_seg[lane * per + j] : 0.0;
        if (part > 0.0) {
            last = lane * per + j;
            if (first == 0x7fffffff && at_end + part >= target) { first = last; first_before = at_end; }
        }
        at_end += part;
    }
    const int last_stretch = __reduce_max_sync(0xffffffffu, last);
    const int found = __reduce_min_sync(0xffffffffu, first), pick = found == 0x7fffffff ? last_stretch : found;
    if (pick >= 0 && pick / per_block == rank && pick % per_block % kWarps == warp) {
        double before = __shfl_sync(0xffffffffu, first_before, pick / per);
        int token = -1, kept_last = -1;
        const int b0 = pick % per_block * stretch, b1 = min(n, b0 + stretch);
        // a window of 128 values: the lane's four
        auto window = [&](int i, const float (&raw)[4]) {
            if (i >= b1 || token >= 0) return;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = i + 4 * lane + e < b1 ? kept_of(raw[e]) : 0.f;
            const double own = ((double)v[0] + (double)v[1]) + ((double)v[2] + (double)v[3]);
            double up = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, up, o);
                if (lane >= o) up += t;
            }
            double reach = before + up - own;                  // the sum in front of the lane's values
            int at = 0x7fffffff, kept = -1;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                reach += (double)v[e];
                if (v[e] > 0.f) {
                    kept = i + 4 * lane + e;
                    if (found != 0x7fffffff && at == 0x7fffffff && reach >= target) at = kept;
                }
            }
            kept_last = max(kept_last, __reduce_max_sync(0xffffffffu, kept));
            at = __reduce_min_sync(0xffffffffu, at);
            if (at != 0x7fffffff) token = at;
            before += __shfl_sync(0xffffffffu, up, 31);
        };
        for (int p0 = b0; p0 < b1 && token < 0; p0 += kStretch) {
            float v[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) fetch(p0 + (k * 32 + lane) * 4, b1, v[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) window(p0 + 128 * k, v[k]);
        }
        // (where rounding leaves the sum short of the target at the stretch's end: its last kept value)
        if (lane == 0) out[row] = i0 + (token >= 0 ? token : kept_last);
    }
    __syncwarp();
    cluster.barrier_wait(std::move(arrival));
    if (last_stretch < 0) {
        // no value has any mass: the first of the maxima (an infinity), the first token where there is none
        int mi = 0x7fffffff;
        for (int st = warp; st < stretches; st += kWarps)
            walk(st, [&](int i, const float (&v)[4], int m) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < m && divided(v[e]) == mx) mi = min(mi, i0 + i + e);
            });
        mi = __reduce_min_sync(0xffffffffu, mi);
        if (lane == 0) s.scratch_i[warp] = mi;
        __syncthreads();
        for (int w = 0; w < kWarps; ++w) mi = min(mi, s.scratch_i[w]);
        if (tid == 0) s.mi = mi;
        cluster.sync();                                       // (the row's blocks are here together)
        if (rank == 0 && tid == 0) {
            for (int r = 1; r < blocks; ++r) mi = min(mi, *cluster.map_shared_rank(&s.mi, r));
            out[row] = mi < vocab ? mi : 0;
        }
        cluster.sync();                                       // (the first block may still read this block's)
    }
}

// How a row is shared out: blocks of its cluster, values of a stretch and of a block's slice (whole stretches).
struct Plan { int blocks, stretch, slice; };
static Plan plan(int vocab) {
    Plan p;
    const int units = (vocab + kStretch - 1) / kStretch;
    p.stretch = kStretch * ((units + kMaxStretches - 1) / kMaxStretches);
    const int stretches = (vocab + p.stretch - 1) / p.stretch;
    p.blocks = 1;
    while (p.blocks < kMaxBlocks && (long long)p.blocks * kSliceTarget < vocab) p.blocks *= 2;
    p.slice = (stretches + p.blocks - 1) / p.blocks * p.stretch;
    return p;
}
static size_t slice_bytes(const Plan& p) { return (size_t)p.slice * 4 <= (size_t)kSliceBytes ? (size_t)p.slice * 4 : 0; }

static int num_sms() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
        cached[dev] = n;
    }
    return cached[dev];
}

// (with tokens to penalise)
LSB_API int lsb_sample_needs_work(int vocab) { return slice_bytes(plan(vocab)) == 0; }

// logits: float [rows, vocab]; work: float [rows, vocab] scratch where there are tokens to penalise and
// lsb_sample_needs_work says so, else unused; params: float [rows, 4] = {temperature, top_p, repetition_penalty, u};
// top_k: int [rows] (0 = off); prev_start: int [rows + 1] offsets into prev_tokens, or null; out: int [rows].
LSB_API int lsb_sample(const float* logits, float* work, int rows, int vocab, const float* params,
                       const int* top_k, const int* prev_start, const int* prev_tokens, int* out,
                       cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0) return (int)cudaErrorInvalidValue;
    // a value's mass is at most 2^44, and never so large that a row's sum leaves 63 bits
    int log2 = 0;
    while (log2 < 31 && (1ll << log2) < vocab) ++log2;
    const float mass_scale = (float)(1ull << (63 - log2 < 44 ? 63 - log2 : 44));
    const Plan p = plan(vocab);
    const double rest = p.slice * kMostRest * kRestScale;    // most that a bucket of a block lacks (half of it is even lanes')
    const int near = rest < 4294967296.0 ? 1 : rest < 2 * 4294967296.0 ? 2 : 0;
    // Two blocks with their slices in shared memory fit an SM, four without.  Rows, us with and without (and with a histogram
    // for each cut): 128,256 logits, 8 blocks a row: 8 27 / 44 (28), 32 31 / 48 (34), 64 50 / 53 (60), 101 67 / 65 (83), 127 82 / 77 (99),
    // 256 156 / 134 (208); 32,000, 4 blocks: 8 19 / 30 (18), 64 22 / 32 (23), 101 29 / 33 (33), 127 34 / 32 (38); 50,257, 8 blocks: 64 40 / 35
    // (45).  So parked up to 2.75 blocks an SM, with twice the registers up to one.
    const size_t smem = slice_bytes(p);
    const long long blocks = (long long)rows * p.blocks;
    if (prev_start || (smem && 4 * blocks <= 11ll * num_sms())) {
        static int configured = -1;
        if (configured < 0) {
            configured = (int)cudaFuncSetAttribute(sample_kernel<512, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSliceBytes);
            if (!configured)
                configured = (int)cudaFuncSetAttribute(sample_kernel<512, true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSliceBytes);
        }
        if (configured) return configured;
        if (!smem && !work) return (int)cudaErrorInvalidValue;
        return lsb_launch(blocks <= num_sms() ? sample_kernel<512, true, 1> : sample_kernel<512, true, 2>, dim3(rows, 1, p.blocks), dim3(512), smem,
                          stream, p.blocks, logits, work, vocab, p.stretch, p.slice, smem ? 1 : 0, mass_scale, near, params, top_k,
                          prev_start, prev_tokens, out);
    }
    return lsb_launch(sample_kernel<256, false, 4>, dim3(rows, 1, p.blocks), dim3(256), 0, stream, p.blocks, logits, work, vocab,
                      p.stretch, p.slice, 0, mass_scale, near, params, top_k, prev_start, prev_tokens, out);
}
