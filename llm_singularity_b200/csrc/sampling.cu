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
// What bounds it is the number of times a row is walked and the blocks that walk it.  A row's logits are
// read once: each block of the cluster keeps its contiguous slice (already divided by the
// temperature) in shared memory.  The cuts are found with histograms over the values, linear in the distance to the
// row's maximum, that the blocks add up through distributed shared memory.  Counts give the bucket of the k-th value; where
// only a few values reach that far, they are collected and both cuts picked among them exactly, by counting.  A cut
// by mass alone takes a histogram of masses, near the maximum first (adding 64-bit masses in shared memory is slow
// where all values of a row take part: 183 us for 128 rows with top-p alone), and the values of the one bucket the cut
// falls into.  A bucket with more than kList values (rows whose values are all but equal, or with outliers that
// stretch the range) is bisected instead, on the order-preserving integer image of the floats, as many as 32 passes
// over the slices.  128 rows of 128,256 logits (greedy, temperature, top-k, top-p and both in turn): 1,425 us
// with one block a row and bisection throughout, 100 us so.
//
// Probabilities are exp(x - max) in 32-bit.  A thread adds its few dozen in 32-bit, everything beyond is added in 64-bit in
// a fixed order; the histogram's masses, which arrive in any order, are 64-bit integers (exp * 2^44, so that even a tail
// of values below 1e-9 counts): the same token every time.
//
// `work` is scratch of the same shape as the logits, used only where a slice does not fit shared memory
// (lsb_sample_needs_work).
#include "common.cuh"

#include <cooperative_groups.h>
#include <float.h>

namespace cg = cooperative_groups;

LSB_DEFINE_STATUS()

typedef unsigned long long u64;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxBlocks = 8;                 // blocks of a row's cluster (the portable size)
constexpr int kSliceTarget = 8192;            // logits a block takes before another one joins the cluster
constexpr int kBuckets = 1024;                // of the histogram, two a thread
constexpr int kList = 1024;                   // values of one bucket that are picked among directly
constexpr int kWhole = 512;                   // values up to the k-th that are, all of them
constexpr int kSliceBytes = 184 * 1024;       // most shared memory for a slice

__device__ __forceinline__ unsigned int ordered(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// (value, index) maximum with the lowest index winning ties
__device__ __forceinline__ void argmax_merge(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

struct Part {                                 // what a block has found in its slice
    float mx, mn;
    int mi;
};

struct Shared {
    Part part;
    double slot[2];                           // a block's count or mass, by turns
    double seg[kWarps];                       // kept mass of each warp's stretch of the slice
    double all_seg[kMaxBlocks * kWarps];      // ... of the whole row
    u64 scratch[kWarps];
    double scratch_d[kWarps];
    float scratch_f[2 * kWarps];
    int scratch_i[kWarps];
    unsigned int cnt[kBuckets];               // this block's histogram
    u64 mass[kBuckets];
    unsigned int tot_cnt[kBuckets];           // the row's, the same in every block
    u64 tot_mass[kBuckets];
    float list[kList];                        // (of the cluster's first block) values of one bucket
    u64 list_mass[kList];
    unsigned int list_n;
    unsigned int thr_k, thr_p;                // the first block's work on the two cuts
    unsigned int cut, cut_mass;               // ... and what it tells the others
    int found;                                // bucket picked by find_bucket, and what stands before it
    u64 before;
};

__device__ __forceinline__ u64 warp_sum(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ u64 block_sum(u64 v, Shared& s) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s.scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    u64 t = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += s.scratch[w];
    return t;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double block_sum(double v, Shared& s) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s.scratch_d[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += s.scratch_d[w];
    return t;
}

// The first bucket at which the running sum of val(b) passes ok(before, inclusive); every thread gets it
// (kBuckets: none) together with the sum before it.
template <typename Val, typename Ok>
__device__ __forceinline__ int find_bucket(Shared& s, u64& before, Val val, Ok ok) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u64 a = val(2 * tid), b = val(2 * tid + 1);
    u64 run = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    __syncthreads();
    if (lane == 31) s.scratch[warp] = run;
    if (tid == 0) { s.found = kBuckets; s.before = 0; }
    __syncthreads();
    u64 base = run - (a + b);
    for (int w = 0; w < warp; ++w) base += s.scratch[w];
    // (the condition turns true once along the buckets: exactly one thread finds the turn)
    if (!ok(base, 0) && ok(base + a, 1)) { s.found = 2 * tid; s.before = base; }
    else if (!ok(base + a, 0) && ok(base + a + b, 1)) { s.found = 2 * tid + 1; s.before = base + a; }
    __syncthreads();
    before = s.before;
    return s.found;
}

// params per row: {temperature, top_p, repetition_penalty, u}
__global__ void __launch_bounds__(kThreads, 2)
sample_kernel(const float* __restrict__ logits, float* __restrict__ work, int vocab, int slice, int slice_in_smem,
              float mass_scale, const float* __restrict__ params, const int* __restrict__ top_ks,
              const int* __restrict__ prev_start, const int* __restrict__ prev_tokens, int* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ Shared s;
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
    float* xs = slice_in_smem ? reinterpret_cast<float*>(dyn) : work + (size_t)row * vocab + i0;
    const int pb = prev_start ? prev_start[row] : 0, pe = prev_start ? prev_start[row + 1] : 0;
    const bool penalised = penalty != 1.0f && pe > pb;
    const bool greedy = temperature == 0.0f;
    const bool cut_k = !greedy && top_k > 0 && top_k < vocab, cut_p = !greedy && top_p < 1.0f;

    // ---- the slice into place (a greedy row without a penalty is only looked at), its extremes
    float mx = -FLT_MAX, mn = FLT_MAX;
    int mi = 0x7fffffff;
    auto see = [&](float x, int i) {
        argmax_merge(mx, mi, x, i0 + i);
        if (x > -INFINITY) mn = fminf(mn, x);
    };
    const bool keep = !greedy || penalised;
    if (penalised) {
        for (int i = tid; i < n; i += kThreads) xs[i] = src[i];
        __syncthreads();
        for (int j = pb; j < pe; ++j) {                       // in order; a token is one thread's alone
            const int t = prev_tokens[j] - i0;
            if (t >= 0 && t < n && t % kThreads == tid) xs[t] = xs[t] > 0.f ? xs[t] / penalty : xs[t] * penalty;
        }
        __syncthreads();
        for (int i = tid; i < n; i += kThreads) {
            const float x = greedy ? xs[i] : xs[i] / temperature;
            if (!greedy) xs[i] = x;
            see(x, i);
        }
    } else if ((reinterpret_cast<uintptr_t>(src) & 15) == 0 && (reinterpret_cast<uintptr_t>(xs) & 15) == 0) {
        const float4* s4 = reinterpret_cast<const float4*>(src);
        const int n4 = n >> 2;
        for (int q0 = tid; q0 < n4; q0 += 4 * kThreads) {     // four 16-byte loads in flight
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (q0 + k * kThreads < n4) v[k] = s4[q0 + k * kThreads];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = q0 + k * kThreads;
                if (q < n4) {
                    if (keep) {
                        v[k].x /= temperature; v[k].y /= temperature; v[k].z /= temperature; v[k].w /= temperature;
                        reinterpret_cast<float4*>(xs)[q] = v[k];
                    }
                    see(v[k].x, 4 * q); see(v[k].y, 4 * q + 1); see(v[k].z, 4 * q + 2); see(v[k].w, 4 * q + 3);
                }
            }
        }
        for (int i = 4 * n4 + tid; i < n; i += kThreads) {
            const float x = keep ? src[i] / temperature : src[i];
            if (keep) xs[i] = x;
            see(x, i);
        }
    } else {
        for (int i = tid; i < n; i += kThreads) {
            const float x = keep ? src[i] / temperature : src[i];
            if (keep) xs[i] = x;
            see(x, i);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        argmax_merge(mx, mi, __shfl_xor_sync(0xffffffffu, mx, o), __shfl_xor_sync(0xffffffffu, mi, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if (lane == 0) { s.scratch_f[warp] = mx; s.scratch_i[warp] = mi; s.scratch_f[kWarps + warp] = mn; }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kWarps; ++w) {
            argmax_merge(mx, mi, s.scratch_f[w], s.scratch_i[w]);
            mn = fminf(mn, s.scratch_f[kWarps + w]);
        }
        s.part = Part{mx, mn, mi};
        s.list_n = 0u;
    }
    cluster.sync();
    {
        mx = -FLT_MAX; mn = FLT_MAX; mi = 0x7fffffff;
        for (int r = 0; r < blocks; ++r) {
            const Part p = *cluster.map_shared_rank(&s.part, r);
            argmax_merge(mx, mi, p.mx, p.mi);
            mn = fminf(mn, p.mn);
        }
    }
    if (greedy) {
        if (rank == 0 && tid == 0) out[row] = mi < vocab ? mi : 0;      // (nothing but -infinities and NaN: the first token)
        cluster.sync();                                       // (a peer may still read this block's part)
        return;
    }

    // exp(x - max), as a number and as an integer; a value that is not a number counts nothing
    auto weight_of = [&](float x) -> float {
        const float e = expf(x - mx);
        return e > 0.f ? e : 0.f;
    };
    auto mass_of = [&](float x) -> u64 { return __float2ull_rn(weight_of(x) * mass_scale); };
    // f(value) for every value of the slice, four a thread and turn
    const int n4 = (reinterpret_cast<uintptr_t>(xs) & 15) == 0 ? n >> 2 : 0;
    auto each = [&](auto f) {
#pragma unroll 2
        for (int i = tid; i < n4; i += kThreads) {
            const float4 v = reinterpret_cast<const float4*>(xs)[i];
            f(v.x); f(v.y); f(v.z); f(v.w);
        }
        for (int i = 4 * n4 + tid; i < n; i += kThreads) f(xs[i]);
    };
    unsigned int thr = 0u;                                    // keep x with ordered(x) >= thr
    if (cut_k || cut_p) {
        // The histogram's buckets are linear in the distance to the maximum, as far as `span`: a larger value never has
        // a later bucket (kBuckets: none).
        float span = INFINITY, inv = mx > mn ? (float)(kBuckets - 1) / (mx - mn) : 0.f;
        auto bucket = [&](float x) {
            const float d = mx - x;
            return d <= span ? min(kBuckets - 1, max(0, (int)(d * inv))) : kBuckets;
        };
        // counts (and masses) of the values that are kept so far, over the whole row
        auto histogram = [&](bool masses) {
            for (int b = tid; b < kBuckets; b += kThreads) { s.cnt[b] = 0u; s.mass[b] = 0ull; }
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
            for (int j = tid; j < share; j += kThreads) {
                const int b = rank * share + j;
                unsigned int c = 0u;
                u64 m = 0ull;
                for (int r = 0; r < blocks; ++r) {
                    c += *cluster.map_shared_rank(&s.cnt[b], r);
                    if (masses) m += *cluster.map_shared_rank(&s.mass[b], r);
                }
                for (int r = 0; r < blocks; ++r) {
                    *cluster.map_shared_rank(&s.tot_cnt[b], r) = c;
                    if (masses) *cluster.map_shared_rank(&s.tot_mass[b], r) = m;
                }
            }
            cluster.sync();
        };
        // the row's sum of val(x) over all slices
        int turn = 0;
        auto row_sum = [&](auto val) -> double {              // (a thread's few values in 32-bit, sums of those in 64-bit)
            float part = 0.f;
            each([&](float x) { part += val(x); });
            const double c = block_sum((double)part, s);
            if (tid == 0) s.slot[turn] = c;
            cluster.sync();
            double t = 0.0;
            for (int r = 0; r < blocks; ++r) t += *cluster.map_shared_rank(&s.slot[turn], r);
            turn ^= 1;
            return t;
        };
        // the values of buckets b0 .. b1 that are kept so far, in the first block's list
        auto collect = [&](int b0, int b1) {
            unsigned int* count = cluster.map_shared_rank(&s.list_n, 0);
            float* list = cluster.map_shared_rank(&s.list[0], 0);
            each([&](float x) {
                const int b = bucket(x);
                if (b >= b0 && b <= b1 && ordered(x) >= thr) {
                    const unsigned int at = atomicAdd(count, 1u);
                    if (at < (unsigned int)kList) list[at] = x;
                }
            });
            cluster.sync();
        };
        // (first block) the r-th largest of the list's m values
        auto pick_kth = [&](int m, u64 r) -> unsigned int {
            if (tid == 0) s.thr_k = 0u;
            __syncthreads();
            for (int i = tid; i < m; i += kThreads) {
                const unsigned int o = ordered(s.list[i]);
                u64 above = 0ull, same = 0ull;
                for (int j = 0; j < m; ++j) {
                    const unsigned int oj = ordered(s.list[j]);
                    above += oj > o;
                    same += oj == o;
                }
                if (above < r && r <= above + same) s.thr_k = o;      // (equal values write the same)
            }
            __syncthreads();
            return s.thr_k;
        };
        // (first block) the smallest of the list's values >= least before which there is no more mass than `most`;
        // list_mass is there, `before` is the mass of larger values that are not in the list
        auto pick_mass = [&](int m, unsigned int least, u64 before, double most) -> unsigned int {
            if (tid == 0) s.thr_p = ordered(mx);
            __syncthreads();
            for (int i = tid; i < m; i += kThreads) {
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
        auto share_out = [&](unsigned int* slot, unsigned int v) {     // (first block, thread 0)
            for (int r = 0; r < blocks; ++r) *cluster.map_shared_rank(slot, r) = v;
        };
        bool done = !cut_p;                                    // nothing is left to be cut behind the k-th value
        bool listed = false;                                   // the list has been used
        if (cut_k) {
            u64 before;
            const u64 k = (u64)top_k;
            histogram(false);
            const int kb = find_bucket(s, before, [&](int b) { return (u64)s.tot_cnt[b]; }, [&](u64 sum, int) { return sum >= k; });
            if (kb < kBuckets && before + s.tot_cnt[kb] <= (u64)kWhole) {
                // a few values up to the k-th: both cuts among them
                collect(0, kb);
                if (rank == 0) {
                    const int m = (int)min(s.list_n, (unsigned int)kList);
                    unsigned int t = pick_kth(m, k);
                    if (cut_p) {
                        u64 tot = 0ull;
                        for (int i = tid; i < m; i += kThreads) {
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
                    if (row_sum([&](float x) { return ordered(x) >= mid ? 1.f : 0.f; }) >= (double)k) lo = mid;
                    else hi = mid - 1u;
                }
                thr = lo;
            }
        }
        if (!done) {
            // the smallest v with mass(x > v) <= top_p * (mass kept so far); everything >= v is kept
            const double tot = row_sum([&](float x) { return ordered(x) >= thr ? weight_of(x) : 0.f; });
            const double most = (double)top_p * tot;
            if (most < 0.0) {
                thr = ordered(mx);                             // (a negative top_p: the maximum alone)
            } else if (tot > 0.0) {
                // Most of the mass lies near the maximum and most of the values do not: the histogram goes 10 down
                // (e^-10 of the maximum's weight) first, all the way if the cut lies further.
                const double most_mass = most * (double)mass_scale;
                u64 before = 0ull;
                int b = kBuckets;
                for (int reach = 0; reach < 2 && b == kBuckets; ++reach) {
                    span = reach == 0 ? 10.f : INFINITY;
                    inv = reach == 0 ? (float)(kBuckets - 1) / span : mx > mn ? (float)(kBuckets - 1) / (mx - mn) : 0.f;
                    histogram(true);
                    b = find_bucket(s, before, [&](int i) { return s.tot_mass[i]; }, [&](u64 sum, int) { return (double)sum > most_mass; });
                }
                if (b < kBuckets && s.tot_cnt[b] <= (unsigned int)kList) {
                    if (listed) {
                        if (rank == 0 && tid == 0) s.list_n = 0u;
                        cluster.sync();
                    }
                    collect(b, b);
                    if (rank == 0) {
                        const int m = (int)min(s.list_n, (unsigned int)kList);
                        for (int i = tid; i < m; i += kThreads) s.list_mass[i] = mass_of(s.list[i]);
                        const unsigned int t = pick_mass(m, thr, before, most_mass);
                        if (tid == 0) share_out(&s.cut_mass, t);
                    }
                    cluster.sync();
                    thr = s.cut_mass;
                } else {
                    unsigned int lo = thr, hi = ordered(mx);
                    while (lo < hi) {
                        const unsigned int mid = lo + (hi - lo) / 2u;
                        const double above = row_sum([&](float x) { return ordered(x) > mid ? weight_of(x) : 0.f; });
                        if (above <= most) hi = mid; else lo = mid + 1u;
                    }
                    thr = lo;
                }
            }
        }
    }

    // ---- inverse CDF in index order: every warp owns a stretch of the slice, its kept mass meets the others'
    constexpr int kPer = kMaxBlocks * kWarps / 32;
    const int stretch = (slice + 4 * kThreads - 1) / (4 * kThreads) * 128;
    const int b0 = min(n, warp * stretch), b1 = min(n, b0 + stretch);
    auto kept_of = [&](float x) -> float { return ordered(x) >= thr ? weight_of(x) : 0.f; };
    // the lane's four values from i on (zeros past the stretch)
    auto four = [&](int i, float (&v)[4]) {
        if (i + 3 < b1 && (reinterpret_cast<uintptr_t>(xs + i) & 15) == 0) {
            const float4 x = *reinterpret_cast<const float4*>(xs + i);
            v[0] = kept_of(x.x); v[1] = kept_of(x.y); v[2] = kept_of(x.z); v[3] = kept_of(x.w);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = i + e < b1 ? kept_of(xs[i + e]) : 0.f;
        }
    };
    float mine = 0.f;
    for (int i = b0 + 4 * lane; i < b1; i += 128) {
        float v[4];
        four(i, v);
        mine += (v[0] + v[1]) + (v[2] + v[3]);
    }
    const double stretch_sum = warp_sum((double)mine);
    if (lane == 0) s.seg[warp] = stretch_sum;
    cluster.sync();
    const int segs = blocks * kWarps;
    if (tid < segs) s.all_seg[tid] = *cluster.map_shared_rank(&s.seg[tid % kWarps], tid / kWarps);
    __syncthreads();
    // (every warp works the answer out for itself; the one whose stretch holds it writes it)
    double part[kPer], sum = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        part[j] = lane * kPer + j < segs ? s.all_seg[lane * kPer + j] : 0.0;
        sum += part[j];
    }
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
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        if (part[j] > 0.0) {
            last = lane * kPer + j;
            if (first == 0x7fffffff && at_end + part[j] >= target) { first = last; first_before = at_end; }
        }
        at_end += part[j];
    }
    const int last_stretch = __reduce_max_sync(0xffffffffu, last);
    const int found = __reduce_min_sync(0xffffffffu, first), pick = found == 0x7fffffff ? last_stretch : found;
    if (pick == rank * kWarps + warp) {
        double before = __shfl_sync(0xffffffffu, first_before, pick / kPer);
        int token = -1, kept_last = -1;
        for (int i = b0; i < b1 && token < 0; i += 128) {
            float v[4];
            four(i + 4 * lane, v);
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
        }
        // (where rounding leaves the sum short of the target at the stretch's end: its last kept value)
        if (lane == 0) out[row] = i0 + (token >= 0 ? token : kept_last);
    } else if (last_stretch < 0 && rank == 0 && tid == 0) {
        out[row] = mi < vocab ? mi : 0;                       // no value has any mass
    }
    cluster.sync();                                           // (a peer may still read this block's sums)
}

// Blocks of a row's cluster, logits of a block's slice and its shared memory (0: the slice lives in `work`).
static void plan(int vocab, int* blocks, int* slice, size_t* smem) {
    int b = 1;
    while (b < kMaxBlocks && (long long)b * kSliceTarget < vocab) b *= 2;
    const int per = ((vocab + b - 1) / b + 3) / 4 * 4;
    *blocks = b;
    *slice = per;
    *smem = (size_t)per * 4 <= kSliceBytes ? (size_t)per * 4 : 0;
}

LSB_API int lsb_sample_needs_work(int vocab) {
    int blocks, slice;
    size_t smem;
    plan(vocab, &blocks, &slice, &smem);
    return smem == 0;
}

// logits: float [rows, vocab]; work: float [rows, vocab] scratch where lsb_sample_needs_work says so, else
// unused; params: float [rows, 4] = {temperature, top_p, repetition_penalty, u}; top_k: int [rows] (0 = off);
// prev_start: int [rows + 1] offsets into prev_tokens, or null; out: int [rows].
LSB_API int lsb_sample(const float* logits, float* work, int rows, int vocab, const float* params,
                       const int* top_k, const int* prev_start, const int* prev_tokens, int* out,
                       cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0) return (int)cudaErrorInvalidValue;
    static int configured = -1;
    if (configured < 0)
        configured = (int)cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSliceBytes);
    if (configured) return configured;
    int blocks, slice;
    size_t smem;
    plan(vocab, &blocks, &slice, &smem);
    if (!smem && !work) return (int)cudaErrorInvalidValue;
    // a value's mass is at most 2^44, and never so large that a row's sum leaves 63 bits
    int log2 = 0;
    while (log2 < 31 && (1ll << log2) < vocab) ++log2;
    const float mass_scale = (float)(1ull << (63 - log2 < 44 ? 63 - log2 : 44));
    return lsb_launch(sample_kernel, dim3(rows, 1, blocks), dim3(kThreads), smem, stream, blocks, logits, work, vocab,
                      slice, smem ? 1 : 0, mass_scale, params, top_k, prev_start, prev_tokens, out);
}
