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
// temperature) in shared memory.  The k-th largest value and the top-p cut are found with one histogram over
// the values, linear from the row's maximum to its minimum, whose counts and masses the blocks add up through
// distributed shared memory; the bucket the cut falls into is then collected (a few values) and the
// cut picked among them exactly, by counting.  A bucket with more than kList values (rows whose values are all
// but equal, or with outliers that stretch the range) is bisected instead, on the order-preserving integer image of the
// floats, as many as 32 passes over the slices.  128 rows of 128,256 logits (greedy, temperature, top-k,
// top-p and both in turn): 1,430 us with one block a row and bisection throughout, MEASURED_US us so.
//
// Probabilities are exp(x - max) in 32-bit; their sums are taken on 64-bit integers (exp * 2^44, so that even a
// tail of values below 1e-9 counts), which makes every sum exact and the same whatever order the blocks add in.
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
    u64 slot[2];                              // a block's count or mass, by turns (bisection)
    u64 seg[kWarps];                          // kept mass of each warp's stretch of the slice
    u64 all_seg[kMaxBlocks * kWarps];         // ... of the whole row
    u64 scratch[kWarps];
    float scratch_f[2 * kWarps];
    int scratch_i[kWarps];
    unsigned int cnt[kBuckets];               // this block's histogram
    u64 mass[kBuckets];
    unsigned int tot_cnt[kBuckets];           // the row's, the same in every block
    u64 tot_mass[kBuckets];
    float list[kList];                        // (of the cluster's first block) values of one bucket
    u64 list_mass[kList];
    unsigned int list_n;
    unsigned int thr_k, thr_p;                // the two cuts, broadcast by the first block
    u64 kept;                                 // ... and the mass of the k-th value's bucket that is kept
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
    if (cut_k || cut_p)
        for (int b = tid; b < kBuckets; b += kThreads) { s.cnt[b] = 0u; s.mass[b] = 0ull; }
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
        if (rank == 0 && tid == 0) out[row] = mi;
        cluster.sync();                                       // (a peer may still read this block's part)
        return;
    }

    // exp(x - max) as an integer; a value that is not a number counts nothing
    auto mass_of = [&](float x) -> u64 {
        const float e = expf(x - mx);
        return e > 0.f ? __float2ull_rn(e * mass_scale) : 0ull;
    };
    unsigned int thr = 0u;                                    // keep x with ordered(x) >= thr
    if (cut_k || cut_p) {
        // ---- the histogram: bucket 0 holds the maximum; a larger value never has a later bucket
        const float inv = mx > mn ? (float)(kBuckets - 1) / (mx - mn) : 0.f;
        auto bucket = [&](float x) { return max(0, (int)fminf((mx - x) * inv, (float)(kBuckets - 1))); };
        for (int i = tid; i < n; i += kThreads) {
            const float x = xs[i];
            const int b = bucket(x);
            atomicAdd(&s.cnt[b], 1u);
            if (cut_p) {
                const u64 m = mass_of(x);
                if (m) atomicAdd(&s.mass[b], m);
            }
        }
        cluster.sync();
        const int share = kBuckets / blocks;                  // (blocks is a power of two)
        for (int j = tid; j < share; j += kThreads) {
            const int b = rank * share + j;
            unsigned int c = 0u;
            u64 m = 0ull;
            for (int r = 0; r < blocks; ++r) {
                c += *cluster.map_shared_rank(&s.cnt[b], r);
                m += *cluster.map_shared_rank(&s.mass[b], r);
            }
            for (int r = 0; r < blocks; ++r) {
                *cluster.map_shared_rank(&s.tot_cnt[b], r) = c;
                *cluster.map_shared_rank(&s.tot_mass[b], r) = m;
            }
        }
        cluster.sync();
        // the row's sum of val(x) over all slices (bisection only)
        int turn = 0;
        auto row_sum = [&](auto val) -> u64 {
            u64 c = 0ull;
            for (int i = tid; i < n; i += kThreads) c += val(xs[i]);
            c = block_sum(c, s);
            if (tid == 0) s.slot[turn] = c;
            cluster.sync();
            u64 t = 0ull;
            for (int r = 0; r < blocks; ++r) t += *cluster.map_shared_rank(&s.slot[turn], r);
            turn ^= 1;
            return t;
        };
        // the values of one bucket that are >= thr, in the first block's list
        auto collect = [&](int b) {
            unsigned int* count = cluster.map_shared_rank(&s.list_n, 0);
            float* list = cluster.map_shared_rank(&s.list[0], 0);
            for (int i = tid; i < n; i += kThreads) {
                const float x = xs[i];
                if (bucket(x) == b && ordered(x) >= thr) {
                    const unsigned int at = atomicAdd(count, 1u);
                    if (at < (unsigned int)kList) list[at] = x;
                }
            }
            cluster.sync();
        };
        int k_bucket = kBuckets;                               // the bucket of the k-th value
        u64 k_mass = 0ull;                                     // mass of its values that are kept
        bool listed = false;                                   // the first block's list holds it
        if (cut_k) {
            u64 before;
            const u64 k = (u64)top_k;
            k_bucket = find_bucket(s, before, [&](int b) { return (u64)s.tot_cnt[b]; },
                                   [&](u64 sum, int) { return sum >= k; });
            if (k_bucket < kBuckets && s.tot_cnt[k_bucket] <= (unsigned int)kList) {
                collect(k_bucket);
                listed = true;
                if (rank == 0) {
                    const int m = (int)min(s.list_n, (unsigned int)kList);
                    const u64 r = k - before;                  // the r-th largest of the list
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
                        if (above < r && r <= above + same) s.thr_k = o;    // (equal values write the same)
                    }
                    __syncthreads();
                    const unsigned int t = s.thr_k;
                    u64 kept = 0ull;
                    if (cut_p)
                        for (int i = tid; i < m; i += kThreads)
                            if (ordered(s.list[i]) >= t) kept += mass_of(s.list[i]);
                    kept = block_sum(kept, s);
                    if (tid == 0)
                        for (int o = 0; o < blocks; ++o) {
                            *cluster.map_shared_rank(&s.thr_k, o) = t;
                            *cluster.map_shared_rank(&s.kept, o) = kept;
                        }
                }
                cluster.sync();
                thr = s.thr_k;
                k_mass = s.kept;
            } else {
                unsigned int lo = 0u, hi = 0xffffffffu;        // count(>= lo) >= k always holds
                while (lo < hi) {
                    const unsigned int mid = lo + (hi - lo) / 2u + ((hi - lo) & 1u);
                    if (row_sum([&](float x) { return (u64)(ordered(x) >= mid); }) >= k) lo = mid;
                    else hi = mid - 1u;
                }
                thr = lo;
                if (cut_p && k_bucket < kBuckets)
                    k_mass = row_sum([&](float x) { return bucket(x) == k_bucket && ordered(x) >= thr ? mass_of(x) : 0ull; });
            }
        }
        if (cut_p) {
            // mass of bucket b that is kept so far: all of it before the k-th value's bucket, none behind
            auto kept_mass = [&](int b) { return b < k_bucket ? s.tot_mass[b] : b == k_bucket ? k_mass : 0ull; };
            const u64 tot = block_sum(kept_mass(2 * tid) + kept_mass(2 * tid + 1), s);
            const double most = (double)top_p * (double)tot;
            // the smallest v with mass(x > v) <= top_p * tot; everything >= v is kept
            u64 before;
            const int b = find_bucket(s, before, kept_mass, [&](u64 sum, int) { return (double)sum > most; });
            if (b == kBuckets) {
                // nothing exceeds it: no mass at all (thr stays), or a negative top_p (the maximum alone)
                if (most < 0.0) thr = ordered(mx);
            } else if (s.tot_cnt[b] <= (unsigned int)kList) {
                if (!(listed && b == k_bucket)) {
                    if (rank == 0 && tid == 0) s.list_n = 0u;
                    cluster.sync();
                    collect(b);
                }
                if (rank == 0) {
                    const int m = (int)min(s.list_n, (unsigned int)kList);
                    if (tid == 0) s.thr_p = ordered(mx);
                    for (int i = tid; i < m; i += kThreads) s.list_mass[i] = mass_of(s.list[i]);
                    __syncthreads();
                    for (int i = tid; i < m; i += kThreads) {
                        const unsigned int o = ordered(s.list[i]);
                        if (o < thr) continue;
                        u64 above = before;
                        for (int j = 0; j < m; ++j)
                            if (ordered(s.list[j]) > o) above += s.list_mass[j];
                        if ((double)above <= most) atomicMin(&s.thr_p, o);
                    }
                    __syncthreads();
                    if (tid == 0)
                        for (int o = 0; o < blocks; ++o) *cluster.map_shared_rank(&s.thr_p, o) = s.thr_p;
                }
                cluster.sync();
                thr = s.thr_p;
            } else {
                unsigned int lo = thr, hi = ordered(mx);
                while (lo < hi) {
                    const unsigned int mid = lo + (hi - lo) / 2u;
                    const u64 above = row_sum([&](float x) { return ordered(x) > mid ? mass_of(x) : 0ull; });
                    if ((double)above <= most) hi = mid; else lo = mid + 1u;
                }
                thr = lo;
            }
        }
    }

    // ---- inverse CDF in index order: every warp owns a stretch of the slice, its kept mass meets the others'
    const int stretch = (slice + kThreads - 1) / kThreads * 32;
    const int b0 = min(n, warp * stretch), b1 = min(n, b0 + stretch);
    auto kept_of = [&](int i) -> u64 {
        const float x = xs[i];
        return ordered(x) >= thr ? mass_of(x) : 0ull;
    };
    u64 mine = 0ull;
    for (int i = b0 + lane; i < b1; i += 32) mine += kept_of(i);
    mine = warp_sum(mine);
    if (lane == 0) s.seg[warp] = mine;
    cluster.sync();
    const int segs = blocks * kWarps;
    if (tid < segs) s.all_seg[tid] = *cluster.map_shared_rank(&s.seg[tid % kWarps], tid / kWarps);
    __syncthreads();
    // (every warp works the answer out for itself; the one whose stretch holds it writes it)
    u64 part[kMaxBlocks * kWarps / 32], sum = 0ull;
#pragma unroll
    for (int j = 0; j < kMaxBlocks * kWarps / 32; ++j) {
        const int at = lane * (kMaxBlocks * kWarps / 32) + j;
        part[j] = at < segs ? s.all_seg[at] : 0ull;
        sum += part[j];
    }
    u64 run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    const u64 total = __shfl_sync(0xffffffffu, run, 31);
    const double target = (double)u * (double)total;
    // the first stretch with mass at whose end the sum reaches the target; if none does (a draw of
    // one or more), the last stretch with mass, and in it the last kept value (the reference's
    // fallback, sampling.cpp:113-116)
    int first = 0x7fffffff, last = -1;
    u64 first_before = 0ull, at_end = run - sum;
#pragma unroll
    for (int j = 0; j < kMaxBlocks * kWarps / 32; ++j) {
        const int at = lane * (kMaxBlocks * kWarps / 32) + j;
        if (part[j]) {
            last = at;
            if (first == 0x7fffffff && (double)(at_end + part[j]) >= target) { first = at; first_before = at_end; }
        }
        at_end += part[j];
    }
    const int pick = __reduce_min_sync(0xffffffffu, first), pick_last = __reduce_max_sync(0xffffffffu, last);
    if (pick == rank * kWarps + warp) {
        const int owner = pick / (kMaxBlocks * kWarps / 32);
        u64 before = __shfl_sync(0xffffffffu, first_before, owner);
        for (int i = b0; i < b1; i += 32) {
            const u64 m = i + lane < b1 ? kept_of(i + lane) : 0ull;
            u64 up = m;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u64 t = __shfl_up_sync(0xffffffffu, up, o);
                if (lane >= o) up += t;
            }
            const unsigned int hit = __ballot_sync(0xffffffffu, m && (double)(before + up) >= target);
            if (hit) {
                if (lane == 0) out[row] = i0 + i + __ffs(hit) - 1;
                break;
            }
            before += __shfl_sync(0xffffffffu, up, 31);
        }
    } else if (pick == 0x7fffffff && pick_last == rank * kWarps + warp) {
        int best = -1;
        for (int i = b0 + lane; i < b1; i += 32)
            if (kept_of(i)) best = i;
        best = __reduce_max_sync(0xffffffffu, best);
        if (lane == 0) out[row] = i0 + best;
    } else if (pick_last < 0 && rank == 0 && tid == 0) {
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
