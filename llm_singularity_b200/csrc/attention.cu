// Causal attention over the paged cache, generic form: any mix of prompt portions and
// single decode tokens, any head size that is a multiple of 16 up to 256, any number of
// heads and groups, 32-bit or bfloat16 storage; all arithmetic in 32-bit.
//
// For request r with q_len = q_start[r+1] - q_start[r] new tokens and kv_len tokens in
// the cache after this step, query row i sits at position p = kv_len - q_len + i and
// sees keys at positions [max(0, p - window + 1), p] (window == 0: from 0).  Query
// head h reads kv head h / (nh / nkv).  Scores (q.k) * scale, softmax by running
// maximum and sum, weighted sum of values, division by the sum at the end.
//
// Two score modifiers that other architectures use are taken here (the reference has neither;
// the tensor-core kernels do not take them, so a mixer that asks for one runs these kernels):
// a soft cap, s <- cap * tanh(s / cap), and a linear position bias per head,
// s <- s - slope[h] * (p - key position), applied in that order before the softmax.
//
// Replaces paged_attention_kernel of the reference (kernels/src/attention.cu:27-172:
// 32 threads per (head, row), per-thread v_acc[128] in registers, shared-memory tree
// merge, one launch per request during prefill, models/llama/llama_model.cpp:603-614).
//
// Two kernels, both with keys and values in tiles of shared memory (as 32-bit, the next tile on its way in registers):
//
// * Single tokens are cache traffic: a block takes a kv head's group of query heads over one of up to eight
//   stretches of the request's keys, and the stretches' sums meet through distributed shared memory.  8 requests
//   of 300 to 1,500 tokens, 32 / 8 heads of 64 in 32-bit (29 MB): 24 us; one warp for each (request, head)
//   walking all of its keys took 1,548 us.  The kernel can rotate the token's queries and key and store the key and value by
//   itself (every block takes them from the projection, one writes the page), which saves a kernel of 4 us in the chain of
//   a step of single tokens whose blocks the SMs hold at once, and asks for its first keys while the projection is computed: a layer at 1B sizes, 8 requests, 110 -> 100 us.
// * Portions are arithmetic: 64 rows (16 queries of 4 heads that share their keys) against a tile, 4 rows by 2 or 4
//   keys a thread for the scores and the same 4 rows for the weighted sum, so that a row's maximum, its sum and its
//   probabilities stay within half a warp; two multiply-adds to an instruction.  The last rows of a portion see the most
//   keys, and few portions leave SMs idle: the tiles of a block's keys are dealt out over a cluster, whose sums meet
//   as those of single tokens do.  500 tokens, the same heads: 83 us (1.0 GFLOP), 91 with a block to all of its
//   keys; 120 tokens after 300 31 and 68, 40 after 300 19 and 50; a warp for each (row, head) took 650 us for the 500.
#include "common.cuh"

#include <cooperative_groups.h>
#include <float.h>
#include <math.h>

#include <type_traits>

namespace cg = cooperative_groups;

LSB_DEFINE_STATUS()

constexpr int kThreads = 256;
constexpr int kMaxHeadDim = 256;
constexpr int kMaxSplits = 8;                   // stretches of a request's keys (a cluster of portable size)

struct AttnParams {
    const void* qkv;                            // q of token t at qkv + t * qkv_stride
    int qkv_stride;
    const void* k_pages;
    const void* v_pages;
    const int* q_start;
    const int* kv_len;
    const int* table_rows;
    const int* block_table;
    int table_stride;
    void* out;                                  // [tokens, nh * hd]
    int nh, nkv, hd, page_size, num_pages;
    float scale;
    int window;
    float softcap;
    const float* slopes;
    int heads;                                  // query heads of a block
    int head_blocks;                            // blocks of a kv head's group
};
// What only some kernels take is no parameter of the others: with it behind theirs the compiler makes them 2 - 5 % slower (64 tokens at
// 500 keys, 8 kv heads of 128: 117.2 -> 122.8 us).
struct SplitParams : AttnParams {
    int splits;                                 // blocks that share out a portion's keys
};
// Single tokens whose projection comes unrotated: dims i and i + rotary_dim / 2 turn by position * inv_freq[i], and the new key and
// value go to their page if `store`.
struct RotatingParams : AttnParams {
    const float* inv_freq;
    int rotary_dim, store;
};

typedef unsigned long long pair32;              // two 32-bit values
__device__ __forceinline__ pair32 twice(float a) {
    pair32 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ void fma2(pair32& acc, pair32 a, pair32 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ pair32 mul2(pair32 a, pair32 b) {
    pair32 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void apart(pair32 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }

// four elements as they lie in memory, and as 32-bit
__device__ __forceinline__ uint4 load_raw(const float* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint2 load_raw(const __nv_bfloat16* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ float4 widen(uint4 v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float4 widen(uint2 v) {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}
template <typename T> struct Raw { typedef uint4 type; };
template <> struct Raw<__nv_bfloat16> { typedef uint2 type; };

// The keys of a tile: at most HDC / 4 pieces of four elements a row, KT rows.
template <typename T, int KT, int HDC>
struct Tile {
    static constexpr int kPieces = KT * HDC / 4 / kThreads;
    typename Raw<T>::type k[kPieces], v[kPieces];

    // off: element offset of each key's row in the page pools, -1 for none
    __device__ __forceinline__ void fetch(const AttnParams& p, const long long* off, int tid) {
        const int per = p.hd >> 2;
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
            const int idx = j * kThreads + tid, row = idx / per;
            k[j] = typename Raw<T>::type{};
            v[j] = typename Raw<T>::type{};
            if (row < KT) {
                const long long o = off[row];
                if (o >= 0) {
                    const long long at = o + (idx - row * per) * 4;
                    k[j] = load_raw(reinterpret_cast<const T*>(p.k_pages) + at);
                    v[j] = load_raw(reinterpret_cast<const T*>(p.v_pages) + at);
                }
            }
        }
    }
    // (returns whether every value of this thread's is a number and finite)
    __device__ __forceinline__ bool park(const AttnParams& p, float* ks, float* vs, int ldk, int tid) const {
        const int per = p.hd >> 2;
        float zero = 0.f;                                      // times a number 0, times anything else NaN
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
            const int idx = j * kThreads + tid, row = idx / per, d = (idx - row * per) * 4;
            if (row < KT) {
                *reinterpret_cast<float4*>(ks + row * ldk + d) = widen(k[j]);
                const float4 w = widen(v[j]);
                *reinterpret_cast<float4*>(vs + row * p.hd + d) = w;
                zero = fmaf(w.x, zero, fmaf(w.y, zero, fmaf(w.z, zero, w.w * zero)));
            }
        }
        return zero == 0.f;
    }
};

// Where the row of key `pos` of kv head g lies in the page pools (elements); -1 and a recorded status if its page
// is not one of the pool's.
__device__ __forceinline__ long long key_offset(const AttnParams& p, const int* table, int g, int pos) {
    const int page = table[pos / p.page_size];
    if (page < 0 || page >= p.num_pages) {
        lsb_set_status(LSB_BAD_PAGE);
        return -1;
    }
    return (((long long)page * p.nkv + g) * p.page_size + pos % p.page_size) * p.hd;
}

__device__ __forceinline__ float modified(const AttnParams& p, float s, float slope, int distance) {
    if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
    return s - slope * (float)distance;
}

// ------------------------------------------------------------------ single tokens
// Most query heads of a block: their sums are kAccs a thread.
constexpr int kAccs = 4;

template <int KT>
static size_t single_smem(int hd, int heads, bool rotates) {
    return ((size_t)KT * (hd + 4) + (size_t)KT * hd + (size_t)heads * hd * 2 + (size_t)heads * (KT + 4) + heads * 4 + (rotates ? 2 * (size_t)hd : 0)) * 4;
}

// P: AttnParams, or RotatingParams to rotate and store.
template <typename T, int KT, int HDC, typename P>
__global__ void __launch_bounds__(kThreads, 2) attention_single_kernel(const P p) {
    constexpr bool ROTATES = std::is_same<P, RotatingParams>::value;
    extern __shared__ __align__(16) float sm[];
    __shared__ long long off[2][KT];
    __shared__ float cs[2][ROTATES ? kMaxHeadDim / 2 : 1];     // cosines and sines of the token's position
    cg::cluster_group cluster = cg::this_cluster();
    lsb_pdl_launch_dependents();
    // The step's metadata and tables are there before its first kernel, so with a rotation all that follows from them is had before
    // the wait for the projection, the first keys and values among it.
    if constexpr (!ROTATES) lsb_pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int splits = (int)gridDim.x, split = (int)blockIdx.x, r = blockIdx.z;
    const int g = blockIdx.y / p.head_blocks, group = p.nh / p.nkv;
    const int h0 = g * group + (int)(blockIdx.y % p.head_blocks) * p.heads;
    const int H = min(p.heads, (g + 1) * group - h0);
    const int t = p.q_start[r];
    if (p.q_start[r + 1] - t != 1) return;                     // (all blocks of the cluster alike)
    const int hd = p.hd, ldk = hd + 4, lds = KT + 4;
    float* ks = sm;
    float* vs = ks + KT * ldk;
    float* qs = vs + KT * hd;                                  // [heads][hd], scaled
    float* os = qs + p.heads * hd;                             // [heads][hd], the stretch's sums
    float* ps = os + p.heads * hd;                             // [heads][KT + 4]
    float* ml = ps + p.heads * lds;                            // running maximum, sum, factor of the last tile; m and l stay
    float* fresh = ml + p.heads * 4;                           // the token's own key and value
    const int pos = p.kv_len[r] - 1;
    const int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    // this block's stretch: whole sixteens of keys
    const int per = ((pos - lo + 1 + splits - 1) / splits + 15) / 16 * 16;
    const int first = lo + split * per, last = min(pos + 1, first + per);     // [first, last), maybe empty
    const int* table = p.block_table + (size_t)p.table_rows[r] * p.table_stride;

    const T* token = reinterpret_cast<const T*>(p.qkv) + (size_t)t * p.qkv_stride;
    bool stores = false;
    int half = 0;
    if constexpr (ROTATES) {
        stores = p.store;
        half = p.rotary_dim >> 1;
        for (int i = tid; i < half; i += kThreads) sincosf((float)pos * p.inv_freq[i], &cs[1][i], &cs[0][i]);
    } else {
        for (int i = tid; i < H * hd; i += kThreads) qs[i] = lsb_to_float(token[(size_t)h0 * hd + i]) * p.scale;
    }
    if (tid < H) { ml[4 * tid] = -FLT_MAX; ml[4 * tid + 1] = 0.f; }
    if (tid < KT) off[0][tid] = first + tid < last ? key_offset(p, table, g, first + tid) : -1;
    float acc[kAccs];
#pragma unroll
    for (int a = 0; a < kAccs; ++a) acc[a] = 0.f;
    __syncthreads();
    Tile<T, KT, HDC> tile;
    if constexpr (!ROTATES) {
        tile.fetch(p, off[0], tid);
    } else {
        // (what its page holds of a key that comes with the projection is not used; one that another layer's kernel writes in this
        // step is waited for)
        const bool early = stores || pos < first || pos >= first + KT;
        if (early) tile.fetch(p, off[0], tid);
        lsb_pdl_wait();
        if (!early) tile.fetch(p, off[0], tid);
        // element d of a head at x, rotated, as the projection's type holds it
        auto turned = [&](const T* x, int d) -> float {
            if (d >= 2 * half) return lsb_to_float(x[d]);
            const int i = d < half ? d : d - half;
            const float x0 = lsb_to_float(x[i]), x1 = lsb_to_float(x[i + half]);
            return lsb_to_float(lsb_from_float<T>(d < half ? x0 * cs[0][i] - x1 * cs[1][i] : x0 * cs[1][i] + x1 * cs[0][i]));
        };
        for (int i = tid; i < H * hd; i += kThreads) qs[i] = turned(token + (size_t)(h0 + i / hd) * hd, i % hd) * p.scale;
        if (stores && pos >= first && pos < last) {
            const long long to = blockIdx.y % p.head_blocks == 0 ? key_offset(p, table, g, pos) : -1;       // (one block writes)
            for (int d = tid; d < hd; d += kThreads) {
                const float u = turned(token + (size_t)(p.nh + g) * hd, d), w = lsb_to_float(token[(size_t)(p.nh + p.nkv + g) * hd + d]);
                fresh[d] = u;
                fresh[hd + d] = w;
                if (to >= 0) {
                    reinterpret_cast<T*>(const_cast<void*>(p.k_pages))[to + d] = lsb_from_float<T>(u);
                    reinterpret_cast<T*>(const_cast<void*>(p.v_pages))[to + d] = lsb_from_float<T>(w);
                }
            }
        }
        __syncthreads();
    }
    for (int base = first, turn = 0; base < last; base += KT, turn ^= 1) {
        tile.park(p, ks, vs, ldk, tid);
        if (stores && pos < last && pos - base < KT) {
            // the token's own key and value over what their page held, by the threads that have just put it there
            const int row = pos - base, pieces = hd >> 2, piece = (tid + kThreads - row * pieces % kThreads) % kThreads;
            if (piece < pieces) {
                *reinterpret_cast<float4*>(ks + row * ldk + piece * 4) = *reinterpret_cast<const float4*>(fresh + piece * 4);
                *reinterpret_cast<float4*>(vs + row * hd + piece * 4) = *reinterpret_cast<const float4*>(fresh + hd + piece * 4);
            }
        }
        const int next = base + KT;
        if (tid < KT) off[turn ^ 1][tid] = next + tid < last ? key_offset(p, table, g, next + tid) : -1;
        __syncthreads();
        if (next < last) tile.fetch(p, off[turn ^ 1], tid);
        for (int i = tid; i < H * KT; i += kThreads) {         // a (head, key) each: whole warps share a head
            const int h = i / KT, k = i % KT;
            float s = -FLT_MAX;
            if (off[turn][k] >= 0) {
                const ulonglong2* a = reinterpret_cast<const ulonglong2*>(qs + h * hd);
                const ulonglong2* b = reinterpret_cast<const ulonglong2*>(ks + k * ldk);
                pair32 s0 = 0ull, s1 = 0ull;
                for (int d = 0; d < hd / 4; d += 4) {          // (hd is a multiple of 16)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const ulonglong2 x = a[d + e], y = b[d + e];
                        fma2(s0, x.x, y.x);
                        fma2(s1, x.y, y.y);
                    }
                }
                float s00, s01, s10, s11;
                apart(s0, s00, s01);
                apart(s1, s10, s11);
                s = modified(p, (s00 + s01) + (s10 + s11), p.slopes ? p.slopes[h0 + h] : 0.f, pos - (base + k));
            }
            ps[h * lds + k] = s;
        }
        __syncthreads();
        for (int h = warp; h < H; h += kThreads / 32) {
            float* row = ps + h * lds;
            float s[KT / 32], mx = -FLT_MAX;
#pragma unroll
            for (int j = 0; j < KT / 32; ++j) { s[j] = row[lane + 32 * j]; mx = fmaxf(mx, s[j]); }
            const float m = ml[4 * h], m_new = fmaxf(m, lsb_warp_max(mx));
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < KT / 32; ++j) {
                const float e = off[turn][lane + 32 * j] >= 0 ? expf(s[j] - m_new) : 0.f;
                row[lane + 32 * j] = e;
                sum += e;
            }
            sum = lsb_warp_sum(sum);
            __syncwarp();
            if (lane == 0) {
                const float corr = expf(m - m_new);            // m == -FLT_MAX first: exp(-huge) = 0
                ml[4 * h] = m_new;
                ml[4 * h + 1] = ml[4 * h + 1] * corr + sum;
                ml[4 * h + 2] = corr;
            }
        }
        __syncthreads();
#pragma unroll
        for (int a = 0; a < kAccs; ++a) {
            const int i = a * kThreads + tid;
            if (i < H * hd) {
                const int h = i / hd, d = i - h * hd;
                const float4* w = reinterpret_cast<const float4*>(ps + h * lds);
                float o = acc[a] * ml[4 * h + 2];
#pragma unroll 4
                for (int k = 0; k < KT / 4; ++k) {
                    const float4 e = w[k];
                    const float* v = vs + 4 * k * hd + d;
                    o = fmaf(e.x, v[0], o);
                    o = fmaf(e.y, v[hd], o);
                    o = fmaf(e.z, v[2 * hd], o);
                    o = fmaf(e.w, v[3 * hd], o);
                }
                acc[a] = o;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < kAccs; ++a)
        if (a * kThreads + tid < H * hd) os[a * kThreads + tid] = acc[a];
    cluster.sync();
    // every block brings its share of the outputs together, stretches in order
    T* out = reinterpret_cast<T*>(p.out) + (size_t)t * p.nh * hd + (size_t)h0 * hd;
    for (int i = split * kThreads + tid; i < H * hd; i += splits * kThreads) {
        const int h = i / hd;
        float m = -FLT_MAX;
        for (int s = 0; s < splits; ++s) m = fmaxf(m, *cluster.map_shared_rank(ml + 4 * h, s));
        float l = 0.f, o = 0.f;
        for (int s = 0; s < splits; ++s) {
            const float f = expf(*cluster.map_shared_rank(ml + 4 * h, s) - m);
            l += f * *cluster.map_shared_rank(ml + 4 * h + 1, s);
            o += f * *cluster.map_shared_rank(os + i, s);
        }
        out[i] = lsb_from_float<T>(o * (l > 0.f ? 1.f / l : 0.f));       // (a sum that is not a number stays none)
    }
    cluster.sync();                                            // (a peer may still read this block's sums)
}

// ------------------------------------------------------------------ portions
constexpr int kRows = 64;                       // (query, head) rows of a block
constexpr int kPortionHeads = 4;                // most query heads of a block

template <int KT>
static size_t portion_smem(int hd) {
    return ((size_t)kRows * (hd + 4) + (size_t)KT * (hd + 4) + (size_t)KT * hd + (size_t)kRows * (KT + 4)) * 4;
}

// P: AttnParams, or SplitParams where a cluster of p.splits blocks shares out the keys of its rows.  (One kernel for both: 500
// tokens at 4,000 keys, 32 / 8 heads of 64 in 32-bit, whole, 746 us where it takes 691.)
template <typename T, int KT, int HDC, typename P>
__global__ void __launch_bounds__(kThreads, HDC <= 128 ? 2 : 1) attention_portion_kernel(const P p) {
    constexpr bool SPLIT = std::is_same<P, SplitParams>::value;
    constexpr int KPT = KT / 16;                // keys of a thread's scores
    constexpr int CPT = HDC / 64;               // groups of four columns of a thread's sums
    extern __shared__ __align__(16) float sm[];
    __shared__ long long off[2][KT];
    __shared__ float slopes[kRows];             // of the rows' heads
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, r = blockIdx.z;
    int splits = 1;
    if constexpr (SPLIT) splits = p.splits;
    const int split = SPLIT ? (int)blockIdx.x % splits : 0;
    const int g = blockIdx.y / p.head_blocks, group = p.nh / p.nkv;
    const int h0 = g * group + (int)(blockIdx.y % p.head_blocks) * p.heads;
    const int H = min(p.heads, (g + 1) * group - h0);
    const int qs0 = p.q_start[r], q_len = p.q_start[r + 1] - qs0;
    const int queries = kRows / p.heads;
    const int i0 = ((int)gridDim.x - 1 - (int)blockIdx.x) / splits * queries;          // the longest rows first
    if (q_len <= 1 || i0 >= q_len) return;                     // (all blocks of the cluster alike)
    const int hd = p.hd, ldk = hd + 4, ldp = KT + 4;
    float* qs = sm;
    float* ks = qs + kRows * ldk;
    float* vs = ks + KT * ldk;
    float* ps = vs + KT * hd;
    const int pos0 = p.kv_len[r] - q_len + i0;                 // of the block's first query
    const int pos_last = min(pos0 + queries, p.kv_len[r]) - 1;
    // this block's tiles: every splits-th
    const int lo = ((p.window > 0 && pos0 - p.window + 1 > 0) ? pos0 - p.window + 1 : 0) + split * KT, stride = SPLIT ? splits * KT : KT;
    const int* table = p.block_table + (size_t)p.table_rows[r] * p.table_stride;

    // row x: query i0 + x / heads, head h0 + x % heads (rows beyond the portion or the group stay zero)
    for (int i = tid; i < kRows * hd; i += kThreads) {
        const int x = i / hd, d = i - x * hd, qi = i0 + x / p.heads, h = x % p.heads;
        qs[x * ldk + d] = qi < q_len && h < H && x / p.heads < queries
            ? lsb_to_float(reinterpret_cast<const T*>(p.qkv)[(size_t)(qs0 + qi) * p.qkv_stride + (size_t)(h0 + h) * hd + d]) * p.scale
            : 0.f;
    }
    if (tid < KT) off[0][tid] = lo + tid <= pos_last ? key_offset(p, table, g, lo + tid) : -1;
    if (p.slopes && tid < kRows) slopes[tid] = tid % p.heads < H ? p.slopes[h0 + tid % p.heads] : 0.f;
    // (a row sees the keys whose distance is below this: one unsigned comparison for both of its ends)
    const unsigned reach = p.window > 0 ? (unsigned)p.window : 0x7fffffffu;
    int pos[4];
    float m[4], l[4];
    pair32 acc[4][2 * CPT];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int x = ty * 4 + i;
        pos[i] = min(pos0 + x / p.heads, pos_last);
        m[i] = -FLT_MAX;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * CPT; ++c) acc[i][c] = 0ull;
    }
    __syncthreads();
    Tile<T, KT, HDC> tile;
    tile.fetch(p, off[0], tid);
    for (int base = lo, turn = 0; base <= pos_last; base += stride, turn ^= 1) {
        const bool finite = tile.park(p, ks, vs, ldk, tid);
        const int next = base + stride;
        if (tid < KT) off[turn ^ 1][tid] = next + tid <= pos_last ? key_offset(p, table, g, next + tid) : -1;
        const bool by_row = __syncthreads_or(!finite);
        if (next <= pos_last) tile.fetch(p, off[turn ^ 1], tid);
        // scores: rows 4 ty + i, keys tx + 16 j
        pair32 s2[4][KPT];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < KPT; ++j) s2[i][j] = 0ull;
#pragma unroll 2
        for (int d = 0; d < hd; d += 4) {
            ulonglong2 a[4], b[KPT];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(qs + (ty * 4 + i) * ldk + d);
#pragma unroll
            for (int j = 0; j < KPT; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ks + (tx + 16 * j) * ldk + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < KPT; ++j) {
                    fma2(s2[i][j], a[i].x, b[j].x);
                    fma2(s2[i][j], a[i].y, b[j].y);
                }
        }
        // a row's 16 threads are half a warp
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float s[KPT], mx = m[i];
            bool seen[KPT];
            const float slope = p.slopes ? slopes[ty * 4 + i] : 0.f;
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const int key = base + tx + 16 * j;
                float u, v;
                apart(s2[i][j], u, v);
                seen[j] = (unsigned)(pos[i] - key) < reach && off[turn][tx + 16 * j] >= 0;
                s[j] = seen[j] ? modified(p, u + v, slope, pos[i] - key) : -FLT_MAX;
                mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float corr = expf(m[i] - mx);                // m == -FLT_MAX first: exp(-huge) = 0
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const float e = seen[j] ? expf(s[j] - mx) : 0.f;
                ps[(ty * 4 + i) * ldp + tx + 16 * j] = e;
                sum += e;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            m[i] = mx;
            l[i] = l[i] * corr + sum;
            const pair32 c2 = twice(corr);
#pragma unroll
            for (int c = 0; c < 2 * CPT; ++c) acc[i][c] = mul2(acc[i][c], c2);
        }
        __syncwarp();                                          // the row's probabilities were written by this warp
        // the weighted sum: columns 4 tx + 64 c
        if (by_row) {
            // an infinity or NaN among the values: a row takes in only the keys it sees (0 times such a value is none)
            for (int k = 0; k < KT; ++k) {
                if (off[turn][k] < 0) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if ((unsigned)(pos[i] - (base + k)) >= reach) continue;
                    const pair32 we = twice(ps[(ty * 4 + i) * ldp + k]);
#pragma unroll
                    for (int c = 0; c < CPT; ++c) {
                        const int d = tx * 4 + 64 * c;
                        if (d < hd) {
                            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vs + k * hd + d);
                            fma2(acc[i][2 * c], we, v.x);
                            fma2(acc[i][2 * c + 1], we, v.y);
                        }
                    }
                }
            }
        } else
#pragma unroll 2
        for (int k = 0; k < KT; k += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(ps + (ty * 4 + i) * ldp + k);
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const int d = tx * 4 + 64 * c;
                if (d < hd) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vs + (k + e) * hd + d);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const pair32 we = twice(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
                            fma2(acc[i][2 * c], we, v.x);
                            fma2(acc[i][2 * c + 1], we, v.y);
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
    if constexpr (SPLIT) {
        cg::cluster_group cluster = cg::this_cluster();
        // the blocks' sums meet: each brings its share of the rows together, blocks in order
        float* os = qs;                                        // [kRows][ldk] (the queries have been used)
        float* ml = ps;                                        // [kRows] (maximum, sum)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = ty * 4 + i;
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const int d = tx * 4 + 64 * c;
                if (d < hd) *reinterpret_cast<ulonglong2*>(os + x * ldk + d) = make_ulonglong2(acc[i][2 * c], acc[i][2 * c + 1]);
            }
            if (tx == 0) { ml[2 * x] = m[i]; ml[2 * x + 1] = l[i]; }
        }
        cluster.sync();
        const int rows = (kRows + splits - 1) / splits, x0 = split * rows, x1 = min(kRows, x0 + rows), per = hd >> 2;
        for (int e = tid; e < (x1 - x0) * per; e += kThreads) {
            const int x = x0 + e / per, d = e % per * 4, qi = i0 + x / p.heads, h = x % p.heads;
            if (qi >= q_len || h >= H || x / p.heads >= queries) continue;
            float top = -FLT_MAX, sum = 0.f, out[4] = {0.f, 0.f, 0.f, 0.f};
            for (int k = 0; k < splits; ++k) top = fmaxf(top, *cluster.map_shared_rank(ml + 2 * x, k));
            for (int k = 0; k < splits; ++k) {
                const float2 of = *reinterpret_cast<const float2*>(cluster.map_shared_rank(ml + 2 * x, k));
                const float4 o = *reinterpret_cast<const float4*>(cluster.map_shared_rank(os + x * ldk + d, k));
                const float f = expf(of.x - top);
                sum += f * of.y;
                out[0] += f * o.x;
                out[1] += f * o.y;
                out[2] += f * o.z;
                out[3] += f * o.w;
            }
            const float inv = sum > 0.f ? 1.f / sum : 0.f;
            T* to = reinterpret_cast<T*>(p.out) + (size_t)(qs0 + qi) * p.nh * hd + (size_t)(h0 + h) * hd + d;
#pragma unroll
            for (int k = 0; k < 4; ++k) to[k] = lsb_from_float<T>(out[k] * inv);
        }
        cluster.sync();                                        // (a peer may still read this block's sums)
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int x = ty * 4 + i, qi = i0 + x / p.heads, h = x % p.heads;
        if (qi >= q_len || h >= H || x / p.heads >= queries) continue;
        const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
        T* o = reinterpret_cast<T*>(p.out) + (size_t)(qs0 + qi) * p.nh * hd + (size_t)(h0 + h) * hd;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            const int d = tx * 4 + 64 * c;
            if (d < hd) {
                float v[4];
                apart(acc[i][2 * c], v[0], v[1]);
                apart(acc[i][2 * c + 1], v[2], v[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) o[d + e] = lsb_from_float<T>(v[e] * inv);
            }
        }
    }
}

// ------------------------------------------------------------------ host side
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

// clusters of consecutive blocks along x
template <typename P>
static int launch_clusters(void (*kernel)(P), dim3 grid, size_t smem, unsigned cluster, const P& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (lsb_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return (int)cudaLaunchKernelEx(&cfg, kernel, p);
}

// Blocks that share out the keys of a portion's rows.  Blocks are taken to run in rounds of `room(s)`, the longest first, the
// lengths falling evenly from the longest to the shortest (tiles of keys).  A block's set-up and end cost it as much as 0.6 of a
// tile, 0.8 where a cluster meets, and clusters have to promise 5 % (all fitted to 57 shapes in one to eight parts: no choice is slower
// than whole blocks there, the geometric mean is 1.3 % above the best).  32 / 8 heads of 64 in 32-bit, us with 1 / 2 / 4 / 8 blocks, the
// choice in front: 500 tokens (2) 97 / 88 / 94 / 142, 240 (2) 53 / 35 / 40 / 71, 40 (1) 15.6 / 20.5 / 16.6 / 21.1, 40 after 300 (6: 22) 59 / 43 / 32 /
// 22, 40 after 3,960 (8) 510 / 261 / 189 / 102, 500 after 3,500 (1) 691 / 701 / 702 / 740, with a window of 1,000 (1) 185 / 200 / 211 / 239;
// 16 / 8 of 256 in bfloat16, 300 after 2,000 (3: 578) 829 / 793 / 640 / 698.
template <typename Room>
static int portion_splits(long long blocks, Room room, int longest, int shortest) {
    int best = 1;
    double least = 0.0;
    for (int s = 1; s <= kMaxSplits && s <= longest; ++s) {
        const long long n = blocks * s, at_once = room(s), rounds = (n + at_once - 1) / at_once;
        if (s > 1 && rounds > 16) break;                       // (the SMs are busy without)
        double cost = ceil((double)longest / s) + (s > 1 ? 0.8 : 0.6);
        for (long long r = 1; r < rounds && r < 64; ++r) {
            const double tiles = (longest - (double)(longest - shortest) * (double)(r * at_once) / (double)n) / s + 0.25;
            cost += (tiles < 1.0 ? 1.0 : tiles) + (s > 1 ? 0.8 : 0.6);
        }
        if (rounds > 64) cost *= (double)rounds / 64.0;
        if (s == 1) cost *= 0.95;
        if (s == 1 || cost < least) { least = cost; best = s; }
    }
    return best;
}
// Blocks of a portion kernel that run at once in clusters of `splits`: fewer than the SMs hold where clusters don't fill a group of SMs.
template <typename T, int KT, int HDC>
static long long portion_room(int hd, int splits) {
    const long long whole = (HDC <= 128 ? 2ll : 1ll) * num_sms();
    static int cached[64][kMaxHeadDim / 16 + 1][kMaxSplits + 1] = {};
    int dev = 0;
    if (splits == 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return whole;
    int& clusters = cached[dev][hd / 16][splits];
    if (clusters == 0) {
        int n = 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(splits);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = portion_smem<KT>(hd);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(attention_portion_kernel<T, KT, HDC, SplitParams>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, attention_portion_kernel<T, KT, HDC, SplitParams>, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            n = (int)(whole / splits);
        }
        clusters = n < 1 ? 1 : n;
    }
    return (long long)clusters * splits;
}
// The blocks from the sizes of a step: `portions` requests of up to max_q_len tokens whose longest context is `keys`, 0 where it is
// not known (a captured launch).  A window bounds what a block walks, whatever the context; without either, the portions
// are taken to be all of their contexts (captured portions of 500: 88 us as a prompt where whole blocks take 97, 701 after 3,500 where
// they take 691; all with the rotary kernel in front).
template <typename T, int KT, int HDC>
static int splits_of_portions(int hd, int nh, int nkv, long long portions, int max_q_len, int keys, int window) {
    const int group = nh / nkv, heads = group < kPortionHeads ? group : kPortionHeads, queries = kRows / heads;
    const long long tiles = (max_q_len + queries - 1) / queries, blocks = tiles * nkv * ((group + heads - 1) / heads) * portions;
    const long long seen = window > 0 ? (long long)window + queries - 1 : 0x7fffffffll;       // most keys of a block
    long long most = keys > max_q_len ? keys : max_q_len, least = most - max_q_len + 1;
    if (window > 0 && keys <= 0) most = least = seen;
    most = most < seen ? most : seen;
    least = least < most ? least : most;
    return portion_splits(blocks, [&](int s) { return portion_room<T, KT, HDC>(hd, s); }, (int)((most + KT - 1) / KT), (int)((least + KT - 1) / KT));
}
LSB_API int lsb_portion_splits(int hd, int nh, int nkv, int portions, int max_q_len, int keys, int window) {
    return hd <= 64    ? splits_of_portions<float, 64, 64>(hd, nh, nkv, portions, max_q_len, keys, window)
           : hd <= 128 ? splits_of_portions<float, 32, 128>(hd, nh, nkv, portions, max_q_len, keys, window)
                       : splits_of_portions<float, 32, 256>(hd, nh, nkv, portions, max_q_len, keys, window);
}

// rot: null, or the rotation of single tokens
template <typename T, int KT, int HDC>
static int launch(AttnParams p, const RotatingParams* rot, int n_requests, int max_q_len, int n_single, int max_keys, int portion_keys,
                  cudaStream_t stream) {
    static int configured = -1;
    const int group = p.nh / p.nkv;
    if (configured < 0) {
        // (the largest any of them asks for: heads of HDC, as many as a block takes of the smallest, 16)
        const auto allow = [](auto kernel) { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024); };
        int rc = allow(attention_single_kernel<T, KT, HDC, AttnParams>);
        if (!rc) rc = allow(attention_single_kernel<T, KT, HDC, RotatingParams>);
        if (!rc) rc = allow(attention_portion_kernel<T, KT, HDC, AttnParams>);
        if (!rc) rc = allow(attention_portion_kernel<T, KT, HDC, SplitParams>);
        configured = rc;
    }
    if (configured) return configured;
    if (n_single > 0) {
        AttnParams s = p;
        s.heads = kAccs * kThreads / p.hd;
        if (s.heads > group) s.heads = group;
        s.head_blocks = (group + s.heads - 1) / s.heads;
        // two blocks an SM, as many stretches as that takes; no stretch shorter than a tile where the longest
        // context is known (a captured launch has to serve any)
        const long long blocks = (long long)n_single * p.nkv * s.head_blocks;
        long long splits = (2ll * num_sms() + blocks / 2) / blocks;
        if (max_keys > 0 && splits > (max_keys + KT - 1) / KT) splits = (max_keys + KT - 1) / KT;
        splits = splits < 1 ? 1 : splits > kMaxSplits ? kMaxSplits : splits;
        if ((long long)p.nkv * s.head_blocks > 65535) return (int)cudaErrorInvalidValue;
        const dim3 grid((unsigned)splits, p.nkv * s.head_blocks, n_requests);
        const size_t smem = single_smem<KT>(p.hd, s.heads, rot != nullptr);
        int rc;
        if (rot) {
            RotatingParams turned = *rot;
            static_cast<AttnParams&>(turned) = s;
            rc = launch_clusters(attention_single_kernel<T, KT, HDC, RotatingParams>, grid, smem, (unsigned)splits, turned, stream);
        } else {
            rc = launch_clusters(attention_single_kernel<T, KT, HDC, AttnParams>, grid, smem, (unsigned)splits, s, stream);
        }
        if (rc) return rc;
    }
    if (max_q_len > 1) {
        p.heads = group < kPortionHeads ? group : kPortionHeads;
        p.head_blocks = (group + p.heads - 1) / p.heads;
        if ((long long)p.nkv * p.head_blocks > 65535) return (int)cudaErrorInvalidValue;
        const int queries = kRows / p.heads;
        const long long tiles = (max_q_len + queries - 1) / queries;
        const int splits = splits_of_portions<T, KT, HDC>(p.hd, p.nh, p.nkv, n_requests > n_single ? n_requests - n_single : 1, max_q_len, portion_keys, p.window);
        if (tiles * splits > 0x7fffffffll) return (int)cudaErrorInvalidValue;
        const dim3 grid((unsigned)(tiles * splits), p.nkv * p.head_blocks, n_requests);
        if (splits == 1) return lsb_launch(attention_portion_kernel<T, KT, HDC, AttnParams>, grid, dim3(kThreads), portion_smem<KT>(p.hd), stream, 1, p);
        SplitParams parts;
        static_cast<AttnParams&>(parts) = p;
        parts.splits = splits;
        return launch_clusters(attention_portion_kernel<T, KT, HDC, SplitParams>, grid, portion_smem<KT>(p.hd), (unsigned)splits, parts, stream);
    }
    return 0;
}

// qkv: [tokens, qkv_stride] with the nh*hd query values first in each row.  softcap: 0 for none; slopes: float [nh] or
// null.  n_single: requests that bring one token; max_keys, portion_keys: the longest context, and of those with more tokens (0: not known,
// the launch is captured).
// inv_freq: null, or the rotation of single tokens (float [rotary_dim / 2]), which come unrotated then, keys and values behind the
// queries in their rows; `store`: and not yet in their pages.
LSB_API int lsb_paged_attention_generic(
    const void* qkv, int qkv_stride, const void* k_pages, const void* v_pages,
    const int* q_start, const int* kv_len, const int* table_rows, const int* block_table,
    int table_stride, void* out, int dtype, int n_requests, int max_q_len, int n_single, int max_keys, int portion_keys,
    int nh, int nkv, int hd, int page_size, int num_pages, float scale, int window,
    float softcap, const float* slopes, const float* inv_freq, int rotary_dim, int store, cudaStream_t stream) {
    if (n_requests <= 0 || max_q_len <= 0) return 0;
    if (hd % 16 || hd <= 0 || hd > kMaxHeadDim || nkv <= 0 || nh % nkv) return (int)cudaErrorInvalidValue;
    if (n_requests > 65535 || nh > 65535) return (int)cudaErrorInvalidValue;
    if (inv_freq && (rotary_dim < 0 || rotary_dim > hd || rotary_dim % 2 || qkv_stride < (nh + 2 * nkv) * hd)) return (int)cudaErrorInvalidValue;
    const AttnParams p{qkv, qkv_stride, k_pages, v_pages, q_start, kv_len, table_rows, block_table, table_stride, out,
                       nh, nkv, hd, page_size, num_pages, scale, window, softcap, slopes, 0, 0};
    RotatingParams rot;
    rot.inv_freq = inv_freq;
    rot.rotary_dim = rotary_dim;
    rot.store = store;
    const RotatingParams* rotation = inv_freq ? &rot : nullptr;
    LSB_DISPATCH_DTYPE(dtype, {
        if (hd <= 64) return launch<T, 64, 64>(p, rotation, n_requests, max_q_len, n_single, max_keys, portion_keys, stream);
        if (hd <= 128) return launch<T, 32, 128>(p, rotation, n_requests, max_q_len, n_single, max_keys, portion_keys, stream);
        return launch<T, 32, 256>(p, rotation, n_requests, max_q_len, n_single, max_keys, portion_keys, stream);
    });
    return 0;
}
