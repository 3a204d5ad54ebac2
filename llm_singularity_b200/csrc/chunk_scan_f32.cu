// The recurrence of csrc/linear_scan.cu for a memory whose fade is one fixed number per head,
//
//     S_t = a S_(t-1) + k_t v_t^T          o_t = S_t^T q_t
//
// on prompt portions, in chunks of 64 tokens.  Within a chunk that starts from the state S,
//
//     o_t = a^(t+1) S^T q_t + sum over s <= t of a^(t-s) (q_t . k_s) v_s
//
// and the chunk's end is a^n S + the sum over s of a^(n-1-s) k_s v_s^T.  Three kernels: what each chunk adds to the state
// (gain), the states the chunks start from, one behind the other (in place of the gains), and the outputs.  Everything is
// held, multiplied and added in 32-bit as the walk does it: q, k and v pass their activation (silu or none) as they are
// staged, the powers of a are rounded once from 64-bit.  The sums form in another order than in the walk, with
// fewer roundings one behind the other.
//
// What bounds it is arithmetic on the 32-bit pipes, then the traffic of shared memory: 8 x 8 outputs a thread read 16
// floats for 64 multiply-adds, as many cycles of the one as of the other.  With 64 tokens a chunk the two products with
// the state (N x V a token each) weigh more than the two within the chunk (64 x (N + V), half of them masked and passed
// over).  16 heads of 128 x 128, 1,500 tokens: 88 us (the pipes of multiply-adds half busy; 31 gains, 24 the chain, 61 outputs
// one by one with cold caches) where the walk takes 477; the tensor cores with operands as pairs of bfloat16 numbers
// took 77, with 16 of the operands' 24 digits.
//
// rows: bfloat16 [tokens, ld]; a head's q and k (head h / share) at q_off, k_off and its v at v_off.  The state is [slot,
// head, V, N] 32-bit, N (channels of q and k) contiguous; N and V multiples of 8 up to 128.  gain: scratch of V x N floats
// a head for each chunk, chunk j of request r at q_start[r] / 64 + r + j.
#include "common.cuh"

LSB_DEFINE_STATUS()

typedef __nv_bfloat16 bf16;

constexpr int kL = 64;               // tokens of a chunk

struct ScanArgs {
    const bf16* rows; long long ld;
    int q_off, k_off, v_off;
    int q_silu, k_silu, v_silu;
    int heads, share, N, V;
    const float* log_decay;          // [heads], natural logarithm
    float q_scale;
    float* state; int n_slots;
    const int *q_start, *table_rows;
    float* out;                      // [tokens, heads * V]
    float* gain;
    int parts;                       // blocks that share out a chunk's value columns
};

__device__ __forceinline__ float silu(float z) { return z * __fdividef(1.f, 1.f + __expf(-z)); }
// eight bfloat16 numbers through their activation, times f
__device__ __forceinline__ void act8(const uint4& raw, bool act, float f, float4& lo, float4& hi) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (act ? silu(v[i]) : v[i]) * f;
    lo = make_float4(v[0], v[1], v[2], v[3]);
    hi = make_float4(v[4], v[5], v[6], v[7]);
}
// put(s, c, raw) for every piece of eight values, c .. c + 7 of `wide` in each of n rows at src, four pieces in flight
// a thread
template <int THREADS, typename Put>
__device__ __forceinline__ void each8(const bf16* src, long long ld, int n, int wide, Put put) {
    const int per = wide / 8, total = n * per;
    for (int w0 = threadIdx.x; w0 < total; w0 += 4 * THREADS) {
        uint4 raw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int w = w0 + u * THREADS, s = w / per;
            if (w < total) raw[u] = *reinterpret_cast<const uint4*>(src + (size_t)s * ld + (w - s * per) * 8);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int w = w0 + u * THREADS, s = w / per;
            if (w < total) put(s, (w - s * per) * 8, raw[u]);
        }
    }
}

// a^i (a = 0: 1, then zeros), the exponent formed in 64-bit
__device__ __forceinline__ float power(const ScanArgs& a, int h, int i) {
    const double e = (double)i * ((double)fmaxf(a.log_decay[h], -1000.f) * 1.4426950408889634), whole = rint(e);
    return ldexpf(exp2f((float)(e - whole)), (int)whole);
}

// a block's chunk and its value columns, VP at most
struct Where { int t0, n, v0, cols; size_t row; };
template <int VP>
__device__ __forceinline__ Where place_of(const ScanArgs& a) {
    const int chunk = (int)blockIdx.x / a.parts, q0 = a.q_start[blockIdx.z], q1 = a.q_start[blockIdx.z + 1];
    Where w;
    w.t0 = q0 + chunk * kL;
    w.n = min(kL, q1 - w.t0);
    w.v0 = (int)blockIdx.x % a.parts * VP;
    w.cols = min(VP, a.V - w.v0);
    w.row = (size_t)(q0 / kL + (int)blockIdx.z + chunk);
    return w;
}

// THREADS: 16 columns of threads, so that a thread has VP / (THREADS / 16) rows of the outputs in fours
template <int NP, int VP, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) chunk_gain_f32_kernel(ScanArgs a) {
    constexpr int TY = THREADS / 16, CN = NP / 64, CV = VP / (4 * TY);
    static_assert(CV > 0, "rows for every thread");
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;                                             // [kL][NP], faded to the chunk's end
    float* vs = ks + kL * NP;                                   // [kL][VP]
    __shared__ float pw[kL];
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const Where at = place_of<VP>(a);
    if (at.n <= 0) return;
    const int h = blockIdx.y, hk = h / a.share, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    if (tid < kL) pw[tid] = power(a, h, tid);
    const bf16* row = a.rows + (size_t)at.t0 * a.ld;
    each8<THREADS>(row + a.v_off + h * a.V + at.v0, a.ld, at.n, at.cols, [&](int s, int c, const uint4& raw) {
        float4* to = reinterpret_cast<float4*>(vs + s * VP + c);
        act8(raw, a.v_silu, 1.f, to[0], to[1]);
    });
    __syncthreads();
    each8<THREADS>(row + a.k_off + hk * a.N, a.ld, at.n, a.N, [&](int s, int c, const uint4& raw) {
        float4* to = reinterpret_cast<float4*>(ks + s * NP + c);
        act8(raw, a.k_silu, pw[at.n - 1 - s], to[0], to[1]);
    });
    __syncthreads();
    // rows 4 ty + 4 TY i, columns 4 tx + 64 j, four by four each (places past V and N hold anything and are not stored)
    float acc[4 * CV][4 * CN];
#pragma unroll
    for (int i = 0; i < 4 * CV; ++i)
#pragma unroll
        for (int j = 0; j < 4 * CN; ++j) acc[i][j] = 0.f;
#pragma unroll 4
    for (int s = 0; s < at.n; ++s) {
        float v[4 * CV], k[4 * CN];
#pragma unroll
        for (int i = 0; i < CV; ++i) *reinterpret_cast<float4*>(v + 4 * i) = *reinterpret_cast<const float4*>(vs + s * VP + 4 * ty + 4 * TY * i);
#pragma unroll
        for (int j = 0; j < CN; ++j) *reinterpret_cast<float4*>(k + 4 * j) = *reinterpret_cast<const float4*>(ks + s * NP + 4 * tx + 64 * j);
#pragma unroll
        for (int i = 0; i < 4 * CV; ++i)
#pragma unroll
            for (int j = 0; j < 4 * CN; ++j) acc[i][j] = fmaf(v[i], k[j], acc[i][j]);
    }
    float* dst = a.gain + ((at.row * a.heads + h) * (size_t)a.V + at.v0) * a.N;
#pragma unroll
    for (int i = 0; i < 4 * CV; ++i) {
        const int v = 4 * ty + 4 * TY * (i / 4) + i % 4;
#pragma unroll
        for (int j = 0; j < CN; ++j) {
            const int n = 4 * tx + 64 * j;
            if (v < at.cols && n < a.N)
                *reinterpret_cast<float4*>(dst + (size_t)v * a.N + n) =
                    make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
        }
    }
}

constexpr int kChainThreads = 128;

// AHEAD: chunks whose loads are in flight at once.  A thread's chain is bound by their latency, so 24 where the longest request has more
// than 8 chunks; for fewer 24 loads would be of the last one again, in registers that other blocks then lack (all three kernels, 16
// heads of 128 x 128, us, with 8 / 24: 65 tokens 42.3 / 44.1, 16 requests of 40 68.5 / 81.5, 500 tokens 49.8 / 51.1, 520 52.3 /
// 51.4, 1,000 70.5 / 65.7, 1,500 84.5 / 77.5, 4,000 226 / 202; a ring of 16, each loaded again as it is used, 1,500 81.7).
template <int AHEAD>
__global__ void __launch_bounds__(kChainThreads) chunk_chain_f32_kernel(ScanArgs a) {
    __shared__ float fade[2];                                   // over a whole chunk, and over the request's last
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const int r = blockIdx.z, h = blockIdx.y;
    const int q0 = a.q_start[r], len = a.q_start[r + 1] - q0;
    const int slot = a.table_rows[r];
    if (len <= 0) return;
    const int chunks = (len + kL - 1) / kL;
    if (threadIdx.x < 2) fade[threadIdx.x] = power(a, h, threadIdx.x ? len - (chunks - 1) * kL : kL);
    __syncthreads();
    const bool known = slot >= 0 && slot < a.n_slots;
    if (!known && threadIdx.x == 0) lsb_set_status(LSB_BAD_ROW);
    const size_t per = (size_t)a.V * a.N;
    const size_t i = ((size_t)blockIdx.x * kChainThreads + threadIdx.x) * 4;
    if (i >= per) return;
    // (a request without a slot starts from zero and leaves nothing)
    float* st = a.state + ((size_t)(known ? slot : 0) * a.heads + h) * per + i;
    float4 cur = known ? *reinterpret_cast<const float4*>(st) : make_float4(0.f, 0.f, 0.f, 0.f);
    float* at = a.gain + ((size_t)(q0 / kL + r) * a.heads + h) * per + i;
    const size_t step = (size_t)a.heads * per;
    for (int s0 = 0; s0 < chunks; s0 += AHEAD) {
        float4 e[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) e[k] = *reinterpret_cast<const float4*>(at + min(s0 + k, chunks - 1) * step);
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (s0 + k < chunks) {
                *reinterpret_cast<float4*>(at + (s0 + k) * step) = cur;
                const float f = fade[s0 + k == chunks - 1];
                cur.x = fmaf(f, cur.x, e[k].x);
                cur.y = fmaf(f, cur.y, e[k].y);
                cur.z = fmaf(f, cur.z, e[k].z);
                cur.w = fmaf(f, cur.w, e[k].w);
            }
        }
    }
    if (known) *reinterpret_cast<float4*>(st) = cur;
}

constexpr int kSlab = 32;            // channels of the state staged at a time, two slabs by turns
constexpr int kKeys = 64;            // channels of the keys staged at a time, two slabs

// Three blocks an SM: queries (values in their place at the end), and two regions that hold slabs of the state, then
// the keys, then (the first) the scores.
template <int NP, int VP>
struct OutLayout {
    static constexpr int LDQ = NP + 4, LDP = kL + 4, LDS = kSlab + 4, LDK = kKeys + 4;    // eight neighbouring rows in eight sets of banks
    static constexpr int kQ = kL * LDQ > kL * VP ? kL * LDQ : kL * VP;
    static constexpr int kRegion = VP * LDS > kL * LDK ? VP * LDS : kL * LDK;
    static_assert(LDP == LDK, "scores take the place of keys");
    static constexpr size_t kTotal = (size_t)(kQ + 2 * kRegion) * 4;
};
__device__ __forceinline__ void copy16(float* to, const float* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}

template <int NP, int VP, int THREADS>
__global__ void __launch_bounds__(THREADS, 3) chunk_output_f32_kernel(ScanArgs a) {
    using L = OutLayout<NP, VP>;
    constexpr int TY = THREADS / 16, R = kL / TY, CV = VP / 64;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                             // [kL][LDQ], at the end the values [kL][VP]
    float* regions = qs + L::kQ;
    __shared__ float pw[kL + 1];
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const Where at = place_of<VP>(a);
    if (at.n <= 0) return;
    const int h = blockIdx.y, hk = h / a.share, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const bf16* row = a.rows + (size_t)at.t0 * a.ld;
    const float* start = a.gain + ((at.row * a.heads + h) * (size_t)a.V + at.v0) * a.N;
    const int slabs = (a.N + kSlab - 1) / kSlab;
    auto copy_slab = [&](int i) {
        if (i < slabs) {
            const int n0 = i * kSlab, per = min(kSlab, a.N - n0) / 4;
            for (int w = tid; w < at.cols * per; w += THREADS) {
                const int v = w / per, c = (w - v * per) * 4;
                // a thread's columns lie sixteen places apart, those of neighbouring threads side by side
                const int place = (v / 64 * 4 + v % 4) * 16 + v / 4 % 16;
                copy16(regions + (i & 1) * L::kRegion + place * L::LDS + c, start + (size_t)v * a.N + n0 + c);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_slab(0);
    copy_slab(1);
    if (tid <= kL) pw[tid] = power(a, h, tid);
    each8<THREADS>(row + a.q_off + hk * a.N, a.ld, at.n, a.N, [&](int s, int c, const uint4& raw) {
        float4* to = reinterpret_cast<float4*>(qs + s * L::LDQ + c);
        act8(raw, a.q_silu, a.q_scale, to[0], to[1]);
    });
    // outputs: tokens ty + TY i, columns 4 tx + 64 c, four each (rows past the chunk's end hold anything and are not stored)
    float acc[R][4 * CV];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < 4 * CV; ++c) acc[i][c] = 0.f;
    for (int slab = 0; slab < slabs; ++slab) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int n0 = slab * kSlab, wide = min(kSlab, a.N - n0);
        const float* st = regions + (slab & 1) * L::kRegion + tx * L::LDS;
        for (int n = 0; n < wide; n += 4) {
            float4 q[R];
#pragma unroll
            for (int i = 0; i < R; ++i) q[i] = *reinterpret_cast<const float4*>(qs + (ty + TY * i) * L::LDQ + n0 + n);
#pragma unroll
            for (int c = 0; c < 4 * CV; ++c) {
                const float4 s = *reinterpret_cast<const float4*>(st + c * 16 * L::LDS + n);
#pragma unroll
                for (int i = 0; i < R; ++i) acc[i][c] = fmaf(q[i].x, s.x, acc[i][c]);
#pragma unroll
                for (int i = 0; i < R; ++i) acc[i][c] = fmaf(q[i].y, s.y, acc[i][c]);
#pragma unroll
                for (int i = 0; i < R; ++i) acc[i][c] = fmaf(q[i].z, s.z, acc[i][c]);
#pragma unroll
                for (int i = 0; i < R; ++i) acc[i][c] = fmaf(q[i].w, s.w, acc[i][c]);
            }
        }
        __syncthreads();                                        // (the slab has been used)
        copy_slab(slab + 2);
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < 4 * CV; ++c) acc[i][c] *= pw[ty + TY * i + 1];
    each8<THREADS>(row + a.k_off + hk * a.N, a.ld, at.n, a.N, [&](int s, int c, const uint4& raw) {
        float4* to = reinterpret_cast<float4*>(regions + c / kKeys * L::kRegion + s * L::LDK + c % kKeys);
        act8(raw, a.k_silu, 1.f, to[0], to[1]);
    });
    __syncthreads();
    float score[R][4];                                          // tokens ty + TY i against tokens tx + 16 j
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) score[i][j] = 0.f;
    for (int n = 0; n < a.N; n += 4) {
        const float* keys = regions + n / kKeys * L::kRegion + tx * L::LDK + n % kKeys;
        float4 q[R];
#pragma unroll
        for (int i = 0; i < R; ++i) q[i] = *reinterpret_cast<const float4*>(qs + (ty + TY * i) * L::LDQ + n);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 k = *reinterpret_cast<const float4*>(keys + 16 * j * L::LDK);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (TY * i + TY > 16 * j) score[i][j] = fmaf(q[i].x, k.x, score[i][j]);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (TY * i + TY > 16 * j) score[i][j] = fmaf(q[i].y, k.y, score[i][j]);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (TY * i + TY > 16 * j) score[i][j] = fmaf(q[i].z, k.z, score[i][j]);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (TY * i + TY > 16 * j) score[i][j] = fmaf(q[i].w, k.w, score[i][j]);
        }
    }
    __syncthreads();
    float* ps = regions;                                      // [kL][LDP]
    float* vs = qs;                                             // [kL][VP]
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int t = ty + TY * i, s = tx + 16 * j;
            ps[t * L::LDP + s] = s <= t ? score[i][j] * pw[t - s] : 0.f;      // (only s <= t < n is used)
        }
    const int fours = (at.n + 3) & ~3;                          // (zeros past the chunk's end, as far as the sums go)
    float zero = 0.f;                                           // times a number 0, times anything else NaN
    each8<THREADS>(row + a.v_off + h * a.V + at.v0, a.ld, at.n, at.cols, [&](int s, int c, const uint4& raw) {
        float4 lo, hi;
        act8(raw, a.v_silu, 1.f, lo, hi);
        zero = fmaf(lo.x, zero, fmaf(lo.y, zero, fmaf(lo.z, zero, lo.w * zero)));
        zero = fmaf(hi.x, zero, fmaf(hi.y, zero, fmaf(hi.z, zero, hi.w * zero)));
        float4* to = reinterpret_cast<float4*>(vs + s * VP + c);
        to[0] = lo;
        to[1] = hi;
    });
    for (int w = at.n * VP + tid; w < fours * VP; w += THREADS) vs[w] = 0.f;
    if (__syncthreads_or(!(zero == 0.f))) {
        // an infinity or NaN among the values: a token takes in only its own past (0 times such a value is none)
        for (int s = 0; s < at.n; ++s) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if (s > ty + TY * i) continue;
                const float p = ps[(ty + TY * i) * L::LDP + s];
#pragma unroll
                for (int c = 0; c < 4 * CV; ++c) acc[i][c] = fmaf(p, vs[s * VP + 4 * tx + 64 * (c / 4) + c % 4], acc[i][c]);
            }
        }
    } else {
        for (int s = 0; s < fours; s += 4) {
            // (rows that lie wholly before s see none of it: their p's are zeros)
            float p[R][4];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (s < TY * i + TY) *reinterpret_cast<float4*>(p[i]) = *reinterpret_cast<const float4*>(ps + (ty + TY * i) * L::LDP + s);
#pragma unroll
            for (int c = 0; c < CV; ++c) {
                float4 v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(vs + (s + e) * VP + 4 * tx + 64 * c);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (s >= TY * i + TY) continue;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        acc[i][4 * c] = fmaf(p[i][e], v[e].x, acc[i][4 * c]);
                        acc[i][4 * c + 1] = fmaf(p[i][e], v[e].y, acc[i][4 * c + 1]);
                        acc[i][4 * c + 2] = fmaf(p[i][e], v[e].z, acc[i][4 * c + 2]);
                        acc[i][4 * c + 3] = fmaf(p[i][e], v[e].w, acc[i][4 * c + 3]);
                    }
                }
            }
        }
    }
    const size_t ldo = (size_t)a.heads * a.V;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (ty + TY * i >= at.n) continue;
#pragma unroll
        for (int c = 0; c < CV; ++c) {
            const int v = 4 * tx + 64 * c;
            if (v < at.cols)
                *reinterpret_cast<float4*>(a.out + (size_t)(at.t0 + ty + TY * i) * ldo + (size_t)h * a.V + at.v0 + v) =
                    make_float4(acc[i][4 * c], acc[i][4 * c + 1], acc[i][4 * c + 2], acc[i][4 * c + 3]);
        }
    }
}

// SMs of the current device (asked once per device).
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

constexpr int kOutThreads = 128;

template <int NP, int VP, int GAIN>
static int run(ScanArgs a, int n_requests, int chunks, cudaStream_t stream) {
    constexpr size_t gain_sm = (size_t)kL * (NP + VP) * 4, out_sm = OutLayout<NP, VP>::kTotal;
    static int configured = -1;
    if (configured < 0) {
        configured = (int)cudaFuncSetAttribute(chunk_gain_f32_kernel<NP, VP, GAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gain_sm);
        if (!configured)
            configured = (int)cudaFuncSetAttribute(chunk_output_f32_kernel<NP, VP, kOutThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_sm);
    }
    if (configured) return configured;
    a.parts = (a.V + VP - 1) / VP;
    const dim3 grid(chunks * a.parts, a.heads, n_requests);
    int rc = lsb_launch(chunk_gain_f32_kernel<NP, VP, GAIN>, grid, dim3(GAIN), gain_sm, stream, 1, a);
    if (rc) return rc;
    const int per = a.V * a.N / 4;
    rc = lsb_launch(chunks > 8 ? chunk_chain_f32_kernel<24> : chunk_chain_f32_kernel<8>,
                    dim3((per + kChainThreads - 1) / kChainThreads, a.heads, n_requests), dim3(kChainThreads), 0, stream, 1, a);
    if (rc) return rc;
    return lsb_launch(chunk_output_f32_kernel<NP, VP, kOutThreads>, grid, dim3(kOutThreads), out_sm, stream, 1, a);
}

LSB_API int lsb_chunk_f32_tokens() { return kL; }

// silu: 1 for queries + 2 for keys + 4 for values that pass it on the way in.  gain: scratch of (tokens / 64 + requests)
// x heads x V x N floats.  q_start and table_rows begin at the first request to be run.
LSB_API int lsb_chunk_scan_f32(const void* rows, long long ld, int q_off, int k_off, int v_off, int heads, int key_heads, int N, int V,
                               const float* log_decay, float q_scale, int silu, float* state, int n_slots, const int* q_start,
                               const int* table_rows, int n_requests, int max_q_len, float* out, float* gain, cudaStream_t stream) {
    if (n_requests <= 0 || max_q_len <= 0) return 0;
    if (N <= 0 || V <= 0 || N % 8 || V % 8 || N > 128 || V > 128 || heads <= 0 || key_heads <= 0 || heads % key_heads || heads > 65535 ||
        n_requests > 65535 || silu < 0 || silu > 7 || !log_decay || !gain)
        return (int)cudaErrorInvalidValue;
    if ((uintptr_t)rows % 16 || ld % 8 || q_off % 8 || k_off % 8 || v_off % 8 || (uintptr_t)state % 16 || (uintptr_t)gain % 16 ||
        (uintptr_t)out % 16)
        return (int)cudaErrorInvalidValue;
    ScanArgs a;
    a.rows = (const bf16*)rows; a.ld = ld;
    a.q_off = q_off; a.k_off = k_off; a.v_off = v_off;
    a.q_silu = silu & 1; a.k_silu = silu & 2; a.v_silu = silu & 4;
    a.heads = heads; a.share = heads / key_heads; a.N = N; a.V = V;
    a.log_decay = log_decay; a.q_scale = q_scale;
    a.state = state; a.n_slots = n_slots; a.q_start = q_start; a.table_rows = table_rows;
    a.out = out; a.gain = gain;
    const int chunks = (max_q_len + kL - 1) / kL;
    // A block of 128 value columns has 8 x 8 outputs a thread and its scores once; 64 columns make twice the blocks, each
    // half as long, which is the better where not every SM has one (16 heads of 128 x 128, us: 48 tokens 59 and 31, 500
    // 68 and 52, 1,000 75 and 84, 1,500 88 and 101).
    const bool wide = V > 64 && (long long)chunks * heads * n_requests > num_sms();
    if (N <= 64) return wide ? run<64, 128, 256>(a, n_requests, chunks, stream) : run<64, 64, 128>(a, n_requests, chunks, stream);
    return wide ? run<128, 128, 256>(a, n_requests, chunks, stream) : run<128, 64, 128>(a, n_requests, chunks, stream);
}
