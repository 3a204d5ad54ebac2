// out[M, N] = x[M, K] * w[N, K]^T of 32-bit values with 32-bit sums, no bit of an operand that could show in one dropped.
// Three kernels, by the number of rows and K; K a multiple of 4 and 16-byte aligned bases (anything else is csrc/gemm.cu's).  An activation of
// a gated product (w's rows alternate gate_i, up_i, out is [M, N / 2]) is applied where the sums meet.  The reference
// hands such products to cublasSgemm (kernels/src/cublas_provider.cpp:36-51) and launches silu(g) * u by itself
// (kernels/src/activations.cu:11-21).
//
// * Up to 16 rows (a decode step) the product is weight traffic.  Weight rows are dealt out over one
//   block per SM, sixteen at most at a time: four to a warp, each row's K in two parts.  A warp copies the weights it
//   needs into a ring of shared memory itself (asynchronously, some 140 KB in flight an SM, the first of them asked for
//   in L2 before the wait on the kernel before, which may be the one that makes w) and shares the rows of x with the three
//   others of its part.  The sums of a group meet once, over lanes by halving exchanges and over the two parts in shared
//   memory, in a fixed order.
//   The four products of a layer at 1B sizes, 8 rows (243 MB): 58 us (4.2 TB/s); as 64 x 64 tiles, 56 of their 64 rows
//   empty and as few as 32 of them: 1,202 us.  (A thread's places of K for all sixteen rows, with no sharing at all, cost
//   four times the exchanges at the end of a group: 89 us.)
//
// * More rows (a prompt), K from 512: the tensor cores.  A 32-bit value is exactly the sum of three bfloat16 values (8
//   bits each of its 24), so a product is nine products of parts; the six that reach 2^-23 of it are taken, the other three
//   are not.  Blocks of 128 x 128 outputs, or 128 x 64 (split_plan, below, has the choice), take x and w as they are by
//   TMA; sixteen warps, two groups by turns, split a stage of 32 along K, x's parts into tensor memory, w's into
//   shared memory.  The tensor core cuts its sums rather than rounding them, so the leading products stay there for
//   128 of K only and are then added up in registers; the five small ones have their own sums, 2^-8 as large.  Where tiles
//   are too few for the SMs, or leave a last round of them half empty, K is shared out over a cluster, whose sums meet in order.
//   Error against 64 bits, 500 x 2,048 x 2,048: 1.4e-7 of the norm, 4.1e-7 by multiply-adds; K = 512 1.3e-7 and 1.6e-7;
//   K = 8,192 1.7e-7 and 8.1e-7 (at K of 100 and 256 the two are alike, which is where the line comes from).  The four
//   products of a layer at 1B sizes, 500 rows (61 GFLOP): 1,491 us by multiply-adds, 470 with all of K a block, 372 so.  What bounds it is the traffic of
//   shared memory and the chain of a stage: 0.66 us where its products take 0.4 (both operands in shared
//   memory: 0.9; one group of eight warps besides: 1.05).  Sums that values which bfloat16 cannot split (infinities, NaN,
//   numbers below 2^-103) could show in and sums that leave the range are done over by multiply-adds at the end, so that
//   they come out as there.
//
// * More rows, smaller K: multiply-adds on the 32-bit pipes.  Eight warps of 64 x 64 outputs (8 x 16 a thread), arranged
//   as a tile of 128 x 256, 128 x 128, 64 x 128 or 64 x 64; in the smaller tiles the warps that are left share out each
//   slice of K and their sums meet at the end, so that few tiles still give an SM eight busy warps.  Slices come by
//   asynchronous copies, three to five in flight.  2,048 x 8,192 x 256: 200 us, 43 TFLOP/s of the 70 that a loop of
//   nothing but multiply-adds reaches here.
//
// A row's sum is taken in an order that is the same from run to run.  M, N and K fix it: which kernel, into how many parts K is cut
// for which of the tiles; so the last digits depend on the number of rows beside a row and, where whole tiles and shared-out
// ones make up one product, on where in it a sum lies.
#include "common.cuh"
#include "gate_act.cuh"

#include <cooperative_groups.h>
#include <cuda.h>

#include <type_traits>

namespace cg = cooperative_groups;

LSB_DEFINE_STATUS()

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// 16 bytes from global to shared memory, zeros where `have` is false (nothing is read then)
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool have) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------ a few rows
constexpr int kRowThreads = 256;
constexpr int kRowsMax = 16;                   // rows of x a block takes
constexpr int kRB = 16;                        // most weight rows of a group: four for each of four warps, twice (two parts of K)
constexpr int kRW = kRB / 4;
// More rows that still go this way, sixteen to a block, where the matrix is so small that a tile's latency shows: up to some
// 48 of them are faster so (us, this way and as tiles of 64 x 64: 17 x 640 x 128 4.9 and 5.7, 48 x 128 x 320 7.5 and 11.3), 64 to
// 128 only along a longer K (64 x 128 x 320 9.7 and 11.5, 128 x 512 x 128 17.0 and 6.1), but the sums are
// the closer ones throughout: K = 128 7.4e-8 of the norm and 9.7e-8, K = 320 8.2e-8 and 1.3e-7.
constexpr int kRowsSmall = 128;
constexpr long long kSmallMatrix = 1 << 18;
constexpr int kKS = 512;                       // K of a stage: two steps of 128 for each part

struct RowsParams {
    const float* x;
    const float* w;
    float* out;
    int M, N, K;
    int per;                                   // weight rows of a group (even for a gated product)
    int groups;
    int act;                                   // of a gated product (0: plain)
};

// MT: rows of x (rounded up), ST: stages of the ring.  Rows 16 blockIdx.y .. of x.
template <int MT, int ST>
__global__ void __launch_bounds__(kRowThreads, 1) gemm_rows_f32_kernel(const RowsParams p) {
    constexpr int V = kRW * MT;                // sums of a thread
    extern __shared__ __align__(16) float ring[];             // [ST][kRB + MT][kKS]
    __shared__ float red[2][2][4][V];          // [by turns][part of K][rows' warp]
    lsb_pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, kg = (tid >> 5) & 1, rg = tid >> 6;
    const int M = min(kRowsMax, p.M - (int)blockIdx.y * kRowsMax);
    const float* x = p.x + (size_t)blockIdx.y * kRowsMax * p.K;
    const int n_out = p.act ? p.N / 2 : p.N;
    float* out = p.out + (size_t)blockIdx.y * kRowsMax * n_out;
    const int chunks = (p.K + kKS - 1) / kKS;
    const int mine = (p.groups - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
    const int total = mine * chunks;
    const int at = kg * 128 + lane * 4;        // this thread's place in a step of 256
    const uint32_t base = smem_u32(ring) + (uint32_t)at * 4u;

    constexpr uint32_t kStage = (kRB + MT) * kKS * 4u;
    // The copies' place, carried along: group, chunk of K and bytes into the ring.  (Found anew for each stage by dividing, and every
    // copy guarded, 16,384 x 2,048 gated took 28.0 us where it takes 23.0 with four rows, 33.7 and 28.3 with eight, 48.9 and 42.2 with
    // twelve; 512 x 2,048 of twelve rows, whose x is copied guarded all the same, 6.9 and 7.0.)
    int to_g = (int)blockIdx.x, to_chunk = 0;
    uint32_t to = 0;
    auto copy_stage = [&]() {
        const int k0 = to_chunk * kKS + at, n0 = to_g * p.per, rows = min(p.per, p.N - n0);
        const float* src = p.w + (size_t)(n0 + rg * kRW) * p.K + k0;
        const float* xs = x + (size_t)rg * p.K + k0;
        const uint32_t st = base + to + (uint32_t)(rg * kRW) * kKS * 4u, sx = base + to + (uint32_t)(kRB + rg) * kKS * 4u;
        const bool whole = to_chunk * kKS + kKS <= p.K;
        if (whole && rg * kRW + kRW <= rows) {
#pragma unroll
            for (int i = 0; i < kRW; ++i, src += p.K) {
                copy16(st + (uint32_t)i * kKS * 4u, src);
                copy16(st + (uint32_t)(i * kKS + 256) * 4u, src + 256);
            }
        } else {
#pragma unroll
            for (int i = 0; i < kRW; ++i, src += p.K) {
                if (rg * kRW + i >= rows) break;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const bool in = k0 + 256 * j < p.K;
                    copy16(st + (uint32_t)(i * kKS + 256 * j) * 4u, in ? src + 256 * j : p.w, in);
                }
            }
        }
        if (whole && M == MT) {
#pragma unroll
            for (int m = 0; m < MT; m += 4, xs += 4 * (size_t)p.K) {
                if (MT < 4 && rg >= MT) break;
                copy16(sx + (uint32_t)m * kKS * 4u, xs);
                copy16(sx + (uint32_t)(m * kKS + 256) * 4u, xs + 256);
            }
        } else {
#pragma unroll
            for (int m = 0; m < MT; m += 4, xs += 4 * (size_t)p.K) {
                if (MT < 4 && rg >= MT) break;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const bool have = rg + m < M && k0 + 256 * j < p.K;
                    copy16(sx + (uint32_t)(m * kKS + 256 * j) * 4u, have ? xs + 256 * j : p.x, have);
                }
            }
        }
        to = to + kStage == ST * kStage ? 0 : to + kStage;
        if (++to_chunk == chunks) { to_chunk = 0; to_g += (int)gridDim.x; }
    };
    auto warm_w = [&](int it) {                // (a lane's 16 bytes are an eighth of a line)
        const int g = (int)blockIdx.x + (it / chunks) * (int)gridDim.x, k0 = it % chunks * kKS + at;
        const int n0 = g * p.per, rows = min(p.per, p.N - n0);
        if (lane & 7) return;
        for (int r = rg * kRW; r < min(rows, rg * kRW + kRW); ++r)
            for (int k = k0; k < min(p.K, k0 + kKS); k += 256)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + (size_t)(n0 + r) * p.K + k));
    };
    // w may be what the kernel before has yet to write: ahead of the wait its first lines are only asked for (L2, where
    // writes go too), and read behind it
    for (int it = 0; it < ST - 1 && it < total; ++it) warm_w(it);
    lsb_pdl_wait();
    for (int it = 0; it < ST - 1; ++it) {
        if (it < total) copy_stage();
        copies_commit();
    }
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.f;
    int chunk = 0, done = 0;
    const float* st = ring + at;
    for (int it = 0; it < total; ++it) {
        copies_wait<ST - 2>();
        // the four warps of this part of K share the rows of x; past this point none still reads the stage before
        asm volatile("bar.sync %0, 128;" ::"r"(1 + kg) : "memory");
        if (it + ST - 1 < total) copy_stage();
        copies_commit();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (chunk * kKS + kg * 128 + 256 * j >= p.K) break;       // (the warp's whole step lies past K)
            float4 wv[kRW];
#pragma unroll
            for (int i = 0; i < kRW; ++i)           // (what stands in rows the group does not have goes into sums of their own)
                wv[i] = *reinterpret_cast<const float4*>(st + (rg * kRW + i) * kKS + 256 * j);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 xv = *reinterpret_cast<const float4*>(st + (kRB + m) * kKS + 256 * j);
#pragma unroll
                for (int i = 0; i < kRW; ++i) {
                    float a = acc[i * MT + m];
                    a = fmaf(wv[i].x, xv.x, a); a = fmaf(wv[i].y, xv.y, a);
                    a = fmaf(wv[i].z, xv.z, a); a = fmaf(wv[i].w, xv.w, a);
                    acc[i * MT + m] = a;
                }
            }
        }
        st = st + kStage / 4 == ring + at + ST * (kStage / 4) ? ring + at : st + kStage / 4;
        if (++chunk < chunks) continue;
        const int n0 = ((int)blockIdx.x + done * (int)gridDim.x) * p.per, rows = min(p.per, p.N - n0);
        // the group's sums: lanes exchange halves until each holds V / 32 of them (or one, by several lanes) ...
        int n = V, first = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if (n > 1) {
                n /= 2;
                const bool upper = lane & o;
                if (upper) first += n;
#pragma unroll
                for (int v = 0; v < V / 2; ++v) {
                    if (v < n) {
                        const float send = upper ? acc[v] : acc[v + n], keep = upper ? acc[v + n] : acc[v];
                        acc[v] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
            } else {
                acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            }
        }
        // ... and the two parts of K
        float(*part)[4][V] = red[done & 1];
#pragma unroll
        for (int v = 0; v < (V >= 32 ? V / 32 : 1); ++v) part[kg][rg][first + v] = acc[v];
        __syncthreads();
        for (int v = tid; v < kRB * MT; v += kRowThreads) {
            const int r = v / MT, m = v % MT, at_r = r % kRW * MT + m;
            if (r >= rows || m >= M || (p.act && (r & 1))) continue;
            const float s = part[0][r / kRW][at_r] + part[1][r / kRW][at_r];
            if (p.act) {
                const float up = part[0][r / kRW][at_r + MT] + part[1][r / kRW][at_r + MT];
                out[(size_t)m * n_out + ((n0 + r) >> 1)] = lsb_gated(s, up, p.act, 0.f);
            } else {
                out[(size_t)m * n_out + n0 + r] = s;
            }
        }
        chunk = 0;
        ++done;
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = 0.f;
    }
}

// ------------------------------------------------------------------ more rows
struct TileParams {
    const float* x;
    const float* w;
    float* out;
    int M, N, K, act;
};

// outputs (m, n .. n + 3), as far as n goes, or what the gated product makes of them (N is even then)
__device__ __forceinline__ void store_four(const TileParams& p, long long m, long long n, float4 v) {
    const bool wide = (p.N & 3) == 0;
    if (p.act) {
        float* d = p.out + m * (p.N / 2) + n / 2;
        const float first = lsb_gated(v.x, v.y, p.act, 0.f);
        if (wide) *reinterpret_cast<float2*>(d) = make_float2(first, lsb_gated(v.z, v.w, p.act, 0.f));
        else {
            d[0] = first;
            if (n + 2 < p.N) d[1] = lsb_gated(v.z, v.w, p.act, 0.f);
        }
        return;
    }
    float* d = p.out + m * p.N + n;
    if (wide) *reinterpret_cast<float4*>(d) = v;
    else {
        d[0] = v.x;
        if (n + 1 < p.N) d[1] = v.y;
        if (n + 2 < p.N) d[2] = v.z;
        if (n + 3 < p.N) d[3] = v.w;
    }
}
__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
    float s = 0.f;
    for (int k = 0; k < K; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
    }
    return s;
}

constexpr int kTileThreads = 256;

// WM x WN warps of 64 x 64 outputs, WK of them on the same outputs with a part of each slice of BK; ST slices in flight
template <int WM, int WN, int WK, int BK, int ST>
struct TileLayout {
    static_assert(WM * WN * WK == 8 && BK % (4 * WK) == 0 && BK % 32 == 0, "eight warps, whole 16-byte pieces of K each");
    static constexpr int BM = 64 * WM, BN = 64 * WN;
    static constexpr int LD = BK + 4;                                 // floats of a row: eight neighbours in eight sets of banks
    static constexpr int kStage = (BM + BN) * LD;
    static constexpr size_t kEnd = (size_t)WK * BM * (BN + 4) * 4;    // the warps' sums, where they meet
    static constexpr size_t kTotal = (size_t)ST * kStage * 4 > kEnd ? (size_t)ST * kStage * 4 : kEnd;
};

template <int WM, int WN, int WK, int BK, int ST>
__global__ void __launch_bounds__(kTileThreads, 1) gemm_tile_f32_kernel(const TileParams p) {
    using L = TileLayout<WM, WN, WK, BK, ST>;
    constexpr int BM = L::BM, BN = L::BN, LD = L::LD;
    constexpr int kRowPieces = BK / 4;                                // 16-byte pieces of a row
    constexpr int kPieces = (BM + BN) * kRowPieces / kTileThreads;
    static_assert((BM + BN) * kRowPieces % kTileThreads == 0 && kTileThreads % kRowPieces == 0, "every piece has a thread");
    extern __shared__ __align__(16) float smem[];
    lsb_pdl_launch_dependents();
    lsb_pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wn = warp / WM % WN, wk = warp / (WM * WN);
    const int lm = lane >> 2, ln = lane & 3;
    const long long m0 = (long long)blockIdx.y * BM, n0 = (long long)blockIdx.x * BN;

    auto copy = [&](int s) {
        const uint32_t st = smem_u32(smem + (s % ST) * L::kStage);
        const int piece = tid % kRowPieces, k = s * BK + piece * 4;
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
            const int row = tid / kRowPieces + j * (kTileThreads / kRowPieces);
            const bool of_x = row < BM;
            const long long r = of_x ? m0 + row : n0 + row - BM;
            const bool have = k < p.K && r < (of_x ? p.M : p.N);
            copy16(st + (uint32_t)(row * LD + piece * 4) * 4u, have ? (of_x ? p.x : p.w) + r * p.K + k : p.x, have);
        }
    };
    // 8 rows (lm, 8 apart) by 16 columns (ln, 4 apart) a thread.  Shared memory gives a warp 128 bytes a cycle
    // whatever is broadcast: 24 floats for 128 multiply-adds keep it at three quarters of the multiply-add pipe's
    // time; 8 x 8 outputs would take as long there as the arithmetic.
    float acc[8][16];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[i][j] = 0.f;
    const int slices = (p.K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < slices) copy(s);
        copies_commit();
    }
    for (int s = 0; s < slices; ++s) {
        copies_wait<ST - 2>();
        __syncthreads();                                              // (nobody still reads the slice before this one)
        if (s + ST - 1 < slices) copy(s + ST - 1);
        copies_commit();
        const float* st = smem + (s % ST) * L::kStage + wk * (BK / WK);
        const float* a0 = st + (wm * 64 + lm) * LD;
        const float* b0 = st + (BM + wn * 64 + ln) * LD;
#pragma unroll
        for (int k = 0; k < BK / WK; k += 4) {
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + 8 * i * LD + k);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float4 b = *reinterpret_cast<const float4*>(b0 + 4 * j * LD + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
            }
        }
    }
    copies_wait<0>();
    __syncthreads();
    // the tile (every warp group's sums) through shared memory, so that whole rows leave
    constexpr int LDT = BN + 4;
    float* tile = smem + (size_t)wk * BM * LDT + (wm * 64 + lm) * LDT + wn * 64 + ln;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) tile[8 * i * LDT + 4 * j] = acc[i][j];
    __syncthreads();
    for (int q = tid; q < BM * BN / 4; q += kTileThreads) {
        const int row = q / (BN / 4), col = q % (BN / 4) * 4;
        float4 v = *reinterpret_cast<const float4*>(smem + row * LDT + col);
#pragma unroll
        for (int w = 1; w < WK; ++w) {
            const float4 o = *reinterpret_cast<const float4*>(smem + (size_t)w * BM * LDT + row * LDT + col);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        const long long m = m0 + row, n = n0 + col;
        if (m >= p.M || n >= p.N) continue;
        store_four(p, m, n, v);
    }
}

// ------------------------------------------------------------------ many rows, on the tensor cores
constexpr int kSplitK = 512;                   // K from which on the split sums are the more exact ones
constexpr int kSM = 128;                       // rows of x of a tile (tensor memory lanes)
constexpr int kSK = 32;                        // K of a stage: 128 bytes of a 32-bit row, 64 of a plane's
constexpr int kSPlanes = 3;
constexpr int kSGroup = 256;                   // eight warps: a row of x or w each thread of a stage
constexpr int kSWorkers = 2 * kSGroup;         // ... and as many for the stage after it
constexpr int kSThreads = kSWorkers + 64;      // ... one warp for the copies, one for the products
constexpr int kSChunk = 4;                     // stages (K = 128) whose leading products meet in tensor memory
constexpr int kSSplits = 8;                    // most blocks of a cluster along K (the portable size)
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// false if the limit ran out or another role gave up
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if ((it & 255u) == 255u) {
            if (*abort_flag) return false;
            __nanosleep(128);
        }
    }
    *abort_flag = 1;
    lsb_set_status(LSB_WAIT_TIMEOUT);
    return false;
}
__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int k, int row) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(k), "r"(row) : "memory");
}
// (the operand of x lies in tensor memory too)
__device__ __forceinline__ void umma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// sums += N columns of tensor memory, one row a lane
template <int N>
__device__ __forceinline__ void tmem_add(uint32_t addr, float (&sums)[N]) {
    static_assert(N == 16 || N == 32, "one load");
    uint32_t r[N];
    if constexpr (N == 32)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                     "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                     "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                       "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                       "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                     : "r"(addr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(addr));
#pragma unroll
    for (int i = 0; i < N; ++i) sums[i] += __uint_as_float(r[i]);
}
// eight columns of tensor memory, one row a lane
__device__ __forceinline__ void tmem_put(uint32_t addr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// A plane of w: rows of 64 bytes with the 64-byte swizzle (16-byte piece j of row r at j ^ (r / 2 & 3)), groups of
// eight rows 512 bytes apart; layout type 4.
__device__ __forceinline__ uint64_t plane_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// Two values as sums of three bfloat16 values: what a rounding leaves is exact, and the third is all that 24 bits leave.
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(b), "f"(a));
    a -= __uint_as_float(m << 16);
    b -= __uint_as_float(m & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(b), "f"(a));
}

// (a number's magnitude as an integer, zeros the largest of all)
__device__ __forceinline__ uint32_t twice_less_one(float v) { return 2u * __float_as_uint(v) - 1u; }
constexpr uint32_t kTiny = 2u * ((127u - 103u) << 23) - 1u;            // of 2^-103

template <int BN>
struct SplitLayout {
    static constexpr int kRows = kSM + BN;
    static constexpr int kRaw = kRows * kSK * 4, kPlane = BN * kSK * 2, kSplit = kSPlanes * kPlane;
    static constexpr int kRing = BN == 128 ? 5 : 6;
    // columns of tensor memory: two chunks' leading sums, the small products', and x's planes of two stages
    static constexpr int kSmall = 2 * BN, kX = 3 * BN, kXPlane = kSK / 2, kXSplit = kSPlanes * kXPlane;
    static_assert(kX + 2 * kXSplit <= 512, "tensor memory");
    static constexpr int LDT = BN + 4;
    static constexpr size_t kTotal = 1024 + (size_t)kRing * kRaw + 2 * kSplit;
    static_assert(kSM * LDT * 4 <= kRing * kRaw, "the sums leave through the ring");
};

// A launch of clusters along K, or of some of a matrix's tiles.
struct PartParams : TileParams {
    int steps;                                 // stages of K a block takes
    int tiles_m, tiles_n, tile0;               // tiles of the matrix, and the first of this launch
};
// Tiles that run side by side share w (rows of tiles first), which is the larger operand then; else x.
template <int BN>
__host__ __device__ __forceinline__ bool rows_first(int M, int N) { return M <= N && (N + BN - 1) / BN <= 65535; }

// P: TileParams (a block for all of K of every tile) or PartParams.  (As one kernel, whole products of a short K took 0.6 us
// a round more: 640 x 2,048 x 512 17.7 -> 18.4 us, 2,000 x 2,048 x 512 34.4 -> 35.9.)
template <int BN, typename P>
__global__ void __launch_bounds__(kSThreads, 1)
gemm_split_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const P p) {
    constexpr bool PARTS = std::is_same<P, PartParams>::value;
    using L = SplitLayout<BN>;
    constexpr int R = L::kRing;
    extern __shared__ unsigned char raw_smem[];
    unsigned char* ring = (unsigned char*)(((uintptr_t)raw_smem + 1023) & ~(uintptr_t)1023);
    unsigned char* planes = ring + (size_t)R * L::kRaw;
    __shared__ uint64_t raw_full[R], raw_empty[R], split_full[2], split_empty[2], acc_full[2], acc_empty[2], done;
    __shared__ uint32_t tmem_slot, least[L::kRows], least_parts[PARTS ? L::kRows : 1];
    __shared__ int abort_flag, any_tiny;
    lsb_pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int m0, n0, splits = 1, first = 0, steps = (p.K + kSK - 1) / kSK;
    if constexpr (PARTS) {
        const int at = p.tile0 + (int)blockIdx.x;
        m0 = rows_first<BN>(p.M, p.N) ? at % p.tiles_m : at / p.tiles_n;
        n0 = rows_first<BN>(p.M, p.N) ? at / p.tiles_m : at % p.tiles_n;
        splits = (int)gridDim.z;
        first = (int)blockIdx.z * p.steps;
        steps = min(p.steps, steps - first);                            // (at least one)
    } else {
        m0 = rows_first<BN>(p.M, p.N) ? blockIdx.x : blockIdx.y;
        n0 = rows_first<BN>(p.M, p.N) ? blockIdx.y : blockIdx.x;
    }
    m0 *= kSM;
    n0 *= BN;
    if (tid < L::kRows) least[tid] = 0xffffffffu;
    if (tid == 0) {
        abort_flag = any_tiny = 0;
        for (int s = 0; s < R; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], kSGroup / 32); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&split_full[s], kSGroup / 32);
            mbar_init(&split_empty[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], kSWorkers / 32);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    constexpr uint32_t kColumns = 512;                                  // (one block an SM)
    if (warp == kSWorkers / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kColumns));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == kSWorkers / 32) {
        if (lsb_elect_one()) {
            const uint32_t base = smem_u32(ring);
            lsb_pdl_wait();
            int it = 0;
            for (; it < steps; ++it) {
                const int s = it % R;
                if (it >= R && !mbar_wait(&raw_empty[s], (uint32_t)(it / R - 1) & 1, &abort_flag)) break;
                mbar_expect(&raw_full[s], L::kRaw);
                tma_rows(base + s * L::kRaw, &map_x, &raw_full[s], (first + it) * kSK, m0);
                tma_rows(base + s * L::kRaw + kSM * kSK * 4, &map_w, &raw_full[s], (first + it) * kSK, n0);
            }
            for (int k = it > R ? it - R : 0; k < it; ++k) {            // (no copy is in flight when the block leaves)
                int ignore = 0;
                mbar_wait(&raw_full[k % R], (uint32_t)(k / R) & 1, &ignore);
            }
        }
    } else if (warp == kSWorkers / 32 + 1) {
        if (lsb_elect_one()) {
            // D 32-bit, A and B bfloat16, both K-major
            constexpr uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(BN >> 3) << 17 | (uint32_t)(kSM >> 4) << 24;
            const uint32_t small = tmem + L::kSmall;
            lsb_pdl_wait();                                             // (a wait's limit is for this kernel's own copies)
            for (int it = 0; it < steps; ++it) {
                const int s = it & 1, c = it / kSChunk;
                if (it % kSChunk == 0 && c >= 2 && !mbar_wait(&acc_empty[c & 1], (uint32_t)(c / 2 - 1) & 1, &abort_flag)) break;
                if (!mbar_wait(&split_full[s], (uint32_t)(it >> 1) & 1, &abort_flag)) break;
                tmem_fence_after();
                const uint32_t at = smem_u32(planes) + s * L::kSplit;
                const uint32_t lead = tmem + (c & 1) * BN;
#pragma unroll
                for (int k = 0; k < kSK / 16; ++k) {                    // 32 bytes along K: +2 in 16-byte units
                    uint32_t a[3];
                    uint64_t b[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        a[i] = tmem + L::kX + s * L::kXSplit + i * L::kXPlane + 8 * k;
                        b[i] = plane_desc(at + i * L::kPlane) + 2 * k;
                    }
                    umma(small, a[0], b[2], idesc, it || k);
                    umma(small, a[2], b[0], idesc, true);
                    umma(small, a[1], b[1], idesc, true);
                    umma(small, a[0], b[1], idesc, true);
                    umma(small, a[1], b[0], idesc, true);
                    umma(lead, a[0], b[0], idesc, it % kSChunk || k);
                }
                umma_commit(&split_empty[s]);
                if (it % kSChunk == kSChunk - 1 || it == steps - 1) umma_commit(&acc_full[c & 1]);
            }
            umma_commit(&done);
            int ignore = 0;
            mbar_wait(&done, 0, &ignore);
        }
    } else {
        lsb_pdl_wait();                                                 // (the output may still be read by the kernel before)
        constexpr int kMine = BN / 4;                                   // columns of a warp, of 32 rows
        float sums[kMine];
#pragma unroll
        for (int i = 0; i < kMine; ++i) sums[i] = 0.f;
        const int q = warp & 3, part = warp >> 2;
        const uint32_t mine = tmem + ((uint32_t)(q * 32) << 16) + part * kMine;
        bool ok = true;
        int taken = 0;
        auto take = [&]() {
            const int c = taken++;
            ok = mbar_wait(&acc_full[c & 1], (uint32_t)(c >> 1) & 1, &abort_flag);
            if (!ok) return;
            tmem_fence_after();
            tmem_add(mine + (c & 1) * BN, sums);
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[c & 1]);
        };
        const int group = warp / (kSGroup / 32), r = tid % kSGroup;     // stages it % 2 == group
        const bool has_row = r < L::kRows;
        uint32_t low = 0xffffffffu;                                     // the least number of the row but zero: twice its bits, less one
        for (int it = group; it < steps && ok; it += 2) {
            const int s = it % R;
            if (!mbar_wait(&raw_full[s], (uint32_t)(it / R) & 1, &abort_flag)) { ok = false; break; }
            if (it >= 2 && !mbar_wait(&split_empty[group], (uint32_t)(it / 2 - 1) & 1, &abort_flag)) { ok = false; break; }
            tmem_fence_after();
            if (has_row) {
                const unsigned char* from = ring + (size_t)s * L::kRaw + r * (kSK * 4);
                unsigned char* to = planes + (size_t)group * L::kSplit + (r - kSM) * (kSK * 2);
                const uint32_t to_x = tmem + ((uint32_t)(q * 32) << 16) + L::kX + group * L::kXSplit;
#pragma unroll
                for (int j = 0; j < kSK / 16; ++j) {                    // sixteen values
                    uint32_t h[8], m[8], l[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 a = *reinterpret_cast<const float4*>(from + (((4 * j + i) ^ (r & 7)) << 4));
                        low = __vimin3_u32(low, twice_less_one(a.x), twice_less_one(a.y));
                        low = __vimin3_u32(low, twice_less_one(a.z), twice_less_one(a.w));
                        split3(a.x, a.y, h[2 * i], m[2 * i], l[2 * i]);
                        split3(a.z, a.w, h[2 * i + 1], m[2 * i + 1], l[2 * i + 1]);
                    }
                    if (r < kSM) {                                      // (whole warps)
                        tmem_put(to_x + 8 * j, h);
                        tmem_put(to_x + L::kXPlane + 8 * j, m);
                        tmem_put(to_x + 2 * L::kXPlane + 8 * j, l);
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            unsigned char* put = to + (((2 * j + i) ^ ((r >> 1) & 3)) << 4);
                            *reinterpret_cast<uint4*>(put) = make_uint4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
                            *reinterpret_cast<uint4*>(put + L::kPlane) = make_uint4(m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]);
                            *reinterpret_cast<uint4*>(put + 2 * L::kPlane) = make_uint4(l[4 * i], l[4 * i + 1], l[4 * i + 2], l[4 * i + 3]);
                        }
                    }
                }
                if (r < kSM) {
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tmem_fence_before();
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) { mbar_arrive(&split_full[group]); mbar_arrive(&raw_empty[s]); }
            // (the chunk before this one: its products have ended by now, and those of the next need its place)
            if (it % kSChunk >= kSChunk - 2 && it >= kSChunk) take();
        }
        const int chunks = (steps + kSChunk - 1) / kSChunk;
        while (taken < chunks && ok) take();
        if (ok) {
            tmem_add(mine + L::kSmall, sums);
            // every product has been issued and waited for, so that the ring is free
            float* row = reinterpret_cast<float*>(ring) + (q * 32 + lane) * L::LDT + part * kMine;
#pragma unroll
            for (int j = 0; j < kMine; j += 4)
                *reinterpret_cast<float4*>(row + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]);
        }
        if (has_row) atomicMin(&least[r], low);
        if (low < kTiny) any_tiny = 1;
        tmem_fence_before();
    }
    __syncwarp();
    // the sums of all stretches of K are there, each in its block; a block brings its share of the rows together
    cg::cluster_group cluster = cg::this_cluster();
    if (PARTS && splits > 1) cluster.sync();
    else __syncthreads();
    if (warp < kSWorkers / 32 && !abort_flag) {
        const float* tile = reinterpret_cast<const float*>(ring);
        int row0 = 0, rows = kSM;
        if constexpr (PARTS) {
            row0 = (int)blockIdx.z * (kSM / splits);
            rows = (int)blockIdx.z == splits - 1 ? kSM - row0 : kSM / splits;
        }
        uint32_t* all_least = PARTS ? least_parts : least;
        // A number below 2^-103 loses less than 2^-125 with the parts that bfloat16 has no normal number for (one that
        // is not below has them all), which is at most K 2^-125 times the largest number of the other operand's row in
        // a sum.  Sums that this could show in are done over; the largest are looked up only where there is such a number.
        float* largest = reinterpret_cast<float*>(planes);              // [kRows] (every product has been waited for)
        bool tiny = any_tiny;
        if constexpr (PARTS)
            for (int k = 0; k < splits && splits > 1; ++k) tiny |= *cluster.map_shared_rank(&any_tiny, k) != 0;
        if (tiny) {
            for (int r = warp; r < L::kRows; r += kSWorkers / 32) {
                const bool of_x = r < kSM;
                if (PARTS && of_x && (r < row0 || r >= row0 + rows)) continue;
                const long long at = of_x ? m0 + r : n0 + r - kSM;
                float big = 0.f;
                if (at < (of_x ? p.M : p.N))
                    for (int k = lane * 4; k < p.K; k += 128) {
                        const float4 a = *reinterpret_cast<const float4*>((of_x ? p.x : p.w) + at * p.K + k);
                        big = fmaxf(fmaxf(big, fmaxf(fabsf(a.x), fabsf(a.y))), fmaxf(fabsf(a.z), fabsf(a.w)));
                    }
                big = lsb_warp_max(big);
                if (lane == 0) {
                    largest[r] = big * ((float)p.K * 0x1p-101f);
                    if constexpr (PARTS) {
                        uint32_t least_of = least[r];
                        for (int k = 0; k < splits && splits > 1; ++k) least_of = min(least_of, *cluster.map_shared_rank(&least[r], k));
                        all_least[r] = least_of;
                    }
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kSWorkers) : "memory");
        }
        for (int e = tid; e < rows * (BN / 4); e += kSWorkers) {
            const int row = row0 + e / (BN / 4), col = e % (BN / 4) * 4;
            if (m0 + row >= p.M || n0 + col >= p.N) continue;
            __align__(16) float v[4];
            const float* at = tile + row * L::LDT + col;
            if (PARTS && splits > 1) {
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                for (int k = 0; k < splits; ++k) {                      // (in order)
                    const float4 a = *reinterpret_cast<const float4*>(cluster.map_shared_rank(at, k));
                    sum.x += a.x; sum.y += a.y; sum.z += a.z; sum.w += a.w;
                }
                *reinterpret_cast<float4*>(v) = sum;
            } else {
                *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(at);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bool over = !(fabsf(v[i]) <= 3.402823466e38f);
                if (tiny)
                    over |= (all_least[row] < kTiny && fabsf(v[i]) < largest[kSM + col + i]) ||
                            (all_least[kSM + col + i] < kTiny && fabsf(v[i]) < largest[row]);
                if (over && n0 + col + i < p.N)
                    v[i] = plain_dot(p.x + (long long)(m0 + row) * p.K, p.w + (long long)(n0 + col + i) * p.K, p.K);
            }
            store_four(p, m0 + row, n0 + col, *reinterpret_cast<float4*>(v));
        }
    }
    __syncwarp();
    if (PARTS && splits > 1) cluster.sync();                            // (a peer may still read this block's sums)
    else __syncthreads();
    if (warp == kSWorkers / 32) {
        tmem_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kColumns));
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

template <int MT, int ST>
static int launch_rows(RowsParams p, cudaStream_t stream) {
    static int configured = -1;
    constexpr size_t smem = (size_t)ST * (kRB + MT) * kKS * 4;
    if (configured < 0)
        configured = (int)cudaFuncSetAttribute(gemm_rows_f32_kernel<MT, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (configured) return configured;
    // groups of as many rows as share the matrix out evenly over the SMs' turns
    const int unit = p.act ? 2 : 1, sms = num_sms();
    const int turns = (p.N + sms * kRB - 1) / (sms * kRB);
    p.per = (p.N + sms * turns - 1) / (sms * turns);
    p.per = (p.per + unit - 1) / unit * unit;
    p.groups = (p.N + p.per - 1) / p.per;
    const int blocks = p.groups < sms ? p.groups : sms;
    return lsb_launch(gemm_rows_f32_kernel<MT, ST>, dim3(blocks, (p.M + kRowsMax - 1) / kRowsMax), dim3(kRowThreads), smem, stream, 1, p);
}

template <int WM, int WN, int WK, int BK, int ST>
static int launch_tile(const TileParams& p, cudaStream_t stream) {
    using L = TileLayout<WM, WN, WK, BK, ST>;
    static int configured = -1;
    if (configured < 0)
        configured = (int)cudaFuncSetAttribute(gemm_tile_f32_kernel<WM, WN, WK, BK, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)L::kTotal);
    if (configured) return configured;
    const dim3 grid((p.N + L::BN - 1) / L::BN, (p.M + L::BM - 1) / L::BM);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    return lsb_launch(gemm_tile_f32_kernel<WM, WN, WK, BK, ST>, grid, dim3(kTileThreads), L::kTotal, stream, 1, p);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

// [rows, K] 32-bit, boxes of [box_rows x 32], 128-byte swizzle, zeros outside
static int map_rows(CUtensorMap* map, const float* ptr, int rows, int K, int box_rows) {
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            return (int)cudaErrorNotSupported;
        encode = (EncodeTiledFn)f;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {(cuuint32_t)kSK, (cuuint32_t)box_rows}, unit[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, unit,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// Blocks of gemm_split_f32_kernel<BN> that run at once in clusters of `splits`.
template <int BN>
static int split_room(int splits) {
    using L = SplitLayout<BN>;
    static int cached[64][kSSplits + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int& room = cached[dev][splits];
    if (room == 0) {
        int clusters = 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, splits);
        cfg.blockDim = dim3(kSThreads);
        cfg.dynamicSmemBytes = L::kTotal;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = splits;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (splits == 1 || cudaFuncSetAttribute(gemm_split_f32_kernel<BN, PartParams>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kTotal) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, gemm_split_f32_kernel<BN, PartParams>, &cfg) != cudaSuccess || clusters <= 0) {
            cudaGetLastError();
            clusters = num_sms() / splits;
        }
        room = clusters * splits < 1 ? 1 : clusters * splits;
    }
    return room;
}

template <int BN>
static int split_maps(const TileParams& p, CUtensorMap* mx, CUtensorMap* mw) {
    static int configured = -1;
    if (configured < 0) {
        configured = (int)cudaFuncSetAttribute(gemm_split_f32_kernel<BN, TileParams>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SplitLayout<BN>::kTotal);
        if (!configured)
            configured = (int)cudaFuncSetAttribute(gemm_split_f32_kernel<BN, PartParams>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SplitLayout<BN>::kTotal);
    }
    if (configured) return configured;
    const int rc = map_rows(mx, p.x, p.M, p.K, kSM);
    return rc ? rc : map_rows(mw, p.w, p.N, p.K, BN);
}
template <int BN>
static int launch_whole(const TileParams& p, cudaStream_t stream) {
    CUtensorMap mx, mw;
    const int rc = split_maps<BN>(p, &mx, &mw);
    if (rc) return rc;
    const unsigned tiles_m = (p.M + kSM - 1) / kSM, tiles_n = (p.N + BN - 1) / BN;
    if (!rows_first<BN>(p.M, p.N) && tiles_m > 65535) return (int)cudaErrorInvalidValue;
    const dim3 grid = rows_first<BN>(p.M, p.N) ? dim3(tiles_m, tiles_n) : dim3(tiles_n, tiles_m);
    return lsb_launch(gemm_split_f32_kernel<BN, TileParams>, grid, dim3(kSThreads), SplitLayout<BN>::kTotal, stream, 1, mx, mw, p);
}
template <int BN>
static int launch_parts(const TileParams& tile, int tile0, int tiles, int splits, cudaStream_t stream) {
    CUtensorMap mx, mw;
    const int rc = split_maps<BN>(tile, &mx, &mw);
    if (rc) return rc;
    PartParams p;
    static_cast<TileParams&>(p) = tile;
    // whole chunks of leading products a block; the last one may have fewer
    const int chunks = (p.K + kSK * kSChunk - 1) / (kSK * kSChunk), per = (chunks + splits - 1) / splits;
    p.steps = per * kSChunk;
    p.tiles_m = (p.M + kSM - 1) / kSM;
    p.tiles_n = (p.N + BN - 1) / BN;
    p.tile0 = tile0;
    const dim3 grid(tiles, 1, (chunks + per - 1) / per);
    return lsb_launch(gemm_split_f32_kernel<BN, PartParams>, grid, dim3(kSThreads), SplitLayout<BN>::kTotal, stream, (int)grid.z, mx, mw, p);
}

LSB_API int lsb_gemm_f32_supported(const void* x, const void* w, int M, int N, int K) {
    return M > 0 && N > 0 && K > 0 && K % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0 && M <= 32 * 65535;
}

// How a split product's tiles go to the SMs: `columns` wide, a block for all of K of the first `whole` of them, a cluster of `splits`
// blocks along K for each of the rest.  A block takes about its fixed part and its stages (fitted to 20 shapes), a cluster some
// 2.5 us more to meet; blocks run in rounds.  500 rows, us, whole and so: 2,048 x 2,048 44 / 31 (two parts), 2,048 x 8,192 161 / 95,
// 16,384 x 2,048 gated 220 / 195 (three whole rounds, the rest in two parts), 3,072 x 2,048 52 / 52 (whole: 96 tiles); 40 rows
// times 2,048 x 8,192 159 / 38 (six parts); 300 times 16,384 x 2,048 160 / 159 (whole).
struct SplitPlan { int columns, splits; long long whole, tiles; };
static SplitPlan split_plan(int M, int N, int K) {
    const int chunks = (K + kSK * kSChunk - 1) / (kSK * kSChunk);
    SplitPlan best{};
    double least = 0.0;
    for (int bn = 64; bn <= 128; bn += 64) {
        const double stage = bn == 64 ? 0.62 : 0.70, fixed = bn == 64 ? 4.8 : 7.0, meet = 2.5;
        const long long tiles = (long long)((M + kSM - 1) / kSM) * ((N + bn - 1) / bn), room = bn == 64 ? split_room<64>(1) : split_room<128>(1);
        const double round = fixed + chunks * kSChunk * stage;
        auto offer = [&](long long whole, int splits, double us) {
            if (splits > 1) us *= 1.03;                        // (in doubt whole)
            if (best.columns == 0 || us < least) { least = us; best = SplitPlan{bn, splits, whole, tiles}; }
        };
        offer(tiles, 1, round * (double)((tiles + room - 1) / room));
        const long long full = tiles / room;
        for (int s = 2; s <= kSSplits && s <= chunks; ++s) {
            const long long at_once = bn == 64 ? split_room<64>(s) : split_room<128>(s);
            const double part = fixed + meet + (chunks + s - 1) / s * kSChunk * stage;
            offer(0, s, part * (double)((tiles * s + at_once - 1) / at_once));
            if (full > 0 && tiles > full * room)
                offer(full * room, s, round * (double)full + part * (double)(((tiles - full * room) * s + at_once - 1) / at_once));
        }
    }
    return best;
}
// The plan as the product makes it, for its tests: columns, blocks along K of the tiles behind `whole`, `whole`, tiles.
LSB_API void lsb_gemm_f32_split_plan(int M, int N, int K, long long* plan) {
    const SplitPlan p = split_plan(M, N, K);
    plan[0] = p.columns;
    plan[1] = p.splits;
    plan[2] = p.whole;
    plan[3] = p.tiles;
}
template <int BN>
static int run_split(const TileParams& p, const SplitPlan& plan, cudaStream_t stream) {
    if (plan.tiles > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    if (plan.splits == 1) return launch_whole<BN>(p, stream);
    if (plan.whole) {
        const int rc = launch_parts<BN>(p, 0, (int)plan.whole, 1, stream);
        if (rc) return rc;
    }
    return launch_parts<BN>(p, (int)plan.whole, (int)(plan.tiles - plan.whole), plan.splits, stream);
}

// act: 0, or the activation of a gated product (1 silu, 2 gelu in its tanh form, 3 none), N even then.
LSB_API int lsb_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int act, cudaStream_t stream) {
    if (!lsb_gemm_f32_supported(x, w, M, N, K) || ((uintptr_t)out % 16)) return (int)cudaErrorInvalidValue;
    if (act < 0 || act > LSB_ACT_NONE || (act && (N & 1))) return (int)cudaErrorInvalidValue;
    if (M <= kRowsMax || (M <= kRowsSmall && (long long)N * K <= kSmallMatrix)) {
        RowsParams p{x, w, out, M, N, K, 0, 0, act};
        if (M == 1) return launch_rows<1, 6>(p, stream);
        if (M == 2) return launch_rows<2, 5>(p, stream);
        if (M <= 4) return launch_rows<4, 5>(p, stream);
        if (M <= 8) return launch_rows<8, 4>(p, stream);
        return launch_rows<16, 3>(p, stream);
    }
    // The tile whose rounds over the SMs cover the least area; a smaller one brings more of x and w a multiply-add and pays
    // its end more often, so it has to win by a few per cent.  At the K that is left for them (below 512) each is the
    // fastest somewhere (128 x 256, 128 x 128, 64 x 128, 64 x 64, us: 1,000 x 8,192 x 256 108 / 114 / 109 / 130; 2,048 x 8,192 x 256
    // 215 / 200 / 218 / 259; 200 x 4,096 x 128 30 / 16 / 9.6 / 11.7; 500 x 512 x 128 29 / 16 / 9.4 / 6.2), and this count finds it within
    // 10 % on most of 120 shapes; along the shortest K it picks too small a tile (500 x 20,000 x 20: 65 us, 128 x 128 29; 2,048 x
    // 2,048 x 64: 28, 128 x 256 18), whose sums are the closer ones: more warps share K out (K = 320, from the smallest tile to the
    // largest: 1.3, 1.7, 2.4 and 3.2e-7 of the norm).
    const TileParams p{x, w, out, M, N, K, act};
    const long long sms = num_sms();
    if (K >= kSplitK) {
        const SplitPlan plan = split_plan(M, N, K);
        return plan.columns == 64 ? run_split<64>(p, plan, stream) : run_split<128>(p, plan, stream);
    }
    const int bm[4] = {128, 128, 64, 64}, bn[4] = {256, 128, 128, 64};
    const double cost[4] = {1.0, 1.0, 1.03, 1.08};
    int best = 0;
    double least = 0.0;
    for (int c = 0; c < 4; ++c) {
        const long long tiles = (long long)((M + bm[c] - 1) / bm[c]) * ((N + bn[c] - 1) / bn[c]);
        const double area = (double)((tiles + sms - 1) / sms) * bm[c] * bn[c] * cost[c];
        if (c == 0 || area < least) { least = area; best = c; }
    }
    switch (best) {
        case 0: return launch_tile<2, 4, 1, 32, 3>(p, stream);
        case 1: return launch_tile<2, 2, 2, 32, 4>(p, stream);
        case 2: return launch_tile<1, 2, 4, 32, 5>(p, stream);
        default: return launch_tile<1, 1, 8, 64, 4>(p, stream);
    }
}
