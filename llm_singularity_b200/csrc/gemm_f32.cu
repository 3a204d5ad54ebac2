// out[M, N] = x[M, K] * w[N, K]^T in true 32-bit: every product a 32-bit multiply-add, no reduced-precision
// matrix mode.  Two kernels, by the number of rows; K a multiple of 4 and 16-byte aligned bases (anything else is
// csrc/gemm.cu's).  An activation of a gated product (w's rows alternate gate_i, up_i, out is [M, N / 2]) is
// applied where the sums meet.  The reference hands such products to cublasSgemm
// (kernels/src/cublas_provider.cpp:36-51) and launches silu(g) * u by itself (kernels/src/activations.cu:11-21).
//
// * Up to 16 rows (a decode step) the product is weight traffic.  Weight rows are dealt out over one
//   block per SM, sixteen at most at a time: four to a warp, each row's K in two parts.  A warp copies the weights it
//   needs into a ring of shared memory itself (asynchronously, some 140 KB in flight an SM, the first of them before
//   the wait on the kernel before) and shares the rows of x with the three others of its part.  The sums of a
//   group meet once, over lanes by halving exchanges and over the two parts in shared memory, in a fixed order.
//   The four products of a layer at 1B sizes, 8 rows (243 MB): 71 us (3.4 TB/s); as 64 x 64 tiles, 56 of their 64 rows
//   empty and as few as 32 of them: 1,202 us.  (A thread's places of K for all sixteen rows, with no sharing at all, cost
//   four times the exchanges at the end of a group: 89 us.)
//
// * More rows (a prompt): arithmetic on the 32-bit pipes.  Eight warps of 64 x 64 outputs (8 x 16 a thread), arranged as a tile of 128 x 256, 128 x 128, 64 x 128 or 64 x 64;
//   in the smaller tiles the warps that are left share out each slice of K and their sums meet at the end, so that
//   a few hundred rows against 2,048 columns still give every SM eight busy warps.  Slices come by asynchronous copies,
//   three to five in flight.  The same four products at 500 rows (61 GFLOP): 1,502 us, 41 TFLOP/s of the 70 that a
//   loop of nothing but multiply-adds reaches here; 64 x 64 tiles of 4 x 4 a thread: 2,104 us.  (Slices fetched through
//   registers, however arranged, exposed their latency: 2,400 us.)
//
// A row's sum is taken in an order that K and the kernel fix, the same from run to run.
#include "common.cuh"
#include "gate_act.cuh"

LSB_DEFINE_STATUS()

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// 16 bytes from global to shared memory, zeros where `have` is false (nothing is read then)
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool have) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------ a few rows
constexpr int kRowThreads = 256;
constexpr int kRowsMax = 16;                   // rows of x a block takes
constexpr int kRB = 16;                        // most weight rows of a group: four for each of four warps, twice (two parts of K)
constexpr int kRW = kRB / 4;
constexpr int kRowsSmall = 128;                // rows that still go this way, sixteen to a block, ...
constexpr long long kSmallMatrix = 1 << 18;    // ... where the matrix is so small that a tile's latency shows
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

    auto copy_w = [&](int it) {
        const int g = (int)blockIdx.x + (it / chunks) * (int)gridDim.x, k0 = it % chunks * kKS + at;
        const int n0 = g * p.per, rows = min(p.per, p.N - n0);
        const uint32_t st = base + (uint32_t)(it % ST) * (kRB + MT) * kKS * 4u;
#pragma unroll
        for (int i = 0; i < kRW; ++i) {
            const int r = rg * kRW + i;
            if (r >= rows) break;
            const float* src = p.w + (size_t)(n0 + r) * p.K;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int k = k0 + 256 * j;
                copy16(st + (uint32_t)(r * kKS + 256 * j) * 4u, k < p.K ? src + k : p.w, k < p.K);
            }
        }
    };
    auto copy_x = [&](int it) {
        const int k0 = it % chunks * kKS + at;
        const uint32_t st = base + ((uint32_t)(it % ST) * (kRB + MT) + kRB) * kKS * 4u;
#pragma unroll
        for (int m = rg; m < MT; m += 4)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int k = k0 + 256 * j;
                const bool have = m < M && k < p.K;
                copy16(st + (uint32_t)(m * kKS + 256 * j) * 4u, have ? x + (size_t)m * p.K + k : p.x, have);
            }
    };
    for (int it = 0; it < ST - 1 && it < total; ++it) copy_w(it);
    lsb_pdl_wait();
    for (int it = 0; it < ST - 1; ++it) {
        if (it < total) copy_x(it);
        copies_commit();
    }
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.f;
    int chunk = 0, done = 0;
    for (int it = 0; it < total; ++it) {
        copies_wait<ST - 2>();
        // the four warps of this part of K share the rows of x; past this point none still reads the stage before
        asm volatile("bar.sync %0, 128;" ::"r"(1 + kg) : "memory");
        if (it + ST - 1 < total) { copy_w(it + ST - 1); copy_x(it + ST - 1); }
        copies_commit();
        const int n0 = ((int)blockIdx.x + done * (int)gridDim.x) * p.per, rows = min(p.per, p.N - n0);
        const float* st = ring + (size_t)(it % ST) * (kRB + MT) * kKS + at;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (chunk * kKS + kg * 128 + 256 * j >= p.K) break;       // (the warp's whole step lies past K)
            float4 wv[kRW];
#pragma unroll
            for (int i = 0; i < kRW; ++i)
                wv[i] = rg * kRW + i < rows ? *reinterpret_cast<const float4*>(st + (rg * kRW + i) * kKS + 256 * j)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
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
        if (++chunk < chunks) continue;
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
    const bool wide = (p.N & 3) == 0;
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
        if (p.act) {                                                   // (N is even)
            float* d = p.out + m * (p.N / 2) + n / 2;
            const float first = lsb_gated(v.x, v.y, p.act, 0.f);
            if (wide) *reinterpret_cast<float2*>(d) = make_float2(first, lsb_gated(v.z, v.w, p.act, 0.f));
            else {
                d[0] = first;
                if (n + 2 < p.N) d[1] = lsb_gated(v.z, v.w, p.act, 0.f);
            }
            continue;
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

LSB_API int lsb_gemm_f32_supported(const void* x, const void* w, int M, int N, int K) {
    return M > 0 && N > 0 && K > 0 && K % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0 && M <= 32 * 65535;
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
    // The tile whose rounds over the SMs cover the least area; a smaller one brings more of x and w a
    // multiply-add and pays its end more often, so it has to win by a few per cent.
    const TileParams p{x, w, out, M, N, K, act};
    const long long sms = num_sms();
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
