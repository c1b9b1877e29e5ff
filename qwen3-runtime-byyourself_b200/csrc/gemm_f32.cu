// True 32-bit matrix product of the check path: Y[M,N] = X[M,K] . W[N,K]^T with float
// operands, fmaf accumulation and no tensor-core mode of reduced precision.
//
// It replaces the reference's single cublasGemmEx call per projection
// (src/ops/linear.cpp:165-193) on the 32-bit path only.  The order of an element's sum
// depends on K and on nothing else - not on M, N or the tile it falls in - so a row's
// result does not depend on which other rows are in the batch, although two kernels share
// the work.  The order, for rows of whole 16-byte packets:
//
//   K is cut into at most 8 ranges (`range_length`); inside a range the even and the odd k
//   are two ascending chains of fmaf, whose sums are added; the ranges' sums are added in
//   ascending order.
//
// Two chains because fma.rn.f32x2 then takes its operands as they lie in memory; ranges
// because warps and blocks can share K without changing the sum.  Shorter chains also round
// less: logits of 4 layers of 8B width are 4.4e-7 away from 64 bits where one chain gave 1.7e-6.
//
//   stream_kernel : up to 8 rows (decode).  Bound by reading W once: 5.6 TB/s over the products of a
//                   decode step of 3 sequences (1.0 ms; tiles of 64 x 64 took 8.9).
//   tile_kernel   : more rows.  Bound by the CUDA cores' fma: 41 TFLOP/s in tiles of 128 x 128 that fill the GPU (1,000 rows, K 2,048,
//                   32,768 wide: 3.25 ms; 3.9 in one ascending chain by tiles of 64 x 64), less where few rows share K over clusters.
//   gemm_tn_kernel: short K, where the tiles above have too few steps to pay for their start.
//
// Rows that are not whole packets, and bfloat16 operands of any width (32-bit accumulation,
// bfloat16 or float output: the products whose width is no multiple of 8, which the
// tensor-core kernels refuse), go to `gemm_tn_kernel` in its other form, one ascending chain.
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

constexpr int MAX_RANGES = 8;

// K per range: a multiple of 32 (the kernels' step).
__host__ __device__ __forceinline__ int range_length(int K) { return ((K + MAX_RANGES - 1) / MAX_RANGES + 31) / 32 * 32; }

__device__ __forceinline__ void copy16(uint32_t to, const void* from, bool inside) {
    // outside: nothing is read, 16 zero bytes are written
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(from), "r"(inside ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// acc = {acc.x + a.x b.x, acc.y + a.y b.y}, each a single rounding (fmaf)
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(uint64_t v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// ---------------------------------------------------------------- few rows
// A block owns 32 rows of W, a lane one of them; a warp walks one range of K, so X is the same address for all lanes.  A
// warp stages 32 k of its 32 rows (whole lines) and of X with asynchronous copies in stages of its own, no barrier between
// warps; the padded row stride (36 words) keeps the lanes' 16-byte reads free of bank conflicts.  The memory's latency at
// full rate needs about 55 KB in flight an SM: two blocks an SM with two stages, or, when the matrix has no more blocks than
// there are SMs, one with four.  Sums of ranges meet in shared memory.
constexpr int S_ROWS = 32, S_WARPS = 8, S_K = 32, S_LD = S_K + 4;

template <int MT> constexpr int stream_stage() { return S_ROWS * S_LD + MT * S_K; }      // floats

template <int MT, int S_STAGES>
__global__ void __launch_bounds__(S_WARPS * 32)
stream_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N, int K, int64_t ldx,
              int64_t ldw, int64_t ldy) {
    extern __shared__ __align__(16) float shared[];
    float* sums = shared + S_WARPS * S_STAGES * stream_stage<MT>();      // [range][MT][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * S_ROWS;
    const int length = range_length(K), ranges = (K + length - 1) / length;
    float* mine = shared + warp * S_STAGES * stream_stage<MT>();
    const uint32_t mine_at = (uint32_t)__cvta_generic_to_shared(mine);
    pdl_launch_dependents();
    pdl_wait();

    const int range = warp;                              // MAX_RANGES == S_WARPS
    const int k_begin = range * length, k_end = min(K, k_begin + length);
    const int steps = range < ranges ? (k_end - k_begin + S_K - 1) / S_K : 0;
    auto fetch = [&](int step) {
        if (step < steps) {
            const int k0 = k_begin + step * S_K;
            const uint32_t at = mine_at + (step % S_STAGES) * (stream_stage<MT>() * 4);
            const int part = (lane & 7) * 4;             // 8 lanes take a row's 128 bytes
            const bool in = k0 + part < k_end;
#pragma unroll
            for (int i = 0; i < S_ROWS / 4; ++i) {
                const int row = i * 4 + (lane >> 3);
                const bool ok = in && n0 + row < N;
                copy16(at + (row * S_LD + part) * 4, ok ? W + (int64_t)(n0 + row) * ldw + k0 + part : W, ok);
            }
#pragma unroll
            for (int i = 0; i < (MT + 3) / 4; ++i) {
                const int row = i * 4 + (lane >> 3);
                const bool ok = in && row < M;
                if (row < MT) copy16(at + (S_ROWS * S_LD + row * S_K + part) * 4, ok ? X + (int64_t)row * ldx + k0 + part : X, ok);
            }
        }
        copies_commit();          // empty groups past the end keep the count of groups in step
    };
    uint64_t acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0;
#pragma unroll
    for (int s = 0; s < S_STAGES - 1; ++s) fetch(s);
    for (int step = 0; step < steps; ++step) {
        copies_wait<S_STAGES - 2>();
        __syncwarp();
        fetch(step + S_STAGES - 1);                     // into the stage that the warp left before the barrier above
        const float* w = mine + (step % S_STAGES) * stream_stage<MT>() + lane * S_LD;
        const float* x = mine + (step % S_STAGES) * stream_stage<MT>() + S_ROWS * S_LD;
#pragma unroll
        for (int k = 0; k < S_K; k += 4) {
            const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + k);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(x + m * S_K + k);
                fma2(acc[m], xv.x, wv.x);
                fma2(acc[m], xv.y, wv.y);
            }
        }
    }
    copies_wait<0>();
    if (range < ranges) {
#pragma unroll
        for (int m = 0; m < MT; ++m) sums[(range * MT + m) * S_ROWS + lane] = both(acc[m]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < MT * S_ROWS; i += S_WARPS * 32) {
        const int m = i / S_ROWS, n = n0 + i % S_ROWS;
        if (m >= M || n >= N) continue;
        float total = sums[i];
        for (int r = 1; r < ranges; ++r) total += sums[r * MT * S_ROWS + i];
        Y[(int64_t)m * ldy + n] = total;
    }
}

template <int MT, int STAGES>
int launch_stream(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldy,
                  cudaStream_t stream) {
    static_assert(S_WARPS == MAX_RANGES, "a warp per range");
    constexpr int SMEM = (S_WARPS * STAGES * stream_stage<MT>() + MAX_RANGES * MT * S_ROWS) * 4;
    static Q3PerDevice configured;
    const cudaError_t e = q3_allow_shared_memory(stream_kernel<MT, STAGES>, SMEM, configured);
    if (e != cudaSuccess) return (int)e;
    return (int)q3_launch(stream_kernel<MT, STAGES>, dim3((N + S_ROWS - 1) / S_ROWS), dim3(S_WARPS * 32), SMEM, stream, X, W, Y, M,
                          N, K, ldx, ldw, ldy);
}

template <int MT>
int launch_stream(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldy,
                  cudaStream_t stream) {
    if ((N + S_ROWS - 1) / S_ROWS <= q3_device_sm_count()) return launch_stream<MT, 4>(X, W, Y, M, N, K, ldx, ldw, ldy, stream);
    return launch_stream<MT, 2>(X, W, Y, M, N, K, ldx, ldw, ldy, stream);
}

// ---------------------------------------------------------------- more rows
// A tile of BM rows of X by 128 rows of W per block, (BM / 16) x 8 elements a thread, both operands staged as they lie in
// memory (rows of 32 k, padded to 36 words: the 16 rows a warp reads at once fall into different banks) in three stages of
// asynchronous copies.  Per 4 k a thread makes 4 BM/16 * 8 multiply-adds from BM/16 + 8 16-byte reads.  The steps of a range are a
// loop of their own, without the code that puts its sum by (in one loop the tiles of 128 rows took 3.75 us a step, 3.5 apart).  When
// there are too few tiles to fill the GPU, the ranges of K are shared out to a cluster's blocks, which leave their sums in shared
// memory and add a share of the tile each, in the order of the ranges.
constexpr int T_N = 128, T_K = 32, T_LD = T_K + 4, T_STAGES = 3;

template <int BM> constexpr int tile_stage() { return (BM + T_N) * T_LD; }               // floats
// Shared memory of a block: the stages, and the sums of its ranges but the last, which lie where the stages were (128 rows: the
// tile's sums).
int tile_bytes(int rows, int ranges, int shares) {
    return T_STAGES * (rows + T_N) * T_LD * 4 + (shares > 1 ? (ranges + shares - 1) / shares - 1 : rows == 128 ? 1 : 0) * rows * T_N * 4;
}

template <int BM>
__global__ void __launch_bounds__(256, BM == 128 ? 1 : 2)
tile_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N, int K, int64_t ldx,
            int64_t ldw, int64_t ldy, int shares) {
    extern __shared__ __align__(16) float shared[];
    constexpr int TM = BM / 16, TN = T_N / 16;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int share = blockIdx.x % shares;
    const int n0 = (blockIdx.x / shares) * T_N, m0 = blockIdx.y * BM;
    const int length = range_length(K), ranges = (K + length - 1) / length;
    const int first = share * ranges / shares, last = (share + 1) * ranges / shares;      // this block's ranges
    const int k_begin = first * length, k_end = min(K, last * length);
    const uint32_t shared_at = (uint32_t)__cvta_generic_to_shared(shared);
    pdl_launch_dependents();
    pdl_wait();

    const int steps = (k_end - k_begin + T_K - 1) / T_K, per_range = length / T_K;
    auto fetch = [&](int step) {
        if (step < steps) {
            const int k0 = k_begin + step * T_K, part = (tid & 7) * 4;
            const uint32_t at = shared_at + (step % T_STAGES) * (tile_stage<BM>() * 4);
            const bool in = k0 + part < k_end;
#pragma unroll
            for (int i = 0; i < (BM + 31) / 32; ++i) {
                const int row = i * 32 + (tid >> 3);
                const bool ok = in && m0 + row < M;
                if (row < BM) copy16(at + (row * T_LD + part) * 4, ok ? X + (int64_t)(m0 + row) * ldx + k0 + part : X, ok);
            }
#pragma unroll
            for (int i = 0; i < T_N / 32; ++i) {
                const int row = i * 32 + (tid >> 3);
                const bool ok = in && n0 + row < N;
                copy16(at + ((BM + row) * T_LD + part) * 4, ok ? W + (int64_t)(n0 + row) * ldw + k0 + part : W, ok);
            }
        }
        copies_commit();
    };
    uint64_t acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0;
#pragma unroll
    for (int s = 0; s < T_STAGES - 1; ++s) fetch(s);
    int done = 0;                                        // ranges that are summed
    for (int step = 0; step < steps;) {
        const int range_end = min(steps, (done + 1) * per_range);
        for (; step < range_end; ++step) {
            copies_wait<T_STAGES - 2>();
            __syncthreads();
            fetch(step + T_STAGES - 1);
            const float* a = shared + (step % T_STAGES) * tile_stage<BM>() + ty * T_LD;
            const float* b = shared + (step % T_STAGES) * tile_stage<BM>() + (BM + tx) * T_LD;
#pragma unroll 2
            for (int k = 0; k < T_K; k += 4) {
                ulonglong2 av[TM];
#pragma unroll
                for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + i * 16 * T_LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(b + j * 16 * T_LD + k);
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        fma2(acc[i][j], av[i].x, bv.x);
                        fma2(acc[i][j], av[i].y, bv.y);
                    }
                }
            }
        }
        // a range is complete
        if (shares == 1 && BM == 128) {              // a block an SM: there is room for the sums so far behind the stages
            float* kept = shared + T_STAGES * tile_stage<BM>() + tid;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float sum = both(acc[i][j]);
                    kept[(i * TN + j) * 256] = done > 0 ? kept[(i * TN + j) * 256] + sum : sum;
                    acc[i][j] = 0;
                }
        } else if (shares == 1) {                    // they wait in Y, where they need neither registers nor shared memory
            float before[TM][TN];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const int m = m0 + i * 16 + ty, n = n0 + j * 16 + tx;
                    before[i][j] = done > 0 && m < M && n < N ? Y[(int64_t)m * ldy + n] : 0.0f;
                }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const int m = m0 + i * 16 + ty, n = n0 + j * 16 + tx;
                    const float sum = both(acc[i][j]);
                    if (m < M && n < N) Y[(int64_t)m * ldy + n] = done > 0 ? before[i][j] + sum : sum;
                    acc[i][j] = 0;
                }
        } else {
            if (first + done + 1 == last) __syncthreads();           // everybody has left the stages
            float* kept = first + done + 1 == last ? shared : shared + T_STAGES * tile_stage<BM>() + done * BM * T_N;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    kept[(i * 16 + ty) * T_N + j * 16 + tx] = both(acc[i][j]);
                    acc[i][j] = 0;
                }
        }
        ++done;
    }
    copies_wait<0>();
    if (shares == 1) {
        if (BM < 128) return;
        const float* kept = shared + T_STAGES * tile_stage<BM>() + tid;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int m = m0 + i * 16 + ty, n = n0 + j * 16 + tx;
                if (m < M && n < N) Y[(int64_t)m * ldy + n] = kept[(i * TN + j) * 256];
            }
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    static_assert(BM * T_N <= T_STAGES * tile_stage<BM>(), "the last range's sums lie where the stages were");
    // four neighbouring sums at a time, all ranges' asked for together
    for (int i = (share * 256 + tid) * 4; i < BM * T_N; i += shares * 256 * 4) {
        const int m = m0 + i / T_N, n = n0 + i % T_N;
        if (m >= M || n >= N) continue;
        float4 part[MAX_RANGES];
        int c = 0, at = 0, to = ranges / shares;         // the share that holds range r, its place there, the share's end
#pragma unroll
        for (int r = 0; r < MAX_RANGES; ++r) {
            part[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r >= ranges) continue;
            if (r == to) {
                at = 0;
                to = (++c + 1) * ranges / shares;
            }
            const float* theirs = cluster.map_shared_rank(shared, c);
            part[r] = *reinterpret_cast<const float4*>(theirs + (r + 1 == to ? 0 : T_STAGES * tile_stage<BM>() + at * BM * T_N) + i);
            ++at;
        }
        float4 sum = part[0];
#pragma unroll
        for (int r = 1; r < MAX_RANGES; ++r) {
            if (r >= ranges) continue;
            sum.x += part[r].x; sum.y += part[r].y; sum.z += part[r].z; sum.w += part[r].w;
        }
        float* y = Y + (int64_t)m * ldy + n;
        y[0] = sum.x;
        if (n + 1 < N) y[1] = sum.y;
        if (n + 2 < N) y[2] = sum.z;
        if (n + 3 < N) y[3] = sum.w;
    }
    cluster.sync();                                      // a block's sums stay until all have read them
}

template <int BM>
int launch_tiles(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldy, int shares,
                 cudaStream_t stream) {
    const int length = range_length(K), ranges = (K + length - 1) / length;
    if ((M + BM - 1) / BM > 65535) return Q3_ERR_TOO_LARGE;
    constexpr int MOST = 227 * 1024;
    static Q3PerDevice configured;
    const cudaError_t e = q3_allow_shared_memory(tile_kernel<BM>, MOST, configured);
    if (e != cudaSuccess) return (int)e;
    const int smem = tile_bytes(BM, ranges, shares);
    const dim3 grid((N + T_N - 1) / T_N * shares, (M + BM - 1) / BM);
    if (shares == 1)
        return (int)q3_launch(tile_kernel<BM>, grid, dim3(256), smem, stream, X, W, Y, M, N, K, ldx, ldw, ldy, shares);
    return (int)q3_launch_cluster(tile_kernel<BM>, grid, dim3(256), smem, stream, dim3(shares, 1, 1), X, W, Y, M, N, K, ldx, ldw,
                                  ldy, shares);
}

// ---------------------------------------------------------------- short rows of K, and rows that are not whole packets
// Tiles of 64 x 64, 4 x 4 elements a thread, staged through registers.  RANGES: the order of sums of the kernels above, for
// packets of float; else one ascending chain.
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// RESIDENT: blocks that an SM must hold (3: at most 80 registers; 0: as the compiler likes, two blocks an SM).
template <bool RANGES, int RESIDENT, typename InT, typename OutT>
__global__ void __launch_bounds__(256, RESIDENT)
gemm_tn_kernel(const InT* __restrict__ X, const InT* __restrict__ W, OutT* __restrict__ Y, int M, int N, int K,
               int64_t ldx, int64_t ldw, int64_t ldy) {
    // RANGES: two tiles, one barrier a tile, the next is fetched under the products of this.  (Rows that are not packets come value by value,
    // and then that costs more than it hides: 64 rows, K 1,001, 1,000 wide 57.7 us, 68.8 with it.)
    __shared__ float Xs[RANGES ? 2 : 1][BK][BM + 4];
    __shared__ float Ws[RANGES ? 2 : 1][BK][BN + 4];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;  // thread tile: rows ty*4.., cols tx*4..
    float acc[TM][TN], odd[TM][TN], total[TM][TN];       // RANGES: chains of the even and of the odd k, the ranges before
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = odd[i][j] = total[i][j] = 0.0f;
    const int length = range_length(K);

    // each thread stages 4 consecutive k of one row of X and one row of W
    const int lr = tid / 4, lk = (tid % 4) * 4;
    alignas(16) float xv[4];
    alignas(16) float wv[4];
    auto fetch = [&](int k0) {
        const int gm = m0 + lr, gn = n0 + lr, gk = k0 + lk;
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = wv[i] = 0.0f;
        if constexpr (RANGES) {
            const InT *px = X + (int64_t)gm * ldx + gk, *pw = W + (int64_t)gn * ldw + gk;
            if (gm < M && gk < K) *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(px);
            if (gn < N && gk < K) *reinterpret_cast<float4*>(wv) = *reinterpret_cast<const float4*>(pw);
        } else {
            if (gm < M) {
                const InT* p = X + (int64_t)gm * ldx + gk;
#pragma unroll
                for (int i = 0; i < 4; ++i) if (gk + i < K) xv[i] = to_f32<InT>(p[i]);
            }
            if (gn < N) {
                const InT* p = W + (int64_t)gn * ldw + gk;
#pragma unroll
                for (int i = 0; i < 4; ++i) if (gk + i < K) wv[i] = to_f32<InT>(p[i]);
            }
        }
    };
    if (RANGES) fetch(0);
    for (int k0 = 0; k0 < K; k0 += BK) {
        const int at = RANGES ? k0 / BK & 1 : 0;
        if (!RANGES) {
            fetch(k0);
            __syncthreads();                             // the previous tile has been consumed
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            Xs[at][lk + i][lr] = xv[i];
            Ws[at][lk + i][lr] = wv[i];
        }
        __syncthreads();
        if (RANGES && k0 + BK < K) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = Xs[at][kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[at][kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float& chain = RANGES && (kk & 1) ? odd[i][j] : acc[i][j];
                    chain = fmaf(a[i], b[j], chain);
                }
        }
        if (RANGES && ((k0 + BK) % length == 0 || k0 + BK >= K)) {       // a range is complete (its length is a multiple of 32)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float sum = acc[i][j] + odd[i][j];
                    total[i][j] = k0 < length ? sum : total[i][j] + sum;
                    acc[i][j] = odd[i][j] = 0.0f;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn < N) Y[(int64_t)gm * ldy + gn] = from_f32<OutT>(RANGES ? total[i][j] : acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------- which tiles, and how many blocks share K
struct Form {
    int rows, shares;             // rows of X of a tile, blocks of a cluster that share K; 0: the 64 x 64 kernel, its blocks of an SM
};

// The form that should be done first: microseconds of the waves of its blocks, from constants fitted to measured products of 9 to 4,000
// rows, widths of 16 to 151,936 and K of 64 to 12,288 (within about a tenth).  What they say: few long rows want K shared, K of 64 or 96
// the small tiles (64 rows of 64 x 64: 4.5 us there, 6.9 in tiles of 64 x 128), and tiles that fill the GPU 128 rows each, whose
// reads of shared memory weigh half as much (1,000 rows, K 2,048, 32,768 wide: 3.25 ms, 3.67 in tiles of 64, 4.6 in small ones).
Form choose_form(int M, int N, int K) {
    struct Cost {
        int rows;
        double alone, paired;     // a step of 32 k of a block alone on its SM, of two that share one
        double range, start;      // the sum of a range put by; start and end of a block
        double meet;              // start and end where the sums meet in a cluster
    };
    constexpr Cost costs[] = {{16, 1.4, 2.55, 0.3, 2.0, 4.2}, {32, 1.5, 2.6, 0.4, 2.0, 4.3}, {64, 2.2, 4.0, 0.93, 1.5, 5.5},
                              {128, 3.5, 0.0, 0.7, 3.0, 0.0}};
    const int64_t sms = q3_device_sm_count();
    const int length = range_length(K), ranges = (K + length - 1) / length;
    const int64_t small_tiles = (int64_t)((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    Form best = {0, 2};
    // small tiles of an SM, two at a time, or three with fewer registers (4,096 wide, 300 rows, K 64: 12.6 and 9.7 us)
    double least = 1e30;
    for (int resident = 2; resident <= 3; ++resident) {
        const double each = small_tiles <= sms ? 1.0 : (double)((small_tiles + resident * sms - 1) / (resident * sms) * resident);
        const double cost = 1.5 + 0.55 * each + (K + BK - 1) / BK * (each == 1.0 ? 0.75 : 0.575 * each);
        if (cost < least) {
            least = cost;
            best = {0, resident};
        }
    }
    for (const Cost& c : costs) {
        if (M <= 16 ? c.rows != 16 : M <= 32 ? c.rows != 32 : c.rows < 64 || (c.rows == 128 && M <= 64)) continue;
        const int64_t tiles = (int64_t)((N + T_N - 1) / T_N) * ((M + c.rows - 1) / c.rows);
        for (int shares = 1; shares <= ranges && (shares == 1 || c.rows < 128); shares *= 2) {
            const int bytes = tile_bytes(c.rows, ranges, shares), per = (ranges + shares - 1) / shares;
            if (bytes > 227 * 1024) continue;
            const bool two = c.rows < 128 && bytes <= 113 * 1024;        // 114 KB a block, 1 KB of them the system's
            const double steps = shares == 1 ? (K + T_K - 1) / T_K : per * (length / T_K);
            const double ends = shares == 1 ? c.start + ranges * c.range : c.meet + (shares < 8 ? 2.0 : 0.0);   // more sums a block
            const int64_t blocks = tiles * shares, slots = two ? 2 * sms : sms, rest = blocks % slots;
            const int64_t apart = shares == 8 ? sms * 3 / 4 : sms;       // blocks that find an SM each: clusters of 8 do not fill them all
            const double cost = (double)(blocks / slots) * (steps * (two ? c.paired : c.alone) + ends) +
                                (rest == 0 ? 0.0 : steps * (two && rest > apart ? c.paired : c.alone) + ends);
            if (cost < least) {
                least = cost;
                best = {c.rows, shares};
            }
        }
    }
    return best;
}

}  // namespace

Q3_EXPORT int q3_gemm_tn_f32(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw,
                             int64_t ldy, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return Q3_ERR_BAD_SIZE;
    const cudaStream_t s = (cudaStream_t)stream;
    if (aligned16(X) && aligned16(W) && ldx % 4 == 0 && ldw % 4 == 0 && K % 4 == 0) {
        // the stream kernel's fma rate lasts for 8 rows at the memory's rate, and no longer for 16
        if (M == 1) return launch_stream<1>(X, W, Y, M, N, K, ldx, ldw, ldy, s);
        if (M == 2) return launch_stream<2>(X, W, Y, M, N, K, ldx, ldw, ldy, s);
        if (M <= 4) return launch_stream<4>(X, W, Y, M, N, K, ldx, ldw, ldy, s);
        if (M <= 8) return launch_stream<8>(X, W, Y, M, N, K, ldx, ldw, ldy, s);
        const Form form = choose_form(M, N, K);
        if (form.rows == 16) return launch_tiles<16>(X, W, Y, M, N, K, ldx, ldw, ldy, form.shares, s);
        if (form.rows == 32) return launch_tiles<32>(X, W, Y, M, N, K, ldx, ldw, ldy, form.shares, s);
        if (form.rows == 64) return launch_tiles<64>(X, W, Y, M, N, K, ldx, ldw, ldy, form.shares, s);
        if (form.rows == 128) return launch_tiles<128>(X, W, Y, M, N, K, ldx, ldw, ldy, form.shares, s);
        const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
        if (grid.y > 65535) return Q3_ERR_TOO_LARGE;
        return (int)q3_launch(form.shares == 3 ? gemm_tn_kernel<true, 3, float, float> : gemm_tn_kernel<true, 0, float, float>, grid,
                              dim3(256), 0, s, X, W, Y, M, N, K, ldx, ldw, ldy);
    }
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return Q3_ERR_TOO_LARGE;
    return (int)q3_launch(gemm_tn_kernel<false, 0, float, float>, grid, dim3(256), 0, (cudaStream_t)stream, X, W, Y, M, N, K,
                          ldx, ldw, ldy);
}

// bfloat16 operands of any width, 32-bit accumulation in one ascending chain over K; Y bfloat16 or float.
Q3_EXPORT int q3_gemm_tn_bf16(const void* X, const void* W, void* Y, int M, int N, int K, int64_t ldx, int64_t ldw,
                              int64_t ldy, int out_is_f32, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return Q3_ERR_BAD_SIZE;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return Q3_ERR_TOO_LARGE;
    if (out_is_f32)
        return (int)q3_launch(gemm_tn_kernel<false, 0, bf16, float>, grid, dim3(256), 0, (cudaStream_t)stream, (const bf16*)X,
                              (const bf16*)W, (float*)Y, M, N, K, ldx, ldw, ldy);
    return (int)q3_launch(gemm_tn_kernel<false, 0, bf16, bf16>, grid, dim3(256), 0, (cudaStream_t)stream, (const bf16*)X,
                          (const bf16*)W, (bf16*)Y, M, N, K, ldx, ldw, ldy);
}
