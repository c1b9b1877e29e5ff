// The two products of routed experts for more than a few tokens per expert (the route, the sort and the sum around
// them, and the form for few tokens, are in moe.cu): every expert's pairs (token, choice) lie one after the other, and
//
//   up   : act[slot] = f(W_gate x, W_up x)      down : y[slot] = W_down act[slot]   (32-bit output)
//
// run as ONE persistent kernel each over the tiles of all experts, on pairs of SMs (tcgen05 cta_group::2), the weights as
// the 256-row operand and the tokens as the other: D[256 rows of W, n tokens].  Experts receive unequal numbers of tokens;
// the token side of the instruction can have any multiple of 16 up to 256, so an expert's tokens are cut into equal
// tiles of at most 256 and a tile costs its tokens rounded up to 64, where a 256-row token side would cost whole
// 256s.  The tile list is walked on the device from the sorted offsets; the host never learns how many tokens an
// expert has.  Bound by the tensor cores with hundreds of tokens per expert, by reading the weights with tens:
//   16 experts of 3,072 at width 4,096, 8,324 pairs: 629 us for the gather and both products, 703 on a GPU at the
//   power cap (1.0 and 0.89 PFLOP/s; 2,924 us with mma.sync tiles of 64 x 64); 500 pairs: 222 us, 0.84 of the rate that reading the weights could have.
//
// Roles in a block: warp 0 the TMA producer, warp 1 tensor memory and (in the pair's first block) the products, warps 2-5
// drain.  The accumulator is double-buffered, so a tile drains under the products of the next.  A block's 128 rows of W are
// 64 rows of the gate and the 64 rows of up of the same features; the gate's lanes then meet up's through shared memory.
// Every wait is bounded (see tma.cuh); what gives up reports into `status`.
#include "common.cuh"
#include "tcgen05.cuh"
#include "tcgen05_pair.cuh"
#include "tma.cuh"

namespace {

constexpr int THREADS = 192, STAGES = 6, BK = 64, ROWS = 128, UMMA_K = 16;
constexpr int MAX_TOKENS = 256, TOKEN_STEP = 64;                      // tokens per tile, its granularity
constexpr int A_BYTES = ROWS * BK * 2, B_BYTES = MAX_TOKENS / 2 * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr uint32_t TMEM_COLS = 2 * MAX_TOKENS;
constexpr int MEET_BYTES = 2 * 32 * 64 * 4;                            // two buffers of 32 tokens x 64 features
enum Mode { DOWN, GATED, RELU2 };

// The tiles of all experts in order; a walker only ever moves forward.
struct Walk {
    const int* offsets;
    int n_real, n_tiles;          // experts, row tiles of one expert
    int e, first, count;          // the expert of the last tile, the number of its first tile, its tokens
    __device__ Walk(const int* o, int experts, int row_tiles) : offsets(o), n_real(experts), n_tiles(row_tiles), e(-1), first(0), count(0) {}
    __device__ int token_tiles() const { return (count + MAX_TOKENS - 1) / MAX_TOKENS; }
    // false: beyond the last tile.  row_tile, slot of the tile's first token, its tokens, the operand's size for them
    __device__ bool at(int tile, int& row_tile, int& slot, int& tokens, int& n) {
        while (e < 0 || tile >= first + token_tiles() * n_tiles) {
            if (e >= 0) first += token_tiles() * n_tiles;
            if (++e >= n_real) {
                e = n_real;
                count = 0;
                return false;
            }
            count = offsets[e + 1] - offsets[e];
        }
        const int tt = token_tiles(), local = tile - first;
        n = ((count + tt - 1) / tt + TOKEN_STEP - 1) / TOKEN_STEP * TOKEN_STEP;
        const int t0 = (local % tt) * n;                    // the token tile varies fastest: neighbours share W in the L2
        row_tile = local / tt;
        slot = offsets[e] + t0;
        tokens = max(0, min(n, count - t0));
        return true;
    }
};

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
expert_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x32, const __grid_constant__ CUtensorMap map_x64,
              const int* __restrict__ offsets,
              void* __restrict__ out, int n_real, int rows, int K, float limit, float alpha, float up_offset, int* __restrict__ status) {
    // rows: features of an expert's output (ff for up, hidden for down)
    extern __shared__ unsigned char smem_raw[];
    constexpr int FEATURES = MODE == GATED ? 128 : 256;                // of the output, per tile
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t meet = base + STAGES * STAGE_BYTES;
    const uint32_t bars = meet + (MODE == GATED ? MEET_BYTES : 0);     // full[S], empty[S], acc_full[2], acc_empty[2], slot
    const uint32_t bar_acc_full = bars + 2 * STAGES * 8, bar_acc_empty = bar_acc_full + 16, tmem_slot = bar_acc_empty + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;
    const int nkb = (K + BK - 1) / BK, n_tiles = (rows + FEATURES - 1) / FEATURES;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x32) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x64) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bars + s * 8, 1);
            mbar_init(bars + (STAGES + s) * 8, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_acc_full + b * 8, 1);
            mbar_init(bar_acc_empty + b * 8, 8);             // one arrival per drain warp of the pair
        }
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                           // the peer's barriers exist before anything signals them
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot) : "memory");
    pdl_wait();

    Walk walk(offsets, n_real, n_tiles);
    int row_tile, slot, tokens, n;
    if (warp == 0) {
        // The whole warp walks and one elected thread copies, as below: what a copy takes is in uniform registers, too.  A block's 128
        // rows of W are one box (the gate's and up's halves one dimension apart), its tokens one or two: with boxes of 64 and 32 rows, five
        // of them a K step from a lane by itself, the copies' issue was what a K step waited for (8,324 pairs of 16
        // experts 3,072 x 4,096 852 us against 703, 3,000 365 / 319; 6,000 of 2,048 x 2,048 278 / 258, 1,400 132 / 124).
        uint32_t it = 0;
        bool ok = true;
        for (int tile = first; ok && walk.at(tile, row_tile, slot, tokens, n); tile += stride) {
            const int half = __shfl_sync(0xffffffffu, n, 0) / 2, x0 = __shfl_sync(0xffffffffu, slot, 0) + (int)rank * half;
            const int w0 = __shfl_sync(0xffffffffu, row_tile, 0) * FEATURES + (int)rank * (FEATURES / 2), e = __shfl_sync(0xffffffffu, walk.e, 0);
            for (int kb = 0; kb < nkb; ++kb, ++it) {
                const uint32_t s = it % STAGES;
                ok = mbar_wait_warp(bars + (STAGES + s) * 8, ((it / STAGES) & 1u) ^ 1u);
                if (!ok) {
                    if (lane == 0) atomicExch(status, 1);
                    break;
                }
                const uint32_t a = base + s * STAGE_BYTES, b = a + A_BYTES;
                const uint32_t full = map_to_rank(bars + s * 8, 0);
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(bars + s * 8, 2 * (A_BYTES + half * BK * 2));       // both blocks' bytes
                    if (MODE == GATED) tma_load_3d_pair(a, &map_w, full, kb * BK, w0, 2 * e);
                    else tma_load_3d_pair(a, &map_w, full, kb * BK, w0, e);
                    int r = 0;
                    for (; r + 64 <= half; r += 64) tma_load_2d_pair(b + r * BK * 2, &map_x64, full, kb * BK, x0 + r);
                    if (r < half) tma_load_2d_pair(b + r * BK * 2, &map_x32, full, kb * BK, x0 + r);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // the whole warp walks and one elected thread issues: descriptors in uniform registers, which the instruction takes
        if (rank == 0) {
            const uint64_t desc0 = desc_k_major(base);
            uint32_t it = 0, local = 0;
            bool ok = true;
            tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);
            for (int tile = first; ok && walk.at(tile, row_tile, slot, tokens, n); tile += stride, ++local) {
                const uint32_t buf = local & 1u, idesc = make_idesc_mn(2 * ROWS, __shfl_sync(0xffffffffu, n, 0));
                ok = mbar_wait_warp(bar_acc_empty + buf * 8, ((local >> 1) & 1u) ^ 1u);      // both blocks have drained it
                if (!ok) {
                    if (lane == 0) atomicExch(status, 4);
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * MAX_TOKENS;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const uint32_t s = it % STAGES;
                    ok = mbar_wait_warp(bars + s * 8, (it / STAGES) & 1u);
                    if (!ok) {
                        if (lane == 0) atomicExch(status, 2);
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = desc0 + (uint64_t)(s * (STAGE_BYTES >> 4)), db = da + (A_BYTES >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k)
                            tc_mma_pair(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        tc_commit_pair(bars + (STAGES + s) * 8);
                    }
                    __syncwarp();
                }
                if (elect_one()) tc_commit_pair(bar_acc_full + buf * 8);
                __syncwarp();
            }
        }
    } else {
        // lane = row of W: a warp writes 32 neighbouring features of a token at once
        const int quarter = warp & 3, row = quarter * 32 + lane;
        uint32_t local = 0;
        for (int tile = first; walk.at(tile, row_tile, slot, tokens, n); tile += stride, ++local) {
            const uint32_t buf = local & 1u;
            const bool landed = mbar_wait(bar_acc_full + buf * 8, (local >> 1) & 1u);
            if (!landed) atomicExch(status, 3);
            uint32_t all;                                     // the four warps meet below: they go on or leave together
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "=r"(all) : "r"((uint32_t)landed) : "memory");
            if (!all) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * MAX_TOKENS;
            uint32_t turn = 0;
#pragma unroll 1
            for (int c = 0; c < tokens; c += 32, turn ^= 1u) {
                uint32_t r[32];
                tc_ld32(acc + (uint32_t)c, r);
                tc_wait_ld();
                const int live = min(32, tokens - c);
                if constexpr (MODE == GATED) {
                    // rows 0..63 are gates, 64..127 the ups of the same features
                    const uint32_t there = meet + turn * (MEET_BYTES / 2) + (uint32_t)(row & 63) * 4u;
                    if (quarter >= 2) {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            asm volatile("st.shared.b32 [%0], %1;" ::"r"(there + (uint32_t)j * 256u), "r"(r[j]) : "memory");
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    const int f = row_tile * FEATURES + (int)rank * 64 + row;
                    if (quarter < 2 && f < rows) {
                        bf16* to = (bf16*)out + (int64_t)(slot + c) * rows + f;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            float u;
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u) : "r"(there + (uint32_t)j * 256u) : "memory");
                            const float g = fminf(__uint_as_float(r[j]), limit);
                            u = fminf(fmaxf(u, -limit), limit);
                            if (j < live) to[(int64_t)j * rows] = __float2bfloat16_rn(g / (1.0f + expf(-alpha * g)) * (u + up_offset));
                        }
                    }
                } else {
                    const int f = row_tile * FEATURES + (int)rank * 128 + row;
                    if (f < rows) {
                        if constexpr (MODE == RELU2) {
                            bf16* to = (bf16*)out + (int64_t)(slot + c) * rows + f;
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                const float v = fmaxf(__uint_as_float(r[j]), 0.0f);
                                if (j < live) to[(int64_t)j * rows] = __float2bfloat16_rn(v * v);
                            }
                        } else {
                            float* to = (float*)out + (int64_t)(slot + c) * rows + f;
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (j < live) to[(int64_t)j * rows] = __uint_as_float(r[j]);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_rank(bar_acc_empty + buf * 8, 0));   // this warp's share is drained
        }
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync();                                           // the peer reads this block's memory and barriers until here
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// x[slot] = h[token of the pair in that slot], 16 bytes a thread: TMA fetches boxes of neighbouring rows.  (17 MB to 68 MB
// written and read back from the L2 for thousands of tokens; 5 % of the products.)
__global__ void __launch_bounds__(256)
gather_tokens_kernel(const uint4* __restrict__ h, const int* __restrict__ pair_of_slot, const int* __restrict__ offsets, int n_real,
                     uint4* __restrict__ x, int top, int packets) {
    pdl_launch_dependents();
    pdl_wait();
    const int slots = offsets[n_real];                        // pairs of identity experts have no slot
    const int64_t total = (int64_t)slots * packets;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int s = (int)(i / packets), c = (int)(i % packets);
        x[i] = h[(int64_t)(pair_of_slot[s] / top) * packets + c];
    }
}

// `count` matrices [rows, K] one after the other, fetched in boxes of [box_count, box_rows, BK] with 128-byte swizzle; beyond a
// matrix's last row a box reads zeros.
bool make_weight_map(CUtensorMap* map, const bf16* W, int count, int rows, int K, int box_rows, int box_count) {
    const Q3EncodeTiled fn = q3_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)count};
    const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)rows * K * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, (cuuint32_t)box_count}, elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
int launch(const bf16* W, const bf16* X, const int* offsets, void* out, int n_pairs, int n_real, int rows, int K, float limit,
           float alpha, float up_offset, int* status, cudaStream_t stream) {
    constexpr int SMEM = STAGES * STAGE_BYTES + (MODE == GATED ? MEET_BYTES : 0) + 1024 + 256;
    constexpr int FEATURES = MODE == GATED ? 128 : 256;
    static Q3PerDevice configured;
    const cudaError_t e = q3_allow_shared_memory(expert_kernel<MODE>, SMEM, configured);
    if (e != cudaSuccess) return (int)e;
    CUtensorMap map_w, map_x32, map_x64;
    if (!make_weight_map(&map_w, W, n_real * (MODE == GATED ? 2 : 1), rows, K, MODE == GATED ? 64 : 128, MODE == GATED ? 2 : 1) ||
        !q3_make_map_bf16(&map_x32, X, n_pairs, K, 32, BK, true) || !q3_make_map_bf16(&map_x64, X, n_pairs, K, 64, BK, true))
        return Q3_ERR_BAD_SIZE;
    // an upper bound on the tiles of all experts together
    const int64_t tiles = ((int64_t)n_pairs / MAX_TOKENS + (n_real < n_pairs ? n_real : n_pairs)) * ((rows + FEATURES - 1) / FEATURES);
    const int pairs = tiles < q3_device_sm_count() / 2 ? (int)tiles : q3_device_sm_count() / 2;
    return (int)q3_launch_cluster(expert_kernel<MODE>, dim3(2 * pairs), dim3(THREADS), (size_t)SMEM, stream, dim3(2, 1, 1), map_w, map_x32, map_x64,
                                  offsets, out, n_real, rows, K, limit, alpha, up_offset, status);
}

}  // namespace

// The experts' two products for any number of pairs; see q3_moe_experts_tc_bf16 for the arguments.  `x` [n_pairs, hidden]:
// room for the pairs' rows of h.  Widths in steps of 8.
Q3_EXPORT int q3_moe_experts_tcgen05_bf16(const void* h, const void* w_gate_up, const void* w_down, const int* offsets,
                                          const int* pair_of_slot, void* x, void* act, float* y, int n_pairs, int n_real, int top,
                                          int hidden, int ff, float limit, float alpha, float up_offset, int gated, int* status,
                                          void* stream_) {
    if (n_pairs <= 0 || n_real <= 0) return 0;
    if (hidden <= 0 || ff <= 0 || hidden % 8 != 0 || ff % 8 != 0 || top <= 0) return Q3_ERR_BAD_SIZE;
    if ((int64_t)n_real * 2 * ff > 0x7fffffff || (int64_t)n_real * hidden > 0x7fffffff) return Q3_ERR_TOO_LARGE;
    if (!aligned16(h) || !aligned16(w_gate_up) || !aligned16(w_down) || !aligned16(x) || !aligned16(act)) return Q3_ERR_MISALIGNED;
    const cudaStream_t stream = (cudaStream_t)stream_;
    const int64_t packets = (int64_t)n_pairs * (hidden / 8), blocks = (packets + 255) / 256, most = (int64_t)q3_device_sm_count() * 8;
    int code = (int)q3_launch(gather_tokens_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, stream, (const uint4*)h,
                              pair_of_slot, offsets, n_real, (uint4*)x, top, hidden / 8);
    if (code != 0) return code;
    const bf16 *wu = (const bf16*)w_gate_up, *wd = (const bf16*)w_down, *xs = (const bf16*)x;
    code = gated ? launch<GATED>(wu, xs, offsets, act, n_pairs, n_real, ff, hidden, limit, alpha, up_offset, status, stream)
                 : launch<RELU2>(wu, xs, offsets, act, n_pairs, n_real, ff, hidden, limit, alpha, up_offset, status, stream);
    if (code != 0) return code;
    return launch<DOWN>(wd, (const bf16*)act, offsets, y, n_pairs, n_real, hidden, ff, limit, alpha, up_offset, status, stream);
}
