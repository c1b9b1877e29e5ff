// A routed feed-forward (mixture of experts) in five kernels, none of which needs the host to know how many
// tokens an expert received, so a step can be captured:
//
//   moe_route   : a block per token, or per four tokens of a long prompt.  Router logits z = W_r h in 32-bit (a warp per
//                 output, a lane's terms in ascending order, then the lanes': one order whatever the step),
//                 scores s = softmax(z) over all outputs, choice scores s + correction, restricted to the
//                 `keep` groups (of `count` equal groups of neighbours) whose best choice score is largest;
//                 the `top` largest choice scores win (ties: the lower index); the weights are their plain
//                 scores s.  The last `identity` outputs are experts without tensors whose output is the
//                 token itself: their weights are summed into id_weight[token].
//                 `by_logit` 1: the `top` largest logits win instead and the weights are the softmax over the chosen
//                 logits only (the correction, if there is one, is a bias on the logits); 2: the scores are sigmoid(z), each output by itself.  `group_pair`: a group's score is
//                 the sum of its two largest choice scores.  The weights are multiplied by `weight_scale`.  With `gate_out`, the router matrix has one more row after the outputs whose logit
//                 is no expert's: gate_out[token] = sigmoid(that logit), the weight of a shared expert.
//   moe_sort    : one block.  Counts the (token, choice) pairs of every real expert, lays the experts out one
//                 after the other (offsets) and gives every pair its place (slot_of_pair, pair_of_slot).
//   moe_up      : act[slot] = f(W_gate x, W_up x) for the pairs of each expert, a tile of TM pairs x 64
//                 columns per block; g = min(gate, limit), u = clamp(up, -limit, limit),
//                 f = g sigmoid(alpha g) (u + up_offset)  (limit = infinity, alpha = 1, up_offset = 0: SiLU(gate) * up).
//                 Experts without a gate: act[slot] = max(W_up x, 0)^2, one matrix instead of two.
//   moe_down    : y[slot] = W_down act[slot], the same tiling, 32-bit output.
//   moe_combine : out[token] = T( sum_k weight_k y[slot(token, k)] + id_weight h[token] + shared_w[token] shared[token] ),
//                 the last term for a shared expert that every token uses (may be absent; without shared_w its weight
//                 is 1).
//
// The products accumulate in 32-bit.  Float tiles run on fmaf in ascending order of k whatever the tile a pair falls into, so
// a token's result does not depend on what else is in the step; bfloat16 tiles run on the tensor cores when the widths are
// multiples of 32, else on fmaf too.  Of the two tensor-core forms (few tokens per expert: `few` below, eight warps' shares of K added;
// more: moe_tcgen05.cu) the step's number of pairs selects one, so there a token's result does hang on the rest of the step, by the
// rounding of sums in another order.
#include "common.cuh"

namespace {

__device__ __forceinline__ bool aligned16_device(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

constexpr int MAX_OUTPUTS = 1024, MANY_OUTPUTS = 256;     // of the router; where four tokens share a block

// What `choose_by_one` does, for up to 32 outputs in one group: lane e has output e's logit.  The same operations in the same
// order, a lane's work being one output's.
__device__ __forceinline__ void choose_by_lanes(float z, const float* __restrict__ correction, int* __restrict__ top_ids, float* __restrict__ top_w,
                                                float* __restrict__ id_weight, int n_out, int n_real, int top, int by_logit, float weight_scale,
                                                int64_t t) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool mine = lane < n_out;
    float choice;
    if (by_logit == 1) {
        if (mine && correction != nullptr) z += correction[lane];
        choice = z;
    } else {
        if (by_logit == 2) {
            z = 1.0f / (1.0f + expf(-z));
        } else {
            const float m = warp_max(mine ? z : -INFINITY);
            z = expf(z - m);
            float sum = 0.0f;
            for (int e = 0; e < n_out; ++e) sum += __shfl_sync(ALL, z, e);
            z *= 1.0f / sum;
        }
        choice = z + (mine && correction != nullptr ? correction[lane] : 0.0f);
    }
    if (!mine) choice = -INFINITY;
    float best_z = 0.0f, sum = 0.0f, idw = 0.0f, w_of_lane = 0.0f;       // w_of_lane: of the place `lane` among the chosen
    int id_of_lane = 0;
    for (int k = 0; k < top; ++k) {
        // the largest choice score, of equal ones the lowest output; none left: output 0
        float best_c = choice;
        int best = choice > -INFINITY ? lane : 32;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float c = __shfl_xor_sync(ALL, best_c, o);
            const int e = __shfl_xor_sync(ALL, best, o);
            if (e < 32 && (best == 32 || c > best_c || (c == best_c && e < best))) {
                best_c = c;
                best = e;
            }
        }
        if (best == 32) best = 0;
        const float zb = __shfl_sync(ALL, z, best);
        if (lane == best) choice = -INFINITY;
        float w;
        if (by_logit == 1) {
            if (k == 0) best_z = zb;
            w = expf(zb - best_z);
            sum += w;
        } else {
            w = zb * weight_scale;
            if (best >= n_real) idw += w;
        }
        if (lane == k) {
            id_of_lane = best;
            w_of_lane = w;
        }
    }
    if (by_logit == 1) {
        w_of_lane *= 1.0f / sum;
        for (int k = 0; k < top; ++k) {
            const float w = __shfl_sync(ALL, w_of_lane, k);
            if (__shfl_sync(ALL, id_of_lane, k) >= n_real) idw += w;
        }
    }
    if (lane < top) {                                    // top <= n_out <= 32
        top_ids[t * top + lane] = id_of_lane;
        top_w[t * top + lane] = w_of_lane;
    }
    if (lane == 0) id_weight[t] = idw;
}

// z [n_out]: a token's logits; choice, group_best, group_kept: room for as many.  By one thread.
__device__ __forceinline__ void choose_by_one(float* z, float* choice, float* group_best, unsigned char* group_kept,
                                              const float* __restrict__ correction, int* __restrict__ top_ids, float* __restrict__ top_w,
                                              float* __restrict__ id_weight, int n_out, int n_real, int top, int group_count, int group_keep,
                                              int by_logit, int group_pair, float weight_scale, int64_t t) {
    if (by_logit == 1) {
        // the largest logits (ties: the lower index), weighted by the softmax over the chosen logits alone
        float best_z = 0.0f, sum = 0.0f;
        for (int e = 0; e < n_out; ++e) {
            if (correction != nullptr) z[e] += correction[e];
            choice[e] = z[e];
        }
        for (int k = 0; k < top; ++k) {
            int best = -1;
            for (int e = 0; e < n_out; ++e)
                if (choice[e] > -INFINITY && (best < 0 || choice[e] > choice[best])) best = e;
            if (best < 0) best = 0;
            if (k == 0) best_z = z[best];
            choice[best] = -INFINITY;
            const float w = expf(z[best] - best_z);
            top_ids[t * top + k] = best;
            top_w[t * top + k] = w;
            sum += w;
        }
        const float inv = 1.0f / sum;
        float idw = 0.0f;
        for (int k = 0; k < top; ++k) {
            top_w[t * top + k] *= inv;
            if (top_ids[t * top + k] >= n_real) idw += top_w[t * top + k];
        }
        id_weight[t] = idw;
        return;
    }
    if (by_logit == 2) {                         // every output's score by itself: sigmoid(z)
        for (int e = 0; e < n_out; ++e) {
            z[e] = 1.0f / (1.0f + expf(-z[e]));
            choice[e] = z[e] + (correction != nullptr ? correction[e] : 0.0f);
        }
    } else {
        float m = -INFINITY, sum = 0.0f;
        for (int e = 0; e < n_out; ++e) m = fmaxf(m, z[e]);
        for (int e = 0; e < n_out; ++e) {
            z[e] = expf(z[e] - m);
            sum += z[e];
        }
        const float inv = 1.0f / sum;
        for (int e = 0; e < n_out; ++e) {
            z[e] *= inv;
            choice[e] = z[e] + (correction != nullptr ? correction[e] : 0.0f);
        }
    }
    if (group_count > 1) {
        // a group's score is its best choice score, or (`group_pair`) the sum of its two best; the `keep` best groups
        // stay (of equal groups the earlier one)
        const int size = n_out / group_count;
        for (int g = 0; g < group_count; ++g) {
            float best = -INFINITY, second = -INFINITY;
            for (int e = 0; e < size; ++e) {
                const float c = choice[g * size + e];
                if (c > best) {
                    second = best;
                    best = c;
                } else if (c > second) {
                    second = c;
                }
            }
            group_best[g] = group_pair && size > 1 ? best + second : best;
            group_kept[g] = 0;
        }
        for (int k = 0; k < group_keep; ++k) {
            int best = -1;
            for (int g = 0; g < group_count; ++g)
                if (!group_kept[g] && (best < 0 || group_best[g] > group_best[best])) best = g;
            group_kept[best] = 1;
        }
        for (int e = 0; e < n_out; ++e)
            if (!group_kept[e / size]) choice[e] = -INFINITY;        // minus infinity, not 0: choice scores can be negative
    }
    float idw = 0.0f;
    for (int k = 0; k < top; ++k) {
        int best = -1;
        for (int e = 0; e < n_out; ++e)
            if (choice[e] > -INFINITY && (best < 0 || choice[e] > choice[best])) best = e;      // ties: the lower index
        if (best < 0) best = 0;                  // fewer candidates than `top` (the caller's sizes rule it out)
        choice[best] = -INFINITY;
        top_ids[t * top + k] = best;
        top_w[t * top + k] = z[best] * weight_scale;
        if (best >= n_real) idw += z[best] * weight_scale;
    }
    id_weight[t] = idw;
}

// The router matrix is read through the L2 once per block, which bounds the kernel for many tokens (one token a block: 140 KB each
// at width 4,096 and 16 outputs): TOKENS tokens a block share it.  4,162 tokens: 71 us with one a block, 64 with four; 8 tokens
// of width 2,048: 7.5 us by eight warps, 5.8 by sixteen with eight packets of a row asked for together.  Sixteen warps are for steps
// whose blocks are all resident at once: of more than 32 outputs one thread chooses while the block waits for it, and then blocks an SM
// count (4,100 tokens of width 96, 300 outputs: 507 us by eight warps, 1,046 by sixteen; 1,000 tokens 243 and 388).
template <typename T, int TOKENS, int OUTPUTS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
moe_route_kernel(const T* __restrict__ h, const T* __restrict__ w_router, const float* __restrict__ correction,
                 int* __restrict__ top_ids, float* __restrict__ top_w, float* __restrict__ id_weight, int64_t n_tokens, int hidden, int n_out,
                 int n_real, int top, int group_count, int group_keep, int by_logit, float* __restrict__ gate_out, int group_pair,
                 float weight_scale) {
    __shared__ float z[TOKENS][OUTPUTS];
    __shared__ float choice[TOKENS][OUTPUTS];
    __shared__ float group_best[TOKENS][OUTPUTS];
    __shared__ unsigned char group_kept[TOKENS][OUTPUTS];
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t0 = (int64_t)blockIdx.x * TOKENS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const T* x[TOKENS];                                  // tokens beyond the last read the last one
#pragma unroll
    for (int n = 0; n < TOKENS; ++n) x[n] = h + min(t0 + n, n_tokens - 1) * hidden;
    // a warp per router output; 16-byte packets when the rows allow it (the order of the sum is fixed either way)
    constexpr int VEC = Pack<T>::N;
    const bool packed = hidden % VEC == 0 && aligned16_device(h) && aligned16_device(w_router);
    const int n_rows = n_out + (gate_out != nullptr ? 1 : 0);
    for (int e = warp; e < n_rows; e += WARPS) {
        const T* w = w_router + (int64_t)e * hidden;
        float dot[TOKENS];
#pragma unroll
        for (int n = 0; n < TOKENS; ++n) dot[n] = 0.0f;
        if (packed) {
#pragma unroll(TOKENS == 1 ? 8 : 2)
            for (int c = lane * VEC; c < hidden; c += 32 * VEC) {
                const Pack<T> wv = load_pack<T>(w + c);
                Pack<T> xv[TOKENS];
#pragma unroll
                for (int n = 0; n < TOKENS; ++n) xv[n] = load_pack<T>(x[n] + c);
#pragma unroll
                for (int n = 0; n < TOKENS; ++n)
#pragma unroll
                    for (int i = 0; i < VEC; ++i) dot[n] = fmaf(wv.get(i), xv[n].get(i), dot[n]);
            }
        } else {
            for (int c = lane; c < hidden; c += 32)
#pragma unroll
                for (int n = 0; n < TOKENS; ++n) dot[n] = fmaf(to_f32<T>(w[c]), to_f32<T>(x[n][c]), dot[n]);
        }
#pragma unroll
        for (int n = 0; n < TOKENS; ++n) {
            const float sum = warp_sum(dot[n]);
            if (lane == 0) z[n][e] = sum;
        }
    }
    __syncthreads();
    const int64_t t = t0 + warp;
    if (warp >= TOKENS || t >= n_tokens) return;
    const int of = TOKENS == 1 ? 0 : warp;               // a number the compiler knows where one token has the block
    if (lane == 0 && gate_out != nullptr) gate_out[t] = 1.0f / (1.0f + expf(-z[of][n_out]));
    if (n_out <= 32 && group_count == 1) {
        choose_by_lanes(lane < n_out ? z[of][lane] : 0.0f, correction, top_ids, top_w, id_weight, n_out, n_real, top, by_logit, weight_scale, t);
        return;
    }
    if (lane == 0)
        choose_by_one(z[of], choice[of], group_best[of], group_kept[of], correction, top_ids, top_w, id_weight, n_out, n_real, top,
                      group_count, group_keep, by_logit, group_pair, weight_scale, t);
}

// counts [E + 1] (the last cell: pairs of identity experts), offsets [E + 1]
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int* __restrict__ top_ids, int n_pairs, int n_real, int* __restrict__ offsets, int* __restrict__ slot_of_pair,
                int* __restrict__ pair_of_slot) {
    extern __shared__ int counts[];            // [n_real] counts, then [n_real + 1] running offsets
    int* start = counts + n_real;
    pdl_launch_dependents();
    pdl_wait();
    for (int e = threadIdx.x; e < n_real; e += blockDim.x) counts[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = top_ids[p];
        if (e < n_real) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < n_real; ++e) {
            start[e] = run;
            offsets[e] = run;
            run += counts[e];
        }
        start[n_real] = run;
        offsets[n_real] = run;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n_real; e += blockDim.x) counts[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = top_ids[p];
        int slot = -1;
        if (e < n_real) {
            slot = start[e] + atomicAdd(&counts[e], 1);
            pair_of_slot[slot] = p;
        }
        slot_of_pair[p] = slot;
    }
}

// Which expert and which of its row tiles block `tile` works on; false: beyond the last tile.
template <int TM>
__device__ __forceinline__ bool find_tile(const int* __restrict__ offsets, int n_real, int tile, int& expert, int& row0, int& rows) {
    int seen = 0;
    for (int e = 0; e < n_real; ++e) {
        const int n = offsets[e + 1] - offsets[e];
        const int tiles = (n + TM - 1) / TM;
        if (tile < seen + tiles) {
            expert = e;
            row0 = offsets[e] + (tile - seen) * TM;
            rows = min(TM, offsets[e + 1] - row0);
            return true;
        }
        seen += tiles;
    }
    return false;
}

constexpr int TN = 64, TK = 32;

// A tile of TM rows of X (gathered through `src_row`) times TN rows of W, accumulated over K in 32-bit on fmaf.
// 256 threads: thread (tx, ty) owns rows ty, ty + 16, ... (TM / 16 of them, at least 1 with TM = 8: ty < 8) and
// columns tx * 4 .. + 3.  DUAL: two weight matrices at once (gate and up).
template <typename T, int TM, bool DUAL>
__device__ __forceinline__ void tile_product(const T* __restrict__ X, int64_t x_stride, const int* src_row, int rows,
                                             const T* __restrict__ W0, const T* __restrict__ W1, int n_cols, int col0, int K,
                                             float (&acc0)[(TM + 15) / 16][4], float (&acc1)[(TM + 15) / 16][4], float* xs, float* ws0,
                                             float* ws1) {
    constexpr int RPT = (TM + 15) / 16;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
    for (int a = 0; a < RPT; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc0[a][b] = acc1[a][b] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += TK) {
        __syncthreads();
        for (int x = tid; x < TM * TK; x += 256) {
            const int rr = x / TK, kk = x % TK;
            xs[rr * (TK + 1) + kk] = (rr < rows && k0 + kk < K) ? to_f32<T>(X[(int64_t)src_row[rr] * x_stride + k0 + kk]) : 0.0f;
        }
        for (int x = tid; x < TN * TK; x += 256) {
            const int cc = x / TK, kk = x % TK;
            const bool ok = col0 + cc < n_cols && k0 + kk < K;
            ws0[cc * (TK + 1) + kk] = ok ? to_f32<T>(W0[(int64_t)(col0 + cc) * K + k0 + kk]) : 0.0f;
            if (DUAL) ws1[cc * (TK + 1) + kk] = ok ? to_f32<T>(W1[(int64_t)(col0 + cc) * K + k0 + kk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < TK; ++kk) {
            float wv0[4], wv1[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                wv0[b] = ws0[(tx * 4 + b) * (TK + 1) + kk];
                if (DUAL) wv1[b] = ws1[(tx * 4 + b) * (TK + 1) + kk];
            }
#pragma unroll
            for (int a = 0; a < RPT; ++a) {
                const int rr = ty + a * 16;
                if (rr < TM) {
                    const float xv = xs[rr * (TK + 1) + kk];
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        acc0[a][b] = fmaf(xv, wv0[b], acc0[a][b]);
                        if (DUAL) acc1[a][b] = fmaf(xv, wv1[b], acc1[a][b]);
                    }
                }
            }
        }
    }
}

template <typename T, int TM, bool GATE>
__global__ void __launch_bounds__(256)
moe_up_kernel(const T* __restrict__ h, const T* __restrict__ w_gate_up, const int* __restrict__ offsets,
              const int* __restrict__ pair_of_slot, T* __restrict__ act, int n_real, int top, int hidden, int ff, float limit,
              float alpha, float up_offset) {
    __shared__ float xs[TM * (TK + 1)], ws0[TN * (TK + 1)], ws1[TN * (TK + 1)];
    __shared__ int src_row[TM];
    pdl_launch_dependents();
    pdl_wait();
    int expert, row0, rows;
    if (!find_tile<TM>(offsets, n_real, blockIdx.y, expert, row0, rows)) return;
    if (threadIdx.x < TM) src_row[threadIdx.x] = threadIdx.x < rows ? pair_of_slot[row0 + threadIdx.x] / top : 0;
    const int col0 = blockIdx.x * TN;
    const T* wg = w_gate_up + (int64_t)expert * (GATE ? 2 : 1) * ff * hidden;      // [gate rows; up rows] of the expert (or up rows alone)
    float g[(TM + 15) / 16][4], u[(TM + 15) / 16][4];
    tile_product<T, TM, GATE>(h, hidden, src_row, rows, wg, GATE ? wg + (int64_t)ff * hidden : nullptr, ff, col0, hidden, g, u, xs, ws0, ws1);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int a = 0; a < (TM + 15) / 16; ++a) {
        const int rr = ty + a * 16;
        if (rr >= rows || rr >= TM) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int c = col0 + tx * 4 + b;
            if (c >= ff) continue;
            if constexpr (!GATE) {
                const float v = fmaxf(g[a][b], 0.0f);
                act[(int64_t)(row0 + rr) * ff + c] = from_f32<T>(v * v);
                continue;
            }
            const float gv = fminf(g[a][b], limit), uv = fminf(fmaxf(u[a][b], -limit), limit);
            act[(int64_t)(row0 + rr) * ff + c] = from_f32<T>(gv / (1.0f + expf(-alpha * gv)) * (uv + up_offset));
        }
    }
}

template <typename T, int TM>
__global__ void __launch_bounds__(256)
moe_down_kernel(const T* __restrict__ act, const T* __restrict__ w_down, const int* __restrict__ offsets, float* __restrict__ y,
                int n_real, int hidden, int ff) {
    __shared__ float xs[TM * (TK + 1)], ws0[TN * (TK + 1)];
    __shared__ int src_row[TM];
    pdl_launch_dependents();
    pdl_wait();
    int expert, row0, rows;
    if (!find_tile<TM>(offsets, n_real, blockIdx.y, expert, row0, rows)) return;
    if (threadIdx.x < TM) src_row[threadIdx.x] = row0 + min((int)threadIdx.x, rows - 1);
    const int col0 = blockIdx.x * TN;
    float acc[(TM + 15) / 16][4], unused[(TM + 15) / 16][4];
    tile_product<T, TM, false>(act, ff, src_row, rows, w_down + (int64_t)expert * hidden * ff, nullptr, hidden, col0, ff, acc, unused,
                               xs, ws0, nullptr);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int a = 0; a < (TM + 15) / 16; ++a) {
        const int rr = ty + a * 16;
        if (rr >= rows || rr >= TM) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int c = col0 + tx * 4 + b;
            if (c < hidden) y[(int64_t)(row0 + rr) * hidden + c] = acc[a][b];
        }
    }
}

// Bound by the bytes of y, the shared expert's rows and the output; rows of whole 16-byte packets in packets (VEC), the slots
// and weights of the token read once.  4,162 tokens of width 4,096, two experts and a shared one: 85.7 us value by value,
// 35.9 in packets; a decode step of 8 tokens of width 2,048: 7.6 and 2.9.  Below 512 the threads of value by value are ahead
// (1,184 tokens of width 96: 2.3 us, 2.5 in packets).
template <typename T, int VEC>
__global__ void moe_combine_kernel(const float* __restrict__ y, const T* __restrict__ h, const int* __restrict__ slot_of_pair,
                                   const float* __restrict__ top_w, const float* __restrict__ id_weight, T* __restrict__ out,
                                   int top, int hidden, const T* __restrict__ shared, const float* __restrict__ shared_w) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const float idw = id_weight[t], sw = shared != nullptr && shared_w != nullptr ? shared_w[t] : 1.0f;
    for (int c = threadIdx.x * VEC; c < hidden; c += blockDim.x * VEC) {
        float v[VEC], from[VEC];
        auto packet = [&](const T* p) {
            if constexpr (VEC == 1) {
                from[0] = to_f32<T>(*p);
            } else {
                const Pack<T> raw = load_pack<T>(p);
#pragma unroll
                for (int i = 0; i < VEC; ++i) from[i] = raw.get(i);
            }
        };
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] = 0.0f;
        if (idw != 0.0f) {
            packet(h + t * hidden + c);
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[i] = idw * from[i];
        }
#pragma unroll 2
        for (int k = 0; k < top; ++k) {
            const int slot = slot_of_pair[t * top + k];
            if (slot < 0) continue;
            const float w = top_w[t * top + k];
            const float* row = y + (int64_t)slot * hidden + c;
            if constexpr (VEC == 1) {
                v[0] = fmaf(w, row[0], v[0]);
            } else {
#pragma unroll
                for (int i = 0; i < VEC; i += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(row + i);
                    v[i] = fmaf(w, r.x, v[i]);
                    v[i + 1] = fmaf(w, r.y, v[i + 1]);
                    v[i + 2] = fmaf(w, r.z, v[i + 2]);
                    v[i + 3] = fmaf(w, r.w, v[i + 3]);
                }
            }
        }
        if (shared != nullptr) {
            packet(shared + t * hidden + c);
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[i] = fmaf(sw, from[i], v[i]);
        }
        if constexpr (VEC == 1) {
            out[t * hidden + c] = from_f32<T>(v[0]);
        } else {
            Pack<T> o;
#pragma unroll
            for (int i = 0; i < VEC; ++i) o.set(i, v[i]);
            store_pack<T>(out + t * hidden + c, o);
        }
    }
}

// ---------------------------------------------------------------- few tokens per expert, on the tensor cores (bfloat16)
// A decode step: what counts is reading every chosen expert's weights once.  A block owns 16 rows of W (8 of the gate and the
// 8 of up of the same features) and up to 8 of an expert's pairs; its 8 warps split K.  As in the few-row product of the
// dense layers a lane reads 16 contiguous bytes of a W row and hands them to mma.m16n8k16 as they come (both operands permute
// k the same way), four blocks of 32 k in flight a warp and three blocks an SM; the warps' sums are added in warp order.
// 8 tokens, 16 experts of 2,048 at width 2,048, two per token (276 MB): both products 65 us from cold caches, 181 with tiles of
// 64 x 64 fed by asynchronous copies of 64 bytes a row, which this replaced.
namespace few {

constexpr int WARPS = 8, IN_FLIGHT = 4, PAIRS = 8;
enum Mode { GATED, RELU2, DOWN };

__device__ __forceinline__ uint4 ld_stream16(const void* p) {
    uint4 v;   // not volatile: the compiler may hoist and batch these loads
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// find_tile by a warp: a lane per expert, 32 experts at a time.
template <int TM>
__device__ __forceinline__ bool find_tile_warp(const int* __restrict__ offsets, int n_real, int tile, int& expert, int& row0, int& rows) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int e0 = 0; e0 < n_real; e0 += 32) {
        const int e = e0 + lane;
        const int begin = offsets[min(e, n_real)], end = offsets[min(e + 1, n_real)];
        const int tiles = (end - begin + TM - 1) / TM;
        int upto = tiles;                                   // tiles of this lane's and all earlier experts of the 32
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned past = __ballot_sync(0xffffffffu, tile < before + upto);
        if (past != 0) {
            const int who = __ffs(past) - 1;
            const int local = tile - before - (__shfl_sync(0xffffffffu, upto, who) - __shfl_sync(0xffffffffu, tiles, who));
            expert = e0 + who;
            row0 = __shfl_sync(0xffffffffu, begin, who) + local * TM;
            rows = min(TM, __shfl_sync(0xffffffffu, end, who) - row0);
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// X [.., K]: h, a row per token (GATED, RELU2), or act, a row per slot (DOWN); `features` of an expert's output.
template <int MODE>
__global__ void __launch_bounds__(WARPS * 32, 3)
expert_kernel(const bf16* __restrict__ X, const bf16* __restrict__ W, const int* __restrict__ offsets, const int* __restrict__ pair_of_slot,
              void* __restrict__ out, int n_real, int top, int features, int K, float limit, float alpha, float up_offset) {
    constexpr int LD = 17, PER_BLOCK = MODE == GATED ? 8 : 16;
    __shared__ float red[WARPS][PAIRS * LD];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane >> 2, tq = lane & 3;
    int expert, row0, rows;
    if (!find_tile_warp<PAIRS>(offsets, n_real, blockIdx.y, expert, row0, rows)) return;
    const int f0 = blockIdx.x * PER_BLOCK, nkb = (K + 31) >> 5;
    const int kb_begin = warp * nkb / WARPS, kb_end = (warp + 1) * nkb / WARPS;

    const bf16* wrow[2];
    bool wok[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int f = MODE == GATED ? f0 + quad : f0 + h * 8 + quad;
        wok[h] = f < features;
        const int64_t row = MODE == GATED ? ((int64_t)expert * 2 + h) * features + f : (int64_t)expert * features + f;
        wrow[h] = W + (wok[h] ? row : 0) * K + tq * 8;
    }
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 w[IN_FLIGHT][2], x[IN_FLIGHT];
    auto load_w = [&](int s, int kb) {
        const int k = kb * 32;
        const bool in = kb < kb_end && k + tq * 8 + 8 <= K;
#pragma unroll
        for (int h = 0; h < 2; ++h) w[s][h] = in && wok[h] ? ld_stream16(wrow[h] + k) : zero;
    };
#pragma unroll
    for (int s = 0; s < IN_FLIGHT; ++s) load_w(s, kb_begin + s);
    const bool xok = quad < rows;
    const int slot = row0 + (xok ? quad : 0);
    const bf16* xrow = X + (int64_t)(MODE == DOWN ? slot : pair_of_slot[slot] / top) * K + tq * 8;
    auto load_x = [&](int s, int kb) {
        const int k = kb * 32;
        const bool in = kb < kb_end && k + tq * 8 + 8 <= K;
        x[s] = in && xok ? *reinterpret_cast<const uint4*>(xrow + k) : zero;
    };
#pragma unroll
    for (int s = 0; s < IN_FLIGHT; ++s) load_x(s, kb_begin + s);
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int kb = kb_begin; kb < kb_end; kb += IN_FLIGHT) {
#pragma unroll
        for (int s = 0; s < IN_FLIGHT; ++s) {
            mma_bf16(acc, w[s][0].x, w[s][1].x, w[s][0].y, w[s][1].y, x[s].x, x[s].y);
            mma_bf16(acc, w[s][0].z, w[s][1].z, w[s][0].w, w[s][1].w, x[s].z, x[s].w);
            load_w(s, kb + s + IN_FLIGHT);           // blocks past the end load zeros, which add nothing
            load_x(s, kb + s + IN_FLIGHT);
        }
    }
    float* mine = red[warp] + tq * 2 * LD + quad;
    mine[0] = acc[0];
    mine[LD] = acc[1];
    mine[8] = acc[2];
    mine[LD + 8] = acc[3];
    __syncthreads();
    for (int i = threadIdx.x; i < PER_BLOCK * PAIRS; i += WARPS * 32) {
        const int r = i / PER_BLOCK, j = i % PER_BLOCK, f = f0 + j;
        if (r >= rows || f >= features) continue;
        float a = 0.0f, b = 0.0f;
#pragma unroll
        for (int v = 0; v < WARPS; ++v) {
            a += red[v][r * LD + j];
            if (MODE == GATED) b += red[v][r * LD + j + 8];
        }
        const int64_t at = (int64_t)(row0 + r) * features + f;
        if constexpr (MODE == DOWN) {
            ((float*)out)[at] = a;
        } else if constexpr (MODE == RELU2) {
            const float v = fmaxf(a, 0.0f);
            ((bf16*)out)[at] = __float2bfloat16_rn(v * v);
        } else {
            const float gv = fminf(a, limit), uv = fminf(fmaxf(b, -limit), limit);
            ((bf16*)out)[at] = __float2bfloat16_rn(gv / (1.0f + expf(-alpha * gv)) * (uv + up_offset));
        }
    }
}

int experts_launch(const bf16* h, const bf16* w_gate_up, const bf16* w_down, const int* offsets, const int* pair_of_slot, bf16* act, float* y,
                   int n_pairs, int n_real, int top, int hidden, int ff, float limit, float alpha, float up_offset, int gated, cudaStream_t stream) {
    // an upper bound on the row tiles of all experts together
    const int tiles = n_pairs < n_real ? n_pairs : (n_pairs + PAIRS - 1) / PAIRS + n_real;
    if (tiles > 65535) return Q3_ERR_TOO_LARGE;
    int code = gated ? (int)q3_launch(expert_kernel<GATED>, dim3((ff + 7) / 8, tiles), dim3(WARPS * 32), 0, stream, h, w_gate_up, offsets,
                                      pair_of_slot, (void*)act, n_real, top, ff, hidden, limit, alpha, up_offset)
                     : (int)q3_launch(expert_kernel<RELU2>, dim3((ff + 15) / 16, tiles), dim3(WARPS * 32), 0, stream, h, w_gate_up, offsets,
                                      pair_of_slot, (void*)act, n_real, top, ff, hidden, limit, alpha, up_offset);
    if (code != 0) return code;
    return (int)q3_launch(expert_kernel<DOWN>, dim3((hidden + 15) / 16, tiles), dim3(WARPS * 32), 0, stream, (const bf16*)act, w_down, offsets,
                          pair_of_slot, (void*)y, n_real, top, hidden, ff, limit, alpha, up_offset);
}
}  // namespace few

template <typename T, int TM>
int moe_experts_launch(const T* h, const T* w_gate_up, const T* w_down, const int* offsets, const int* pair_of_slot, T* act, float* y,
                       int n_pairs, int n_real, int top, int hidden, int ff, float limit, float alpha, float up_offset, int gated, cudaStream_t stream) {
    const int tiles = (n_pairs + TM - 1) / TM + n_real;         // an upper bound on the row tiles of all experts together
    if (tiles > 65535) return Q3_ERR_TOO_LARGE;
    int code = (int)q3_launch(gated ? moe_up_kernel<T, TM, true> : moe_up_kernel<T, TM, false>, dim3((ff + TN - 1) / TN, tiles), dim3(256), 0, stream, h, w_gate_up, offsets,
                              pair_of_slot, act, n_real, top, hidden, ff, limit, alpha, up_offset);
    if (code != 0) return code;
    return (int)q3_launch(moe_down_kernel<T, TM>, dim3((hidden + TN - 1) / TN, tiles), dim3(256), 0, stream, act, w_down, offsets, y,
                          n_real, hidden, ff);
}

}  // namespace

#define Q3_MOE_EXPORTS(SUFFIX, T)                                                                                         \
    Q3_EXPORT int q3_moe_route_##SUFFIX(const void* h, const void* w_router, const float* correction, int* top_ids,       \
                                        float* top_w, float* id_weight, int64_t n_tokens, int hidden, int n_out, int n_real, \
                                        int top, int group_count, int group_keep, int by_logit, float* gate_out,           \
                                        int group_pair, float weight_scale, void* stream) {                                                                   \
        if (n_tokens <= 0) return 0;                                                                                      \
        if (n_out <= 0 || n_out >= MAX_OUTPUTS || top <= 0 || top > n_out || n_real < 0 || n_real > n_out || \
            group_count <= 0 || n_out % group_count != 0 || group_keep <= 0 || group_keep > group_count ||                \
            n_tokens > 0x7fffffffLL)                                                                                      \
            return Q3_ERR_BAD_SIZE;                                                                                       \
        /* four tokens a block where that leaves every SM two blocks */                                                   \
        if (n_out < MANY_OUTPUTS && n_tokens >= 8 * (int64_t)q3_device_sm_count())                                        \
            return (int)q3_launch(moe_route_kernel<T, 4, MANY_OUTPUTS, 8>, dim3((unsigned)((n_tokens + 3) / 4)), dim3(256), 0, (cudaStream_t)stream, \
                                  (const T*)h, (const T*)w_router, correction, top_ids, top_w, id_weight, n_tokens, hidden, n_out, \
                                  n_real, top, group_count, group_keep, by_logit, gate_out, group_pair, weight_scale);    \
        /* sixteen warps a token while all tokens' blocks are resident at once, else eight */                             \
        if (n_tokens <= 4 * (int64_t)q3_device_sm_count())                                                                \
            return (int)q3_launch(moe_route_kernel<T, 1, MAX_OUTPUTS, 16>, dim3((unsigned)n_tokens), dim3(512), 0, (cudaStream_t)stream, \
                                  (const T*)h, (const T*)w_router, correction, top_ids, top_w, id_weight, n_tokens, hidden, n_out, \
                                  n_real, top, group_count, group_keep, by_logit, gate_out, group_pair, weight_scale);    \
        return (int)q3_launch(moe_route_kernel<T, 1, MAX_OUTPUTS, 8>, dim3((unsigned)n_tokens), dim3(256), 0, (cudaStream_t)stream, \
                              (const T*)h, (const T*)w_router, correction, top_ids, top_w, id_weight, n_tokens, hidden, n_out, \
                              n_real, top, group_count, group_keep, by_logit, gate_out, group_pair, weight_scale);        \
    }                                                                                                                     \
    Q3_EXPORT int q3_moe_experts_##SUFFIX(const void* h, const void* w_gate_up, const void* w_down, const int* offsets,   \
                                          const int* pair_of_slot, void* act, float* y, int n_pairs, int n_real, int top, \
                                          int hidden, int ff, float limit, float alpha, float up_offset, int gated, void* stream) {                   \
        if (n_pairs <= 0 || n_real <= 0) return 0;                                                                        \
        if (n_pairs <= 64)                                                                                                \
            return moe_experts_launch<T, 8>((const T*)h, (const T*)w_gate_up, (const T*)w_down, offsets, pair_of_slot,    \
                                            (T*)act, y, n_pairs, n_real, top, hidden, ff, limit, alpha, up_offset, gated,            \
                                            (cudaStream_t)stream);                                                        \
        return moe_experts_launch<T, 32>((const T*)h, (const T*)w_gate_up, (const T*)w_down, offsets, pair_of_slot,       \
                                         (T*)act, y, n_pairs, n_real, top, hidden, ff, limit, alpha, up_offset, gated, (cudaStream_t)stream); \
    }                                                                                                                     \
    Q3_EXPORT int q3_moe_combine_##SUFFIX(const float* y, const void* h, const int* slot_of_pair, const float* top_w,     \
                                          const float* id_weight, void* out, int64_t n_tokens, int top, int hidden,       \
                                          const void* shared, const float* shared_w, void* stream) {                      \
        if (n_tokens <= 0) return 0;                                                                                      \
        if (n_tokens > 0x7fffffffLL) return Q3_ERR_BAD_SIZE;                                                              \
        constexpr int V = Pack<T>::N;                                                                                     \
        if (hidden % V == 0 && hidden >= 512 && aligned16(y) && aligned16(h) && aligned16(out) && (shared == nullptr || aligned16(shared))) { \
            const int threads = hidden / V >= 256 ? 256 : (hidden / V + 31) / 32 * 32;                                    \
            return (int)q3_launch(moe_combine_kernel<T, V>, dim3((unsigned)n_tokens), dim3(threads), 0, (cudaStream_t)stream, y, \
                                  (const T*)h, slot_of_pair, top_w, id_weight, (T*)out, top, hidden, (const T*)shared, shared_w); \
        }                                                                                                                 \
        return (int)q3_launch(moe_combine_kernel<T, 1>, dim3((unsigned)n_tokens), dim3(hidden >= 1024 ? 256 : 128), 0,    \
                              (cudaStream_t)stream, y, (const T*)h, slot_of_pair, top_w, id_weight, (T*)out, top, hidden, \
                              (const T*)shared, shared_w);                                                                \
    }

Q3_EXPORT int q3_moe_sort(const int* top_ids, int n_pairs, int n_real, int* offsets, int* slot_of_pair, int* pair_of_slot,
                          void* stream) {
    if (n_pairs <= 0) return 0;
    if (n_real < 0 || n_real > 4096) return Q3_ERR_BAD_SIZE;
    return (int)q3_launch(moe_sort_kernel, dim3(1), dim3(1024), (size_t)(2 * n_real + 1) * sizeof(int), (cudaStream_t)stream, top_ids,
                          n_pairs, n_real, offsets, slot_of_pair, pair_of_slot);
}

// bfloat16 with both widths in steps of 32 (and 16-byte aligned rows) on the tensor cores: any number of pairs, made for few
// per expert (q3_moe_experts_tcgen05_bf16 is for more).
Q3_EXPORT int q3_moe_experts_tc_bf16(const void* h, const void* w_gate_up, const void* w_down, const int* offsets,
                                     const int* pair_of_slot, void* act, float* y, int n_pairs, int n_real, int top, int hidden, int ff,
                                     float limit, float alpha, float up_offset, int gated, void* stream) {
    if (n_pairs <= 0 || n_real <= 0) return 0;
    if (hidden % 32 != 0 || ff % 32 != 0 || hidden <= 0 || ff <= 0) return Q3_ERR_BAD_SIZE;
    if (!aligned16(h) || !aligned16(w_gate_up) || !aligned16(w_down) || !aligned16(act)) return Q3_ERR_MISALIGNED;
    return few::experts_launch((const bf16*)h, (const bf16*)w_gate_up, (const bf16*)w_down, offsets, pair_of_slot, (bf16*)act, y, n_pairs,
                               n_real, top, hidden, ff, limit, alpha, up_offset, gated, (cudaStream_t)stream);
}

Q3_MOE_EXPORTS(f32, float)
Q3_MOE_EXPORTS(bf16, bf16)
