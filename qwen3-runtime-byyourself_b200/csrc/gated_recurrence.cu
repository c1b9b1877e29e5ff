// Linear attention whose forget gate also decides what is written (HGRN2), with a fixed-size state per sequence:
//
//     f_t = low + (1 - low) * sigmoid(z_t + bias)          per head and channel, low the gate's lower bound
//     S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T            (S: [d, vd] per head, float32, one per cache slot)
//     o_t = S_t^T q_t,   q_t = SiLU(projection)
//
// A row of the projection holds, head by head, the H*d values of q, the H*d of z and the H*vd of v.
//
//   gated_scan    : one block per (head, sequence, tile of up to 16 columns of the state: columns do not depend
//                   on one another) walks the sequence's new tokens in order with its share of the state in
//                   registers: thread (j, r) owns column j of the tile and the rows r * ROWS .. r * ROWS + ROWS - 1 (up
//                   to 8 rows; the threads of a column add their partial outputs through shared memory); it reads the
//                   state from the slot's row before the first token and writes it back after the last.  The
//                   tokens arrive a stage (up to 16) at a time: while the threads walk a stage, each by itself,
//                   the projection rows of the next stage are already on their way into registers; they are activated
//                   into shared memory between the two barriers of a stage, so a token costs no barrier of its own
//                   and no wait for global memory.  The launch depends on the sizes only, never on the step: a
//                   token's output is the same bits however the sequence was cut.  Gate, state and o are 32-bit whatever T.
//   gated_scan_wide : the same sums to the bit for d and vd multiples of 8: a thread has 8 rows of four columns, two rows
//                   at a time in the paired 32-bit arithmetic of this architecture.
//   gated_step    : the same for a step in which every sequence brings one token, with the same sums to the bit.
//   head_rms_norm : out = T( o / sqrt(mean(o^2) + eps) * w ) over the vd values of every (token, head); one weight
//                   vector for all heads.
#include "common.cuh"

namespace {

constexpr int COL_TILE = 16;      // columns of the state per block
constexpr int MAX_ROWS = 8;       // rows of the state per thread
constexpr int MAX_STAGE = 16;     // tokens fetched together
constexpr int PRE_QF = 8;         // values of q and of the gate that a thread holds for the next stage
constexpr int PRE_V = 2;          // values of v

// Sigmoid for the gate and the query's SiLU: exact division and expf in the 32-bit path; with bfloat16 inputs the
// hardware's exponential and reciprocal (32-bit, a few units in the last place).
template <typename T> __device__ __forceinline__ float sigmoid_of(float z) { return 1.0f / (1.0f + expf(-z)); }
template <> __device__ __forceinline__ float sigmoid_of<bf16>(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }

template <typename T, int ROWS>
__global__ void __launch_bounds__(512)
gated_scan_kernel(const T* __restrict__ proj, float* __restrict__ state, const float* __restrict__ low, const float* __restrict__ bias,
                  const int* __restrict__ seq_start, const int* __restrict__ seq_slots, float* __restrict__ out, int H, int d, int vd,
                  int R, int vt, int stage) {
    extern __shared__ __align__(16) float smem[];
    const int dp = R * ROWS;                 // d rounded up to whole threads: the rows beyond d hold q = 0
    float* q_s = smem;                       // [stage][dp]
    float* f_s = q_s + stage * dp;           // [stage][dp]
    float* v_s = f_s + stage * dp;           // [stage][vt]
    float* red = v_s + stage * vt;           // [stage][R][vt]
    pdl_launch_dependents();
    const int head = blockIdx.x, seq = blockIdx.y, col0 = blockIdx.z * vt;
    const int tid = threadIdx.x, nthreads = blockDim.x, jt = tid % vt, j = col0 + jt, r = tid / vt;
    const bool live = r < R && j < vd;
    const int64_t cols = 2 * (int64_t)H * d + (int64_t)H * vd;
    // which values of a stage this thread fetches: x = tid + k * nthreads < stage * d (q and gate), < stage * vt (v);
    // the token and the channel of each, found once (token << 16 | channel; a token beyond the stage: none)
    float lo_r[PRE_QF], bias_r[PRE_QF];
    int at_qf[PRE_QF], at_v[PRE_V];
#pragma unroll
    for (int k = 0; k < PRE_QF; ++k) {
        const int x = tid + k * nthreads;
        const int i = x % d;
        at_qf[k] = x < stage * d ? (x / d) << 16 | i : MAX_STAGE << 16;
        lo_r[k] = x < stage * d ? low[head * d + i] : 0.0f;
        bias_r[k] = x < stage * d ? bias[head * d + i] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < PRE_V; ++k) {
        const int x = tid + k * nthreads;
        at_v[k] = x < stage * vt ? (x / vt) << 16 | (x % vt) : MAX_STAGE << 16;
    }
    for (int x = tid; x < 2 * stage * dp; x += nthreads) smem[x] = 0.0f;        // the padding rows stay 0
    pdl_wait();
    float* S_g = state + ((int64_t)seq_slots[seq] * H + head) * d * vd;
    float S[ROWS];
#pragma unroll
    for (int n = 0; n < ROWS; ++n) {
        const int i = r * ROWS + n;
        S[n] = live && i < d ? S_g[(int64_t)i * vd + j] : 0.0f;
    }
    const int t_begin = seq_start[seq], t_end = seq_start[seq + 1];
    T q_raw[PRE_QF], f_raw[PRE_QF], v_raw[PRE_V];
    auto fetch = [&](int t0) {
        const int n_stage = min(stage, t_end - t0);
#pragma unroll
        for (int k = 0; k < PRE_QF; ++k) {
            const int tt = at_qf[k] >> 16, i = at_qf[k] & 0xffff;
            if (tt < n_stage) {
                const T* row = proj + (int64_t)(t0 + tt) * cols + i;
                q_raw[k] = row[(int64_t)head * d];
                f_raw[k] = row[(int64_t)(H + head) * d];
            }
        }
#pragma unroll
        for (int k = 0; k < PRE_V; ++k) {
            const int tt = at_v[k] >> 16, c = at_v[k] & 0xffff;
            if (tt < n_stage && col0 + c < vd)
                v_raw[k] = proj[(int64_t)(t0 + tt) * cols + 2 * (int64_t)H * d + (int64_t)head * vd + col0 + c];
        }
    };
    auto activate = [&](int t0) {
        const int n_stage = min(stage, t_end - t0);
#pragma unroll
        for (int k = 0; k < PRE_QF; ++k) {
            const int tt = at_qf[k] >> 16, i = at_qf[k] & 0xffff;
            if (tt < n_stage) {
                const float qz = to_f32<T>(q_raw[k]), fz = to_f32<T>(f_raw[k]);
                q_s[tt * dp + i] = qz * sigmoid_of<T>(qz);
                f_s[tt * dp + i] = lo_r[k] + (1.0f - lo_r[k]) * sigmoid_of<T>(fz + bias_r[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < PRE_V; ++k) {
            const int tt = at_v[k] >> 16, c = at_v[k] & 0xffff;
            if (tt < n_stage) v_s[tt * vt + c] = col0 + c < vd ? to_f32<T>(v_raw[k]) : 0.0f;
        }
    };
    if (t_begin < t_end) fetch(t_begin);
    __syncthreads();                                     // the zeros are in place
    if (t_begin < t_end) activate(t_begin);
    __syncthreads();
    for (int t0 = t_begin; t0 < t_end; t0 += stage) {
        const int n_stage = min(stage, t_end - t0);
        if (t0 + stage < t_end) fetch(t0 + stage);       // on its way while this stage is walked
        if (live) {
#pragma unroll 2
            for (int tt = 0; tt < n_stage; ++tt) {
                const float v = v_s[tt * vt + jt];
                const float* fr = f_s + tt * dp + r * ROWS;
                const float* qr = q_s + tt * dp + r * ROWS;
                float part0 = 0.0f, part1 = 0.0f;
                if constexpr (ROWS % 4 == 0) {
#pragma unroll
                    for (int n = 0; n < ROWS; n += 4) {
                        const float4 f4 = *reinterpret_cast<const float4*>(fr + n), q4 = *reinterpret_cast<const float4*>(qr + n);
                        S[n] = fmaf(f4.x, S[n] - v, v);          // f S + (1 - f) v
                        S[n + 1] = fmaf(f4.y, S[n + 1] - v, v);
                        S[n + 2] = fmaf(f4.z, S[n + 2] - v, v);
                        S[n + 3] = fmaf(f4.w, S[n + 3] - v, v);
                        part0 = fmaf(S[n], q4.x, part0);
                        part1 = fmaf(S[n + 1], q4.y, part1);
                        part0 = fmaf(S[n + 2], q4.z, part0);
                        part1 = fmaf(S[n + 3], q4.w, part1);
                    }
                } else {
#pragma unroll
                    for (int n = 0; n < ROWS; ++n) {
                        S[n] = fmaf(fr[n], S[n] - v, v);
                        part0 = fmaf(S[n], qr[n], part0);
                    }
                }
                red[(tt * R + r) * vt + jt] = part0 + part1;
            }
        }
        __syncthreads();
        for (int x = tid; x < n_stage * vt; x += nthreads) {
            const int tt = x / vt, c = x % vt;
            if (col0 + c < vd) {
                float o = 0.0f;
                for (int rr = 0; rr < R; ++rr) o += red[(tt * R + rr) * vt + c];
                out[((int64_t)(t0 + tt) * H + head) * vd + col0 + c] = o;
            }
        }
        if (t0 + stage < t_end) activate(t0 + stage);    // everybody has left the stage's q, gate and v
        __syncthreads();
    }
    if (live) {
#pragma unroll
        for (int n = 0; n < ROWS; ++n) {
            const int i = r * ROWS + n;
            if (i < d) S_g[(int64_t)i * vd + j] = S[n];
        }
    }
}

// The scan for states of whole packets.  The tokens of a sequence are a serial chain, so the length of a token's step counts:
// the threads that walk the state do nothing else, and as many helpers fetch and activate the stage after and add up the
// outputs of the stage before, with one barrier a stage.  A walker has eight rows of four columns, so that a gate or query
// value read from shared memory serves four, and takes rows in pairs (fma.rn.f32x2: each half is the scalar operation, so a
// pair of rows holds the two chains of a column's sum as they are).  The longest sequences start first.
// Prompts of 2,048 + 911 + 1,203 tokens, 32 heads of 128 x 128: 1,058 us by threads of one column that do everything, 490 here.
__device__ __forceinline__ uint64_t two(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void one_each(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

constexpr int WIDE_STAGE = 8;     // tokens fetched together
constexpr int WIDE_PACKETS = 5;   // packets of them a helper holds
constexpr int WIDE_TILE = 32;     // columns of the state per block
constexpr int WIDE_RANKED = 64;   // sequences up to which the longest start first

template <typename T>
__global__ void __launch_bounds__(512)
gated_scan_wide_kernel(const T* __restrict__ proj, float* __restrict__ state, const float* __restrict__ low, const float* __restrict__ bias,
                       const int* __restrict__ seq_start, const int* __restrict__ seq_slots, float* __restrict__ out, int H, int d, int vd,
                       int n_seqs, int walkers) {
    constexpr int P = Pack<T>::N, VT = WIDE_TILE;
    extern __shared__ __align__(16) float smem[];
    __shared__ int which;
    const int R = d / 8, per_token = 2 * d + VT, stage_floats = WIDE_STAGE * per_token, red_floats = WIDE_STAGE * R * VT;
    float* red = smem + 2 * stage_floats;              // [2][stage][R][VT]; before it, [2]: q [stage][d], gates [stage][d], v [stage][VT]
    float* low_s = red + 2 * red_floats;               // [d]
    float* bias_s = low_s + d;                         // [d]
    pdl_launch_dependents();
    const int head = blockIdx.x, col0 = blockIdx.y * VT, tid = threadIdx.x;
    const int64_t cols = 2 * (int64_t)H * d + (int64_t)H * vd;
    for (int i = tid; i < d; i += blockDim.x) {
        low_s[i] = low[head * d + i];
        bias_s[i] = bias[head * d + i];
    }
    pdl_wait();
    // The blockIdx.z-th longest sequence (of equal ones the earlier first).  Finding it takes every block n_seqs comparisons a
    // thread, and with many sequences blocks enough follow one another to fill the gaps of the longest: beyond WIDE_RANKED they
    // come as they are.  (1,500 sequences of 3 tokens, 32 heads of 128 x 128: 179 ms ranked, 2.3 ms as they come.)
    const bool ranked = n_seqs > 1 && n_seqs <= WIDE_RANKED;
    if (ranked) {
        for (int i = tid; i < n_seqs; i += blockDim.x) {
            const int mine = seq_start[i + 1] - seq_start[i];
            int rank = 0;
            for (int k = 0; k < n_seqs; ++k) {
                const int n = seq_start[k + 1] - seq_start[k];
                rank += n > mine || (n == mine && k < i);
            }
            if (rank == (int)blockIdx.z) which = i;
        }
    }
    __syncthreads();
    const int seq = ranked ? which : (int)blockIdx.z, t_begin = seq_start[seq], n_tokens = seq_start[seq + 1] - t_begin;
    if (n_tokens == 0) return;
    const int stages = (n_tokens + WIDE_STAGE - 1) / WIDE_STAGE;

    if (tid >= walkers) {
        // ---------------- helpers
        const int id = tid - walkers, n_helpers = blockDim.x - walkers;
        // a stage's packets: all of q, then all of the gates, then the block's columns of v, so that a warp's are of one kind
        const int q_packets = WIDE_STAGE * d / P, v_packets = WIDE_STAGE * VT / P;
        int token[WIDE_PACKETS], kind[WIDE_PACKETS], place[WIDE_PACKETS], channel[WIDE_PACKETS];   // place: of its first value in the stage
        const T* src[WIDE_PACKETS];                    // in the first token's row of the sequence
#pragma unroll
        for (int k = 0; k < WIDE_PACKETS; ++k) {
            const int x = id + k * n_helpers;
            kind[k] = x < q_packets ? 0 : x < 2 * q_packets ? 1 : 2;
            const int y = x - kind[k] * q_packets, width = kind[k] < 2 ? d : VT, i = y * P % width;
            token[k] = kind[k] < 2 || (y < v_packets && col0 + i < vd) ? y * P / width : WIDE_STAGE;
            channel[k] = i;
            place[k] = kind[k] * WIDE_STAGE * d + y * P;
            const int64_t column = kind[k] == 0 ? (int64_t)head * d + i : kind[k] == 1 ? (int64_t)(H + head) * d + i
                                                                                       : 2 * (int64_t)H * d + (int64_t)head * vd + col0 + i;
            src[k] = proj + (int64_t)(t_begin + token[k]) * cols + column;
        }
        Pack<T> raw[WIDE_PACKETS];
        auto fetch = [&](int st) {
            const int n_stage = min(WIDE_STAGE, n_tokens - st * WIDE_STAGE);
#pragma unroll
            for (int k = 0; k < WIDE_PACKETS; ++k)
                if (token[k] < n_stage) raw[k] = load_pack<T>(src[k] + (int64_t)st * WIDE_STAGE * cols);
        };
        auto activate = [&](int st) {
            const int n_stage = min(WIDE_STAGE, n_tokens - st * WIDE_STAGE);
#pragma unroll
            for (int k = 0; k < WIDE_PACKETS; ++k) {
                if (token[k] >= n_stage) continue;
                float v[P];
#pragma unroll
                for (int e = 0; e < P; ++e) v[e] = raw[k].get(e);
                if (kind[k] == 0) {
#pragma unroll
                    for (int e = 0; e < P; ++e) v[e] *= sigmoid_of<T>(v[e]);
                } else if (kind[k] == 1) {
                    float lo[P], b[P];
#pragma unroll
                    for (int e = 0; e < P; e += 4) {
                        const float4 l4 = *reinterpret_cast<const float4*>(low_s + channel[k] + e), b4 = *reinterpret_cast<const float4*>(bias_s + channel[k] + e);
                        lo[e] = l4.x; lo[e + 1] = l4.y; lo[e + 2] = l4.z; lo[e + 3] = l4.w;
                        b[e] = b4.x; b[e + 1] = b4.y; b[e + 2] = b4.z; b[e + 3] = b4.w;
                    }
#pragma unroll
                    for (int e = 0; e < P; ++e) v[e] = lo[e] + (1.0f - lo[e]) * sigmoid_of<T>(v[e] + b[e]);
                }
                float* to = smem + (st & 1) * stage_floats + place[k];
#pragma unroll
                for (int e = 0; e < P; e += 4) *reinterpret_cast<float4*>(to + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
            }
        };
        auto add_up = [&](int st) {
            const int n_stage = min(WIDE_STAGE, n_tokens - st * WIDE_STAGE), col = id % VT;
            const float* from = red + (st & 1) * red_floats + col;
            if (col0 + col >= vd) return;
            for (int tt = id / VT; tt < n_stage; tt += n_helpers / VT) {
                float o = 0.0f;
#pragma unroll 8
                for (int rr = 0; rr < R; ++rr) o += from[(tt * R + rr) * VT];
                out[((int64_t)(t_begin + st * WIDE_STAGE + tt) * H + head) * vd + col0 + col] = o;
            }
        };
        fetch(0);
        activate(0);
        if (stages > 1) fetch(1);
        __syncthreads();
        for (int st = 0; st < stages; ++st) {
            if (st + 1 < stages) activate(st + 1);
            if (st + 2 < stages) fetch(st + 2);
            if (st > 0) add_up(st - 1);
            __syncthreads();
        }
        add_up(stages - 1);
        return;
    }

    // ---------------- walkers
    const int c = (tid % (VT / 4)) * 4, r = tid / (VT / 4);
    const bool live = r < R && col0 + c < vd;
    uint64_t S[4][4];                                  // rows 2 n and 2 n + 1 of the thread's eight, its four columns
    float* S_g = state + ((int64_t)seq_slots[seq] * H + head) * d * vd + (int64_t)r * 8 * vd + col0 + c;
    if (live) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const float4 a = *reinterpret_cast<const float4*>(S_g + (int64_t)(2 * n) * vd), b = *reinterpret_cast<const float4*>(S_g + (int64_t)(2 * n + 1) * vd);
            S[n][0] = two(a.x, b.x);
            S[n][1] = two(a.y, b.y);
            S[n][2] = two(a.z, b.z);
            S[n][3] = two(a.w, b.w);
        }
    }
    __syncthreads();
    for (int st = 0; st < stages; ++st) {
        const int n_stage = min(WIDE_STAGE, n_tokens - st * WIDE_STAGE);
        if (live) {
            const float* q_s = smem + (st & 1) * stage_floats + r * 8;
            const float* f_s = q_s + WIDE_STAGE * d;
            const float* v_s = smem + (st & 1) * stage_floats + 2 * WIDE_STAGE * d + c;
            float* to = red + (st & 1) * red_floats + r * VT + c;
#pragma unroll 2
            for (int tt = 0; tt < n_stage; ++tt) {
                const float4 v4 = *reinterpret_cast<const float4*>(v_s + tt * VT);
                const uint64_t v2[4] = {two(v4.x, v4.x), two(v4.y, v4.y), two(v4.z, v4.z), two(v4.w, v4.w)};
                const uint64_t nv2[4] = {two(-v4.x, -v4.x), two(-v4.y, -v4.y), two(-v4.z, -v4.z), two(-v4.w, -v4.w)};
                uint64_t part[4] = {0ull, 0ull, 0ull, 0ull};             // the sums over even and over odd rows
#pragma unroll
                for (int n = 0; n < 4; n += 2) {
                    const ulonglong2 f2 = *reinterpret_cast<const ulonglong2*>(f_s + tt * d + 2 * n);
                    const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(q_s + tt * d + 2 * n);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        S[n][e] = fma2(f2.x, add2(S[n][e], nv2[e]), v2[e]);                      // f S + (1 - f) v
                        part[e] = fma2(S[n][e], q2.x, part[e]);
                        S[n + 1][e] = fma2(f2.y, add2(S[n + 1][e], nv2[e]), v2[e]);
                        part[e] = fma2(S[n + 1][e], q2.y, part[e]);
                    }
                }
                float even[4], odd[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) one_each(part[e], even[e], odd[e]);
                *reinterpret_cast<float4*>(to + tt * R * VT) = make_float4(even[0] + odd[0], even[1] + odd[1], even[2] + odd[2], even[3] + odd[3]);
            }
        }
        __syncthreads();
    }
    if (live) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            float4 a, b;
            one_each(S[n][0], a.x, b.x);
            one_each(S[n][1], a.y, b.y);
            one_each(S[n][2], a.z, b.z);
            one_each(S[n][3], a.w, b.w);
            *reinterpret_cast<float4*>(S_g + (int64_t)(2 * n) * vd) = a;
            *reinterpret_cast<float4*>(S_g + (int64_t)(2 * n + 1) * vd) = b;
        }
    }
}

// A step in which every sequence brings one token: bound by reading and writing the state once.  A block takes 64 columns
// of one head's state (32 where that leaves SMs without a block), a thread 8 neighbouring rows of 4 columns: eight 16-byte
// loads in flight a thread, whole lines a warp.  The sums are those of the scan, to the bit: 8 rows in two chains, then the
// groups of 8 in order.  8 sequences, 16 heads of 128 x 128: 4.1 us, 20.2 by the scan.
template <typename T>
__global__ void __launch_bounds__(256)
gated_step_kernel(const T* __restrict__ proj, float* __restrict__ state, const float* __restrict__ low, const float* __restrict__ bias,
                  const int* __restrict__ seq_start, const int* __restrict__ seq_slots, float* __restrict__ out, int H, int d, int vd, int tile) {
    __shared__ float q_s[256], f_s[256], red[32][64];
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.x, seq = blockIdx.y, col0 = blockIdx.z * tile, tid = threadIdx.x;
    const int packets = tile / 4, groups = d / 8, c = (tid % packets) * 4;
    float* S_g = state + ((int64_t)seq_slots[seq] * H + head) * d * vd + col0 + c;
    const int64_t t = seq_start[seq];
    if (t == seq_start[seq + 1]) return;
    const T* row = proj + t * (2 * (int64_t)H * d + (int64_t)H * vd);
    const bool live = col0 + c < vd;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (live) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = to_f32<T>(row[2 * (int64_t)H * d + (int64_t)head * vd + col0 + c + e]);
    }
    float4 S[8];
    int g = tid / packets;
    auto load = [&]() {
#pragma unroll
        for (int n = 0; n < 8; ++n) S[n] = *reinterpret_cast<const float4*>(S_g + (int64_t)(g * 8 + n) * vd);
    };
    if (live && g < groups) load();
    if (tid < d) {
        const float qz = to_f32<T>(row[(int64_t)head * d + tid]), fz = to_f32<T>(row[(int64_t)(H + head) * d + tid]);
        const float lo = low[head * d + tid];
        q_s[tid] = qz * sigmoid_of<T>(qz);
        f_s[tid] = lo + (1.0f - lo) * sigmoid_of<T>(fz + bias[head * d + tid]);
    }
    __syncthreads();
    for (bool first = true; live && g < groups; g += blockDim.x / packets, first = false) {
        if (!first) load();
        float part0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, part1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float f = f_s[g * 8 + n], q = q_s[g * 8 + n];
            float* s = &S[n].x;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[e] = fmaf(f, s[e] - v[e], v[e]);
                if (n & 1) part1[e] = fmaf(s[e], q, part1[e]); else part0[e] = fmaf(s[e], q, part0[e]);
            }
            *reinterpret_cast<float4*>(S_g + (int64_t)(g * 8 + n) * vd) = S[n];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) red[g][c + e] = part0[e] + part1[e];
    }
    __syncthreads();
    if (tid < tile && col0 + tid < vd) {
        float o = 0.0f;
        for (int r = 0; r < groups; ++r) o += red[r][tid];
        out[(t * H + head) * vd + col0 + tid] = o;
    }
}

template <typename T>
int gated_scan_launch(const T* proj, float* state, const float* low, const float* bias, const int* seq_start, const int* seq_slots,
                      float* out, int n_seqs, int H, int d, int vd, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (H <= 0 || d <= 0 || vd <= 0 || d > 256 || vd > 256 || n_seqs > 65535) return Q3_ERR_BAD_SIZE;
    // The scan for whole packets, but for small states of many sequences, where its 160 threads a block and more find little to do (512
    // sequences of 2 tokens, 2 heads of 16 x 16: 3.9 us below, 9.0 there; 64 of 16 and fewer: level), and for 32-bit heads beyond
    // 128 in fewer blocks than there are SMs, where its helpers hold the walkers up (one sequence of 2,048 tokens, 8 heads of 256 x 256:
    // 596 us below, 716 there; four of 700 tokens, 256 blocks: ahead there).
    const int64_t wide_blocks = (int64_t)H * ((vd + WIDE_TILE - 1) / WIDE_TILE) * n_seqs;
    const bool wide = (d >= 32 || n_seqs <= WIDE_RANKED) && (sizeof(T) == 2 || d <= 128 || wide_blocks >= q3_device_sm_count());
    if (wide && d % 8 == 0 && vd % 8 == 0 && aligned16(proj) && aligned16(state)) {
        // walkers of 8 rows x 4 columns in whole warps; helpers: 128, or 256 where a stage has more than three packets each
        const int walkers = ((d / 8) * (WIDE_TILE / 4) + 31) / 32 * 32, packets = WIDE_STAGE * (2 * d + WIDE_TILE) / Pack<T>::N;
        const int helpers = packets <= 3 * 128 ? 128 : 256;      // (32-bit, 16 heads of 128 x 128, 2,048 tokens: 640 us with 128, 432 with 256)
        static_assert(WIDE_PACKETS * 256 >= WIDE_STAGE * (2 * 256 + WIDE_TILE) / 4, "a stage's packets of 32-bit values, d = 256");
        const size_t bytes = (size_t)(2 * WIDE_STAGE * (2 * d + WIDE_TILE + (d / 8) * WIDE_TILE) + 2 * d) * sizeof(float);   // at most 102 KB
        static Q3PerDevice configured;
        const cudaError_t e = q3_allow_shared_memory(gated_scan_wide_kernel<T>, 112 * 1024, configured);
        if (e != cudaSuccess) return (int)e;
        return (int)q3_launch(gated_scan_wide_kernel<T>, dim3(H, (vd + WIDE_TILE - 1) / WIDE_TILE, n_seqs), dim3(walkers + helpers), bytes,
                              stream, proj, state, low, bias, seq_start, seq_slots, out, H, d, vd, n_seqs, walkers);
    }
    const int vt = min(vd, COL_TILE);
    const int R = (d + MAX_ROWS - 1) / MAX_ROWS;       // threads that share a column: up to 32
    const int need = (d + R - 1) / R;                  // rows a thread: up to 8
    const int rows = need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : 8;
    const int threads = ((vt * R + 31) / 32) * 32;     // up to 512
    const int stage = max(1, min(MAX_STAGE, min(PRE_QF * threads / d, PRE_V * threads / vt)));
    const size_t smem = (size_t)stage * (2 * R * rows + vt + R * vt) * sizeof(float);      // at most 66 KB
    const dim3 grid(H, n_seqs, (vd + vt - 1) / vt);
#define Q3_SCAN(ROWS)                                                                                                        \
    do {                                                                                                                     \
        if (smem > 48 * 1024) {                                                                                              \
            const cudaError_t e = cudaFuncSetAttribute(gated_scan_kernel<T, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                       (int)smem);                                                           \
            if (e != cudaSuccess) return (int)e;                                                                             \
        }                                                                                                                    \
        return (int)q3_launch(gated_scan_kernel<T, ROWS>, grid, dim3(threads), smem, stream, proj, state, low, bias,         \
                              seq_start, seq_slots, out, H, d, vd, R, vt, stage);                                           \
    } while (0)
    if (rows == 1) Q3_SCAN(1);
    if (rows == 2) Q3_SCAN(2);
    if (rows == 4) Q3_SCAN(4);
    Q3_SCAN(8);
#undef Q3_SCAN
}

template <typename T>
int gated_step_launch(const T* proj, float* state, const float* low, const float* bias, const int* seq_start, const int* seq_slots,
                      float* out, int n_seqs, int H, int d, int vd, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (H <= 0 || d <= 0 || vd <= 0 || d > 256 || vd > 256 || d % 8 != 0 || vd % 4 != 0 || n_seqs > 65535) return Q3_ERR_BAD_SIZE;
    if (!aligned16(state)) return gated_scan_launch<T>(proj, state, low, bias, seq_start, seq_slots, out, n_seqs, H, d, vd, stream);
    const int tile = (int64_t)H * n_seqs * ((vd + 63) / 64) >= q3_device_sm_count() ? 64 : 32;
    // a thread for every packet of the state, for every q and gate and for every output, 256 at most (512 sequences, 2 heads of
    // 16 x 16: 3.2 us with these threads, 5.7 with 256)
    const int held = (d / 8) * (tile / 4), need = held > d ? held : d, threads = need >= 256 ? 256 : ((need > tile ? need : tile) + 31) / 32 * 32;
    return (int)q3_launch(gated_step_kernel<T>, dim3(H, n_seqs, (vd + tile - 1) / tile), dim3(threads), 0, stream, proj, state, low, bias,
                          seq_start, seq_slots, out, H, d, vd, tile);
}

// One warp per (token, head).
template <typename T>
__global__ void head_rms_norm_kernel(const float* __restrict__ o, const float* __restrict__ w, T* __restrict__ out, int64_t n_rows, int vd,
                                     float eps) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n_rows) return;
    const int lane = threadIdx.x & 31;
    const float* x = o + row * vd;
    float sq = 0.0f;
    for (int c = lane; c < vd; c += 32) sq += x[c] * x[c];
    const float inv = rsqrtf(warp_sum(sq) / (float)vd + eps);
    for (int c = lane; c < vd; c += 32) out[row * vd + c] = from_f32<T>(x[c] * inv * w[c]);
}

}  // namespace

#define Q3_GATED_EXPORTS(SUFFIX, T)                                                                                         \
    Q3_EXPORT int q3_gated_scan_##SUFFIX(const void* proj, float* state, const float* low, const float* bias,              \
                                         const int* seq_start, const int* seq_slots, float* out, int n_seqs, int heads,    \
                                         int d, int vd, void* stream) {                                                    \
        return gated_scan_launch<T>((const T*)proj, state, low, bias, seq_start, seq_slots, out, n_seqs, heads, d, vd,      \
                                    (cudaStream_t)stream);                                                                 \
    }                                                                                                                       \
    Q3_EXPORT int q3_gated_step_##SUFFIX(const void* proj, float* state, const float* low, const float* bias,              \
                                         const int* seq_start, const int* seq_slots, float* out, int n_seqs, int heads,    \
                                         int d, int vd, void* stream) {                                                    \
        return gated_step_launch<T>((const T*)proj, state, low, bias, seq_start, seq_slots, out, n_seqs, heads, d, vd,      \
                                    (cudaStream_t)stream);                                                                 \
    }                                                                                                                       \
    Q3_EXPORT int q3_head_rms_norm_##SUFFIX(const float* o, const float* w, void* out, int64_t n_rows, int vd, float eps,   \
                                            void* stream) {                                                                \
        if (n_rows <= 0) return 0;                                                                                          \
        if (vd <= 0 || (n_rows + 7) / 8 > 0x7fffffffLL) return Q3_ERR_BAD_SIZE;                                             \
        return (int)q3_launch(head_rms_norm_kernel<T>, dim3((unsigned)((n_rows + 7) / 8)), dim3(256), 0,                    \
                              (cudaStream_t)stream, o, w, (T*)out, n_rows, vd, eps);                                        \
    }

Q3_GATED_EXPORTS(f32, float)
Q3_GATED_EXPORTS(bf16, bf16)
