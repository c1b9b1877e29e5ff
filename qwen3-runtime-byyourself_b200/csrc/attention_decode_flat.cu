// Decode attention over the paged cache for bfloat16, the whole of a decode step in one launch: norm and rotation of the
// new queries and key, the write of key and value into the cache, attention over every cached key, and the joining of the
// parts of a row (src/ops/gqa_attention.cu:84-153, src/model/self_attention.cpp:147-152).
//
// A row is one (sequence, kv head): the pages of 64 keys that its query reads, with the query heads of the group as the
// eight columns of mma.m16n8k16 (keys and values are its 16-row operands).  Rows are cut into parts of at most `c` pages,
// c being the smallest number that gives no more parts than blocks are resident at once: contexts of unequal length take
// about as long as equal ones of the same total.  Where there are more rows than blocks, or long ones that leave many blocks
// without, c is smaller and a block takes several parts, if that should be ahead (`time_of`); short rows beyond the grid are taken
// whole.  Every block finds c and its parts from the positions by itself; c, and with it the order of a row's sums, hangs on the
// lengths of all sequences of the step.
//   warp 4     copies the pages' K and V panels (16 KB each at head size 128, contiguous) by TMA into a ring.
//   warps 0-3  take 16 of a page's 64 keys each, with an online softmax of their own, and meet at the end of the part.
//              A page is a chain of dependent steps - score products, maximum, exponentials, value products - of 0.65 us for a
//              block by itself and about 1.25 for one of three on an SM (from steps whose busiest block had 60 to 500 pages), so what
//              counts is how many blocks are on an SM: three with a ring of two pages.
// A row that one block holds whole is finished there.  Of a row that is cut, every block leaves its sums in
// `parts` and counts itself at the row's counter; the one that comes last adds them up, in the order of the parts - a
// fixed order whichever comes last - and sets the counter back to zero.  Nobody waits for another block.
//
// Bound by its chain of steps with short contexts, by memory with long ones: 64 sequences of 130 tokens, 32 heads over 8 of 128, 17 us
// for 34 MB where the form of attention_decode.cu, which does not split so many rows and runs them in two waves, takes 29; 64 of 60 to
// 8,000 tokens 170 and 218; one of 24,000 among 63 of 100 43 and 257 (250 here with whole rows); 96 of 4,000 230 and 252 (6.9 TB/s);
// 64 of 16,000 620 and 630.  Equal rows that are a little more than the grid are its worst: 64 of 6,000 257 and 246.
#include <cuda.h>

#include "common.cuh"
#include "decode_head.cuh"
#include "tma.cuh"

#ifndef Q3_HEAD_DIM
#error "compile with -DQ3_HEAD_DIM=<64 or 128>"
#endif

namespace {

constexpr int D = Q3_HEAD_DIM;
static_assert(D == 64 || D == 128, "pages are copied in swizzled halves of 64 columns");
constexpr int PAGE = Q3_PAGE_TOKENS;
static_assert(PAGE == 64, "each of the four warps takes 16 keys of a page");
constexpr int WARPS = 4, KEYS = PAGE / WARPS, THREADS = WARPS * 32 + 32;
constexpr int BARS_BYTES = 128;                    // the ring's barriers and one word
constexpr int MAX_G = 8;                              // query heads of a kv head
constexpr int HALF_BYTES = PAGE * 128, PANEL_BYTES = (D / 64) * HALF_BYTES, STAGE_BYTES = 2 * PANEL_BYTES;
constexpr int MAX_STAGES = 4;
constexpr int MT = D / 16, KT = D / 16;             // tiles of 16 values of the output, of a score's dot
constexpr int LDO = D + 4;                          // a result row in shared memory: the lanes' stores fall into different banks
constexpr int MIN_PART = 4;                         // pages below which a row is not cut
constexpr int MAX_WAVES = 8;                        // parts of a block, where rows are cut
constexpr int LONG_ROW = 48;                        // pages of the longest row from which more rows than blocks are cut
constexpr int BLOCKS_PER_SM = 3;
constexpr int MERGE = 12;                           // parts of a row added up in one round

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void meet() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }

// Byte offset of the 16-byte packet `c` of row `r` inside a panel: halves of 64 columns, the packets of a row exchanged by
// the row's index (the 128-byte swizzle of the copy).
__device__ __forceinline__ uint32_t packet(int r, int c) {
    return (uint32_t)((c >> 3) * HALF_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

// Floats between the parts' sums: [G][D], then (max, sum) [G][2], whole 16-byte packets.
__host__ __device__ constexpr int part_floats(int G) { return (G * (D + 2) + 3) / 4 * 4; }

struct Args {
    const bf16* qkv;               // [tokens, (nq + 2 nkv) * D]: the projection output as it is
    bf16* k_pages;
    bf16* v_pages;
    bf16* out;                     // [tokens, nq * D]
    float* parts;                  // [MAX_WAVES blocks][part_floats(G)], 16-byte aligned
    int* counters;                 // [tokens * nkv], zero between launches
    const float* q_norm_w;         // [D] or null
    const float* k_norm_w;
    const float* cos_tab;          // [positions, rot / 2] or null
    const float* sin_tab;
    const int* token_seq;
    const int* token_pos;
    const int* page_table;
    int pages_per_seq, n_tokens, nq, nkv, window, stages, rot, write_kv;
    float eps, scale_log2;
    int* status;
};

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// A mask for a register of two bfloat16 values, of keys `key` and `key` + 1: all ones where the key lies in [lo, pos].
__device__ __forceinline__ uint32_t keys_seen(int key, int lo, int pos) {
    return (key >= lo && key <= pos ? 0x0000ffffu : 0u) | (key + 1 >= lo && key + 1 <= pos ? 0xffff0000u : 0u);
}

// Pages that the query of token t reads, from page `first` on.
struct Row {
    int pos, lo, first, n;
    __device__ __forceinline__ Row(const Args& a, int t) {
        pos = a.token_pos[t];
        lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
        first = lo / PAGE;
        n = pos / PAGE + 1 - first;
    }
};
__device__ __forceinline__ int pages_of(const Args& a, int t) { return t < a.n_tokens ? Row(a, t).n : 0; }
__device__ __forceinline__ int parts_of(int n, int c) { return (n + c - 1) / c; }

// Parts of all rows together when a row is cut into parts of at most c pages (by one warp).
__device__ __forceinline__ int count_parts(const Args& a, int c, int lane, int mine) {
    int count = 0;
    for (int base = 0; base < a.n_tokens; base += 32) {
        const int n = base == 0 ? mine : pages_of(a, base + lane);
        count += __reduce_add_sync(0xffffffffu, n > 0 ? parts_of(n, c) : 0);
    }
    return count * a.nkv;
}

// Pages of the busiest block when every block takes whole rows, every gridDim.x-th (by one warp).
__device__ __forceinline__ int busiest_block(const Args& a, int lane) {
    int most = 0;
    for (int block = lane; block < (int)gridDim.x; block += 32) {
        int pages = 0;
        for (int row = block; row < a.n_tokens * a.nkv; row += (int)gridDim.x) pages += Row(a, row / a.nkv).n;
        most = max(most, pages);
    }
    return __reduce_max_sync(0xffffffffu, most);
}

// What a step takes, in microseconds, from the pages of its busiest block and of all blocks on average.  (Fitted to measured steps of 56 to
// 128 sequences of 8 kv heads, 60 to 24,000 tokens, with whole rows and cut ones: within a tenth for most.)
__device__ __forceinline__ float time_of(float busiest, float share) { return 0.65f * busiest + 1.25f * share; }

// Long rows that fill the grid badly - more of them than blocks, so that some blocks have a row when the others are done, or a little
// more than half as many: several parts a block where that should be ahead.  A part more is 6 us of starts and ends, a part of a row
// 0.5 where they are added up.  Returns the pages of a part.  (Not inlined: steps of short rows, which do not come here, took 1 us longer.)
__device__ __noinline__ int cut_long_rows(const Args& a, int c, int most, int share, int first_pages) {
    const int grid = gridDim.x, lane = threadIdx.x & 31;
    const float as_is = a.n_tokens * a.nkv > grid ? time_of(busiest_block(a, lane), share) : time_of(c, share) + 6.0f + 0.5f * parts_of(most, c);
    float least = 0.93f * as_is;
    for (int m = 1; m <= MAX_WAVES - 2; ++m) {
        const int smaller = max(MIN_PART, (share + m - 1) / m), parts = count_parts(a, smaller, lane, first_pages);
        const float time = time_of(share + 0.5f * smaller, share) + 6.0f * ((parts + grid - 1) / grid) + 0.5f * parts_of(most, smaller);
        if (parts <= MAX_WAVES * grid && time < least) {
            least = time;
            c = smaller;
        }
    }
    return c;
}

__global__ void __launch_bounds__(THREADS, BLOCKS_PER_SM)
decode_flat_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Args a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int G = a.nq / a.nkv, stages = a.stages;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // behind the ring: the barriers and a word; then, by turns, the prepared queries [8][D] with the new key and value, and
    // the warps' results [4][G][LDO] with their (max, sum) pairs
    const uint32_t ring = smem_u32(smem), full = ring + stages * STAGE_BYTES, empty = full + 8 * MAX_STAGES;
    int* last_one = reinterpret_cast<int*>(smem + stages * STAGE_BYTES + 16 * MAX_STAGES);
    bf16* prep = reinterpret_cast<bf16*>(smem + stages * STAGE_BYTES + BARS_BYTES);
    float* sm_o = reinterpret_cast<float*>(prep);
    float* sm_ml = sm_o + WARPS * G * LDO;

    pdl_launch_dependents();
    if (ring & 1023u) {                          // the swizzled panels need 1024-byte alignment
        if (threadIdx.x == 0) atomicExch(a.status, 18);
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full + s * 8, 1);
            mbar_init(empty + s * 8, WARPS);
        }
        mbar_init_fence();
    }

    // every warp finds c for itself
    const int first_pages = pages_of(a, lane);
    int c, most = 0;
    {
        int64_t total = 0;
        for (int base = 0; base < a.n_tokens; base += 32) {
            const int n = base == 0 ? first_pages : pages_of(a, base + lane);
            total += __reduce_add_sync(0xffffffffu, n);
            most = max(most, __reduce_max_sync(0xffffffffu, n));
        }
        const int grid = gridDim.x, share = (int)((total * a.nkv + grid - 1) / grid);
        int lo = max(MIN_PART, share);
        int hi = max(lo, most);                  // whole rows: as many parts as there are rows, whether they fit or not
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (count_parts(a, mid, lane, first_pages) <= grid) hi = mid;
            else lo = mid + 1;
        }
        c = lo;
        if (most >= LONG_ROW) c = cut_long_rows(a, c, most, share, first_pages);
    }
    __syncthreads();                             // the barriers are set up

    const bool producer = warp == WARPS;
    // The pages and the step's positions do not depend on the kernel before this one when the new token's key and value are this
    // kernel's own to write; a layer that reads another layer's cache finds them there once the kernels before are done.
    if (producer && !a.write_kv) pdl_wait();
    const int quad = lane >> 2, tq = lane & 3;
    int s = 0;                                   // place in the ring
    uint32_t phase = 0;
    bool ok = true, waited = false;
    // this block's parts: of a list that is longer than the grid every gridDim.x-th
    int before = 0, chunk = blockIdx.x;      // parts of the tokens before `base`
    for (int base = 0; base < a.n_tokens; base += 32) {
        const int n = base == 0 ? first_pages : pages_of(a, base + lane);
        int upto = n > 0 ? parts_of(n, c) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int all = before + __shfl_sync(0xffffffffu, upto, 31) * a.nkv;
        for (; chunk < all; chunk += (int)gridDim.x) {
            const int found = __ffs(__ballot_sync(0xffffffffu, before + upto * a.nkv > chunk)) - 1;
            const int t = base + found, past = found > 0 ? __shfl_sync(0xffffffffu, upto, max(found - 1, 0)) : 0;
            const Row row(a, t);
            const int k = parts_of(row.n, c), at = chunk - before - past * a.nkv;
            const int kvh = at / k, part = at % k;
            const int begin = (int)((int64_t)part * row.n / k), end = (int)((int64_t)(part + 1) * row.n / k);
            const int* pages = a.page_table + (int64_t)a.token_seq[t] * a.pages_per_seq + row.first;

            if (producer) {
                for (int p0 = begin; p0 < end && ok; p0 += 32) {
                    const int mine = p0 + lane < end ? pages[p0 + lane] : 0;
                    const int m = min(32, end - p0);
                    for (int j = 0; j < m; ++j) {
                        const int page = __shfl_sync(0xffffffffu, mine, j);
                        if (!mbar_wait(empty + s * 8, phase ^ 1u)) {
                            if (lane == 0) atomicExch(a.status, 1);
                            ok = false;
                            break;
                        }
                        if (lane == 0) {
                            const uint32_t dst = ring + s * STAGE_BYTES, bar = full + s * 8;
                            const int y = (page * a.nkv + kvh) * PAGE;
                            mbar_expect_tx(bar, STAGE_BYTES);
#pragma unroll
                            for (int h = 0; h < D / 64; ++h) tma_load_2d(dst + h * HALF_BYTES, &map_k, bar, h * 64, y);
#pragma unroll
                            for (int h = 0; h < D / 64; ++h) tma_load_2d(dst + PANEL_BYTES + h * HALF_BYTES, &map_v, bar, h * 64, y);
                        }
                        __syncwarp();
                        if (++s == stages) {
                            s = 0;
                            phase ^= 1u;
                        }
                    }
                }
                continue;
            }

            // the projections, the output of the kernel before, are read from here on
            if (!waited) pdl_wait();
            else meet();                             // the results of the part before have been read
            waited = true;
            // the block that holds the row's last page owns the new token's key and value
            const int pos = row.pos;
            const bool owner = a.write_kv && end == row.n;
            const bf16* src = a.qkv + (int64_t)t * (a.nq + 2 * a.nkv) * D;
            for (int g = warp; g < G; g += WARPS)
                prepare_head<D>(src + (int64_t)(kvh * G + g) * D, prep + g * D, a.q_norm_w, a.cos_tab, a.sin_tab, pos, a.eps, a.rot, lane);
            if (owner) {
                if (warp == G % WARPS)
                    prepare_head<D>(src + (int64_t)(a.nq + kvh) * D, prep + MAX_G * D, a.k_norm_w, a.cos_tab, a.sin_tab, pos, a.eps, a.rot, lane);
                if (warp == (G + 1) % WARPS)
                    for (int i = lane; i < D; i += 32) prep[(MAX_G + 1) * D + i] = src[(int64_t)(a.nq + a.nkv + kvh) * D + i];
            }
            meet();
            if (owner) {       // into the cache for the steps to come; this step reads them from `prep`
                const int64_t to = (((int64_t)pages[row.n - 1] * a.nkv + kvh) * PAGE + pos % PAGE) * D;
                for (int i = threadIdx.x; i < D; i += WARPS * 32) {
                    a.k_pages[to + i] = prep[MAX_G * D + i];
                    a.v_pages[to + i] = prep[(MAX_G + 1) * D + i];
                }
            }
            // the group's queries as columns: column g = head kvh*G + g (columns >= G are zero)
            uint32_t qb[KT][2];
#pragma unroll
            for (int kt = 0; kt < KT; ++kt) {
                qb[kt][0] = quad < G ? *reinterpret_cast<const uint32_t*>(prep + quad * D + kt * 16 + tq * 2) : 0u;
                qb[kt][1] = quad < G ? *reinterpret_cast<const uint32_t*>(prep + quad * D + kt * 16 + tq * 2 + 8) : 0u;
            }
            float o[MT][4];                                  // value 16 mt + quad [+8] of heads 2 tq and 2 tq + 1
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) o[mt][0] = o[mt][1] = o[mt][2] = o[mt][3] = 0.0f;
            float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};   // of those heads; l_run: this lane's keys

            for (int p = begin; p < end; ++p) {
                const uint32_t kbuf = ring + s * STAGE_BYTES, vbuf = kbuf + PANEL_BYTES, bar = s * 8;
                unsigned char* stage = smem + s * STAGE_BYTES;
                if (ok && !mbar_wait(full + bar, phase)) {
                    ok = false;
                    if (lane == 0) atomicExch(a.status, 2);
                }
                if (++s == stages) {
                    s = 0;
                    phase ^= 1u;
                }
                // the new token's own key and value: not in the cache when this page was asked for
                if (owner && p == row.n - 1 && (pos % PAGE) / KEYS == warp) {
                    const int r = pos % PAGE;
                    for (int i = lane; i < D / 8; i += 32) {
                        *reinterpret_cast<uint4*>(stage + packet(r, i)) = *reinterpret_cast<const uint4*>(prep + MAX_G * D + i * 8);
                        *reinterpret_cast<uint4*>(stage + PANEL_BYTES + packet(r, i)) = *reinterpret_cast<const uint4*>(prep + (MAX_G + 1) * D + i * 8);
                    }
                    fence_proxy_async();             // the stage is the copy engine's again afterwards
                    __syncwarp();
                }
                // scores of this warp's 16 keys against the group's heads, in two chains
                float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
                const int krow = warp * KEYS + (lane & 15);
#pragma unroll
                for (int kt = 0; kt < KT; kt += 2) {
                    uint32_t ka[4], kb[4];
                    ldmatrix_x4(ka, kbuf + packet(krow, 2 * kt + (lane >> 4)));
                    ldmatrix_x4(kb, kbuf + packet(krow, 2 * kt + 2 + (lane >> 4)));
                    mma_bf16(sc, ka, qb[kt][0], qb[kt][1]);
                    mma_bf16(sd, kb, qb[kt + 1][0], qb[kt + 1][1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[e] = (sc[e] + sd[e]) * a.scale_log2;
                // keys outside [lo, pos]; sc[0], sc[1] are of key page*64 + warp*16 + quad, sc[2], sc[3] of the eighth after it
                const int key0 = (row.first + p) * PAGE;
                const bool edge = key0 < row.lo || key0 + PAGE - 1 > pos;
                if (edge) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int key = key0 + warp * KEYS + quad + h * 8;
                        if (key < row.lo || key > pos) sc[2 * h] = sc[2 * h + 1] = -INFINITY;
                    }
                }
                float alpha[2], m_use[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float mx = fmaxf(sc[j], sc[2 + j]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    const float m_new = fmaxf(m_run[j], mx);
                    m_use[j] = m_new == -INFINITY ? 0.0f : m_new;      // no key seen yet
                    alpha[j] = exp2f(m_run[j] - m_use[j]);
                    m_run[j] = m_new;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[e] = exp2f(sc[e] - m_use[e & 1]);
#pragma unroll
                for (int j = 0; j < 2; ++j) l_run[j] = l_run[j] * alpha[j] + (sc[j] + sc[2 + j]);
                const uint32_t pb0 = transpose_8x8(pack_bf16(sc[0], sc[1])), pb1 = transpose_8x8(pack_bf16(sc[2], sc[3]));
                // o = o * alpha + V^T . P over this warp's 16 keys; no maximum has moved: nothing to multiply
                if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        o[mt][0] *= alpha[0]; o[mt][1] *= alpha[1];
                        o[mt][2] *= alpha[0]; o[mt][3] *= alpha[1];
                    }
                }
                const int vrow = warp * KEYS + (lane & 7) + ((lane >> 4) << 3);
                if (edge) {
                    // what the page holds outside [lo, pos] was left by whoever had it before: its weight is zero, and zero times an
                    // infinity or a NaN would not be zero
                    const int key = key0 + warp * KEYS + tq * 2;
                    const uint32_t near = keys_seen(key, row.lo, pos), far = keys_seen(key + 8, row.lo, pos);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        uint32_t va[4];
                        ldmatrix_x4_trans(va, vbuf + packet(vrow, 2 * mt + ((lane >> 3) & 1)));
                        va[0] &= near; va[1] &= near; va[2] &= far; va[3] &= far;
                        mma_bf16(o[mt], va, pb0, pb1);
                    }
                } else {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        uint32_t va[4];
                        ldmatrix_x4_trans(va, vbuf + packet(vrow, 2 * mt + ((lane >> 3) & 1)));
                        mma_bf16(o[mt], va, pb0, pb1);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + bar);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                l_run[j] += __shfl_xor_sync(0xffffffffu, l_run[j], 4);
                l_run[j] += __shfl_xor_sync(0xffffffffu, l_run[j], 8);
                l_run[j] += __shfl_xor_sync(0xffffffffu, l_run[j], 16);
            }

            // the warps' results meet where the queries were
            meet();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int g = 2 * tq + j;
                if (g >= G) continue;
                float* to = sm_o + (warp * G + g) * LDO + quad;
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    to[mt * 16] = o[mt][j];
                    to[mt * 16 + 8] = o[mt][2 + j];
                }
                if (quad == 0) {
                    sm_ml[(warp * G + g) * 2 + 0] = m_run[j];
                    sm_ml[(warp * G + g) * 2 + 1] = l_run[j];
                }
            }
            meet();
            float* mine = a.parts + (int64_t)chunk * part_floats(G);
            bf16* out = a.out + ((int64_t)t * a.nq + kvh * G) * D;
            for (int idx = threadIdx.x; idx < G * D; idx += WARPS * 32) {
                const int g = idx / D, col = idx % D;
                float m = -INFINITY;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) m = fmaxf(m, sm_ml[(w * G + g) * 2]);
                float acc = 0.0f, l = 0.0f;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) {
                    const float mw = sm_ml[(w * G + g) * 2];
                    const float f = mw == -INFINITY ? 0.0f : exp2f(mw - m);
                    acc += f * sm_o[(w * G + g) * LDO + col];
                    l += f * sm_ml[(w * G + g) * 2 + 1];
                }
                if (k == 1) {
                    out[idx] = __float2bfloat16_rn(acc / l);
                } else {
                    mine[idx] = acc;
                    if (col == 0) {
                        mine[G * D + 2 * g] = m;
                        mine[G * D + 2 * g + 1] = l;
                    }
                }
            }
            if (k > 1) {
                __threadfence();
                meet();
                if (threadIdx.x == 0) {
                    int* counter = a.counters + (int64_t)t * a.nkv + kvh;
                    const int came = atomicAdd(counter, 1);
                    *last_one = came == k - 1;
                    if (came == k - 1) *counter = 0;
                }
                meet();
                if (*last_one) {
                    __threadfence();
                    // Four values a thread and MERGE parts' packets asked for together: a row of one long sequence has some fifty
                    // parts, and a round of loads takes about a microsecond whatever it brings.
                    const float* parts = a.parts + (int64_t)(chunk - part) * part_floats(G);
                    for (int idx = threadIdx.x * 4; idx < G * D; idx += WARPS * 32 * 4) {
                        const int g = idx / D;
                        float m = -INFINITY, l = 0.0f;
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                        for (int b = 0; b < k; b += MERGE) {
                            float ms[MERGE], ls[MERGE], top = m;
                            float4 os[MERGE];
#pragma unroll
                            for (int i = 0; i < MERGE; ++i) {
                                ms[i] = -INFINITY;
                                ls[i] = 0.0f;
                                os[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (b + i < k) {
                                    const float* from = parts + (int64_t)(b + i) * part_floats(G);
                                    os[i] = __ldcg(reinterpret_cast<const float4*>(from + idx));
                                    ms[i] = __ldcg(from + G * D + 2 * g);
                                    ls[i] = __ldcg(from + G * D + 2 * g + 1);
                                }
                            }
#pragma unroll
                            for (int i = 0; i < MERGE; ++i) top = fmaxf(top, ms[i]);
                            const float use = top == -INFINITY ? 0.0f : top, f = exp2f(m - use);
                            l *= f;
                            acc.x *= f; acc.y *= f; acc.z *= f; acc.w *= f;
#pragma unroll
                            for (int i = 0; i < MERGE; ++i) {
                                const float w = exp2f(ms[i] - use);      // 0 where the part has seen no key
                                l += w * ls[i];
                                acc.x += w * os[i].x; acc.y += w * os[i].y; acc.z += w * os[i].z; acc.w += w * os[i].w;
                            }
                            m = top;
                        }
                        out[idx] = __float2bfloat16_rn(acc.x / l);
                        out[idx + 1] = __float2bfloat16_rn(acc.y / l);
                        out[idx + 2] = __float2bfloat16_rn(acc.z / l);
                        out[idx + 3] = __float2bfloat16_rn(acc.w / l);
                    }
                }
            }
        }
        before = all;
    }
    if (producer || !waited) pdl_wait();         // a grid is done only after the one before it
}

int behind_ring(int G) {
    const int prep = (MAX_G + 2) * D * 2, results = WARPS * G * (LDO + 2) * 4;
    return BARS_BYTES + (prep > results ? prep : results);
}
// Blocks of an SM: three where a ring of two pages and what lies behind it fit three times into its 228 KB (1 KB of each block's
// is the system's), else two.
int blocks_per_sm(int G) { return 2 * STAGE_BYTES + behind_ring(G) <= 75 * 1024 ? BLOCKS_PER_SM : 2; }

}  // namespace

// Blocks of a launch: as many as are resident at once.
Q3_EXPORT int q3_attention_decode_flat_blocks(int group) { return blocks_per_sm(group) * q3_device_sm_count(); }

// Float32 elements of `parts`; `counters` holds n_tokens * nkv ints, zero before the first launch and left zero by each.
Q3_EXPORT int64_t q3_attention_decode_flat_parts(int group) {
    return (int64_t)MAX_WAVES * q3_attention_decode_flat_blocks(group) * part_floats(group) + 4;      // 4: to a 16-byte boundary
}

Q3_EXPORT int q3_attention_decode_flat_bf16(const void* qkv, void* k_pages, void* v_pages, void* out, float* parts, int* counters,
                                            const float* q_norm_w, const float* k_norm_w, const float* cos_tab,
                                            const float* sin_tab, float eps, const int* token_seq, const int* token_pos,
                                            const int* page_table, int pages_per_seq, int64_t n_tokens, int64_t n_cache_pages, int nq,
                                            int nkv, float scale, int window, int write_kv, int rotary_dim, int* status, void* stream_) {
    if (n_tokens <= 0) return 0;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || nq / nkv > MAX_G || n_cache_pages <= 0) return Q3_ERR_BAD_SIZE;
    if ((cos_tab == nullptr) != (sin_tab == nullptr)) return Q3_ERR_BAD_SIZE;
    if (rotary_dim <= 0) rotary_dim = D;
    if (rotary_dim % 2 != 0 || rotary_dim > D) return Q3_ERR_BAD_SIZE;
    if (n_tokens > 65535 || nkv > 65535 || n_tokens * nkv > 1 << 24 || n_cache_pages * nkv * PAGE > 0x7fffffff) return Q3_ERR_TOO_LARGE;
    if (!aligned16(qkv) || !aligned16(k_pages) || !aligned16(v_pages)) return Q3_ERR_MISALIGNED;
    static Q3PerDevice configured;
    cudaError_t e = q3_allow_shared_memory(decode_flat_kernel, 112 * 1024, configured);
    if (e != cudaSuccess) return (int)e;
    const int G = nq / nkv, rows = (int)(n_cache_pages * nkv * PAGE);
    CUtensorMap map_k, map_v;
    if (!q3_make_map_bf16(&map_k, k_pages, rows, D, PAGE, 64, true) || !q3_make_map_bf16(&map_v, v_pages, rows, D, PAGE, 64, true))
        return Q3_ERR_BAD_SIZE;
    Args a;
    a.qkv = (const bf16*)qkv; a.k_pages = (bf16*)k_pages; a.v_pages = (bf16*)v_pages; a.out = (bf16*)out;
    a.parts = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(parts) + 15) & ~(uintptr_t)15);
    a.counters = counters;
    a.q_norm_w = q_norm_w; a.k_norm_w = k_norm_w; a.cos_tab = cos_tab; a.sin_tab = sin_tab;
    a.token_seq = token_seq; a.token_pos = token_pos; a.page_table = page_table;
    a.pages_per_seq = pages_per_seq; a.n_tokens = (int)n_tokens; a.nq = nq; a.nkv = nkv; a.window = window;
    a.rot = rotary_dim; a.write_kv = write_kv; a.eps = eps; a.scale_log2 = scale * 1.4426950408889634f; a.status = status;
    a.stages = ((blocks_per_sm(G) == 3 ? 75 : 112) * 1024 - behind_ring(G)) / STAGE_BYTES;
    if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
    return (int)q3_launch(decode_flat_kernel, dim3(q3_attention_decode_flat_blocks(G)), dim3(THREADS),
                          (size_t)(a.stages * STAGE_BYTES + behind_ring(G)), (cudaStream_t)stream_, map_k, map_v, a);
}
