// Attention over the paged cache in float32 for the usual forms: key and value heads of one size (64 or 128), pages of 64
// positions, all keys or a span of them (`first_visible_key`), a factor on the result.  The other forms of the score, other
// sizes and both spans at once stay with `attention_generic.cu`, whose arithmetic this is: float32 dot products times the
// scale, accurate exponentials, float32 sums, the token at position p sees the keys 0..p of its slot (attention.rs:92-121).
//
// A block owns a tile of up to ROWS rows of one sequence and one kv head (a row is a query head of that kv head at one
// token: row = token * n_rep + head) and walks pages of 64 keys, so a page is read once for all the query heads that share
// it and once per 64 / n_rep tokens, where a block per (token, head) read it each time: scores as a product of register
// tiles (rows / 16 by 4 per thread) out of shared memory, online softmax by 16 threads per row, then the values likewise.
// The next page's keys are copied (cp.async) while this page's values are summed, its values while its scores are.
// The pages of a tile can be dealt out over the blocks of a cluster, which merge through distributed shared memory in the
// order of their ranks: steps of few tokens have too few tiles to fill the GPU.
//
// What bounds it: FFMA, with about as much shared-memory traffic.  333 tokens of 14 heads of 64 over 2 kv heads: 239 us with a
// block per (token, head), 33 with these tiles, 21 with two blocks per tile.
#include "cluster.cuh"

using namespace ri;

namespace {

constexpr int THREADS = 256, KEYS = 64;

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The weight of a key that the row does not see: such a key may hold anything, NaN too, and its value is left out.  A key that is
// seen and whose weight is so small that it is 0 takes part (0 times an infinity is NaN): its weight is never the negative zero.
constexpr float UNSEEN = -0.f;
__device__ __forceinline__ bool unseen(float weight) { return __float_as_uint(weight) == 0x80000000u; }

// over the 16 threads that share a row
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The blocks of a cluster hold, each for the pages it had, a row's maximum and sum (ml) and its weighted values (res, not yet
// divided): the ranks share the rows' channels out, four at a time, and add what the others hold in the order of the ranks.
template <int HD, int ROWS, int LD, typename Write>
__device__ __forceinline__ void merge(const float* res, const float* ml, int rank, int splits, int row0, int n_rows, float out_scale,
                                      Write write) {
    cluster_sync();
    for (int i = rank * THREADS + (int)threadIdx.x; i < ROWS * (HD / 4); i += splits * THREADS) {
        const int r = i / (HD / 4), d = (i % (HD / 4)) * 4;
        if (row0 + r >= n_rows) continue;
        float top = -INFINITY, pm[8], pl[8];
        float4 po[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {            // all reads at once: a trip to a peer costs as much for eight as for one
            const bool there = p < splits;
            pm[p] = there ? peer_float(ml + r, p) : -INFINITY;
            pl[p] = there ? peer_float(ml + ROWS + r, p) : 0.f;
            po[p] = there ? peer_float4(res + r * LD + d, p) : make_float4(0.f, 0.f, 0.f, 0.f);
            top = fmaxf(top, pm[p]);
        }
        float sum = 0.f;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const float f = expf(pm[p] - top);
            sum = fmaf(pl[p], f, sum);
            v.x = fmaf(po[p].x, f, v.x);
            v.y = fmaf(po[p].y, f, v.y);
            v.z = fmaf(po[p].z, f, v.z);
            v.w = fmaf(po[p].w, f, v.w);
        }
        const float inv = out_scale / sum;
        write(row0 + r, d, make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv));
    }
    cluster_sync();                              // a peer may still be reading this block's part
}

// floats of shared memory: queries, keys and values padded by four floats a row (rows then start in different banks), weights
constexpr int smem_floats(int hd, int rows) { return (rows + 2 * KEYS) * (hd + 4) + rows * (KEYS + 4) + 2 * rows; }

template <int HD, int ROWS>
__global__ void __launch_bounds__(THREADS)
attn_f32_kernel(const float* q, int q_ld, const float* __restrict__ kcache, const float* __restrict__ vcache,
                const int* __restrict__ page_table, int max_pages, const int* __restrict__ seq_slot,
                const int* __restrict__ seq_start, const int* __restrict__ cu_seqlens, float* __restrict__ out, int out_ld,
                int n_rep, int n_kv, float scale, int span, float out_scale, int splits) {
    constexpr int RI = ROWS / 16;                // rows per thread: ty, ty + 16, ...
    constexpr int CJ = HD / 64;                  // runs of four channels per thread: 4 tx + 64 j
    constexpr int LD = HD + 4, LP = KEYS + 4;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                            // [ROWS][LD]; at the end the block's result
    float* ks = qs + ROWS * LD;                  // [KEYS][LD]
    float* vs = ks + KEYS * LD;                  // [KEYS][LD]
    float* ps = vs + KEYS * LD;                  // [ROWS][LP]
    float* ml = ps + ROWS * LP;                  // [2][ROWS]

    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int rank = splits > 1 ? (int)cluster_rank() : 0;
    const int tile = (int)blockIdx.x / splits, kvh = blockIdx.y, seq = blockIdx.z;
    let_next_kernel_start();
    wait_for_previous_kernels();
    const int first_tok = cu_seqlens[seq], n_tok = cu_seqlens[seq + 1] - first_tok;
    const int n_rows = n_tok * n_rep, row0 = tile * ROWS;
    if (row0 >= n_rows) return;                  // a whole cluster at once: its blocks share the tile
    const int start = seq_start[seq];
    const int* pages = page_table + (size_t)seq_slot[seq] * max_pages;

    for (int i = tid; i < ROWS * (HD / 4); i += THREADS) {
        const int r = i / (HD / 4), d = (i % (HD / 4)) * 4, row = row0 + r;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n_rows)
            v = load_written(q + (size_t)(first_tok + row / n_rep) * q_ld + (size_t)(kvh * n_rep + row % n_rep) * HD + d);
        *reinterpret_cast<float4*>(qs + r * LD + d) = v;
    }

    int pos[RI], low[RI];                        // this thread's rows: position and first visible key (a row beyond the step sees none)
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int row = row0 + ty + 16 * i;
        pos[i] = row < n_rows ? start + row / n_rep : -1;
        low[i] = row < n_rows ? first_visible_key(pos[i], span) : 0;
    }
    const int last_pos = start + (min(row0 + ROWS, n_rows) - 1) / n_rep;
    const int page_end = last_pos / KEYS + 1;
    int page = first_visible_key(start + row0 / n_rep, span) / KEYS + rank;

    auto fetch = [&](float* dst, const float* cache, int p) {
        if (p < page_end) {
            int at = pages[p];
            if (!RI_BLOCK_IN_LIMIT(at, RI_LIMIT_PAGES, RI_CHECK_PAGE)) at = 0;      // checked build: recorded, read from a page that exists
            const float* src = cache + ((size_t)at * n_kv + kvh) * KEYS * HD;
#pragma unroll
            for (int i = 0; i < KEYS * HD / 4 / THREADS; ++i) {
                const int e = (i * THREADS + tid) * 4;
                copy16(dst + (e / HD) * LD + e % HD, src + e);
            }
        }
        copies_commit();
    };
    fetch(ks, kcache, page);
    fetch(vs, vcache, page);

    float m[RI], l[RI], o[RI][CJ][4];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < CJ; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[i][j][c] = 0.f;
    }

    for (; page < page_end; page += splits) {
        copies_wait<1>();
        __syncthreads();                         // keys (and, the first time, queries) are there
        float s[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            float4 a[RI], b[4];
#pragma unroll
            for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty + 16 * i) * LD + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * LD + d);
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                    s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                    s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                    s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                }
        }
        // softmax: the 16 threads of a row hold 4 keys each
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            float top = -INFINITY;
            bool seen[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = page * KEYS + tx + 16 * j;
                seen[j] = key <= pos[i] && key >= low[i];
                s[i][j] = seen[j] ? s[i][j] * scale : -INFINITY;
                top = fmaxf(top, s[i][j]);
            }
            const float m_new = fmaxf(m[i], row_max(top));
            const float ref = m_new == -INFINITY ? 0.f : m_new;        // no visible key yet: every weight is exp(-inf) = 0
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = seen[j] ? expf(s[i][j] - ref) : UNSEEN;
                ps[(ty + 16 * i) * LP + tx + 16 * j] = p;
                sum += p;
            }
            const float alpha = expf(m[i] - ref);
            l[i] = l[i] * alpha + row_sum(sum);
            m[i] = m_new;
#pragma unroll
            for (int j = 0; j < CJ; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) o[i][j][c] *= alpha;
        }
        __syncthreads();                         // the keys are used up, the weights are there
        fetch(ks, kcache, page + splits);
        copies_wait<1>();
        __syncthreads();                         // the values are there
#pragma unroll 4
        for (int kk = 0; kk < KEYS; kk += 4) {
            float4 p[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) p[i] = *reinterpret_cast<const float4*>(ps + (ty + 16 * i) * LP + kk);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float4 v[CJ];
#pragma unroll
                for (int j = 0; j < CJ; ++j) v[j] = *reinterpret_cast<const float4*>(vs + (kk + u) * LD + 4 * tx + 64 * j);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const float w = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                    if (!unseen(w)) {
#pragma unroll
                        for (int j = 0; j < CJ; ++j) {
                            o[i][j][0] = fmaf(w, v[j].x, o[i][j][0]);
                            o[i][j][1] = fmaf(w, v[j].y, o[i][j][1]);
                            o[i][j][2] = fmaf(w, v[j].z, o[i][j][2]);
                            o[i][j][3] = fmaf(w, v[j].w, o[i][j][3]);
                        }
                    }
                }
            }
        }
        __syncthreads();                         // values and weights are used up
        fetch(vs, vcache, page + splits);
    }
    copies_wait<0>();

    auto write = [&](int row, int d, const float4& v) {
        *reinterpret_cast<float4*>(out + (size_t)(first_tok + row / n_rep) * out_ld + (size_t)(kvh * n_rep + row % n_rep) * HD + d) = v;
    };
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int row = row0 + ty + 16 * i;
            if (row >= n_rows) continue;
            const float inv = out_scale / l[i];
#pragma unroll
            for (int j = 0; j < CJ; ++j)
                write(row, 4 * tx + 64 * j, make_float4(o[i][j][0] * inv, o[i][j][1] * inv, o[i][j][2] * inv, o[i][j][3] * inv));
        }
        return;
    }
    __syncthreads();                             // a block without pages comes here while its queries are still being stored
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int r = ty + 16 * i;
#pragma unroll
        for (int j = 0; j < CJ; ++j)
            *reinterpret_cast<float4*>(qs + r * LD + 4 * tx + 64 * j) = make_float4(o[i][j][0], o[i][j][1], o[i][j][2], o[i][j][3]);
        if (tx == 0) {
            ml[r] = m[i];
            ml[ROWS + r] = l[i];
        }
    }
    merge<HD, ROWS, LD>(qs, ml, rank, splits, row0, n_rows, out_scale, write);
}

// Few rows (single tokens): a block still walks pages of 64 keys, but every thread takes its part of a page straight from memory
// into registers, the next page's while this one is worked on, and shared memory holds only queries and weights.  Four threads
// share a key (each a quarter of its channels) and meet all rows with it; a warp per row forms the softmax; then a thread
// owns four channels of a few keys' values.  What bounds a step is the latency of a block's few pages: 16-row tiles of the kernel
// above, which read every key through shared memory for all of their rows, took 17.1 us for four sequences of up to 700 positions
// (6 query heads per kv head of 128, eight blocks each; the generic kernel 112); with this one the 28-layer step around it went
// from 2,286 to 1,989 us.  Positions, slots, pages and a first page that lies wholly before the step are read before the wait for the
// kernel before: the chain of four dependent reads and the page's own is over when the queries come (with the float32 rotary kernel's
// reads done likewise, 1,963 -> 1,894 us, products as they were).
template <int HD, int ROWS>
constexpr int few_smem_floats() { return ROWS * HD + 2 * ROWS * (KEYS + 4) + 4 * ROWS + 1024 / HD * ROWS * HD; }

template <int HD, int ROWS>
__global__ void __launch_bounds__(THREADS)
attn_f32_few_kernel(const float* q, int q_ld, const float* __restrict__ kcache, const float* __restrict__ vcache,
                    const int* __restrict__ page_table, int max_pages, const int* __restrict__ seq_slot,
                    const int* __restrict__ seq_start, const int* __restrict__ cu_seqlens, float* __restrict__ out, int out_ld,
                    int n_rep, int n_kv, float scale, int span, float out_scale, int splits) {
    constexpr int KN = HD / 16;                  // four-channel pieces of a key per thread
    constexpr int GROUPS = 1024 / HD;            // groups of keys whose values are summed side by side
    constexpr int VN = KEYS / GROUPS;            // keys per group
    constexpr int LP = KEYS + 4;
    constexpr int WARPS = THREADS / 32;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                            // [ROWS][HD]; at the end the block's result
    float* ps = qs + ROWS * HD;                  // two of [ROWS][LP]
    float* factor = ps + 2 * ROWS * LP;          // two of [ROWS]: what a row's sums so far are multiplied by
    float* ml = factor + 2 * ROWS;               // [2][ROWS]
    float* parts = ml + 2 * ROWS;                // [GROUPS][ROWS][HD]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = splits > 1 ? (int)cluster_rank() : 0;
    const int kvh = blockIdx.y, seq = blockIdx.z;
    let_next_kernel_start();
    // positions, slots and pages are fixed before the step, and so are the keys and values of pages that lie wholly before it
    const int first_tok = cu_seqlens[seq], n_tok = cu_seqlens[seq + 1] - first_tok;
    const int n_rows = n_tok * n_rep;            // at most ROWS
    if (n_rows == 0) {                           // a whole cluster at once
        wait_for_previous_kernels();             // (who waits for this kernel waits for those before it too)
        return;
    }
    const int start = seq_start[seq];
    const int* pages = page_table + (size_t)seq_slot[seq] * max_pages;
    const int page_end = (start + n_tok - 1) / KEYS + 1;
    int page = first_visible_key(start, span) / KEYS + rank;

    const int key = tid >> 2, quarter = tid & 3, channel = (tid % (HD / 4)) * 4, group = tid / (HD / 4);
    float4 kr[KN], vr[VN];
    auto row_of = [&](int p) -> size_t {
        int at = pages[p];
        if (!RI_BLOCK_IN_LIMIT(at, RI_LIMIT_PAGES, RI_CHECK_PAGE)) at = 0;      // checked build: recorded, read from a page that exists
        return ((size_t)at * n_kv + kvh) * KEYS;
    };
    auto fetch_keys = [&](int p) {
        if (p >= page_end) return;
        const float* src = kcache + (row_of(p) + key) * HD + quarter * 4;
#pragma unroll
        for (int i = 0; i < KN; ++i) kr[i] = load_written(src + 16 * i);
    };
    auto fetch_values = [&](int p) {
        if (p >= page_end) return;
        const float* src = vcache + (row_of(p) + group * VN) * HD + channel;
#pragma unroll
        for (int i = 0; i < VN; ++i) vr[i] = load_written(src + i * HD);
    };
    const bool older = (page + 1) * KEYS <= start;
    if (older) {
        fetch_keys(page);
        fetch_values(page);
    }
    wait_for_previous_kernels();
    if (!older) {
        fetch_keys(page);
        fetch_values(page);
    }
    for (int i = tid * 4; i < ROWS * HD; i += THREADS * 4) {
        const int r = i / HD, d = i % HD;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n_rows) v = load_written(q + (size_t)(first_tok + r / n_rep) * q_ld + (size_t)(kvh * n_rep + r % n_rep) * HD + d);
        *reinterpret_cast<float4*>(qs + i) = v;
    }
    __syncthreads();

    constexpr int OWN = ROWS / WARPS;            // rows whose softmax this warp forms: warp, warp + WARPS
    float m[OWN], l[OWN], o[ROWS][4];
#pragma unroll
    for (int i = 0; i < OWN; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[r][c] = 0.f;

    for (int turn = 0; page < page_end; page += splits, turn ^= 1) {
        float* p = ps + turn * ROWS * LP;
        float* f = factor + turn * ROWS;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r >= n_rows) break;
            float dot = 0.f;
#pragma unroll
            for (int i = 0; i < KN; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(qs + r * HD + quarter * 4 + 16 * i);
                dot = fmaf(a.x, kr[i].x, fmaf(a.y, kr[i].y, fmaf(a.z, kr[i].z, fmaf(a.w, kr[i].w, dot))));
            }
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
            if ((r & 3) == quarter) p[r * LP + key] = dot;
        }
        fetch_keys(page + splits);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < OWN; ++i) {
            const int r = warp + i * WARPS;
            if (r >= n_rows) continue;           // uniform over the warp
            const int pos = start + r / n_rep, low = first_visible_key(pos, span);
            float s[2], top = -INFINITY;
            bool seen[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int k = page * KEYS + lane + 32 * j;
                seen[j] = k <= pos && k >= low;
                s[j] = seen[j] ? p[r * LP + lane + 32 * j] * scale : -INFINITY;
                top = fmaxf(top, s[j]);
            }
            const float m_new = fmaxf(m[i], warp_max(top));
            const float ref = m_new == -INFINITY ? 0.f : m_new;        // no visible key yet: every weight is exp(-inf) = 0
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float e = seen[j] ? expf(s[j] - ref) : UNSEEN;
                p[r * LP + lane + 32 * j] = e;
                sum += e;
            }
            const float alpha = expf(m[i] - ref);
            l[i] = l[i] * alpha + warp_sum(sum);
            m[i] = m_new;
            if (lane == 0) f[r] = alpha;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r >= n_rows) break;
            const float alpha = f[r];
#pragma unroll
            for (int c = 0; c < 4; ++c) o[r][c] *= alpha;
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                const float w = p[r * LP + group * VN + i];
                if (!unseen(w)) {
                    o[r][0] = fmaf(w, vr[i].x, o[r][0]);
                    o[r][1] = fmaf(w, vr[i].y, o[r][1]);
                    o[r][2] = fmaf(w, vr[i].z, o[r][2]);
                    o[r][3] = fmaf(w, vr[i].w, o[r][3]);
                }
            }
        }
        fetch_values(page + splits);
        // the next page's scores go to the other half of `ps`; this half is written again behind the next barrier
    }

#pragma unroll
    for (int i = 0; i < OWN; ++i)
        if (lane == 0) {
            ml[warp + i * WARPS] = m[i];
            ml[ROWS + warp + i * WARPS] = l[i];
        }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        *reinterpret_cast<float4*>(parts + (group * ROWS + r) * HD + channel) = make_float4(o[r][0], o[r][1], o[r][2], o[r][3]);
    __syncthreads();
    auto write = [&](int row, int d, const float4& v) {
        *reinterpret_cast<float4*>(out + (size_t)(first_tok + row / n_rep) * out_ld + (size_t)(kvh * n_rep + row % n_rep) * HD + d) = v;
    };
    for (int i = tid * 4; i < n_rows * HD; i += THREADS * 4) {
        float4 v = *reinterpret_cast<const float4*>(parts + i);
#pragma unroll
        for (int g = 1; g < GROUPS; ++g) {
            const float4 u = *reinterpret_cast<const float4*>(parts + g * ROWS * HD + i);
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        if (splits == 1) {
            const float inv = out_scale / ml[ROWS + i / HD];
            write(i / HD, i % HD, make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv));
        } else {
            *reinterpret_cast<float4*>(qs + i) = v;
        }
    }
    if (splits > 1) merge<HD, ROWS, HD>(qs, ml, rank, splits, 0, n_rows, out_scale, write);
}

template <int HD, int ROWS>
int launch(const float* q, int q_ld, const float* kcache, const float* vcache, const int* page_table, int max_pages, const int* seq_slot,
           const int* seq_start, const int* cu_seqlens, float* out, int out_ld, int n_seqs, int max_new, int n_rep, int n_kv, float scale,
           int span, float out_scale, int splits, cudaStream_t stream) {
    constexpr bool FEW = ROWS <= 16;
    constexpr size_t SMEM = (FEW ? few_smem_floats<HD, ROWS>() : smem_floats(HD, ROWS)) * sizeof(float);
    auto kernel = [] {
        if constexpr (FEW) return attn_f32_few_kernel<HD, ROWS>;
        else return attn_f32_kernel<HD, ROWS>;
    }();
    static PerDeviceOnce once;
    if (int rc = raise_dynamic_smem(kernel, (int)SMEM, once, "attention_f32")) return rc;
    const long long tiles = FEW ? 1 : ((long long)max_new * n_rep + ROWS - 1) / ROWS;
    if (tiles * splits > 0x7fffffffLL) return fail("attention_f32: %lld row tiles", tiles);
    return launch_cluster("attention_f32", kernel, dim3((unsigned)(tiles * splits), n_kv, n_seqs), THREADS, SMEM, splits,
                          stream, q, q_ld, kcache, vcache, page_table, max_pages, seq_slot, seq_start, cu_seqlens, out, out_ld, n_rep, n_kv,
                          scale, span, out_scale, splits);
}

}  // namespace

// `span`: see `first_visible_key`; `splits`: blocks (1..8) that share the pages of a row tile; `max_new`: the most tokens any of
// the step's sequences brings.  Steps of up to 16 rows per kv head and sequence take the kernel for few rows, others tiles of 64.
RI_API int ri_attention_f32(const float* q, int q_ld, const float* kcache, const float* vcache, const int* page_table, int max_pages,
                            const int* seq_slot, const int* seq_start, const int* cu_seqlens, float* out, int out_ld, int n_seqs,
                            int max_new, int n_heads, int n_kv, int hd, int page_size, float scale, int span, float out_scale, int splits,
                            cudaStream_t stream) {
    if (n_seqs <= 0 || max_new <= 0) return 0;
    if (n_kv <= 0 || n_heads % n_kv) return fail("attention_f32: %d heads are not a multiple of %d kv heads", n_heads, n_kv);
    if (page_size != KEYS) return fail("attention_f32: pages of %d positions (64 are wanted)", page_size);
    if (hd != 64 && hd != 128) return fail("attention_f32: head size %d", hd);
    if (q_ld % 4 || out_ld % 4 || ((uintptr_t)q | (uintptr_t)out | (uintptr_t)kcache | (uintptr_t)vcache) % 16)
        return fail("attention_f32: rows must be whole, aligned 16-byte pieces");
    if (splits < 1 || splits > 8) return fail("attention_f32: %d blocks per row tile", splits);
    if (n_kv > 65535 || n_seqs > 65535) return fail("attention_f32: %d kv heads, %d sequences exceed the grid limit", n_kv, n_seqs);
    const int n_rep = n_heads / n_kv;
    const long long rows = (long long)max_new * n_rep;
#define RI_RUN(HD, ROWS)                                                                                                            \
    return launch<HD, ROWS>(q, q_ld, kcache, vcache, page_table, max_pages, seq_slot, seq_start, cu_seqlens, out, out_ld, n_seqs,   \
                            max_new, n_rep, n_kv, scale, span, out_scale, splits, stream)
    if (hd == 64) {
        if (rows <= 8) RI_RUN(64, 8);
        if (rows <= 16) RI_RUN(64, 16);
        RI_RUN(64, 64);
    }
    if (rows <= 8) RI_RUN(128, 8);
    if (rows <= 16) RI_RUN(128, 16);
    RI_RUN(128, 64);
#undef RI_RUN
}

RI_DEFINE_LAST_ERROR()
