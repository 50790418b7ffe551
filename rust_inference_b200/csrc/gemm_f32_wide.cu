// out[M, N] = X[M, K] * W[N, K]^T for float32 operands of many rows (prompts), on the tensor cores without giving up 32 bits: the
// arithmetic of `gemm_f32.cu`'s kernel for more than a few rows (three bfloat16 parts per operand, eight products of parts, sums of 64
// steps of K added to float32 registers), cut so that less work goes into a multiply-add:
//
//   - X is cut once, by a kernel before this one, into three bfloat16 matrices that TMA brings into shared memory; in that kernel
//     every tile of rows of W cuts X again.
//   - The grid is persistent, and the epilogue runs from registers: the next tile's weights are cut and its first products made meanwhile.
//   - A tile's width follows the rows there are (a multiple of 16 up to 128): 333 rows are three tiles of 112.
//   - Eight such sums go onto one register before it joins a sum in tensor memory, which keeps long sums as close to 64 bits as several
//     pieces of K would (relative error, rows of N(0, 1) times rows of N(0, 1/K), in brackets with one running sum of the blocks:
//     0.90e-7 at K = 896, 1.04e-7 (1.16e-7) at 4,864, 1.17e-7 (1.77e-7) at 18,944).
//
// What bounds it: per 64 steps of K the cutting of W (four warps, about 1,900 clocks) up to 64 rows and, beyond, shared memory (the
// parts of W stored, those of X arriving, the reads of 32 MMAs): 2,080 clocks at 64 rows, 2,540 at 128, where the tensor core needs
// 1,024 and 2,048.  us, before (X cut in every tile) -> now: 333 x 151,936 x 896 1,000 -> 643, 333 x 4,864 x 896 gated 81 -> 59, 333 x 896 x
// 4,864 56 -> 46, 256 x 8,960 x 1,536 gated 126 -> 107, 512 x 1,536 x 8,960 208 -> 123.
//
// Per block of K: four warps read 128 x 64 numbers of W, cut them and store the parts (128-byte swizzle); one thread brings the parts
// of X; one thread issues the MMAs; eight warps add the sums to registers, two per 32 rows of W.  Both operands lie in one of two
// stages.  Sums keep a fixed order, so a product's bits do not change from run to run.
//
// K may be cut over the blocks of a cluster (few tiles); the pieces meet through distributed shared memory in a fixed order.
// Sums that came out infinite or NaN are computed again with FFMA as plain float32 sums; finite ones beside them keep their bits.
#include "cluster.cuh"
#include "gemm_f32_common.cuh"
#include "tcgen05_common.cuh"

using namespace ri;
using namespace ri::f32;
using namespace ri::tc;

namespace {

constexpr int ROWS = 128, BK = 64, PART = ROWS * BK * 2;
constexpr int STAGES = 2, W_STAGE = 3 * PART;
constexpr int MAX_TN = 128, HALF_MAX = MAX_TN / 2;           // rows of X per tile; columns an adding warp holds
constexpr int GROUP = 8;                                     // blocks of K whose sums go onto one register before it joins the sum in tensor memory
constexpr int ADD_WARPS = 8, CUT_WARPS = 4, TMA_WARP = ADD_WARPS + CUT_WARPS, MMA_WARP = TMA_WARP + 1;
// Warps come in fours that share out the block's registers (16 x 32 x 128 at launch): the adding ones hold a tile's sums.
constexpr int THREADS = 16 * 32, LAUNCH_REGS = 128, ADD_REGS = 176, CUT_REGS = 96, ISSUE_REGS = 64;
static_assert(8 * ADD_REGS + 4 * CUT_REGS + 4 * ISSUE_REGS <= 16 * LAUNCH_REGS, "a warp waits for registers that the block does not have");
constexpr int S_COL = MAX_TN, SUM_COL = 3 * MAX_TN;          // tensor memory: the large products' sums, two buffers of the small ones', the groups' sum
enum Status { ST_CUT_TIMEOUT = 41, ST_MMA_TIMEOUT = 42, ST_ADD_TIMEOUT = 43 };

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// X [M, K] -> parts [3][M][ld] (the leading parts, the middle ones, the rest; zeros beyond K), four numbers per thread.
__global__ void __launch_bounds__(256)
cut_rows_kernel(const float* X, __nv_bfloat16* parts, int M, int K, int ld) {
    let_next_kernel_start();
    wait_for_previous_kernels();
    const int per_row = ld / 4;
    const size_t total = (size_t)M * per_row, plane = (size_t)M * ld;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t m = i / per_row;
        const int k = (int)(i - m * per_row) * 4;
        const float4 v = k < K ? load_written(X + m * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint2 hi, mid, lo;
        cut(make_float2(v.x, v.y), hi.x, mid.x, lo.x);
        cut(make_float2(v.z, v.w), hi.y, mid.y, lo.y);
        uint2* to = reinterpret_cast<uint2*>(parts + m * ld + k);
        to[0] = hi;
        to[plane / 4] = mid;
        to[plane / 2] = lo;
    }
}

// The row of W (gated: of W or W2) that is row r of the tile whose first feature is f0.  A gated tile has 64 features: of every 32
// rows the first 16 are gate rows and the others the up rows of the same features, so that both lie in one warp.
template <bool DUAL>
__device__ __forceinline__ int feature_of(int f0, int r) { return f0 + (DUAL ? (r >> 5) * 16 + (r & 15) : r); }
template <bool DUAL>
__device__ __forceinline__ const float* weight_row(const float* W, const float* W2, int f0, int r, int K) {
    return (DUAL && (r & 16) ? W2 : W) + (size_t)feature_of<DUAL>(f0, r) * K;
}

// `finish`; an element that is added to is added to once, by an instruction that returns nothing, so that nobody waits for its old value
// (read first: 2 to 8% of a product whose K is cut; the comparison below: 1 to 2%).  That instruction takes subnormal operands and results for zeros.  From |v| = 2^-100 on
// this changes no sum: a subnormal is less than half of v's last place, and what two such numbers leave of each other is a multiple of
// 2^-124.  Smaller v are added the ordinary way.
template <int MODE>
__device__ __forceinline__ void put_out(float* out, size_t o, int f, float v, float up, const float* __restrict__ bias, const Forms& forms) {
    if (MODE == 2) {
        if (fabsf(v) < 0x1p-100f) out[o] += v;
        else atomicAdd(out + o, v);
    } else {
        finish<MODE>(out, o, f, v, up, bias, forms);
    }
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_wide_kernel(const __grid_constant__ CUtensorMap map_x, const float* X, const float* __restrict__ W, const float* __restrict__ W2,
                     const float* __restrict__ bias, float* out, int M, int N, int K, int tn, int tok_tiles, int tiles, int splits,
                     int* status) {
    constexpr bool DUAL = MODE == 3;
    constexpr int FEATS = DUAL ? ROWS / 2 : ROWS;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[STAGES], done[STAGES], read_out;
    __shared__ float again[ADD_WARPS][4 * 32];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag, any_failed;

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;             // stages: three parts of W, three of X
    const uint32_t x_bytes = (uint32_t)tn * BK * 2, stage_bytes = W_STAGE + 3 * x_bytes;
    float* pieces = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));      // [tn][128], over the stages at the end
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = splits > 1 ? (int)cluster_rank() : 0;
    const int first = (int)blockIdx.x / splits, step = (int)gridDim.x / splits;            // tiles first, first + step, ...
    const int total_kb = (K + BK - 1) / BK;
    const int kb0 = (int)((long long)total_kb * rank / splits);
    const int n_kb = (int)((long long)total_kb * (rank + 1) / splits) - kb0;               // >= 1: splits <= total_kb

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), CUT_WARPS + 1);    // the warps that cut W, and what announces the bytes of X
            mbar_init(smem_u32(&done[s]), 1);                // a block's products: its stage is free, its sums may be read
        }
        mbar_init(smem_u32(&read_out), ADD_WARPS);           // the sums have been read
        abort_flag = any_failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (splits > 1) cluster_arrive();            // flags and barriers are set up
    let_next_kernel_start();

    if (warp >= ADD_WARPS && warp < TMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CUT_REGS));
        // ---- read, cut and store W: 16 threads per row of 64 floats, rows row, row + 8, ... ----
        const int tid = (int)threadIdx.x - ADD_WARPS * 32;
        const int k4 = tid & 15, row = tid >> 4;
        constexpr int PER = ROWS / (CUT_WARPS * 2);
        const uint32_t col = (uint32_t)(row * 128 + ((k4 * 8) ^ ((row & 7) << 4)));
        // One address per matrix and tile: row r of a plain tile is row f0 + r of W; of a gated one rows with bit 4 are W2's.
        const size_t stride = (size_t)8 * K;
        const float *w1 = W, *w2 = W;
        uint32_t has = 0;                                    // a bit for every one of the thread's rows that exists
        auto enter = [&](int f0) {
            has = 0;
            if (f0 < 0) return;
            w1 = W + (size_t)(f0 + row) * K + k4 * 4;
            if (DUAL) w2 = W2 + (size_t)(f0 + row) * K + k4 * 4;
#pragma unroll
            for (int i = 0; i < PER; ++i) has |= (feature_of<DUAL>(f0, row + 8 * i) < N ? 1u : 0u) << i;
        };
        auto load = [&](int i, int k) {                      // gated: of every four steps of 8 rows two are W's, two W2's
            const float* p = !DUAL ? w1 + (size_t)i * stride : ((i & 2) ? w2 : w1) + (size_t)((i >> 2) * 2 + (i & 1)) * stride;
            return ((has >> i) & 1) && k4 * 4 + k < K ? load_weight(p + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 wv[PER];
        int tile = first;
        enter(tile < tiles ? tile / tok_tiles * FEATS : -1);
#pragma unroll
        for (int i = 0; i < PER; ++i) wv[i] = load(i, kb0 * BK);
        uint32_t g = 0;
        for (bool alive = true; tile < tiles && alive; tile += step)
            for (int b = 0; b < n_kb; ++b, ++g) {
                const uint32_t s = g % STAGES;
                if (!mbar_wait(smem_u32(&done[s]), ((g / STAGES) & 1u) ^ 1u)) {
                    if (!abort_flag && lane == 0) report(status, ST_CUT_TIMEOUT);
                    abort_flag = 1;
                }
                if (abort_flag) { alive = false; break; }
                // the registers take the next 64 of K, of this tile or of the next, as soon as they are cut
                int k = (kb0 + b + 1) * BK;
                if (b + 1 == n_kb) {
                    enter(tile + step < tiles ? (tile + step) / tok_tiles * FEATS : -1);
                    k = kb0 * BK;
                }
                const uint32_t stage = base + s * stage_bytes + col;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    put(stage + (uint32_t)(i * 8 * 128), PART, wv[i]);
                    wv[i] = load(i, k);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the MMA reads what was just stored
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full[s]));
            }
    } else if (warp >= TMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGS));
        if (warp == TMA_WARP) {
            // ---- the parts of X ----
            if (lane == 0) {
                wait_for_previous_kernels();
                uint32_t g = 0;
                bool alive = true;
                for (int tile = first; tile < tiles && alive; tile += step) {
                    const int t0 = tile % tok_tiles * tn;
                    for (int b = 0; b < n_kb; ++b, ++g) {
                        const uint32_t s = g % STAGES;
                        if (!mbar_wait(smem_u32(&done[s]), ((g / STAGES) & 1u) ^ 1u) || abort_flag) {
                            if (!abort_flag) report(status, ST_CUT_TIMEOUT);
                            abort_flag = 1;
                            alive = false;
                            break;
                        }
                        mbar_expect_tx(smem_u32(&full[s]), 3 * x_bytes);
                        for (int p = 0; p < 3; ++p)
                            tma_load_3d(base + s * stage_bytes + W_STAGE + p * x_bytes, &map_x, smem_u32(&full[s]), (kb0 + b) * BK, t0, p);
                    }
                }
                // no copy into this block's shared memory may be in flight when it leaves: what was read by a finished product has
                // landed, and where something gave up the wait runs out
                for (uint32_t j = g > STAGES ? g - STAGES : 0; j < g; ++j)
                    if (!mbar_wait(smem_u32(&full[j % STAGES]), (j / STAGES) & 1u)) { report(status, ST_CUT_TIMEOUT); break; }
            }
        } else if (warp == MMA_WARP) {
            // ---- the products of a block of K, the small ones first, the large one into sums of its own ----
            // (the whole warp goes through this, one lane issues: see `umma_by`)
            const uint32_t leader = elect_one();
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tn >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
            const uint64_t a_desc = make_smem_desc(base), b_desc = make_smem_desc(base + W_STAGE);
            constexpr int PA[7] = {1, 2, 2, 0, 1, 1, 0}, PB[7] = {2, 1, 0, 2, 1, 0, 1};      // parts of W and of X
            const uint64_t x_part = (uint64_t)(x_bytes >> 4);
            uint32_t g = 0;
            bool ok = true;
            for (int tile = first; tile < tiles && ok; tile += step)
                for (int b = 0; b < n_kb && ok; ++b, ++g) {
                    const uint32_t s = g % STAGES;
                    ok = mbar_wait_warp(smem_u32(&full[s]), (g / STAGES) & 1u);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((s * stage_bytes) >> 4);
                    const uint64_t a0 = a_desc + off, b0 = b_desc + off;
                    // the small sums of two blocks ago were read before the large one of the last began
                    const uint32_t small = tmem + S_COL + (g & 1u) * MAX_TN;
#pragma unroll
                    for (int p = 0; p < 7; ++p)
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            umma_by(leader, small, a0 + (uint64_t)(PA[p] * (PART >> 4) + 2 * k), b0 + PB[p] * x_part + 2 * k, idesc,
                                    p > 0 || k > 0);
                    if (g > 0) {
                        ok = mbar_wait_warp(smem_u32(&read_out), (g - 1) & 1u);
                        tc_fence_after();
                    }
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_by(leader, tmem, a0 + 2 * k, b0 + 2 * k, idesc, k > 0);
                    umma_commit_by(leader, smem_u32(&done[s]));
                }
            if (!ok) {
                if (!abort_flag && lane == 0) report(status, ST_MMA_TIMEOUT);
                abort_flag = 1;
            }
            // tensor memory is given back below: what was issued has finished
            if (g > 0) mbar_wait(smem_u32(&done[(g - 1) % STAGES]), ((g - 1) / STAGES) & 1u);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ADD_REGS));
        // ---- add the sums onto registers, write the tile: a thread owns a row of W (a TMEM lane) and half of the rows of X ----
        const int q = warp & 3, part = warp >> 2, half = tn / 2;     // q: the TMEM lanes this warp may read
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * half);
        const uint32_t sum_row = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(SUM_COL + part * HALF_MAX);
        wait_for_previous_kernels();                                 // `out` and X come from earlier kernels
        const Forms forms = load_forms<MODE>(bias);
        uint32_t g = 0;
        for (int tile = first; tile < tiles; tile += step) {
            const int t0 = tile % tok_tiles * tn + part * half, f0 = tile / tok_tiles * FEATS;
            float acc[HALF_MAX];
#pragma unroll
            for (int c = 0; c < HALF_MAX; ++c) acc[c] = 0.f;
            for (int b = 0; b < n_kb; ++b, ++g) {
                const bool landed = !abort_flag && mbar_wait(smem_u32(&done[g % STAGES]), (g / STAGES) & 1u);
                if (!landed && lane == 0) {
                    if (!abort_flag) report(status, ST_ADD_TIMEOUT);
                    abort_flag = 1;
                }
                if (__any_sync(0xffffffffu, abort_flag)) break;
                tc_fence_after();
                const uint32_t small_at = S_COL + (g & 1u) * MAX_TN;
#pragma unroll
                for (int c0 = 0; c0 < HALF_MAX; c0 += 16) {
                    if (c0 >= half) break;
                    uint32_t large[16], small[16];
                    tmem_ld16(trow + (uint32_t)c0, large);
                    tmem_ld16(trow + small_at + (uint32_t)c0, small);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(large[j]) + __uint_as_float(small[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&read_out));
                // a sum of GROUP blocks joins those before it: fewer roundings of a large sum
                const bool first_group = b < GROUP, last = b + 1 == n_kb;
                if ((b % GROUP == GROUP - 1 || last) && !(first_group && last)) {
#pragma unroll
                    for (int c0 = 0; c0 < HALF_MAX; c0 += 16) {
                        if (c0 >= half) break;
                        uint32_t sum[16];
                        if (!first_group) {
                            tmem_ld16(sum_row + (uint32_t)c0, sum);
                            tmem_wait_ld();
#pragma unroll
                            for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(sum[j]);
                        }
                        if (!last) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                sum[j] = __float_as_uint(acc[c0 + j]);
                                acc[c0 + j] = 0.f;
                            }
                            tmem_st16(sum_row + (uint32_t)c0, sum);
                        }
                    }
                    tmem_wait_st();
                }
            }
            if (__any_sync(0xffffffffu, abort_flag)) break;
            const int f = feature_of<DUAL>(f0, q * 32 + lane);
            const int columns = min(half, M - t0);                    // <= 0: rows of X that do not exist
            bool finite = true;
#pragma unroll
            for (int c = 0; c < HALF_MAX; ++c) {
                acc[c] *= DOWN;
                if (c < columns) finite &= fabsf(acc[c]) <= LARGEST;
            }
            if (__any_sync(0xffffffffu, !finite && f < N)) {
                float* buf = again[warp];
#pragma unroll 1
                for (int c0 = 0; c0 < HALF_MAX; c0 += 4) {           // the registers go round, four columns at the front at a time
#pragma unroll
                    for (int j = 0; j < 4; ++j) buf[j * 32 + lane] = acc[j];
                    __syncwarp();
                    if (c0 < columns)
                        sum_again(buf, 32, X, t0 + c0, min(4, columns - c0), f < N, K, kb0 * BK, min(K, (kb0 + n_kb) * BK),
                                  [&](int r) { return weight_row<DUAL>(W, W2, f0, q * 32 + r, K); });
#pragma unroll
                    for (int c = 0; c < HALF_MAX - 4; ++c) acc[c] = acc[c + 4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[HALF_MAX - 4 + j] = buf[j * 32 + lane];
                    __syncwarp();
                }
            }
            if (splits > 1) {                                         // one tile; the last MMAs have finished: nothing reads the stages
#pragma unroll
                for (int c = 0; c < HALF_MAX; ++c)
                    if (c < half) pieces[(part * half + c) * ROWS + q * 32 + lane] = acc[c];
            } else if (DUAL) {
                // the halves of a warp hold gate and up sums of the same features: each finishes every other row of X
#pragma unroll
                for (int c = 0; c < HALF_MAX; c += 2) {
                    if (c >= columns) break;
                    const bool upper = (lane & 16) != 0;
                    const float other = __shfl_xor_sync(0xffffffffu, upper ? acc[c] : acc[c + 1], 16);
                    const int t = t0 + c + (upper ? 1 : 0);
                    if (f < N && t < M) finish<MODE>(out, (size_t)t * N + f, f, upper ? other : acc[c], upper ? acc[c + 1] : other, bias, forms);
                }
            } else if (f < N) {
#pragma unroll
                for (int c0 = 0; c0 < HALF_MAX; c0 += 8) {
                    if (c0 >= columns) break;
                    float* to = out + (size_t)(t0 + c0) * N + f;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c0 + j < columns) put_out<MODE>(to, (size_t)j * N, f, acc[c0 + j], 0.f, bias, forms);
                }
            }
        }
    }
    __syncwarp();
    wait_for_previous_kernels();          // every thread may read and write `out` below
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (splits == 1) return;
    cluster_wait();                              // the peers have started
    if (abort_flag && threadIdx.x == 0) set_in_all(&any_failed, splits);
    cluster_sync();
    const bool failed = any_failed != 0;         // one block without its piece: none writes a sum that lacks it
    const Forms forms = load_forms<MODE>(bias);
    const int t0 = first % tok_tiles * tn, f0 = first / tok_tiles * FEATS;
    // four features at a time, so that a thread's reads of all pieces are on their way together
    const int items = tn * FEATS / 4 / splits, from = items * rank;                    // tn * FEATS is a multiple of 1,024
    for (int i = from + (int)threadIdx.x; i < from + items && !failed; i += THREADS) {
        const int c = i / (FEATS / 4), fl = (i - c * (FEATS / 4)) * 4, f = f0 + fl;
        if (t0 + c >= M || f >= N) continue;
        const int at = c * ROWS + (DUAL ? (fl >> 4) * 32 + (fl & 15) : fl);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f), up = v;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            if (p >= splits) break;
            const float4 x = peer_float4(pieces + at, (uint32_t)p);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
            if (DUAL) {
                const float4 y = peer_float4(pieces + at + 16, (uint32_t)p);
                up.x += y.x; up.y += y.y; up.z += y.z; up.w += y.w;
            }
        }
        const float vs[4] = {v.x, v.y, v.z, v.w}, ups[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (f + j < N) put_out<MODE>(out, (size_t)(t0 + c) * N + f + j, f + j, vs[j], ups[j], bias, forms);
    }
    cluster_sync();                              // a peer may still be reading this block's pieces
}

constexpr int smem_bytes(int tn) { return 1024 + STAGES * (W_STAGE + 3 * tn * BK * 2); }

// How a product is cut: rows of X per tile and blocks along K, by the run of the fullest SM.  Nanoseconds: a block of K takes 800 + 5.3 tn,
// but no less than 1,220; a tile's epilogue 2,000 (gated 4,500); one whose pieces meet in a cluster 6,000.  Over 14 shapes of 33 to 512
// rows the plan is within 3% of the best of all widths and cuts.
struct Plan { int tn, splits; long long cost; };
int blocks_at_once(int splits) {
    static PerDeviceOnce once;
    if (raise_dynamic_smem(gemm_f32_wide_kernel<1>, smem_bytes(MAX_TN), once, "gemm_f32") != 0) return 128;
    return blocks_alone((const void*)gemm_f32_wide_kernel<1>, THREADS, smem_bytes(MAX_TN), splits);
}
Plan plan(int M, int N, int K, bool dual) {
    const int feats = dual ? ROWS / 2 : ROWS, total_kb = (K + BK - 1) / BK;
    const long long feat_tiles = (N + feats - 1) / feats;
    Plan best{0, 1, 0};
    const int columns = (M + MAX_TN - 1) / MAX_TN;
    for (int c = columns; c <= columns + 3; ++c) {
        const int tn = ((M + c - 1) / c + 15) / 16 * 16;
        const long long block = tn < 80 ? 1220 : 800 + 53 * tn / 10, tiles = feat_tiles * ((M + tn - 1) / tn);
        for (int s = 1; s <= 8 && s <= total_kb; s *= 2) {
            const long long at_once = blocks_at_once(s);
            const long long rounds = (tiles * s + at_once - 1) / at_once;
            const long long cost = rounds * ((total_kb + s - 1) / s * block + (s > 1 ? 6000 : dual ? 4500 : 2000));
            if (best.tn == 0 || cost < best.cost) best = Plan{tn, s, cost};
        }
    }
    return best;
}

int encode_parts(CUtensorMap* map, const void* parts, int M, int ld, int tn) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail("gemm_f32: cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[3] = {(cuuint64_t)ld, (cuuint64_t)M, 3};
    cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)M * ld * 2};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)tn, 1};
    cuuint32_t elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(parts), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail("gemm_f32: cuTensorMapEncodeTiled failed (code %d)", (int)r);
    return 0;
}

template <int MODE>
int launch(const Plan& p, const CUtensorMap& map, const float* X, const float* W, const float* W2, const float* bias, float* out, int M,
           int N, int K, int* status, cudaStream_t stream) {
    constexpr int FEATS = MODE == 3 ? ROWS / 2 : ROWS;
    static PerDeviceOnce once;
    if (int rc = raise_dynamic_smem(gemm_f32_wide_kernel<MODE>, smem_bytes(MAX_TN), once, "gemm_f32")) return rc;
    const int tok_tiles = (M + p.tn - 1) / p.tn;
    const long long tiles = (long long)tok_tiles * ((N + FEATS - 1) / FEATS);
    if (tiles * p.splits > 0x7fffffffLL) return fail("gemm_f32: %lld tiles", tiles);
    const unsigned blocks = p.splits > 1 ? (unsigned)(tiles * p.splits) : (unsigned)(tiles < sm_count() ? tiles : sm_count());
    return launch_cluster("gemm_f32 (wide)", gemm_f32_wide_kernel<MODE>, dim3(blocks), THREADS, (size_t)smem_bytes(p.tn), p.splits, stream, map,
                          X, W, W2, bias, out, M, N, K, p.tn, tok_tiles, (int)tiles, p.splits, status);
}

}  // namespace

// Columns of the three bfloat16 matrices that a product of K takes as scratch, [3][M][that many].
RI_API int ri_gemm_f32_wide_ld(int K) { return (K + 7) / 8 * 8; }

// `mode`: the epilogue, as in `ri_gemm_f32`; parts: bfloat16 [3][part_rows][ri_gemm_f32_wide_ld(K)], 16-byte aligned, overwritten: so many
// rows of X are cut and multiplied at a time, in stretches of about equal length.
// tn, splits (0: the plan's): rows of X per tile, a multiple of 16 up to 128, and blocks along K, 1, 2, 4 or 8; for tests.
RI_API int ri_gemm_f32_wide(const float* X, const float* W, const float* W2, const float* bias, float* out, void* parts, int part_rows,
                            int mode, int M, int N, int K, int tn, int splits, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4) return fail("gemm_f32: K must be a positive multiple of 4, found %d", K);
    if (((uintptr_t)X | (uintptr_t)W | (uintptr_t)W2 | (uintptr_t)parts) % 16) return fail("gemm_f32: operands must be 16-byte aligned");
    if (mode == 3 && W2 == nullptr) return fail("gemm_f32: the gated epilogue needs a second matrix");
    if (mode == 2 && bias != nullptr) return fail("gemm_f32: the residual epilogue takes no bias");
    if ((mode == 4 || mode == 5) && bias == nullptr) return fail("gemm_f32: epilogue %d needs its constants", mode);
    if (mode < 0 || mode > 5) return fail("gemm_f32: unknown epilogue mode %d", mode);
    if (part_rows <= 0) return fail("gemm_f32: parts of %d rows", part_rows);
    const int ld = ri_gemm_f32_wide_ld(K), total_kb = (K + BK - 1) / BK;
    const int stretches = M / part_rows + (M % part_rows != 0), most = M / stretches + (M % stretches != 0);
    for (int m0 = 0; m0 < M; m0 += most) {
        const int rows = M - m0 < most ? M - m0 : most;
        const float* x = X + (size_t)m0 * K;
        float* to = out + (size_t)m0 * N;
        Plan p = plan(rows, N, K, mode == 3);
        if (tn > 0) p.tn = tn;
        if (splits > 0) p.splits = splits;
        if (p.tn % 16 || p.tn > MAX_TN || p.splits > total_kb || (p.splits != 1 && p.splits != 2 && p.splits != 4 && p.splits != 8))
            return fail("gemm_f32: no tiles of %d rows cut into %d", p.tn, p.splits);
        CUtensorMap map;
        if (int rc = encode_parts(&map, parts, rows, ld, p.tn)) return rc;
        // (waits for the products of the stretch before, which read the parts)
        const long long items = (long long)rows * (ld / 4);
        const cudaError_t e = launch_dependent(cut_rows_kernel, dim3((unsigned)(items + 255 < 256LL * 4096 ? (items + 255) / 256 : 4096)), 256,
                                               0, stream, x, (__nv_bfloat16*)parts, rows, K, ld);
        if (int rc = check_launch(e, "gemm_f32 (cut)")) return rc;
        int rc = 0;
        switch (mode) {
            case 0:
            case 1: rc = launch<1>(p, map, x, W, W2, bias, to, rows, N, K, status, stream); break;
            case 2: rc = launch<2>(p, map, x, W, W2, bias, to, rows, N, K, status, stream); break;
            case 3: rc = launch<3>(p, map, x, W, W2, bias, to, rows, N, K, status, stream); break;
            case 4: rc = launch<4>(p, map, x, W, W2, bias, to, rows, N, K, status, stream); break;
            default: rc = launch<5>(p, map, x, W, W2, bias, to, rows, N, K, status, stream);
        }
        if (rc) return rc;
    }
    return 0;
}

RI_DEFINE_LAST_ERROR()
