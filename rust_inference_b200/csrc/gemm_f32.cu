// out[M, N] = X[M, K] * W[N, K]^T for float32 operands with float32 results, in two kernels that between them take
// M up to 64 (K a multiple of 4 and 16-byte aligned operands: rows are read 16 bytes at a time; `gemm_simt.cu` has the rest).
//
// Few rows of X (a decode step, up to FEW_MAX): the product is a read of W.  A warp owns a few rows of W, its lanes run
// along K with 16-byte asynchronous copies into a ring of their own (or loads), several steps ahead, and every weight meets all rows of X,
// which lie in shared memory too; FFMA, float32 sums.  K is cut over the thread blocks of a cluster when N alone has too few
// rows to keep the memory busy; the pieces meet through distributed shared memory in a fixed order, so a product's bits do
// not change from run to run.
//
// More rows (up to 64; beyond, `gemm_f32_wide.cu`): the tensor cores, without giving up 32 bits.  A float32 number is the exact sum of three bfloat16 numbers
// (its leading 8 significant bits, the next 8 and the last 8), so x * w is the sum of nine products of bfloat16 numbers,
// each exact in the tensor core.  The last one (low * low) is below 2^-30 of the whole and is left out; the other eight are added.
// Eight warps read both operands, cut them and put the parts into shared memory as the MMA wants them (128-byte swizzle); eight
// MMAs per 16 steps of K add up 64 steps of K in tensor memory, the seven small products in a sum of their own: the tensor
// core's additions truncate, which would cost the large product's sum its last bits with every small one.  Then eight warps
// add both sums onto float32 registers and the next 64 steps start from zero, so that truncated sums never run over more.
// Off from 64 bits (root mean square over that of the results; in brackets one running FFMA sum, `gemm_simt.cu`), rows of
// N(0, 1) times rows of N(0, 1/K): 0.75e-7 at K = 128 (2.0e-7), 0.94e-7 at 896 (5.4e-7), 1.1e-7 at 4,864 (12e-7), 1.4e-7 at 18,944
// (25e-7); all-positive rows 0.81e-7 at 896 (4.2e-7), where sums are too small by 0.67e-7 on average; rows with one entry 0.25e-7
// (0.25e-7), with 2 of 896 0.36e-7 (0.31e-7: every block's sum is rounded for itself), with 4 0.46e-7 (0.41e-7), with 16 0.62e-7
// (0.76e-7).  The kernel for few rows: 0.7e-7 to 1.8e-7 dense, 0.25e-7, 0.38e-7, 0.49e-7 and 0.64e-7 for those few entries.
// A number that is infinite or NaN has no such parts (they turn every sum that they meet infinite or NaN): sums that came out
// so are computed again with FFMA, as a plain float32 sum; finite ones beside them keep their bits.
//
// Epilogues as in `gemm_simt.cu` (0 and 1 are the same here: float32 with a bias): 2 out += acc, 3 gated, 4 an activation,
// 5 silu for the first columns.
#include "cluster.cuh"
#include "gemm_f32_common.cuh"
#include "tcgen05_common.cuh"

using namespace ri;
using namespace ri::f32;
using namespace ri::tc;

namespace {

// ---------------------------------------------------------------------------------------------------------------------
// Few rows of X.
//
// Bound by the read of W.  Every lane copies its 16 bytes of a row and step into a ring in shared memory and reads only what it
// copied itself, so no warp waits for another: 3 or 7 steps of 512 bytes a row are on their way per warp (up to four rows of X; 2 or 3
// beyond; 24 to 56 KiB per block), across groups of rows and before the wait for the kernel before.  Loads into registers (4 or 2 steps of
// them; RING false) do the same on paper and took a step of a 0.5B-sized decoder from 797 to 887 us, depending on an unused branch; they
// are left where X leaves a ring too little room (`few_plan`).  X comes by such copies too.  Where K is cut over a cluster the pieces go straight to
// the block that finishes an output, which reads them behind one meeting point.  A decode step of a 1.5B-sized decoder and 4 sequences:
// 1,988 -> about 1,885 us, 0.5B-sized 933 -> 790 (1 sequence), 1,406 -> 1,270 (8).  Asking for the following weights to come into the L2
// before the wait as well cost 1%.  A weight costs one FFMA per row of X and a 16-byte read of X from shared memory per RW of them:
// with RW = 2 up to four rows and 4 beyond, both stay below what the memory delivers (23 bytes per clock and SM).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int FEW_MAX = 16;
constexpr int FEW_THREADS = 256, FEW_WARPS = FEW_THREADS / 32;
constexpr int STEP = 128;                      // floats of K that a warp reads per step and row: 16 bytes per lane

// 16 bytes into shared memory; not `in`: zeros, and nothing is read
__device__ __forceinline__ void copy16_or_zeros(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__host__ __device__ constexpr int few_ring_floats(int rw, int u) { return FEW_WARPS * u * rw * STEP; }

// a[0 .. n) of every lane, summed over the lanes: afterwards lane l holds in a[0 .. n/32) (n < 32: in a[0]) the sums number
// `lane_first` .. ; every exchange halves what a lane still carries
template <int N>
__device__ __forceinline__ int reduce_lanes(float (&a)[N], int lane) {
    int first = 0, n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            const int half = n / 2;
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i >= half) break;
                const float give = upper ? a[i] : a[i + half], keep = upper ? a[i + half] : a[i];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
            if (upper) first += half;
            n = half;
        } else {
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
        }
    }
    return first;
}

template <int MT, int RW, int U, int MODE, bool RING>
__global__ void __launch_bounds__(FEW_THREADS, MT > 8 ? 2 : 3)
gemm_f32_few_kernel(const float* X, const float* __restrict__ W, const float* __restrict__ W2,
                    const float* __restrict__ bias, float* out, int M, int N, int K, int steps, int splits) {
    constexpr bool DUAL = MODE == 3;
    constexpr int FEATS = DUAL ? RW / 2 : RW;                // features per warp (gated: a gate row and an up row each)
    constexpr int GROUP = FEW_WARPS * FEATS;                 // features per block
    constexpr int SUMS = FEW_WARPS * RW * MT;
    extern __shared__ __align__(16) float smem[];
    __shared__ float sums[2][SUMS + 16];                     // whole products; K cut: the pieces of this block's outputs, block by block

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* ring = smem + warp * (U * RW * STEP) + lane * 4;  // [U][RW][STEP] per warp; a lane reads only what it copied itself
    float* xs = smem + (RING ? few_ring_floats(RW, U) : 0);  // [MT][this block's stretch of K]
    const int rank = splits > 1 ? (int)cluster_rank() : 0;
    const int first_step = (int)((long long)steps * rank / splits);
    const int ns = (int)((long long)steps * (rank + 1) / splits) - first_step;      // >= 1: splits <= steps
    const int k0 = first_step * STEP, width = ns * STEP;
    const int groups = (N + GROUP - 1) / GROUP, stride = (int)gridDim.x / splits;

    // the next step's weights on their way into a slot of the ring: steps of this group of rows, then of the block's next group
    int group = (int)blockIdx.x / splits, copy_group = group, copy_step = 0;
    auto copy_next = [&](int slot) {
        if (copy_group < groups) {
            const int k = k0 + copy_step * STEP + lane * 4;
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int f = copy_group * GROUP + warp * FEATS, row = min(DUAL ? f + r / 2 : f + r, N - 1);
                const float* base = (DUAL && (r & 1)) ? W2 : W;
                copy16_or_zeros(ring + (slot * RW + r) * STEP, base + (k < K ? (size_t)row * K + k : 0), k < K);
            }
            if (++copy_step == ns) {
                copy_step = 0;
                copy_group += stride;
            }
        }
        copies_commit();
    };
    // without the ring: U steps in registers
    float4 held[RING ? 1 : U][RW];
    auto load = [&](float4 (&w)[RW], int group, int step) {
        const int k = k0 + step * STEP + lane * 4, f = group * GROUP + warp * FEATS;
        const bool in = step < ns && k < K && group < groups;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int row = min(DUAL ? f + r / 2 : f + r, N - 1);
            const float* base = (DUAL && (r & 1)) ? W2 : W;
            w[r] = in ? load_weight(base + (size_t)row * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };

    let_next_kernel_start();
    if (splits > 1) cluster_arrive();
#pragma unroll
    for (int u = 0; u < (RING ? U - 1 : U); ++u) {           // weights: written by no kernel
        if constexpr (RING) copy_next(u); else load(held[u], group, u);
    }
    wait_for_previous_kernels();
    // X: asynchronous copies too, all on their way at once (rows and columns beyond X become zeros)
    for (int m = 0, k = threadIdx.x * 4;; k += FEW_THREADS * 4) {
        while (k >= width && m < MT) {
            k -= width;
            ++m;
        }
        if (m == MT) break;
        const bool in = m < M && k0 + k < K;                 // width is a multiple of 4: the four belong to one row
        copy16_or_zeros(xs + m * width + k, in ? X + (size_t)m * K + k0 + k : X, in);
    }
    copies_commit();
    copies_wait<0>();
    const Forms forms = load_forms<MODE>(bias);
    // outputs (feature of the group, row of X), the feature fastest; the cluster's blocks share them out
    constexpr int TOTAL = GROUP * MT;
    const int each = (TOTAL + splits - 1) / splits, from = min(TOTAL, each * rank), to = min(TOTAL, from + each);
    __syncthreads();
    if (splits > 1) cluster_wait();              // every block of the cluster is there: its shared memory may be written

    int slot = 0, used = U - 1;                  // this step's slot, and the one of the step before it: free
    for (int turn = 0; group < groups; group += stride, turn ^= 1) {
        float old = 0.f;                         // what this thread's output is added to
        if (MODE == 2 && RING) {
            const int i = from + threadIdx.x, m = i / GROUP, f = group * GROUP + i - m * GROUP;
            if (i < to && m < M && f < N) old = out[(size_t)m * N + f];
        }
        float acc[RW * MT];
#pragma unroll
        for (int i = 0; i < RW * MT; ++i) acc[i] = 0.f;
        const float* x0 = xs + lane * 4;
        auto multiply = [&](const float4 (&w)[RW], const float* x0) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(x0 + m * width);
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    float a = acc[r * MT + m];
                    a = fmaf(w[r].x, x.x, a);
                    a = fmaf(w[r].y, x.y, a);
                    a = fmaf(w[r].z, x.z, a);
                    a = fmaf(w[r].w, x.w, a);
                    acc[r * MT + m] = a;
                }
            }
        };
        if constexpr (RING) {
            for (int s = 0; s < ns; ++s, x0 += STEP) {
                copies_wait<U - 2>();
                float4 w[RW];
#pragma unroll
                for (int r = 0; r < RW; ++r) w[r] = *reinterpret_cast<const float4*>(ring + (slot * RW + r) * STEP);
                copy_next(used);
                used = slot;
                slot = slot == U - 1 ? 0 : slot + 1;
                multiply(w, x0);
            }
        } else {
            const int ns_up = (ns + U - 1) / U * U;
            for (int s0 = 0; s0 < ns_up; s0 += U) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (s0 + u < ns) multiply(held[u], x0 + (s0 + u) * STEP);
                    // the registers just used take the step U further on, of this group of rows or of the next
                    const int next = s0 + u + U;
                    if (next < ns_up) load(held[u], group, next);
                    else load(held[u], group + stride, next - ns_up);
                }
            }
        }
        const int at = reduce_lanes(acc, lane);
        constexpr int HELD = RW * MT >= 32 ? RW * MT / 32 : 1;
        if (RW * MT >= 32 || (lane & (32 / (RW * MT) - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < HELD; ++i) {
                if (splits == 1) {
                    sums[turn][warp * RW * MT + at + i] = acc[i];
                } else {                         // to the block that finishes this output
                    const int r = (at + i) / MT, m = (at + i) % MT;
                    const int o = m * GROUP + warp * FEATS + (DUAL ? r / 2 : r), owner = o / each;
                    store_peer_float(&sums[turn][(DUAL ? 2 : 1) * (rank * each + o - owner * each) + (DUAL ? r & 1 : 0)], (uint32_t)owner, acc[i]);
                }
            }
        }
        if (splits > 1) cluster_sync(); else __syncthreads();
        for (int i = from + threadIdx.x; i < to; i += FEW_THREADS) {
            const int m = i / GROUP, fl = i - m * GROUP, f = group * GROUP + fl;
            if (m >= M || f >= N) continue;
            float v = 0.f, up = 0.f;
            if (splits > 1) {
                for (int p = 0; p < splits; ++p) {
                    const float* piece = &sums[turn][(DUAL ? 2 : 1) * (p * each + i - from)];
                    v += piece[0];
                    if (DUAL) up += piece[1];
                }
            } else {
                const int slot = ((fl / FEATS) * RW + (fl % FEATS) * (DUAL ? 2 : 1)) * MT + m;
                v = sums[turn][slot];
                if (DUAL) up = sums[turn][slot + MT];
            }
            const size_t o = (size_t)m * N + f;
            if (MODE == 2) out[o] = (RING && i < from + FEW_THREADS ? old : out[o]) + v;
            else finish<MODE>(out, o, f, v, up, bias, forms);
        }
        // the other half of `sums` is next: whoever writes this half again has passed the barrier of the turn between
    }
}

constexpr int FEW_SMEM_MAX = 200 * 1024, SM_SMEM = 228 * 1024;

// Slots of a warp's ring, with the X of a block in `x_bytes`, and blocks per SM: the deeper ring while three blocks still fit an SM (one row
// of X: 887 -> 760 us a step as above with 8 slots).
constexpr int few_slots_least(int rw) { return rw == 2 ? 4 : 3; }
constexpr int few_slots_most(int rw) { return rw == 2 ? 8 : 4; }
int few_slots(int rw, long long x_bytes) {
    return x_bytes + 4ll * few_ring_floats(rw, few_slots_most(rw)) <= 74 * 1024 ? few_slots_most(rw) : few_slots_least(rw);
}
constexpr int few_held(int rw) { return rw == 2 ? 4 : 2; }            // steps in registers, without a ring
int few_per_sm(int rows, int rw, long long smem) {         // (its own sums and 1 KB of the system's lie in a block's shared memory too)
    return max(1, min(rows > 8 ? 2 : 3, (int)(SM_SMEM / (smem + 8 * (FEW_WARPS * rw * rows + 16) + 1024))));
}

// How a product of few rows is cut: blocks along K (0: another kernel), and whether the weights come through the ring.  A ring takes 32 or
// 48 KB of a block that X may need; where fewer blocks fit an SM for it, registers are the better place.  us, ring / registers: 8 x 14,336
// x 4,096 gated 150 / 105, 16 x 11,008 x 2,048 gated 91 / 61, 8 x 3,584 x 18,944 123 / 104, 16 x 32,000 x 2,048 127 / 82, 4 x 2,048 x
// 40,960 123 / 86; where as many fit it is the ring: 8 x 8,960 x 1,536 gated 23 / 32, 8 x 4,608 x 3,584 15 / 22.  Over 230 shapes of 1 to
// 16 rows the plan is on average within 5% of the best of both and all cuts.  (9 rows and more of which one block fills an SM without a
// ring go to the tensor cores: 16 x 4,096 x 22,016 139 us, 270 from registers.)
struct FewPlan { int splits; bool ring; };
FewPlan few_plan(int rows, int rw, int group, int N, int K) {
    const int steps = (K + STEP - 1) / STEP, groups = (N + group - 1) / group;
    FewPlan best{0, true};
    long long best_cost = 0;
    for (int ring = 1; ring >= 0; --ring)
        for (int s = 1; s <= 8 && s <= steps; s *= 2) {
            const int per = (steps + s - 1) / s;
            const long long x_bytes = (long long)rows * per * STEP * 4;
            const long long smem = x_bytes + (ring ? 4ll * few_ring_floats(rw, few_slots(rw, x_bytes)) : 0);
            const int per_sm = few_per_sm(rows, rw, smem);
            if (smem > FEW_SMEM_MAX || (!ring && rows > 8 && per_sm == 1)) continue;
            const int resident = per_sm * sm_count() / s;      // clusters
            // rounds of the persistent grid times the steps of one, and what a round costs besides (about three steps; four where the
            // pieces meet across blocks); registers for 5% less
            const long long rounds = (groups + resident - 1) / resident;
            const long long cost = rounds * (per + (s > 1 ? 4 : 3)) * (ring ? 95 : 100);
            if (best.splits == 0 || cost < best_cost) {
                best = FewPlan{s, ring != 0};
                best_cost = cost;
            }
        }
    return best;
}

template <int MT, int RW, int U, int MODE, bool RING>
int launch_few(const float* X, const float* W, const float* W2, const float* bias, float* out, int M, int N, int K, int splits,
               cudaStream_t stream) {
    constexpr int GROUP = FEW_WARPS * (MODE == 3 ? RW / 2 : RW);
    const int steps = (K + STEP - 1) / STEP, groups = (N + GROUP - 1) / GROUP;
    const long long x_bytes = (long long)MT * ((steps + splits - 1) / splits) * STEP * 4;
    if constexpr (RING && U == few_slots_least(RW))
        if (few_slots(RW, x_bytes) != U) return launch_few<MT, RW, few_slots_most(RW), MODE, true>(X, W, W2, bias, out, M, N, K, splits, stream);
    const size_t smem = (size_t)x_bytes + (RING ? 4 * few_ring_floats(RW, U) : 0);
    auto kernel = gemm_f32_few_kernel<MT, RW, U, MODE, RING>;
    static PerDeviceOnce once;
    if (int rc = raise_dynamic_smem(kernel, FEW_SMEM_MAX, once, "gemm_f32")) return rc;
    const int clusters = max(1, min(groups, few_per_sm(MT, RW, smem) * sm_count() / splits));
    return launch_cluster("gemm_f32 (few rows)", kernel, dim3(clusters * splits), FEW_THREADS, smem, splits, stream, X, W, W2, bias, out, M, N,
                          K, steps, splits);
}
template <int MT, int RW, int MODE>
int launch_few(const FewPlan& p, const float* X, const float* W, const float* W2, const float* bias, float* out, int M, int N, int K,
               cudaStream_t stream) {
    return p.ring ? launch_few<MT, RW, few_slots_least(RW), MODE, true>(X, W, W2, bias, out, M, N, K, p.splits, stream)
                  : launch_few<MT, RW, few_held(RW), MODE, false>(X, W, W2, bias, out, M, N, K, p.splits, stream);
}

// ---------------------------------------------------------------------------------------------------------------------
// Many rows of X: three bfloat16 parts per operand on the tensor cores.
//
// A tile is 128 rows of W (gated: 64 gate rows and the 64 up rows of the same features) by TN rows of X, up to 64 (beyond, the kernel of
// `gemm_f32_wide.cu` puts less work into a multiply-add: X is cut here once for every tile of rows of W).  What bounds a
// block of 64 steps of K is the cutting, eight warps with a few dependent instructions per number, and shared memory (32 MMAs that
// read 4 KiB of W and TN * 32 bytes of X each, and the parts' writes: at TN = 64 2,100 clocks against 1,024 of the tensor core).
// 64 x 4,864 x 896 gated takes 29 us, 64 x 896 x 4,864 24.  Parts rounded instead of cut off, with six products, took as long and left
// a single product off by up to 1.4 x 2^-24.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int ROWS = 128, BK = 64, PART = ROWS * BK * 2, STAGES = 2, SPLIT_MAX = 64;
constexpr int CUT_WARPS = 8, CUT_THREADS = CUT_WARPS * 32, ADD_WARPS = 8;
constexpr int SPLIT_THREADS = CUT_THREADS + ADD_WARPS * 32;
enum Status { ST_CUT_TIMEOUT = 41, ST_MMA_TIMEOUT = 42, ST_ADD_TIMEOUT = 43 };

// Infinite or NaN sums of a tile computed again over the block's piece of K: a warp takes 32 neighbouring features and four rows of X.
// (A call of its own: inside the kernel it takes registers from the loops that always run.)
template <int TN, bool DUAL>
__device__ __noinline__ void sums_again(float* pieces, const float* X, const float* W, const float* W2, int M, int N, int K, int f0, int k_begin,
                                        int k_end) {
    constexpr int FEATS = DUAL ? ROWS / 2 : ROWS;
    for (int g = threadIdx.x >> 5; g < TN / 4 * (ROWS / 32); g += SPLIT_THREADS / 32) {
        const int c0 = g / (ROWS / 32) * 4, r0 = g % (ROWS / 32) * 32;
        sum_again(pieces + c0 * ROWS + r0, ROWS, X, c0, min(4, M - c0), f0 + (r0 + (int)(threadIdx.x & 31)) % FEATS < N, K, k_begin, k_end,
                  [&](int r) { return (DUAL && r0 + r >= FEATS ? W2 : W) + (size_t)(f0 + (DUAL ? (r0 + r) % FEATS : r0 + r)) * K; });
    }
}

template <int TN, int MODE>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_f32_split_kernel(const float* X, const float* __restrict__ W, const float* __restrict__ W2,
                      const float* __restrict__ bias, float* out, int M, int N, int K, int splits, int* status) {
    constexpr bool DUAL = MODE == 3;
    constexpr int FEATS = DUAL ? ROWS / 2 : ROWS;
    constexpr int X_PART = TN * BK * 2;
    constexpr int STAGE = 3 * (PART + X_PART);
    constexpr int ACC = 2 * TN;                  // tensor memory columns of a block of K: the large products' sums, the small ones'
    constexpr int TMEM_COLS = 2 * ACC;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag, odd_flag, any_failed;

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    float* pieces = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));      // [TN][128], over the stages at the end
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = splits > 1 ? (int)cluster_rank() : 0;
    const int f0 = (int)blockIdx.x / splits * FEATS;             // one tile holds all rows of X: M <= TN
    const int total_kb = (K + BK - 1) / BK;
    const int kb0 = (int)((long long)total_kb * rank / splits);
    const int n_kb = (int)((long long)total_kb * (rank + 1) / splits) - kb0;        // >= 1: splits <= total_kb

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), CUT_WARPS);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&acc_full[i]), 1);
            mbar_init(smem_u32(&acc_empty[i]), ADD_WARPS);
        }
        abort_flag = 0;
        odd_flag = any_failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == CUT_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (splits > 1) cluster_arrive();            // flags and barriers are set up
    let_next_kernel_start();

    if (warp < CUT_WARPS) {
        // ---- read, cut, store: 16 threads per row of 64 floats ----
        const int k4 = threadIdx.x & 15, row = threadIdx.x >> 4;             // rows row, row + 16, ...
        const uint32_t col = (uint32_t)(row * 128 + ((k4 * 8) ^ ((row & 7) << 4)));
        constexpr int WN = ROWS / 16, XN = TN / 16;
        // a thread's rows are 16 apart: one address per matrix, and a bit for every row that exists
        const size_t stride = (size_t)16 * K;
        const float* xp = X + (size_t)row * K;
        const float* wp = W + (size_t)(f0 + row) * K;
        const float* wp2 = DUAL ? W2 + (size_t)(f0 + row) * K : nullptr;
        uint32_t w_has = 0, x_has = 0;
#pragma unroll
        for (int i = 0; i < WN; ++i) w_has |= (f0 + (row + 16 * i) % FEATS < N ? 1u : 0u) << i;
#pragma unroll
        for (int i = 0; i < XN; ++i) x_has |= (row + 16 * i < M ? 1u : 0u) << i;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        int k = kb0 * BK + k4 * 4;
        auto load_w = [&](int i, bool in) {
            const float* p = DUAL && i >= WN / 2 ? wp2 + (size_t)(i - WN / 2) * stride : wp + (size_t)i * stride;
            return in && ((w_has >> i) & 1) ? load_weight(p + k) : zero;
        };
        auto load_x = [&](int i, bool in) {
            return in && ((x_has >> i) & 1) ? load_written(xp + (size_t)i * stride + k) : zero;
        };
        float4 wv[WN], xv[XN];
#pragma unroll
        for (int i = 0; i < WN; ++i) wv[i] = load_w(i, k < K);
        wait_for_previous_kernels();
#pragma unroll
        for (int i = 0; i < XN; ++i) xv[i] = load_x(i, k < K);
        for (int b = 0; b < n_kb; ++b) {
            const int s = b % STAGES;
            if (!mbar_wait(smem_u32(&empty_bar[s]), (uint32_t)((b / STAGES) & 1) ^ 1u)) {
                if (!abort_flag && lane == 0) report(status, ST_CUT_TIMEOUT);
                abort_flag = 1;
            }
            if (abort_flag) break;
            k += BK;
            const bool more = b + 1 < n_kb && k < K;             // these registers take the next 64 of K as soon as they are cut
            const uint32_t stage = base + (uint32_t)(s * STAGE) + col;
#pragma unroll
            for (int i = 0; i < WN; ++i) {
                put(stage + (uint32_t)(i * 16 * 128), PART, wv[i]);
                wv[i] = load_w(i, more);
            }
#pragma unroll
            for (int i = 0; i < XN; ++i) {
                put(stage + 3 * PART + (uint32_t)(i * 16 * 128), X_PART, xv[i]);
                xv[i] = load_x(i, more);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the MMA reads what was just stored
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
        }
    } else {
        // ---- add the sums of 64 steps onto float32 registers: a thread owns a row of W (a TMEM lane) ----
        // The first of these warps also issues the MMAs, two blocks of K ahead of the one being added (a warp of its own for
        // that would leave every thread fewer registers than the sums of 128 columns take).
        constexpr int COLS = TN / 2;                             // four warps add the first half of the columns, four the second
        const int q = warp & 3, part = (warp - CUT_WARPS) >> 2;  // q: the TMEM lanes this warp may read
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * COLS);
        const uint64_t a_desc = make_smem_desc(base), b_desc = make_smem_desc(base + 3 * PART);
        int issued = 0;
        const uint32_t leader = elect_one();
        auto issue = [&](int b) {                                // the whole warp goes through, one lane issues
            const int s = b % STAGES, buf = b & 1;
            if (!(mbar_wait_warp(smem_u32(&acc_empty[buf]), (uint32_t)((b >> 1) & 1) ^ 1u) &&
                  mbar_wait_warp(smem_u32(&full_bar[s]), (uint32_t)((b / STAGES) & 1)))) {
                if (lane == 0) report(status, ST_MMA_TIMEOUT);
                abort_flag = 1;
                return;
            }
            tc_fence_after();
            const uint64_t off = (uint64_t)((uint32_t)(s * STAGE) >> 4);
            const uint32_t acc = tmem + (uint32_t)(buf * ACC);
            // (part of W, part of X), the smallest products first; the last is the large one
            constexpr int PRODUCTS = 8, PA[PRODUCTS] = {1, 2, 2, 0, 1, 1, 0, 0}, PB[PRODUCTS] = {2, 1, 0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int p = 0; p < PRODUCTS; ++p) {
                const bool large = p == PRODUCTS - 1;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_by(leader, large ? acc : acc + TN, a_desc + off + (uint64_t)(PA[p] * (PART >> 4) + 2 * k),
                            b_desc + off + (uint64_t)(PB[p] * (X_PART >> 4) + 2 * k), IDESC, (p > 0 && !large) || k > 0);
            }
            umma_commit_by(leader, smem_u32(&empty_bar[s]));
            umma_commit_by(leader, smem_u32(&acc_full[buf]));
            issued = b + 1;
        };
        if (warp == CUT_WARPS)
            for (int b = 0; b < 2 && b < n_kb && !__any_sync(0xffffffffu, abort_flag); ++b) issue(b);
        __syncwarp();
        float acc[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
        for (int b = 0; b < n_kb; ++b) {
            const int buf = b & 1;
            const bool landed = !abort_flag && mbar_wait(smem_u32(&acc_full[buf]), (uint32_t)((b >> 1) & 1));
            if (!landed && lane == 0) {
                if (!abort_flag) report(status, ST_ADD_TIMEOUT);
                abort_flag = 1;
            }
            if (__any_sync(0xffffffffu, abort_flag)) {
                // the MMAs on their way have to finish before tensor memory is given back
                if (warp == CUT_WARPS && lane == 0)
                    for (int i = max(0, issued - 2); i < issued; ++i) mbar_wait(smem_u32(&acc_full[i & 1]), (uint32_t)((i >> 1) & 1));
                break;
            }
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16) {
                uint32_t large[16], small[16];
                tmem_ld16(trow + (uint32_t)(buf * ACC + c0), large);
                tmem_ld16(trow + (uint32_t)(buf * ACC + TN + c0), small);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(large[j]) + __uint_as_float(small[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
            if (warp == CUT_WARPS && b + 2 < n_kb) issue(b + 2);
            __syncwarp();
        }
        // the last MMAs have finished: nothing reads the stages any more
        if (!abort_flag) {
            bool finite = true;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                pieces[(part * COLS + c) * ROWS + q * 32 + lane] = acc[c] * DOWN;
                finite &= fabsf(acc[c]) <= LARGEST;
            }
            if (!finite) odd_flag = 1;
        }
    }
    __syncwarp();
    wait_for_previous_kernels();          // every thread may read and write `out` below
    tc_fence_before();
    __syncthreads();
    if (warp == CUT_WARPS) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
    }
    bool failed = abort_flag != 0;
    if (odd_flag && !failed) {
        sums_again<TN, DUAL>(pieces, X, W, W2, M, N, K, f0, kb0 * BK, min(K, (kb0 + n_kb) * BK));
        __syncthreads();
    }
    if (splits > 1) {
        cluster_wait();                          // the peers have started
        if (failed && threadIdx.x == 0) set_in_all(&any_failed, splits);
        cluster_sync();
        failed = any_failed != 0;                // one block without its piece: none writes a sum that lacks it
    }
    const Forms forms = load_forms<MODE>(bias);
    const int from = TN * FEATS / splits * rank, to = from + TN * FEATS / splits;      // TN * FEATS is a multiple of 8
    for (int i = from + (int)threadIdx.x; i < to && !failed; i += SPLIT_THREADS) {
        const int c = i / FEATS, fl = i - c * FEATS, f = f0 + fl;
        if (c >= M || f >= N) continue;
        const int at = c * ROWS + fl;
        float v = 0.f, up = 0.f;
        if (splits > 1) {
            for (int p = 0; p < splits; ++p) {
                v += peer_float(pieces + at, (uint32_t)p);
                if (DUAL) up += peer_float(pieces + at + FEATS, (uint32_t)p);
            }
        } else {
            v = pieces[at];
            if (DUAL) up = pieces[at + FEATS];
        }
        finish<MODE>(out, (size_t)c * N + f, f, v, up, bias, forms);
    }
    if (splits > 1) cluster_sync();          // a peer may still be reading this block's pieces
}

template <int TN, int MODE>
int launch_split(const float* X, const float* W, const float* W2, const float* bias, float* out, int M, int N, int K, int* status,
                 cudaStream_t stream) {
    constexpr int FEATS = MODE == 3 ? ROWS / 2 : ROWS;
    constexpr int SMEM = STAGES * 3 * (PART + TN * BK * 2) + 1024;
    static PerDeviceOnce once;
    if (int rc = raise_dynamic_smem(gemm_f32_split_kernel<TN, MODE>, SMEM, once, "gemm_f32")) return rc;
    const long long tiles = (N + FEATS - 1) / FEATS;
    const int total_kb = (K + BK - 1) / BK;
    // K over the blocks of a cluster while that shortens the run of the fullest SM: rounds of the grid (one block per SM;
    // clusters of eight leave some SMs out) times blocks of K, plus what a tile costs besides (about three blocks of K, one
    // more where pieces meet)
    int splits = 1;
    long long best = 0;
    for (int s = 1; s <= 8 && s <= total_kb; s *= 2) {
        const long long at_once = s == 8 ? 128 : s == 4 ? 144 : sm_count();
        const long long cost = ((tiles * s + at_once - 1) / at_once) * ((total_kb + s - 1) / s + 3 + (s > 1));
        if (s == 1 || cost < best) { splits = s; best = cost; }
    }
    if (tiles * splits > 0x7fffffffLL) return fail("gemm_f32: %lld tiles", tiles);
    return launch_cluster("gemm_f32", gemm_f32_split_kernel<TN, MODE>, dim3((unsigned)(tiles * splits)), SPLIT_THREADS, SMEM, splits, stream, X, W,
                          W2, bias, out, M, N, K, splits, status);
}

template <int MODE>
int dispatch(const float* X, const float* W, const float* W2, const float* bias, float* out, int M, int N, int K, int* status,
             int few_max, cudaStream_t stream) {
    // Up to 16 rows the read of W past them is the faster one everywhere it was tried (us, few rows against tensor cores):
    // 16 x 8,960 x 1,536 gated 37.7 / 42.3, 16 x 1,536 x 8,960 33.0 / 34.6, 16 x 151,936 x 896 153 / 234, 4 x 8,960 x 1,536 gated
    // 22.5 / 41.7 (16.9 at the memory's rate; the FFMA kernel of square tiles: 160).
    if (M <= few_max) {
        const int rows = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
        const int rw = rows <= 4 ? 2 : 4;
        const FewPlan p = few_plan(rows, rw, FEW_WARPS * (MODE == 3 ? rw / 2 : rw), N, K);
        if (p.splits > 0) {
            if (rows == 1) return launch_few<1, 2, MODE>(p, X, W, W2, bias, out, M, N, K, stream);
            if (rows == 2) return launch_few<2, 2, MODE>(p, X, W, W2, bias, out, M, N, K, stream);
            if (rows == 4) return launch_few<4, 2, MODE>(p, X, W, W2, bias, out, M, N, K, stream);
            if (rows == 8) return launch_few<8, 4, MODE>(p, X, W, W2, bias, out, M, N, K, stream);
            return launch_few<16, 4, MODE>(p, X, W, W2, bias, out, M, N, K, stream);
        }
    }
    if (M <= 32) return launch_split<32, MODE>(X, W, W2, bias, out, M, N, K, status, stream);
    return launch_split<64, MODE>(X, W, W2, bias, out, M, N, K, status, stream);
}

}  // namespace

// `mode`: the epilogue; `few_max`: up to how many rows the kernel for few rows is taken (0: never; at most 16; negative:
// the default).
RI_API int ri_gemm_f32(const float* X, const float* W, const float* W2, const float* bias, float* out, int mode, int M, int N, int K,
                       int few_max, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4) return fail("gemm_f32: K must be a positive multiple of 4, found %d", K);
    if (((uintptr_t)X | (uintptr_t)W | (uintptr_t)W2) % 16) return fail("gemm_f32: operands must be 16-byte aligned");
    if (mode == 3 && W2 == nullptr) return fail("gemm_f32: the gated epilogue needs a second matrix");
    if (mode == 2 && bias != nullptr) return fail("gemm_f32: the residual epilogue takes no bias");
    if ((mode == 4 || mode == 5) && bias == nullptr) return fail("gemm_f32: epilogue %d needs its constants", mode);
    if (M > SPLIT_MAX) return fail("gemm_f32: %d rows exceed %d", M, SPLIT_MAX);
    if (few_max < 0 || few_max > FEW_MAX) few_max = FEW_MAX;
    switch (mode) {
        case 0:
        case 1: return dispatch<1>(X, W, W2, bias, out, M, N, K, status, few_max, stream);
        case 2: return dispatch<2>(X, W, W2, bias, out, M, N, K, status, few_max, stream);
        case 3: return dispatch<3>(X, W, W2, bias, out, M, N, K, status, few_max, stream);
        case 4: return dispatch<4>(X, W, W2, bias, out, M, N, K, status, few_max, stream);
        case 5: return dispatch<5>(X, W, W2, bias, out, M, N, K, status, few_max, stream);
    }
    return fail("gemm_f32: unknown epilogue mode %d", mode);
}

RI_DEFINE_LAST_ERROR()
