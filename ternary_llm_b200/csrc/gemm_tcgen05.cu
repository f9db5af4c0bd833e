// Prompt GEMM  C[M,N] = A[M,K] . W^T  on the 5th-generation tensor cores (sm_100a).
//
// W is ternary with one FP16 scale per 128 weights along K.  The product scale * t is exactly
// representable in FP16, so the weight operand is expanded to FP16 {-s, 0, +s} and a plain
// FP16 x FP16 -> FP32 contraction over the whole K gives the reference result with nothing but
// FP32 accumulation rounding.
//
// Bound: the tensor pipe for long prompts (4 clocks a token of a tile and scale group); the chain of
// expansion, MMA and hand-overs, about 600 clocks a scale group, for tiles of few tokens.  A tile is
// 128 features x TM tokens, TM any multiple of 16 up to 256: the launch picks the TM (and a split of K)
// with which the tiles come out even over the SMs.  One persistent CTA per SM, whose warps run ahead
// of one another over the tiles' scale groups:
//   * one warp loads the activations by TMA, a scale group (two boxes of 64 columns, 128-byte swizzled rows) a
//     stage, three to eight stages; another one the packed codes, one box of 8 row blocks x 544 bytes per scale
//     group, six ahead.  (Read by the expanders from global memory one group ahead, a group took a
//     microsecond whatever the tile, the latency of a load from HBM.)
//   * twelve warps expand: one thread per feature row = one lane of tensor memory, three warps per
//     lane quarter on every third group (28672 x 4096, 37 tokens: two sets 30.4 us, three 26.5, four 26.1).
//     The codes c = t + 1 of two weights are the selector of one PRMT into the byte table {-s, 0, +s}, which
//     yields the FP16 pair; tcgen05.st writes it.  The expanded weights are the MMA's A operand in TENSOR
//     MEMORY and never touch shared memory.
//   * one warp issues tcgen05.mma (kind::f16, M=128, N=TM, K=16) into one of two accumulators (one beyond 192 tokens).  A stage is one
//     wait (activations and weights arrive on one barrier), eight MMAs and one commit, and the warp's loop is
//     uniform with an elected lane for the MMAs: as the loop of one thread, with a barrier and a commit for
//     either operand, the issue alone took 2000 clocks a stage;
//   * four warps empty the other accumulator with tcgen05.ld and store C (a lane is an output feature, so a
//     warp stores 32 adjacent features of one token at a time).
// Tensor memory: the accumulators of TM columns (a multiple of 32 apart), then two to four weight
// stages of 64 columns.
// Too few tiles for the SMs: K is split over the CTAs of a cluster; each leaves its FP32 sums in its
// shared memory, and each adds all of them, in rank order, for its share of the tokens.
// All mbarrier waits are bounded; a wait that gives up sets the device error flag, every role waits for
// its own copies and MMAs (bounded again) and falls through to the common exit.
//
// us among a few launches (weights from HBM), with a CTA a tile of 32 to 256 tokens and without all this -> now: 4096 x 4096, 40 tokens
// 13.8 -> 9.4, 300: 26.5 -> 15.2, 1024: 29.6 -> 26.8; 4096 x 14336, 40: 30.1 -> 17.1, 300: 60 -> 33.7; 28672 x 4096, 300: 103 -> 60,
// 2048: 372 -> 335 (1436 TFLOP/s; single launches 320 to 330); 2048 x 8192, 300: 29.3 -> 16.1, 2048: 53.8 -> 46.2.
#include <climits>
#include <mutex>

#include "common.cuh"
#include "launch.cuh"
#include "packed_layout.cuh"
#include "tcgen05.cuh"

namespace tllm {

namespace gemm {

constexpr int kTileN = 128;          // features per tile (MMA M, TMEM lanes)
constexpr int kBoxK = 64;            // columns per activation box (128 bytes of FP16)
constexpr int kACols = kGroup / 2;   // tensor-memory columns of a weight stage (FP16 pairs)
constexpr int kMaxTm = 256;
constexpr int kMaxTm2 = 192;         // of two accumulators beside the weights
constexpr int kMaxB = 8;             // activation stages, upper bound
constexpr int kMaxA = 4;             // weight stages, upper bound
constexpr int kCodes = 6;            // scale groups of codes in shared memory
constexpr int kCodeBytes = kTileN / kTileRows * kTileBytes;
constexpr int kSets = 3;             // sets of four expander warps
constexpr int kOutWarp = 4 + 4 * kSets;
constexpr int kThreads = (kOutWarp + 4) * 32;        // warps 0-3: activations, MMA, codes, none; expanders; four for outputs
constexpr int kTmemCols = 512;
// All of it for every tile: a CTA that takes the whole tensor memory shares its SM with no other kernel's that needs some.
constexpr size_t kSmem = 226 * 1024;
constexpr int kMaxSplit = 8;

struct Args {
    RowsOut out[TLLM_MAX_FUSED];     // row ranges of the matrix and where they go; unused ones start past every row
    int M, N, groups;                // tokens; rows of W; K / 128
    int mt, tiles, split;            // token tiles; tiles; CTAs per tile
    uint32_t over_split;             // 2^32 / split rounded up: the upper word of a product with it is a quotient
    int tm, acc_stride, na, nb;      // tokens per tile; columns between accumulators; weight and activation stages (na <= nb)
    int accs;                        // accumulators: two, or one for tiles of more than kMaxTm2 tokens
    int* err;
};

// kind::f16 instruction descriptor: FP16 x FP16 -> FP32, both operands K-major, M = 128
__device__ __forceinline__ uint32_t make_idesc(int tm)
{
    return (1u << 4) | ((uint32_t)(tm >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
}

__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
enum Special { kClusterRank, kClusterId, kClusters };
template <Special S>
__device__ __forceinline__ uint32_t special_register()
{
    uint32_t r;
    if constexpr (S == kClusterRank) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    else if constexpr (S == kClusterId) asm("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    else asm("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}

// A place in a ring of n slots: the slot and the parity of its uses.
struct Ring {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void step(int n, int by = 1)
    {
        slot += by;
        while (slot >= n) {
            slot -= n;
            phase ^= 1;
        }
    }
};

__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Args a)
{
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the 128-byte swizzle atoms
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * kMaxB + 2 * kCodes + 5];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tm = a.tm, nb = a.nb, na = a.na;
    // the CTAs of a cluster share a tile; from registers and by a multiplication, because divisions here are in front of everything
    const int split = a.split, rank = (int)special_register<kClusterRank>(), first = (int)special_register<kClusterId>();
    const int step = (int)special_register<kClusters>();
    const int it0 = split > 1 ? (int)__umulhi(rank * a.groups, a.over_split) : 0;    // scale groups of this CTA
    const int nst = (split > 1 ? (int)__umulhi((rank + 1) * a.groups, a.over_split) : a.groups) - it0;
    const int box_bytes = tm * kBoxK * 2, stage_bytes = 2 * box_bytes;
    constexpr int rb_tile = kTileN / kTileRows;                                        // row blocks of a tile
    uint8_t* codes = smem + nb * stage_bytes;

    const uint32_t bar0 = smem_u32(bars);
    // full: a stage's activations (one arrival and their bytes) and expanded weights (four warps); done: its MMAs
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto done = [&](int s) { return bar0 + 8u * (kMaxB + s); };
    auto full_c = [&](int s) { return bar0 + 8u * (2 * kMaxB + s); };
    auto empty_c = [&](int s) { return bar0 + 8u * (2 * kMaxB + kCodes + s); };
    auto acc_full = [&](int s) { return bar0 + 8u * (2 * kMaxB + 2 * kCodes + s); };
    auto acc_empty = [&](int s) { return bar0 + 8u * (2 * kMaxB + 2 * kCodes + 2 + s); };
    const uint32_t drained = bar0 + 8u * (2 * kMaxB + 2 * kCodes + 4);

    if (tid == 0) {
        prefetch_map(&map_w);
        prefetch_map(&map_x);
        for (int s = 0; s < kMaxB; s++) {
            mbar_init(full(s), 5);
            mbar_init(done(s), 1);
        }
        for (int s = 0; s < kCodes; s++) {
            mbar_init(full_c(s), 1);
            mbar_init(empty_c(s), 4);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(acc_full(s), 1);
            mbar_init(acc_empty(s), 4);
        }
        mbar_init(drained, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // only now: a following kernel that took this SM's tensor memory first would wait for this one with it
    pdl_launch_dependents();
    const uint32_t tmem = tmem_base_slot;
    volatile int* abortp = &abort_flag;
    int never = 0;

    if (warp == 0) {
        // ---------------- activations ----------------
        const bool leader = elect_one();
        pdl_wait();
        Ring b;
        bool ok = true;
        for (int tile = first; ok && tile < a.tiles; tile += step) {
            const int m0 = (tile % a.mt) * tm;
            for (int it = 0; it < nst; it++) {
                if (!(ok = mbar_wait(done(b.slot), b.phase ^ 1, abortp))) break;
                const uint32_t dst = smem_u32(smem + b.slot * stage_bytes);
                if (leader) {
                    mbar_expect_tx(full(b.slot), stage_bytes);
                    tma_load_2d(dst, &map_x, (it0 + it) * kGroup, m0, full(b.slot));
                    tma_load_2d(dst + box_bytes, &map_x, (it0 + it) * kGroup + kBoxK, m0, full(b.slot));
                }
                b.step(nb);
            }
        }
        if (!ok) {
            // The copies in flight land before the CTA leaves; a stage's barrier cannot tell that any more (its weights
            // may never come), so a millisecond passes instead of their microseconds.
            abort_flag = 1;
            for (int i = 0; i < 1000; i++) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const bool leader = elect_one();
        pdl_wait();
        const uint32_t idesc = make_idesc(tm);
        Ring b, w, acc;
        bool ok = true;
        for (int tile = first; ok && tile < a.tiles; tile += step) {
            if (!(ok = mbar_wait(acc_empty(acc.slot), acc.phase ^ 1, abortp))) break;
            const uint32_t d = tmem + acc.slot * a.acc_stride;
            for (int it = 0; it < nst; it++) {
                if (!(ok = mbar_wait(full(b.slot), b.phase, abortp))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t d0 = make_sw128_desc(smem_u32(smem + b.slot * stage_bytes));
                const uint64_t d1 = make_sw128_desc(smem_u32(smem + b.slot * stage_bytes) + box_bytes);
                const uint32_t a_t = tmem + a.accs * a.acc_stride + w.slot * kACols, more = it > 0 ? 1u : 0u;
                if (leader) {
#pragma unroll
                    for (int k = 0; k < kGroup / 16; k++)          // 32 bytes (2 in the descriptor) inside the 128-byte swizzled row
                        mma_ts(d, a_t + k * 8, (k < 4 ? d0 : d1) + (k & 3) * 2, idesc, k ? 1u : more);
                    mma_commit(done(b.slot));
                }
                b.step(nb);
                w.step(na);
            }
            if (leader) mma_commit(acc_full(acc.slot));
            acc.step(a.accs);
        }
        if (!ok) abort_flag = 1;
        if (leader) mma_commit(drained);
        __syncwarp();
        mbar_wait(drained, 0, &never);
    } else if (warp == 2) {
        // ---------------- packed codes (constants: not behind the kernel before) ----------------
        const bool leader = elect_one();
        Ring c;
        int used = 0;
        bool ok = true;
        for (int tile = first; ok && tile < a.tiles; tile += step) {
            const int rb = tile / a.mt * rb_tile;
            for (int it = 0; it < nst; it++) {
                if (used == kCodes) pdl_wait();              // from here on a wait depends on the kernel before
                if (!(ok = mbar_wait(empty_c(c.slot), c.phase ^ 1, abortp))) break;
                const uint32_t dst = smem_u32(codes + c.slot * kCodeBytes);
                if (leader) {
                    mbar_expect_tx(full_c(c.slot), kCodeBytes);
                    tma_load_2d(dst, &map_w, (it0 + it) * (kTileBytes / 4), rb, full_c(c.slot));
                }
                c.step(kCodes);
                used = min(used + 1, kCodes);
            }
        }
        if (!ok) abort_flag = 1;
        for (; used > 0; used--) {                           // no copy outlives the CTA
            c.slot = c.slot ? c.slot - 1 : kCodes - 1;
            if (c.slot == kCodes - 1) c.phase ^= 1;
            mbar_wait(full_c(c.slot), c.phase, &never);
        }
    } else if (warp >= 4 && warp < kOutWarp) {
        // ---------------- expanders ----------------
        const int set = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
        const int rbl = row >> 4, r16 = row & 15;             // row block of the tile and row inside it
        const int gq = r16 & 7, h = r16 >> 3;
        // this row's code words of MMA lane t: the pair (column halves j2 = 0, 1) at word index
        // (gq*4 + t)*4 + 2h, one 64-bit load per t; each word holds all four 32-column steps
        const uint8_t* cp = codes + rbl * kTileBytes + gq * 64 + h * 8;
        const uint8_t* sp = codes + rbl * kTileBytes + kTileCodeBytes + tile_scale_index(r16) * 2;
        const uint32_t lane_base = tmem + ((uint32_t)(row & ~31) << 16) + a.accs * a.acc_stride;   // this warp's 32 lanes
        Ring c, w, f, past;                                  // codes; weight stage; stage; the stage that had the weight stage before
        c.step(kCodes, set);
        w.step(na, set);
        f.step(nb, set);
        past.slot = (set + kMaxA * kSets - na) % kSets;      // of the set's first scale group from na on (nb is at least 3)
        bool ok = true;
        int g = 0, turn = 0;                                 // scale groups of this CTA so far; whose the next one is
        for (int tile = first; ok && tile < a.tiles; tile += step) {
            for (int it = 0; it < nst; it++, g++) {
                const bool mine = turn == set;
                turn = turn + 1 == kSets ? 0 : turn + 1;
                if (!mine) continue;
                if (!(ok = mbar_wait(full_c(c.slot), c.phase, abortp))) break;
                uint2 cur[4];
#pragma unroll
                for (int t = 0; t < 4; t++) cur[t] = *reinterpret_cast<const uint2*>(cp + c.slot * kCodeBytes + t * 16);
                const uint32_t sbits = *reinterpret_cast<const unsigned short*>(sp + c.slot * kCodeBytes);
                // PRMT table of this row: bytes 0,1 = -s (code 0), 2,3 = 0 (code 1), 4,5 = +s (code 2)
                const uint32_t tab_lo = sbits ^ 0x8000u, tab_hi = sbits;
                if (g >= na) {
                    if (g < na + kSets) pdl_wait();          // from here on a wait depends on the kernel before
                    if (!(ok = mbar_wait(done(past.slot), past.phase, abortp))) break;
                    past.step(nb, kSets);
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_t = lane_base + w.slot * kACols;
#pragma unroll
                for (int m = 0; m < 4; m++) {                 // 32 K per step -> 16 columns; step m is code field m
                    uint32_t r[16];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
#pragma unroll
                        for (int j2 = 0; j2 < 2; j2++) {
                            // four codes (K offsets 32m + 16*j2 + 4t .. +3) in the low two bits of each byte;
                            // selector nibbles 2c, 2c+1 per weight: one PRMT makes an FP16 pair {-s,0,+s}
                            const uint32_t s = (((j2 ? cur[t].y : cur[t].x) >> (2 * m)) & 0x03030303u) * 0x22u + 0x10101010u;
                            r[8 * j2 + 2 * t] = prmt(tab_lo, tab_hi, s);
                            r[8 * j2 + 2 * t + 1] = prmt(tab_lo, tab_hi, s >> 16);
                        }
                    }
                    tmem_st16(a_t + m * 16, r);
                    if (m == 0) {
                        // the slot may be refilled now: this store's operands came from every load of it (an arrival behind
                        // loads still in flight let the next group's codes overtake them)
                        __syncwarp();
                        if (lane == 0) mbar_arrive(empty_c(c.slot));
                        c.step(kCodes, kSets);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full(f.slot));
                f.step(nb, kSets);
                w.step(na, kSets);
            }
        }
        if (!ok) abort_flag = 1;
    } else if (warp >= kOutWarp) {
        // ---------------- outputs ----------------
        pdl_wait();
        const int row = (warp & 3) * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(row & ~31) << 16);
        Ring acc;
        bool ok = true;
        for (int tile = first; tile < a.tiles; tile += step) {
            ok = mbar_wait(acc_full(acc.slot), acc.phase, abortp) && !*abortp;
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m0 = (tile % a.mt) * tm, mv = min(tm, a.M - m0);
            const int n = tile / a.mt * kTileN + row;
            half* y = a.out[0].y;
            int r0 = 0, rows = a.out[0].rows;
#pragma unroll
            for (int i = 1; i < TLLM_MAX_FUSED; i++)
                if (n >= a.out[i].row0) {
                    y = a.out[i].y;
                    r0 = a.out[i].row0;
                    rows = a.out[i].rows;
                }
            y += (size_t)m0 * rows + (n - r0);
            float* part = reinterpret_cast<float*>(smem) + row;
            const uint32_t d = lane_base + acc.slot * a.acc_stride;
            if (split > 1) {
                for (int c = 0; c < mv; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(d + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c + j < mv) part[(c + j) * kTileN] = __uint_as_float(v[j]);
                }
            } else {
                for (int c = 0; c < mv; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(d + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (n >= a.N) continue;
                    // whole chunks without a test per token, a running pointer: the stores' instructions bound short tiles
                    // (16384 x 2048, 1000 tokens: 62.5 -> 53.9 us)
                    half* yc = y + (size_t)c * rows;
                    if (c + 32 <= mv) {
#pragma unroll
                        for (int j = 0; j < 32; j++, yc += rows) *yc = __float2half_rn(__uint_as_float(v[j]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++, yc += rows)
                            if (c + j < mv) *yc = __float2half_rn(__uint_as_float(v[j]));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(acc.slot));
            acc.step(a.accs);
        }
        if (!ok) abort_flag = 1;
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (split > 1) {
        // each CTA adds the cluster's sums for its share of the tile's tokens: a warp takes a token, a lane four rows
        pdl_wait();
        cluster_sync();
        const int m0 = (first % a.mt) * tm, mv = min(tm, a.M - m0);
        const int t0 = rank * mv / split, t1 = (rank + 1) * mv / split;
        const int row = lane * 4;
        const int n = first / a.mt * kTileN + row;
        half* y = a.out[0].y;
        int r0 = 0, rows = a.out[0].rows;
#pragma unroll
        for (int i = 1; i < TLLM_MAX_FUSED; i++)
            if (n >= a.out[i].row0) {
                y = a.out[i].y;
                r0 = a.out[i].row0;
                rows = a.out[i].rows;
            }
        for (int t = t0 + warp; t < t1; t += kThreads / 32) {
            const uint32_t at = smem_u32(smem) + (uint32_t)(t * kTileN + row) * 4;
            float4 p[kMaxSplit], v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int z = 0; z < kMaxSplit; z++)
                if (z < split) {
                    uint32_t peer;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(z));
                    p[z] = ld_cluster(peer);
                }
#pragma unroll
            for (int z = 0; z < kMaxSplit; z++)
                if (z < split) {
                    v.x += p[z].x;
                    v.y += p[z].y;
                    v.z += p[z].z;
                    v.w += p[z].w;
                }
            const half o[4] = {__float2half_rn(v.x), __float2half_rn(v.y), __float2half_rn(v.z), __float2half_rn(v.w)};
            half* yp = y + (size_t)(m0 + t) * rows + (n - r0);
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (n + j < a.N && !*abortp) yp[j] = o[j];
        }
        cluster_sync();                                      // nobody leaves while its sums are still read
    }
    if (abort_flag && tid == 0) atomicExch(a.err, TLLM_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

struct Device {
    int sms = 0;
    int slots[kMaxSplit + 1] = {};       // CTAs that run at the same time in clusters of that size
};

static Device* device()
{
    static Device devices[64];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    Device& d = devices[dev];
    if (!d.sms) {
        int sms = 0;
        if (cudaFuncSetAttribute(gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        for (int c = 1; c <= kMaxSplit; c++) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at;
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = c;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.gridDim = dim3((unsigned)(sms / c * c));
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kSmem;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_kernel, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            d.slots[c] = n * c;
        }
        d.sms = sms;
    }
    return &d;
}

// Tokens per tile and CTAs per tile: the least time in clocks of
//   rounds of tiles x scale groups x the largest of 580 and 500 + 2.45 a token (chain) and 4.6 a token (MMA)
//   + 31 a CTA (they start one after the other) + what a launch has around them: first loads 3000, the last tile's outputs 16 a
//     token, those of every tile 21 a token where one accumulator has to be emptied first, a cluster's sums 3000 + 33 a token
//     (beyond 192 tokens 1000 more).
// Fitted to 1949 times of 231 products (14 matrices, 33 to 2048 tokens): what it takes is within 4 % of the quickest of them but
// for five products of 512 or 3072 features (10 %).  With tiles of up to 192 tokens alone 4096 x 4096, 1024 tokens, needed two
// rounds of 128-token tiles, 32.9 us in place of 27.3; 2048 x 8192, 2048 tokens 58.5, now 45.6; 14336 x 14336, 256 tokens 97, now 77.
static void choose(Args& a, int nt, const Device& d)
{
    long long best = LLONG_MAX;
    for (int mt = (a.M + kMaxTm - 1) / kMaxTm, end = (a.M + kMaxTm2 - 1) / kMaxTm2 + 16; mt <= end; mt++) {
        const int tm = ((a.M + mt - 1) / mt + 15) / 16 * 16;
        if ((a.M + tm - 1) / tm != mt) continue;
        const bool one = tm > kMaxTm2;
        const long long chain = 500 + 49 * tm / 20, mma = 23 * tm / 5, stage = mma > chain ? mma : chain > 580 ? chain : 580;
        const long long tiles = (long long)nt * mt;
        if (tiles > INT_MAX / kMaxSplit) break;
        for (int c = 1; c <= kMaxSplit; c++) {
            if (c > 1 && (tiles * c > d.slots[c] || a.groups < 2 * c)) continue;
            const long long rounds = c > 1 ? 1 : (tiles + d.sms - 1) / d.sms, ctas = tiles * c < d.sms ? tiles * c : d.sms;
            const long long cost = rounds * ((a.groups + c - 1) / c) * stage + 31 * ctas + 3000 + 16 * tm + (one ? (rounds - 1) * 21 * tm : 0) +
                                   (c > 1 ? 3000 + 33 * tm + (one ? 1000 : 0) : 0);
            if (cost < best) {
                best = cost;
                a.mt = mt;
                a.tm = tm;
                a.tiles = (int)tiles;
                a.split = c;
            }
        }
    }
}

static bool encode(EncodeTiledFn enc, CUtensorMap* map, CUtensorMapDataType type, const void* base, cuuint64_t inner, cuuint64_t outer,
                   cuuint64_t stride, int box_inner, int box_outer, CUtensorMapSwizzle swizzle)
{
    const cuuint64_t dims[2] = {inner, outer}, strides[1] = {stride};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer}, estr[2] = {1, 1};
    return enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace gemm

// A: half [M,K] row-major (16-byte aligned), packed: prepared weights, possibly matrices packed back to back (every row
// count but the last a multiple of 16); out[i]: rows row0 .. row0 + rows of them go to y[M, rows].
int launch_gemm_tcgen05(const half* A, const uint8_t* packed, const RowsOut* out, int nout, int M, int K, cudaStream_t stream)
{
    using namespace gemm;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from this driver");
    int* err = device_error_flag();
    Device* dev = device();
    if (!err || !dev) return fail(TLLM_ERR_LAUNCH, "device scratch unavailable");
    if (nout < 1 || nout > TLLM_MAX_FUSED) return fail(TLLM_ERR_SHAPE, "gemm_tcgen05: %d outputs", nout);
    Args a = {};
    for (int i = 0; i < TLLM_MAX_FUSED; i++) {
        if (i < nout) a.out[i] = out[i];
        else a.out[i].row0 = INT_MAX;
    }
    a.M = M;
    a.N = out[nout - 1].row0 + out[nout - 1].rows;
    a.groups = K / kGroup;
    const int nrb = (a.N + kTileRows - 1) / kTileRows;
    choose(a, (a.N + kTileN - 1) / kTileN, *dev);
    if (!a.split) return fail(TLLM_ERR_SHAPE, "gemm_tcgen05: M=%d N=%d K=%d: too many tiles", M, a.N, K);
    a.over_split = (uint32_t)((0x100000000ull + a.split - 1) / a.split);         // of one CTA not used
    a.err = err;
    a.acc_stride = (a.tm + 31) / 32 * 32;
    a.accs = a.tm > kMaxTm2 ? 1 : 2;
    a.na = (kTmemCols - a.accs * a.acc_stride) / kACols;
    if (a.na > kMaxA) a.na = kMaxA;
    a.nb = (int)((kSmem - 1024 - kCodes * kCodeBytes) / (a.tm * kGroup * 2));
    if (a.nb > kMaxB) a.nb = kMaxB;
    if (a.na > a.nb) a.na = a.nb;        // weights of a scale group are announced on its stage's barrier
    CUtensorMap map_x, map_w;
    if (!encode(enc, &map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, A, K, M, (cuuint64_t)K * sizeof(half), kBoxK, a.tm, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode(enc, &map_w, CU_TENSOR_MAP_DATA_TYPE_UINT32, packed, (cuuint64_t)a.groups * (kTileBytes / 4), nrb,
                (cuuint64_t)a.groups * kTileBytes, kTileBytes / 4, kTileN / kTileRows, CU_TENSOR_MAP_SWIZZLE_NONE))
        return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled failed");
    const int grid = a.split > 1 ? a.tiles * a.split : (a.tiles < dev->sms ? a.tiles : dev->sms);
    return launch_pdl_cluster("gemm_tcgen05", gemm_kernel, a.split, dim3((unsigned)grid), dim3(kThreads), kSmem, stream, map_x, map_w, a);
}

}  // namespace tllm
