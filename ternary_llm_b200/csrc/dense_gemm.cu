// Dense BF16 GEMM on the 5th-generation tensor cores (sm_100a): Y[M, N] = X[M, K] . W[N, K]^T
// with FP32 accumulation in tensor memory and the element-wise tail of the operator (bias,
// activation, gated product, per-head gate) in the epilogue.
//
// A tile is 128 tokens x TN features, or 256 tokens x TN features of a pair of CTAs (PAIR,
// cta_group::2): each loads its 128 tokens and half of the features' weights and keeps the sums of
// its tokens, the first one issues the MMAs of both.  What bounds a tile is the copies of its operands into
// shared memory (64 bytes a clock and SM): 48 KB for 64 columns of K and 256 features, 32 KB a CTA of a
// pair.  Gate and up of 8192 x 2048, 2000 tokens: 92 -> 81 us in a prompt (1.66 PFLOP/s, where cuBLAS reaches 1.63 at
// 8192^3 by itself), 101 -> 90 in a row of its own; in tiles of 64
// and 128 features what bounded was the loop of one thread that issued the MMAs (2048 x 8192, 100 tokens
// 40.5 -> 29.2 us with the loop run by a warp and one elected lane).
// Where tiles are few, the CTAs of a cluster share one, each a part of K (SPLIT); they send one another
// their sums of the tokens that the other finishes, and add them in rank order.
// One persistent CTA per SM walks tiles with three roles
// that run ahead of one another: a TMA producer (K-major tiles of 64 columns, 128-byte swizzle;
// out-of-range rows and columns read as zero, so no size needs to divide a tile), a warp
// whose elected lane issues tcgen05.mma kind::f16 (M = 128, of a pair 256, N = TN, K = 16) into one of two accumulators in
// tensor memory, and eight epilogue warps that empty the other one: a TMEM lane is a token, the
// rows pass through a small shared-memory tile per warp so that global stores are whole lines.
// A gated feed-forward loads TN/2 gate rows and the TN/2 up rows with the same numbers into one
// tile, so both factors of a product meet in the same thread.  Tiles also run over the entries
// of a block-diagonal or per-head product (column offset in X and Y, row offset in W).  All
// mbarrier waits are bounded; a wait that gives up sets the device error flag, the roles wait
// for their own copies and MMAs (bounded again), and TMEM is freed.  The CTAs of a pair give up together: the
// copies of both count on the first one's barriers, so it waits for what either has issued (pair_drain.cuh)
// before both leave.
#include <mutex>

#include "dense.cuh"
#include "launch.cuh"
#include "pair_drain.cuh"
#include "tcgen05.cuh"

namespace tllm {

namespace {

using namespace gemm;

constexpr int kTok = 128;            // tokens per CTA (MMA M, TMEM lanes)
constexpr int kBlkK = 64;            // K per stage: one 128-byte swizzled row
constexpr int kEpiWarps = 8;         // two per quarter of the TMEM lanes, taking turns at 32 columns
constexpr int kThr = 128 + 32 * kEpiWarps;

constexpr int kStageLd = 20;         // words per row of an epilogue warp's tile: 16 of data (16 FP32 or 32 BF16 columns)

enum Way { kSingle, kPair, kSplit };      // a CTA a tile; two CTAs a tile of 256 tokens; K of a tile over the CTAs of a cluster

template <int TN, Way WAY>
struct DCfg {
    static constexpr bool PAIR = WAY == kPair;
    static constexpr int kXBytes = kTok * kBlkK * 2;
    static constexpr int kWBytes = TN * kBlkK * 2 / (PAIR ? 2 : 1);
    static constexpr int kStage = kXBytes + kWBytes;
    static constexpr int kStages = PAIR ? (TN == 256 ? 6 : 8) : WAY == kSplit ? 6 : (TN == 256) ? 4 : (TN == 128) ? 6 : 8;
    static constexpr int kEpiBytes = kEpiWarps * 32 * kStageLd * 4;
    static constexpr size_t kSums = WAY == kSplit ? (size_t)TN * kTok * 4 : 0;      // what the cluster's CTAs send
    static constexpr size_t kSmem = (size_t)kStages * kStage + kEpiBytes + kSums + 1024;
};

struct DenseEpi {
    void* y;
    const float* bias;
    const bf16* gate;
    int ldy, y_batch, gate_ld;
    int M, N, K, x_batch, w_rows;
    int mt, nt, tiles;             // tiles along the tokens, along the features, in all
    int split;                     // CTAs that share a tile's K, a power of two
    int act, glu, y_f32, vec, bias_vec;
    float act_param;
    int act_lo, act_hi, f32_from, ldy2, vec2;
    float* y2;
    const int *group, *groups;
    int* err;
};

template <int TN, bool PAIR>
__device__ __forceinline__ uint32_t idesc_bf16()
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)((PAIR ? 2 * kTok : kTok) >> 4) << 24);
}

template <bool PAIR>
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    if constexpr (PAIR)
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
    else
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// arrives, once everything issued so far is complete, at this barrier of the CTA, or of both CTAs of the pair
template <bool PAIR>
__device__ __forceinline__ void commit(uint32_t bar)
{
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        mma_commit(bar);
}
// the copy's bytes count on `bar`, of the pair's first CTA for both
template <bool PAIR>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    if constexpr (PAIR)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
    else
        tma_load_2d(dst, map, x, y, bar);
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t in_first_cta(uint32_t addr) { return in_cta(addr, 0); }
__device__ __forceinline__ void store_cluster(uint32_t addr, int v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// counts bytes that no copy will bring
__device__ __forceinline__ void complete_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// all threads of the CTA, or of the pair
template <bool PAIR>
__device__ __forceinline__ void sync_all()
{
    __syncwarp();
    if constexpr (PAIR) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}

template <int TN, Way WAY>
__global__ void __launch_bounds__(kThr, 1)
dense_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const DenseEpi a)
{
    constexpr bool PAIR = WAY == kPair, SPLIT = WAY == kSplit;
    using Cfg = DCfg<TN, WAY>;
    constexpr int kStages = Cfg::kStages, kStage = Cfg::kStage, kXBytes = Cfg::kXBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * kStages + 4];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag, other_count;            // of a pair: stages that the second CTA filled, tiles that the first one committed
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int outs = a.glu ? TN / 2 : TN;              // output features of a tile
    const int rank = PAIR ? blockIdx.x & 1 : 0;        // CTA of the pair: its half of the tile's tokens and of its rows of W
    const int first_tile = PAIR ? blockIdx.x >> 1 : SPLIT ? blockIdx.x / a.split : blockIdx.x;
    const int step_tiles = PAIR ? gridDim.x >> 1 : gridDim.x;                  // SPLIT: one tile
    const int nk_all = (a.K + kBlkK - 1) / kBlkK;
    // SPLIT: this CTA's part of K and, of its tile's tokens, those that it finishes
    const int part = SPLIT ? blockIdx.x & (a.split - 1) : 0, k0 = SPLIT ? part * nk_all / a.split : 0;
    const int nk = (SPLIT ? (part + 1) * nk_all / a.split : nk_all) - k0;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
    auto acc_full = [&](int i) { return bar0 + 8u * (2 * kStages + i); };
    auto acc_empty = [&](int i) { return bar0 + 8u * (2 * kStages + 2 + i); };

    if (tid == 0) {
        prefetch_map(&map_x);
        prefetch_map(&map_w);
        for (int s = 0; s < kStages; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(acc_full(i), 1);
            mbar_init(acc_empty(i), PAIR ? 2 * kEpiWarps : 32 * kEpiWarps);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(&tmem_slot)), "r"(2 * TN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(&tmem_slot)), "r"(2 * TN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<PAIR || SPLIT>();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    volatile int* abortp = &abort_flag;
    int fills = 0;                                     // stages that this warp's producer filled
    auto give_up = [&]() {
        abort_flag = 1;
        if constexpr (PAIR) store_cluster(in_cta(smem_u32(&abort_flag), rank ^ 1), 1);
    };
    int never = 0;
    pdl_wait();
    // tile -> first token, first feature, batch entry, entry of W; tokens vary fastest (neighbours
    // share W), with grouped rows those of one entry
    const int tiles = a.group ? min(*a.groups, a.mt) * a.nt : a.tiles;
    auto where = [&](int tile, int& m0, int& n0, int& z, int& entry) {
        if (a.group) {
            const int* g = a.group + 3 * (tile / a.nt);
            const int first = g[1], count = g[2], r = tile - first * a.nt, n = r / count;
            m0 = (first + r - n * count) * kTok;
            n0 = n * outs;
            z = 0;
            entry = g[0];
            return;
        }
        m0 = (tile % a.mt) * (PAIR ? 2 * kTok : kTok) + rank * kTok;
        tile /= a.mt;
        n0 = (tile % a.nt) * outs;
        entry = z = tile / a.nt;
    };

    float* sums = reinterpret_cast<float*>(smem + (size_t)kStages * kStage + Cfg::kEpiBytes);       // SPLIT
    auto head_gate = [&](int mrow, int z) {
        return (a.gate && mrow + lane < a.M) ? sigmoid_f(__bfloat162float(a.gate[(size_t)(mrow + lane) * a.gate_ld + z])) : 1.f;
    };
    // Epilogue of 32 columns from column c of a tile on (features n0 + c ..), whose sums `read` gives for this lane's row, mrow + lane
    // of the nrows from mrow on; st: a tile of this warp in shared memory.
    const int ew = warp - 4;
    uint32_t* st = reinterpret_cast<uint32_t*>(smem + (size_t)kStages * kStage) + ew * 32 * kStageLd;
    const int sr = lane >> 2, sw = (lane & 3) * 4;       // row (of eight) and words this lane stores
    auto finish = [&](int c, int ncols, int n0, int z, int mrow, int nrows, float hg, auto read) {
        // 32 columns go one way: the limits of the activation and of y2 are multiples of 64
        const bool second = n0 + c >= a.f32_from, y_f32 = a.y_f32 || second;
        const int act = n0 + c >= a.act_lo && n0 + c < a.act_hi && !second ? a.act : kActNone;
        const int wcols = y_f32 ? 1 : 2;         // columns per staged word
        float f[32];
        read(c, f);
        if (a.glu) {
            float u[32];
            read(TN / 2 + c, u);
            apply_act_n<32>(act, f);
#pragma unroll
            for (int j = 0; j < 32; j++) f[j] *= u[j];
        } else {
            if (a.bias) {
                const float* bp = a.bias + (size_t)z * a.N + n0 + c;
                if (a.bias_vec && c + 32 <= ncols) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 t = __ldg(reinterpret_cast<const float4*>(bp) + j);
                        f[4 * j] += t.x;
                        f[4 * j + 1] += t.y;
                        f[4 * j + 2] += t.z;
                        f[4 * j + 3] += t.w;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c + j < ncols) f[j] += __ldg(bp + j);
                }
            }
            apply_act_n<32>(act, f, a.act_param);
            if (a.gate) {
#pragma unroll
                for (int j = 0; j < 32; j++) f[j] *= hg;
            }
        }
        // through shared memory, 16 words of a row at a time: FP32 in two halves, BF16 at once
#pragma unroll
        for (int part = 0; part < 2; part++) {
            if (part == 1 && !y_f32) break;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int e = 4 * j + q;
                    if (y_f32) {
                        w[q] = __float_as_uint(f[part * 16 + e]);
                    } else {
                        const __nv_bfloat162 t = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
                        w[q] = *reinterpret_cast<const uint32_t*>(&t);
                    }
                }
                *reinterpret_cast<uint4*>(st + lane * kStageLd + 4 * j) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            __syncwarp();
            const int col = c + part * 16 + sw * wcols;      // first of this lane's columns inside the tile
            if (col < ncols) {
                const bool vec = (second ? a.vec2 : a.vec) && col + 4 * wcols <= ncols;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int rr = r * 8 + sr, m = mrow + rr;
                    if (m >= a.M || rr >= nrows) break;
                    const uint4 t = *reinterpret_cast<const uint4*>(st + rr * kStageLd + sw);
                    const size_t o = second ? (size_t)m * a.ldy2 + n0 + col - a.f32_from
                                            : (size_t)m * a.ldy + (size_t)z * a.y_batch + n0 + col;
                    if (vec) {
                        if (y_f32) *reinterpret_cast<uint4*>((second ? a.y2 : static_cast<float*>(a.y)) + o) = t;
                        else *reinterpret_cast<uint4*>(static_cast<bf16*>(a.y) + o) = t;
                    } else {
                        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
                        for (int q = 0; q < 4 * wcols && col + q < ncols; q++) {
                            if (y_f32) (second ? a.y2 : static_cast<float*>(a.y))[o + q] = __uint_as_float(w[q]);
                            else static_cast<uint16_t*>(a.y)[o + q] = (uint16_t)(w[q >> 1] >> ((q & 1) * 16));
                        }
                    }
                }
            }
        }
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        const bool leader = elect_one();
        int s = 0, phase = 1;                            // stage, parity that means empty
        bool ok = true;
        for (int tile = first_tile; ok && tile < tiles; tile += step_tiles) {
            int m0, n0, z, entry;
            where(tile, m0, n0, z, entry);
            const int wr0 = entry * a.w_rows + n0, wr1 = a.glu ? wr0 + a.N : wr0 + TN / 2, x0 = z * a.x_batch;
            for (int k = 0; k < nk; k++) {
                if (!(ok = mbar_wait(empty(s), phase, abortp))) break;
                if (leader) {
                    if (rank == 0) mbar_expect_tx(full(s), PAIR ? 2 * kStage : kStage);
                    const uint32_t dst = smem_u32(smem + (size_t)s * kStage), bar = PAIR ? in_first_cta(full(s)) : full(s);
                    load_tile<PAIR>(dst, &map_x, x0 + (k0 + k) * kBlkK, m0, bar);
                    load_tile<PAIR>(dst + kXBytes, &map_w, (k0 + k) * kBlkK, rank ? wr1 : wr0, bar);
                    if (!PAIR) load_tile<PAIR>(dst + kXBytes + TN / 2 * kBlkK * 2, &map_w, (k0 + k) * kBlkK, wr1, bar);
                }
                fills++;
                if (++s == kStages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
        if (!ok) give_up();
        __syncwarp();
        // normally the MMAs consume every stage; after an abort the copies still in flight
        // must land before the shared memory goes away (of a pair: below, for both CTAs)
        if constexpr (PAIR) {
            if (leader && rank) store_cluster(in_cta(smem_u32(&other_count), 0), fills);
        } else if (*abortp) {
            for (int f = max(0, fills - kStages); f < fills; f++) mbar_wait(full(f % kStages), (f / kStages) & 1, &never);
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------- MMA issuer ----------------
        const bool leader = elect_one();
        const uint32_t idesc = idesc_bf16<TN, PAIR>();
        int s = 0, phase = 0, i = 0;                     // i: tiles of this CTA so far
        bool ok = true;
        for (int tile = first_tile; ok && tile < tiles; tile += step_tiles, i++) {
            const int buf = i & 1;
            if (!(ok = mbar_wait(acc_empty(buf), ((i >> 1) & 1) ^ 1, abortp))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + buf * TN;
            for (int k = 0; k < nk; k++) {
                if (!(ok = mbar_wait(full(s), phase, abortp))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t xd = make_sw128_desc(smem_u32(smem + (size_t)s * kStage)), wd = make_sw128_desc(smem_u32(smem + (size_t)s * kStage + kXBytes));
                const uint32_t more = k > 0;
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < kBlkK / 16; kk++)          // 32 bytes (2 in the descriptor) inside the swizzled row
                        mma_ss<PAIR>(acc, xd + kk * 2, wd + kk * 2, idesc, kk ? 1u : more);
                    commit<PAIR>(empty(s));
                }
                if (++s == kStages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            // arrives after everything issued so far, on the abort path too
            if (leader) commit<PAIR>(acc_full(buf));
        }
        if (!ok) give_up();
        if constexpr (PAIR)
            if (leader) store_cluster(in_cta(smem_u32(&other_count), 1), i);
        __syncwarp();
        // the last accumulators complete before TMEM and shared memory are given up
        for (int j = i > 2 ? i - 2 : 0; j < i; j++)
            if (!mbar_wait(acc_full(j & 1), (j >> 1) & 1, &never)) give_up();
    } else if (warp >= 4) {
        // ---------------- epilogue ----------------
        const int row0 = (ew & 3) * 32, half = ew >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)row0 << 16);
        int i = 0;
        for (int tile = first_tile; tile < tiles; tile += step_tiles, i++) {
            const int buf = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(acc_full(buf), (i >> 1) & 1, abortp))) {
                give_up();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int m0, n0, z, entry;
            where(tile, m0, n0, z, entry);
            const int mrow = m0 + row0;
            const uint32_t acc = lane_base + buf * TN;
            auto read = [&](int c, float (&f)[32]) {
                uint32_t v[32];
                __syncwarp();
                tmem_ld32(acc + c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 32; j++) f[j] = __uint_as_float(v[j]);
            };
            if constexpr (SPLIT) {
                // this CTA's sums of a row to the CTA that finishes it: [CTA][column][row]
                const int rows = kTok / a.split, to = (row0 + lane) / rows;
                uint32_t peer;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_u32(sums + part * TN * rows + (row0 + lane) % rows)), "r"(to));
                if (mrow < a.M)
                    for (int c = half * 32; c < TN; c += 64) {
                        float f[32];
                        read(c, f);
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer + (uint32_t)((c + j) * rows * 4)), "f"(f[j]) : "memory");
                    }
                break;
            }
            const float hg = head_gate(mrow, z);
            const int ncols = min(outs, a.N - n0);
            if (mrow < a.M)
#pragma unroll 1
                for (int c = half * 32; c < ncols; c += 64) finish(c, ncols, n0, z, mrow, 32, hg, read);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if constexpr (PAIR) {
                __syncwarp();
                if (lane == 0) arrive_cluster(in_first_cta(acc_empty(buf)));
            } else {
                mbar_arrive(acc_empty(buf));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<PAIR || SPLIT>();                           // of a pair: nothing of one CTA is used by the other any more
    if constexpr (PAIR) {
        if (abort_flag) {                                // of both CTAs: the copies of either and the last arrivals come before they leave
            if (rank == 0 && warp == 0) {
                for (int f = pair_fills_begin(fills, other_count, kStages); f < pair_fills_end(fills, other_count); f++) {
                    const PairFill p = pair_fill(f, fills, other_count, kStages);
                    if (lane == 0 && p.unarmed) mbar_expect_tx(full(p.stage), kStage);
                    if (lane == 0 && p.lacks) complete_tx(full(p.stage), kStage);
                    mbar_wait(full(p.stage), p.parity, &never);
                }
            } else if (rank == 1 && warp == 1) {
                for (int j = max(0, other_count - 2); j < other_count; j++) mbar_wait(acc_full(j & 1), (j >> 1) & 1, &never);
            }
            sync_all<true>();
        }
    }
    if constexpr (SPLIT) {
        if (warp >= 4 && !abort_flag) {
            const int rows = kTok / a.split, nrows = min(32, rows), groups = rows / nrows, per = (outs + 31) / 32;
            int m0, n0, z, entry;
            where(first_tile, m0, n0, z, entry);
            const int ncols = min(outs, a.N - n0);
            for (int i = ew; i < groups * per; i += kEpiWarps) {
                const int c = i / groups * 32, r0 = i % groups * 32, mrow = m0 + part * rows + r0;
                if (c >= ncols || mrow >= a.M) continue;
                finish(c, ncols, n0, z, mrow, nrows, head_gate(mrow, z), [&](int col, float (&f)[32]) {
                    const float* p = sums + col * rows + r0 + lane % nrows;
#pragma unroll
                    for (int j = 0; j < 32; j++) f[j] = 0.f;
                    for (int q = 0; q < a.split; q++, p += TN * rows)
#pragma unroll
                        for (int j = 0; j < 32; j++) f[j] += p[j * rows];
                });
            }
        }
    }
    if (abort_flag && tid == 0) atomicExch(a.err, TLLM_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TN) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TN) : "memory");
    }
}

int encode(EncodeTiledFn enc, CUtensorMap* map, const bf16* p, int cols, int rows, int ld, int box_rows)
{
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(bf16)};
    const cuuint32_t box[2] = {(cuuint32_t)kBlkK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(p), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TLLM_ERR_LAUNCH, "dense_gemm: cuTensorMapEncodeTiled failed with %d", (int)r);
    return TLLM_OK;
}

template <int TN, Way WAY>
int launch_tn(EncodeTiledFn enc, const LinearArgs<bf16>& l, DenseEpi e, int sms, cudaStream_t stream)
{
    CUtensorMap mx, mw;
    int st;
    if ((st = encode(enc, &mx, l.x, (l.batch - 1) * l.x_batch + l.K, l.M, l.ldx, kTok))) return st;
    if ((st = encode(enc, &mw, l.w, l.K, (l.group ? l.entries : l.batch) * l.w_rows, l.ldw, TN / 2))) return st;
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr[dev]) {
        cudaFuncSetAttribute(dense_gemm_kernel<TN, WAY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DCfg<TN, WAY>::kSmem);
        attr[dev] = true;
    }
    const int outs = l.glu ? TN / 2 : TN;
    const int tokens = WAY == kPair ? 2 * kTok : kTok, per = WAY == kPair ? 2 : WAY == kSplit ? e.split : 1;
    e.mt = (l.M + tokens - 1) / tokens;
    e.nt = (l.N + outs - 1) / outs;
    e.tiles = e.mt * e.nt * l.batch;
    const int grid = (WAY == kSplit || e.tiles < sms / per ? e.tiles : sms / per) * per;
    return launch_pdl_cluster("dense_gemm", dense_gemm_kernel<TN, WAY>, per, dim3(grid), dim3(kThr), DCfg<TN, WAY>::kSmem, stream, mx, mw, e);
}

}  // namespace

// The way of a product: the tile's features, whether pairs of CTAs share a tile, and the CTAs that share its K.
DenseWay dense_way(const LinearArgs<bf16>& l, int sms)
{
    const long long mt = (l.M + kTok - 1) / kTok;
    auto tiles = [&](int tn, long long m) {
        const int outs = l.glu ? tn / 2 : tn;
        return m * ((l.N + outs - 1) / outs) * l.batch;
    };
    DenseWay r = {64, false, 1};
    if (l.group) {                           // their number is known on the device alone: the widest tile that still gives most SMs one
        r.features = tiles(256, mt) * 10 >= 7LL * sms ? 256 : tiles(128, mt) * 10 >= 7LL * sms ? 128 : 64;
        return r;
    }
    // The quickest by rounds of tiles: 64 columns of K take 0.21, 0.27, 0.39 us in a tile of 64, 128, 256 features (its operands' 24,
    // 32, 48 KB through 64 bytes a clock), 0.235 and 0.36 in a pair's tile of 128 and 256 (24 and 32 KB a CTA); the outputs of a tile
    // 0.8 and 0.02 a feature (twice that where rows of Y are no whole 16-byte pieces), of gated pairs 1.6 and 0.016, beside the next tile's product; a launch 2.5, of pairs 4.  us measured with 64, 128, 256, pair 128, pair
    // 256, the one taken in brackets: 2000 tokens 2048 x 2048 31 22 (20) 20 21, 8192 x 2048 gated 183 116 96 107 (89), 4096 x 128
    // 16.2 16.2 (15.2) 18.8 17.0; 1000 tokens 2048 x 8192 55 35 53 (31) 48; 300 tokens 4096 x 4096 30 21 32 (19) 30, 14336 x 4096 gated
    // 128 85 (83) 95 89; 100 tokens 8192 x 2048 (12.3) 14.4 20.7 14.3 19.8.  Gated and short: 400 tokens 4864 x 512 13.2 (10.1) 11.6 12.1 12.4; 64
    // tokens 12032 x 200 11.4 (8.9).
    const struct { int tn; bool pair; double step; } way[] = {{64, false, 0.21}, {128, false, 0.27}, {256, false, 0.39}, {128, true, 0.235}, {256, true, 0.36}};
    const size_t es = l.y_f32 ? 4 : 2;
    const double ragged = l.ldy * es % 16 || l.y_batch * es % 16 ? 2. : 1.;              // rows of Y are stored element by element
    auto outputs = [&](int tn) { return l.glu ? 1.6 + 0.016 * tn : ragged * (0.8 + 0.02 * tn); };
    double best = 0.;
    for (const auto& w : way) {
        if (w.pair && mt == 1) continue;
        const long long at_once = w.pair ? sms / 2 : sms, n = tiles(w.tn, w.pair ? (mt + 1) / 2 : mt);
        const double product = (l.K + kBlkK - 1) / kBlkK * w.step, output = outputs(w.tn);
        const double t = (double)((n + at_once - 1) / at_once) * (product > output ? product : output) + (product > output ? output : product) + (w.pair ? 4. : 2.5);
        if (best == 0. || t < best) {
            best = t;
            r.features = w.tn;
            r.pair = w.pair;
        }
    }
    // Few tiles: K over a cluster's CTAs while all of them run at once; exchanging the sums takes 3.7 us.  One CTA a tile / so, 100
    // tokens: 2048 x 8192 29 / 15, 4096 x 14336 48 / 32, 2048 x 2048 10.6 / 9.7, 2048 x 1024 7.5 / 8.6.
    const long long n = tiles(64, mt), most[3] = {sms, sms * 8 / 9, sms * 4 / 5};
    for (int i = 0, split = 2; i < 3 && n * split <= most[i]; i++, split *= 2) {
        const int steps = (l.K + kBlkK - 1) / kBlkK;
        if (steps < split) break;
        const double t = (steps + split - 1) / split * 0.21 + outputs(64) + 2.5 + 3.7;
        if (t < best) {
            best = t;
            r = {64, false, split};
        }
    }
    return r;
}

int launch_dense_gemm_tcgen05(const LinearArgs<bf16>& l, cudaStream_t stream)
{
    if (l.M == 0 || l.N == 0 || l.batch == 0) return TLLM_OK;
    // K offsets of a TMA box must start on 16-byte boundaries, rows as well
    if (l.K < 8 || l.K % 8 || l.ldw % 8 || l.ldx % 8 || l.x_batch % 8)
        return fail(TLLM_ERR_SHAPE, "dense_gemm: K=%d ldw=%d ldx=%d x_batch=%d must be multiples of 8", l.K, l.ldw, l.ldx, l.x_batch);
    if ((reinterpret_cast<uintptr_t>(l.x) | reinterpret_cast<uintptr_t>(l.w)) & 15)
        return fail(TLLM_ERR_ALIGN, "dense_gemm: operands must be 16-byte aligned");
    if (l.group && (l.batch != 1 || !l.groups)) return fail(TLLM_ERR_SHAPE, "dense_gemm: grouped rows with %d batch entries", l.batch);
    if ((l.act_lo | (l.act_hi == INT_MAX ? 0 : l.act_hi) | (l.f32_from == INT_MAX ? 0 : l.f32_from)) % 64 ||
        ((l.act_lo || l.act_hi != INT_MAX || l.f32_from != INT_MAX) && (l.glu || l.batch != 1)))
        return fail(TLLM_ERR_SHAPE, "dense_gemm: column ranges %d..%d and %d", l.act_lo, l.act_hi, l.f32_from);
    if (l.w_rows < (l.glu ? 2 : 1) * l.N) return fail(TLLM_ERR_SHAPE, "dense_gemm: %d rows of W for N=%d", l.w_rows, l.N);
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from this driver");
    DenseEpi e = {};
    e.y = l.y;
    e.bias = l.bias;
    e.gate = l.gate;
    e.ldy = l.ldy;
    e.y_batch = l.y_batch;
    e.gate_ld = l.gate_ld;
    e.M = l.M;
    e.N = l.N;
    e.K = l.K;
    e.x_batch = l.x_batch;
    e.w_rows = l.w_rows;
    e.act = l.act;
    e.glu = l.glu;
    e.y_f32 = l.y_f32;
    const size_t es = l.y_f32 ? 4 : 2;
    e.vec = ((l.ldy * es) % 16 == 0 && (l.y_batch * es) % 16 == 0 && (reinterpret_cast<uintptr_t>(l.y) & 15) == 0);
    e.bias_vec = l.N % 4 == 0 && (reinterpret_cast<uintptr_t>(l.bias) & 15) == 0;
    e.act_param = l.act_param;
    e.act_lo = l.act_lo;
    e.act_hi = l.act_hi;
    e.f32_from = l.f32_from;
    e.y2 = l.y2;
    e.ldy2 = l.ldy2;
    e.vec2 = l.ldy2 % 4 == 0 && (reinterpret_cast<uintptr_t>(l.y2) & 15) == 0;
    e.group = l.group;
    e.groups = l.groups;
    e.err = device_error_flag();
    if (!e.err) return fail(TLLM_ERR_LAUNCH, "device scratch unavailable");
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return fail(TLLM_ERR_LAUNCH, "dense_gemm: no current device");
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    const DenseWay r = dense_way(l, sms[dev]);
    e.split = r.split;
    if (r.features == 256) return r.pair ? launch_tn<256, kPair>(enc, l, e, sms[dev], stream) : launch_tn<256, kSingle>(enc, l, e, sms[dev], stream);
    if (r.features == 128) return r.pair ? launch_tn<128, kPair>(enc, l, e, sms[dev], stream) : launch_tn<128, kSingle>(enc, l, e, sms[dev], stream);
    if (r.split > 1) return launch_tn<64, kSplit>(enc, l, e, sms[dev], stream);
    return launch_tn<64, kSingle>(enc, l, e, sms[dev], stream);
}

}  // namespace tllm
