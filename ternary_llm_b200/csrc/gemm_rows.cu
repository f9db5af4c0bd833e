// Products of a few activation rows (4..32) with a ternary matrix, C[M, N] = A[M, K] . W^T.
//
// Bound: the weight stream and, at these sizes, the latencies of a launch.  A tcgen05 tile of 128
// features walks its weights through tensor memory one scale group at a time, a chain of about a
// microsecond per group that a decode batch cannot fill; here every warp expands its own weights
// into mma.sync.m16n8k16 operand registers, so that all SMs stream at once and no step waits for
// another warp.  scale * t is exact in FP16, so this is the same FP16 contraction with FP32 sums as
// the tcgen05 kernel's (gemm_tcgen05.cu).
//
//   * A CTA owns RG * R row blocks of 16 features and a range of scale groups; warp (rg, kw) takes R
//     row blocks and every KW-th group.  A lane's 16 bytes of codes per (row block, group) are four
//     whole A fragments' worth: the byte j, field f of a word is column 32f + 16*j2 + 4t + j
//     (packed_layout.cuh), so MMA (f, j2) contracts sixteen neighbouring columns with the columns
//     4t..4t+3 in lane t's four slots, and the B fragment is one 8-byte piece of an activation row.
//   * Codes and scales go from global memory into registers, D groups ahead, and the first D are
//     requested before the wait on the previous kernel.
//   * Activations pass through shared memory in stages of KW groups, cp.async, three stages; rows are
//     padded by 32 bytes so that a fragment load touches every bank once.
//   * The KW partial sums of a CTA meet in shared memory.  Where there are too few row blocks for the
//     SMs, a cluster of C CTAs splits the groups; its CTAs add one another's sums over the cluster's
//     shared memory, in rank order, each for a share of the outputs.
#include <climits>

#include "launch.cuh"
#include "packed_layout.cuh"

namespace tllm {

namespace {

constexpr int kThreads = 256;
constexpr int kStages = 3;
constexpr int kRowWarps = 2, kGroupWarps = 4;        // RG and KW

struct RowsArgs {
    const uint8_t* packed;
    const half* x;                           // [m, cols]
    RowsOut out[TLLM_MAX_FUSED];             // row ranges of the matrix and where they go; unused ones start past every row
    int m, cols, groups, nrb, split;
};

__device__ __forceinline__ uint32_t sm32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 ldg_stream(const void* p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_word(const void* p)
{
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

template <int NB, int RG, int KW> struct Shape {
    static constexpr int kR = 2;                                     // row blocks per warp
    static constexpr int kAhead = 3;                                 // groups per warp whose weights are in flight
    static constexpr int kRows = RG * kR * kTileRows;                // features per CTA
    static constexpr int kLd = KW * kGroup + 16;                     // halves per staged activation row
    static constexpr int kStage = NB * 8 * kLd;                      // halves per stage
    static constexpr int kLdRed = kRows + 4;                         // floats per vector of the partial sums
    static constexpr size_t kX = (size_t)kStages * kStage * sizeof(half);
    static constexpr size_t kRed = (size_t)(KW + 1) * NB * 8 * kLdRed * sizeof(float);
    static constexpr size_t kSmem = kX > kRed ? kX : kRed;
    static_assert(RG * KW * 32 == kThreads, "eight warps");
};

template <int NB, int RG, int KW>
__global__ void __launch_bounds__(kThreads, 2)
gemm_rows_kernel(const RowsArgs a)
{
    using S = Shape<NB, RG, KW>;
    constexpr int R = S::kR, kAhead = S::kAhead;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    half* xs = reinterpret_cast<half*>(smem_raw);
    float* red = reinterpret_cast<float*>(smem_raw);                 // after the last group
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3;
    const int kw = warp % KW, rg = warp / KW;
    const int rank = blockIdx.x % a.split, tile = blockIdx.x / a.split;
    const int g0 = (int)((long long)rank * a.groups / a.split), ng = (int)((long long)(rank + 1) * a.groups / a.split) - g0;
    const int nst = (ng + KW - 1) / KW, mine = (ng - kw + KW - 1) / KW;        // stages; groups of this warp
    const int rb0 = (tile * RG + rg) * R;

    const uint8_t* wp[R];
#pragma unroll
    for (int r = 0; r < R; r++)      // row blocks past the matrix repeat the last one and are not stored
        wp[r] = a.packed + ((size_t)min(rb0 + r, a.nrb - 1) * a.groups + g0 + kw) * kTileBytes;
    uint4 cw[kAhead][R];
    uint32_t sw[kAhead][R];
    auto load = [&](int i, uint4 (&c)[R], uint32_t (&s)[R]) {
        if (i < mine) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint8_t* p = wp[r] + (size_t)i * (KW * kTileBytes);
                c[r] = ldg_stream(p + lane * 16);
                s[r] = ldg_word(p + kTileCodeBytes + gq * 4);
            }
        }
    };
#pragma unroll
    for (int d = 0; d < kAhead; d++) load(d, cw[d], sw[d]);

    float acc[R][NB][4];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[r][n][e] = 0.f;

    pdl_wait();
    auto stage = [&](int i) {
        if (i < nst) {
            const uint32_t dst = sm32(xs + (i % kStages) * S::kStage);
            const int c0 = (g0 + i * KW) * kGroup, cend = (g0 + ng) * kGroup;
            constexpr int kPieces = KW * kGroup / 8;
            for (int p = tid; p < NB * 8 * kPieces; p += kThreads) {
                const int n = p / kPieces, c = (p - n * kPieces) * 8;
                const bool v = n < a.m && c0 + c < cend;
                copy16(dst + (n * S::kLd + c) * 2, v ? a.x + (size_t)n * a.cols + c0 + c : a.x, v);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; i++) stage(i);

    for (int i0 = 0; i0 < nst; i0 += kAhead) {
#pragma unroll
        for (int d = 0; d < kAhead; d++) {
            const int i = i0 + d;
            if (i >= nst) break;
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            __syncthreads();                             // stage i is here, stage i - 1 is free
            stage(i + kStages - 1);
            if (i < mine) {
                const half* xr = xs + (i % kStages) * S::kStage + gq * S::kLd + kw * kGroup + 4 * t;
                uint32_t lo[R][2], hi[R][2];
#pragma unroll
                for (int r = 0; r < R; r++) {            // byte table of a row: -s, 0, +s for the codes 0, 1, 2
                    lo[r][0] = (sw[d][r] & 0xffffu) ^ 0x8000u;
                    hi[r][0] = sw[d][r];
                    hi[r][1] = sw[d][r] >> 16;
                    lo[r][1] = hi[r][1] ^ 0x8000u;
                }
#pragma unroll
                for (int f = 0; f < 4; f++)
#pragma unroll
                    for (int j2 = 0; j2 < 2; j2++) {
                        uint2 b[NB];
#pragma unroll
                        for (int n = 0; n < NB; n++) b[n] = *reinterpret_cast<const uint2*>(xr + n * 8 * S::kLd + 32 * f + 16 * j2);
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            const uint32_t s0 = (((j2 ? cw[d][r].y : cw[d][r].x) >> (2 * f)) & 0x03030303u) * 0x22u + 0x10101010u;
                            const uint32_t s1 = (((j2 ? cw[d][r].w : cw[d][r].z) >> (2 * f)) & 0x03030303u) * 0x22u + 0x10101010u;
                            const uint32_t fr[4] = {prmt(lo[r][0], hi[r][0], s0), prmt(lo[r][1], hi[r][1], s1),
                                                    prmt(lo[r][0], hi[r][0], s0 >> 16), prmt(lo[r][1], hi[r][1], s1 >> 16)};
#pragma unroll
                            for (int n = 0; n < NB; n++) mma_f16(acc[r][n], fr, b[n].x, b[n].y);
                        }
                    }
            }
            load(i + kAhead, cw[d], sw[d]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // ---- the KW partial sums of the CTA, then those of the cluster ------------------------------
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                red[((size_t)kw * NB * 8 + n * 8 + 2 * t + (e & 1)) * S::kLdRed + (rg * R + r) * kTileRows + gq + 8 * (e >> 1)] = acc[r][n][e];
    __syncthreads();
    float* part = red + KW * NB * 8 * S::kLdRed;
    const int row0 = tile * S::kRows;
    auto store = [&](int e, float v) {
        const int n = e / S::kRows, row = row0 + e - n * S::kRows;
        half* y = a.out[0].y;
        int first = 0, rows = a.out[0].rows;
#pragma unroll
        for (int i = 1; i < TLLM_MAX_FUSED; i++)
            if (row >= a.out[i].row0) {
                y = a.out[i].y;
                first = a.out[i].row0;
                rows = a.out[i].rows;
            }
        if (row - first < rows) y[(size_t)n * rows + row - first] = __float2half_rn(v);
    };
    for (int e = tid; e < a.m * S::kRows; e += kThreads) {
        const int n = e / S::kRows, row = e - n * S::kRows;
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < KW; k++) v += red[((size_t)k * NB * 8 + n) * S::kLdRed + row];
        if (a.split == 1) store(e, v);
        else part[n * S::kLdRed + row] = v;
    }
    if (a.split > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        for (int e = rank * kThreads + tid; e < a.m * S::kRows; e += a.split * kThreads) {
            const int n = e / S::kRows, row = e - n * S::kRows;
            const uint32_t at = sm32(part + n * S::kLdRed + row);
            float p[8], v = 0.f;
#pragma unroll
            for (int z = 0; z < 8; z++) {
                p[z] = 0.f;
                if (z < a.split) {
                    uint32_t peer;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(z));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(p[z]) : "r"(peer) : "memory");
                }
            }
#pragma unroll
            for (int z = 0; z < 8; z++)
                if (z < a.split) v += p[z];
            store(e, v);
        }
        // nobody leaves while its sums are still read
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// CTAs that run at the same time on the current device, two per SM; 0 without one.
int cta_slots()
{
    static int sms[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return 2 * sms[dev];
}

// CTAs that share the scale groups of a tile: as many, a power of two, as run at the same time and have two of them per warp.
int split_of(int tiles, int groups, int slots)
{
    int split = 1;
    while (split < 8 && tiles * split * 2 <= slots && groups >= split * 2 * kGroupWarps) split *= 2;
    return split;
}

template <int NB>
int launch(RowsArgs a, cudaStream_t stream)
{
    using S = Shape<NB, kRowWarps, kGroupWarps>;
    auto kernel = gemm_rows_kernel<NB, kRowWarps, kGroupWarps>;
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return fail(TLLM_ERR_LAUNCH, "gemm_rows: no current device");
    if (!attr[dev]) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
        attr[dev] = true;
    }
    const int tiles = (a.nrb + S::kRows / kTileRows - 1) / (S::kRows / kTileRows);
    a.split = split_of(tiles, a.groups, cta_slots());
    return launch_pdl_cluster("gemm_rows", kernel, a.split, dim3((unsigned)(tiles * a.split)), dim3(kThreads), S::kSmem, stream, a);
}

}  // namespace

// Matrices packed back to back (every row count but the last a multiple of 16) as one.
int launch_gemm_rows(const uint8_t* packed, const half* x, const RowsOut* out, int nout, int m, int cols, cudaStream_t stream)
{
    if (m < 1 || m > kRowsMax || nout < 1 || nout > TLLM_MAX_FUSED) return fail(TLLM_ERR_BATCH, "gemm_rows: m=%d outputs=%d", m, nout);
    RowsArgs a = {};
    for (int i = 0; i < TLLM_MAX_FUSED; i++) {
        if (i < nout) a.out[i] = out[i];
        else a.out[i].row0 = INT_MAX;
    }
    a.packed = packed;
    a.x = x;
    a.m = m;
    a.cols = cols;
    a.groups = cols / kGroup;
    a.nrb = (out[nout - 1].row0 + out[nout - 1].rows + kTileRows - 1) / kTileRows;
    switch ((m + 7) / 8) {
        case 1: return launch<1>(a, stream);
        case 2: return launch<2>(a, stream);
        case 3: return launch<3>(a, stream);
        default: return launch<4>(a, stream);
    }
}

// Where the lines lie.  A CTA here walks its share of the scale groups, one after the other (0.35 us each beside 3 us a launch for
// 8 rows, 0.42 for 16): the time is steps = groups / split x rounds of CTAs, and the split falls from eight to one as the rows grow past
// 2368, 4736 and 9472.  The GEMV and the tcgen05 kernel divide their work more evenly.  us among launches of the same kind, weights
// larger than L2, other / here:
//   m = 1..3: one GEMV pass is as quick (2048 x 2048, m = 3: 5.6 / 3.2; 14336 x 4096: 7.9 / 12.5), and its block fixed point answers
//     a non-finite activation with NaN in every output
//   m = 4, one GEMV pass: with four or more CTAs a tile 4096 x 2048 5.7 / 3.9, 4096 x 8192 9.1 / 8.2, 4096 x 14336 13.9 / 12.9; with
//     fewer up to eight steps 8192 x 2048 5.5 / 5.2, 16384 x 1024 4.7 / 4.2, behind them 6144 x 4096 7.2 / 7.6, 8192 x 14336
//     17.1 / 22.9, 14336 x 14336 21.8 / 42.0; longer rows than 20480 leave the GEMV passes of two vectors: 8192 x 24576 64 / 37
//   m = 5..8, two GEMV passes: two or more CTAs a tile 8192 x 4096 14.2 / 8.3, 8192 x 14336 31.9 / 23.2; one and up to 32 steps 16384 x
//     4096 17.0 / 13.6; more: 10240 x 6144, m = 5 16.6 / 18.3; 28672 x 4096, m = 8 21.3 / 24.3
//   m = 9..16, tcgen05: eight CTAs a tile 2048 x 28672 18.1 / 15.9; two or four up to 16 steps 8192 x 4096 10.8 / 9.7, 4096 x 8192 11.3 /
//     9.8; more 3072 x 14336 13.5 / 14.6, 3072 x 28672 21.4 / 26.3; one up to 8 steps 16384 x 1024 6.1 / 5.1, 16 steps 10240 x 2048
//     8.0 / 8.4
//   m = 17..24: eight CTAs a tile, or up to 8 steps in two: 4096 x 4096 9.0 / 8.0; 4096 x 8192 11.8 / 12.1
//   m = 25..32: up to 8 steps in four: 2048 x 2048 6.6 / 6.5; 6144 x 4096 10.7 / 13.9
bool linear_takes_rows(int m, int rows, int cols)
{
    if (m < 4 || m > kRowsMax) return false;
    const int slots = cta_slots(), groups = cols / kGroup, per = Shape<1, kRowWarps, kGroupWarps>::kRows, tiles = (rows + per - 1) / per;
    if (!slots || !groups) return false;
    const int split = split_of(tiles, groups, slots);
    const long long rounds = ((long long)tiles * split + slots - 1) / slots, steps = (groups + split - 1) / split * rounds;
    if (m == 4) return split >= 4 || steps <= 8 || cols > 20480;
    if (m <= 8) return split >= 2 || steps <= 32 || cols > 20480;
    if (m <= 16) return split == 8 || steps <= (split > 1 ? 16 : 8);
    if (m <= 24) return split == 8 || (split > 1 && steps <= 8);
    return split >= 4 && steps <= 8;
}

// Matrices packed back to back on this kernel or the tcgen05 GEMM (m > 8, or where this one is taken).
int launch_linear_out(const uint8_t* packed, const half* x, const RowsOut* out, int nout, int m, int cols, cudaStream_t stream)
{
    if (linear_takes_rows(m, out[nout - 1].row0 + out[nout - 1].rows, cols)) return launch_gemm_rows(packed, x, out, nout, m, cols, stream);
    return launch_gemm_tcgen05(x, packed, out, nout, m, cols, stream);
}

int launch_linear_f16(const uint8_t* packed, const half* x, half* y, int m, int rows, int cols, cudaStream_t stream)
{
    const RowsOut out = {y, 0, rows};
    if (m > 8 || linear_takes_rows(m, rows, cols)) return launch_linear_out(packed, x, &out, 1, m, cols, stream);
    return launch_gemv_packed(packed, x, y, m, rows, cols, stream);
}

}  // namespace tllm
