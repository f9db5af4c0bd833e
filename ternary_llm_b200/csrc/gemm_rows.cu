// Products of a few activation rows (4..32; one in a decode step) with a ternary matrix, C[M, N] = A[M, K] . W^T.
//
// Bound: the weight stream and, at these sizes, the latencies of a launch.  A tcgen05 tile of 128
// features walks its weights through tensor memory one scale group at a time, a chain of about a
// microsecond per group that a decode batch cannot fill; here every warp expands its own weights
// into mma.sync.m16n8k16 operand registers, so that all SMs stream at once and no step waits for
// another warp.  A code is exact in FP16 and its scale joins the group's sum in FP32: FP16 products with FP32
// sums, as in the tcgen05 kernel (gemm_tcgen05.cu), whose weights carry their scale.
//
//   * A CTA owns RG * R row blocks of 16 features and a range of scale groups; warp (rg, kw) takes R
//     row blocks and every KW-th group.  A lane's 16 bytes of codes per (row block, group) are four
//     whole A fragments' worth: the byte j, field f of a word is column 32f + 16*j2 + 4t + j
//     (packed_layout.cuh), so MMA (f, j2) contracts sixteen neighbouring columns with the columns
//     4t..4t+3 in lane t's four slots, and the B fragment is one 8-byte piece of an activation row.
//   * Codes and scales go from global memory into registers, D groups ahead, and the first D are
//     requested before the wait on the previous kernel.
//   * A code becomes -1, 0 or +1 in FP16 by one logical and one FP16 instruction for two weights (code_f16),
//     without the scale: the group's sums are multiplied by it in FP32 when they join the others.  (As a byte table
//     of -s, 0, +s, ten instructions of the slower integer pipe for eight weights instead of five, the pipe was the
//     bound: 4096 x 14336, four rows, 12.7 us; 9.6 here = 1.6 TB/s of weights.)
//   * Activations pass through shared memory in stages of KW groups, cp.async, three stages; rows are
//     padded by 32 bytes so that a fragment load touches every bank once.
//   * The KW partial sums of a CTA meet in shared memory.  Where there are too few row blocks for the
//     SMs, a cluster of C CTAs splits the groups; a CTA sends its sums to the CTAs that finish them, one barrier
//     of the cluster later they are added in rank order.
#include <climits>

#include "launch.cuh"
#include "layer.cuh"
#include "packed_layout.cuh"

namespace tllm {

namespace {

constexpr int kThreads = 256;
constexpr int kStages = 3;
constexpr int kRowWarps = 2, kGroupWarps = 4;        // RG and KW

// A cluster's CTAs along x, the tiles along y and, where they are more than a grid may be high, z: of the few that this is too many
// nothing is stored.
dim3 grid_of(int split, int tiles)
{
    const int nz = (tiles + 65534) / 65535;
    return dim3(split, (tiles + nz - 1) / nz, nz);
}

struct RowsArgs {
    const uint8_t* packed;
    const half* x;                           // [m, cols]
    RowsOut out[TLLM_MAX_FUSED];             // row ranges of the matrix and where they go; unused ones start past every row
    int m, cols, groups, nrb;
    int split, share;                        // CTAs that share a tile's groups; features that one of them finishes, at most
    uint32_t over_split, over_share;         // 2^32 over the two, rounded up: the upper word of a product with it is a quotient
};

__device__ __forceinline__ uint32_t sm32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}
// Two codes of 0, 1, 2 in the field f of a word's halves as the FP16 numbers -1, 0, +1: placed in the mantissa of 1024 they are
// 1024 + 4^f c, from which one multiplication and addition without rounding makes c - 1.
template <int SHIFT>
__device__ __forceinline__ uint32_t code_f16(uint32_t w, int f)
{
    uint32_t v;                                              // one instruction for and, or: the compiler makes two of the constants
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(w >> SHIFT), "r"(0x00030003u << (2 * f)), "r"(0x64006400u));
    const float m = 1.0f / (float)(1 << (2 * f));
    const half2 r = __hfma2(*reinterpret_cast<const half2*>(&v), __float2half2_rn(m), __float2half2_rn(-1024.0f * m - 1.0f));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
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
    static constexpr int kAhead = NB == 4 ? 2 : 3;                   // groups per warp whose weights are in flight (registers)
    static constexpr int kRows = RG * kR * kTileRows;                // features per CTA
    static constexpr int kLd = KW * kGroup + 16;                     // halves per staged activation row
    static constexpr int kStage = NB * 8 * kLd;                      // halves per stage
    static constexpr int kLdRed = kRows + 4;                         // floats per vector of the partial sums
    static constexpr size_t kX = (size_t)kStages * kStage * sizeof(half);
    static constexpr size_t kRed = (size_t)KW * NB * 8 * kLdRed * sizeof(float);
    static constexpr size_t kMain = kX > kRed ? kX : kRed;
    static constexpr size_t kSmem = kMain + (size_t)NB * 8 * (kRows + 8) * sizeof(float);   // and what the cluster's CTAs send

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
    if (a.split > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3;
    const int kw = warp % KW, rg = warp / KW;
    const int rank = blockIdx.x, tile = blockIdx.z * gridDim.y + blockIdx.y;
    const int g0 = a.split > 1 ? __umulhi(rank * a.groups, a.over_split) : 0;
    const int ng = (a.split > 1 ? __umulhi((rank + 1) * a.groups, a.over_split) : a.groups) - g0;
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
    // a thread's piece (8 columns) of every fourth row; what lies behind the rows and the groups is left as it is, its sums go nowhere
    constexpr int kPieces = KW * kGroup / 8, kPass = kThreads / kPieces;
    static_assert(kThreads % kPieces == 0 && kPass == 4, "whole rows");
    const int piece = tid % kPieces, n0 = tid / kPieces;
    const half* src = a.x + (size_t)n0 * a.cols + g0 * kGroup + piece * 8;
    int left = ng * kGroup - piece * 8;                  // columns from this piece on
    const uint32_t dst0 = sm32(xs) + (uint32_t)(n0 * S::kLd + piece * 8) * 2;
    uint32_t slot = 0;
    const size_t pass = (size_t)kPass * a.cols;
    auto stage = [&]() {
        if (left > 0) {
            const half* p = src;
#pragma unroll
            for (int u = 0; u < NB * 8 / kPass; u++, p += pass)
                if (n0 + u * kPass < a.m) copy16(dst0 + slot + u * (kPass * S::kLd * 2), p);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        src += KW * kGroup;
        left -= KW * kGroup;
        slot = slot == (kStages - 1) * S::kStage * 2 ? 0 : slot + S::kStage * 2;
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; i++) stage();

    int at = 0;                                          // of stage i in shared memory
    for (int i0 = 0; i0 < nst; i0 += kAhead) {
#pragma unroll
        for (int d = 0; d < kAhead; d++) {
            const int i = i0 + d;
            if (i >= nst) break;
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            __syncthreads();                             // stage i is here, stage i - 1 is free
            stage();
            if (i < mine) {
                const half* xr = xs + at + gq * S::kLd + kw * kGroup + 4 * t;
                float sum[R][NB][4];
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int n = 0; n < NB; n++)
#pragma unroll
                        for (int e = 0; e < 4; e++) sum[r][n][e] = 0.f;
                // bytes 0, 2, 1, 3: columns 4t, 4t + 1 at the same bits of a word's halves, 4t + 2 and 4t + 3 eight bits above
                uint32_t w[R][4];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    w[r][0] = prmt(cw[d][r].x, 0, 0x3120);
                    w[r][1] = prmt(cw[d][r].y, 0, 0x3120);
                    w[r][2] = prmt(cw[d][r].z, 0, 0x3120);
                    w[r][3] = prmt(cw[d][r].w, 0, 0x3120);
                }
#pragma unroll
                for (int j2 = 0; j2 < 2; j2++)
#pragma unroll
                    for (int f = 0; f < 4; f++) {
                        uint2 b[NB];
#pragma unroll
                        for (int n = 0; n < NB; n++) b[n] = *reinterpret_cast<const uint2*>(xr + n * 8 * S::kLd + 32 * f + 16 * j2);
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            const uint32_t fr[4] = {code_f16<0>(w[r][j2], f), code_f16<0>(w[r][2 + j2], f), code_f16<8>(w[r][j2], f),
                                                    code_f16<8>(w[r][2 + j2], f)};
#pragma unroll
                            for (int n = 0; n < NB; n++) mma_f16(sum[r][n], fr, b[n].x, b[n].y);
                        }
                    }
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float2 sc = __half22float2(*reinterpret_cast<const half2*>(&sw[d][r]));     // rows gq, gq + 8
#pragma unroll
                    for (int n = 0; n < NB; n++)
#pragma unroll
                        for (int e = 0; e < 4; e++) acc[r][n][e] = fmaf(e < 2 ? sc.x : sc.y, sum[r][n][e], acc[r][n][e]);
                }
            }
            load(i + kAhead, cw[d], sw[d]);
            at = at == (kStages - 1) * S::kStage ? 0 : at + S::kStage;
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
    const int row0 = tile * S::kRows;
    auto store = [&](int n, int r, float v) {
        const int row = row0 + r;
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
    // CTA z of the cluster finishes the features f of all rows with f * split / kRows == z: from first(z) on
    float* sent = reinterpret_cast<float*>(smem_raw + S::kMain);      // [CTA of the cluster][row][feature of the share]
    auto first = [&](int z) { return (int)__umulhi(z * S::kRows + a.split - 1, a.over_split); };
    if (a.split > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");       // all of them run
    const int share = a.share;
    static_assert(kThreads % S::kRows == 0, "a thread's feature is the same in every pass");
    const int row = tid % S::kRows, to = row * a.split / S::kRows;
    uint32_t peer = 0;
    if (a.split > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(sm32(sent + rank * (NB * 8) * share + row - first(to))), "r"(to));
    for (int n = tid / S::kRows; n < a.m; n += kThreads / S::kRows) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < KW; k++) v += red[((size_t)k * NB * 8 + n) * S::kLdRed + row];
        if (a.split == 1) store(n, row, v);
        else asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer + n * share * 4), "f"(v) : "memory");
    }
    if (a.split > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int f0 = first(rank), mine_f = first(rank + 1) - f0;
        for (int e = tid; e < a.m * share; e += kThreads) {
            const int n = __umulhi(e, a.over_share), f = e - n * share;
            if (f >= mine_f) continue;
            float v = 0.f;
            for (int z = 0; z < a.split; z++) v += sent[z * (NB * 8) * share + e];
            store(n, f0 + f, v);
        }
    }
}

constexpr int kMaxSplit = 8;
// ---- one vector ---------------------------------------------------------------------------------
// A decode step's products of one vector on the same codes and cuts.  The whole share of the vector lies in shared memory before the
// first group, made there from what the step has (RowInput), so that there is no barrier between the groups and no launch for a norm
// or a SwiGLU; all lanes of a quarter read the same activations, and the MMA's eight columns are the same.
struct OneArgs {
    const uint8_t* packed;
    RowVector x;
    half* y;
    int rows, cols, groups, nrb, split, share;
    uint32_t over_split;
};

constexpr int kOneAhead = 4;
constexpr size_t kOneSmem = 40 * 1024;                 // shared memory that needs no attribute

template <int INPUT>
__global__ void __launch_bounds__(kThreads, 2)
gemm_row_kernel(const OneArgs a)
{
    constexpr int R = 2, RG = kRowWarps, KW = kGroupWarps, kRows = RG * R * kTileRows;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    half* xs = reinterpret_cast<half*>(smem_raw);        // the vector (kRowNorm), or its share
    __shared__ float red[KW][kRows], sent[kMaxSplit * kRows], sums[kThreads / 32];
    pdl_launch_dependents();
    if (a.split > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3;
    const int kw = warp % KW, rg = warp / KW;
    const int rank = blockIdx.x, tile = blockIdx.z * gridDim.y + blockIdx.y;
    const int g0 = a.split > 1 ? __umulhi(rank * a.groups, a.over_split) : 0;
    const int ng = (a.split > 1 ? __umulhi((rank + 1) * a.groups, a.over_split) : a.groups) - g0;
    const int mine = (ng - kw + KW - 1) / KW;
    const int rb0 = (tile * RG + rg) * R;

    const uint8_t* wp[R];
#pragma unroll
    for (int r = 0; r < R; r++)      // row blocks past the matrix repeat the last one and are not stored
        wp[r] = a.packed + ((size_t)min(rb0 + r, a.nrb - 1) * a.groups + g0 + kw) * kTileBytes;
    uint4 cw[kOneAhead][R];
    uint32_t sw[kOneAhead][R];
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
    for (int d = 0; d < kOneAhead; d++) load(d, cw[d], sw[d]);

    pdl_wait();
    const uint4 *xa = reinterpret_cast<const uint4*>(a.x.a), *xb = reinterpret_cast<const uint4*>(a.x.b);
    uint4* x8 = reinterpret_cast<uint4*>(xs);
    const half* mine_x = xs;                             // of the first group
    if (INPUT == kRowNorm) {
        // the arithmetic of the norm operator: sum rounded to FP16, mean of squares and scaling in FP32, one rounding of the result
        const int n8 = a.cols >> 3;
        const bool keeps = a.x.res_out && rank == 0 && tile == 0;
        float ss = 0.f;
        for (int i = tid; i < n8; i += kThreads) {
            uint4 v = xa[i];
            half* vh = reinterpret_cast<half*>(&v);
            if (xb) {
                const uint4 br = xb[i];
                const half* bh = reinterpret_cast<const half*>(&br);
#pragma unroll
                for (int j = 0; j < 8; j++) vh[j] = __float2half_rn(__half2float(vh[j]) + __half2float(bh[j]));
                if (keeps) reinterpret_cast<uint4*>(a.x.res_out)[i] = v;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float f = __half2float(vh[j]);
                ss += f * f;
            }
            x8[i] = v;
        }
        ss = warp_sum(ss);
        if (lane == 0) sums[warp] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int i = 0; i < kThreads / 32; i++) ss += sums[i];
        const float rinv = rsqrtf(ss / (float)a.cols + a.x.eps);
        for (int i = tid; i < n8; i += kThreads) {
            uint4 v = x8[i];
            const uint4 wr = reinterpret_cast<const uint4*>(a.x.w)[i];
            half* vh = reinterpret_cast<half*>(&v);
            const half* wh = reinterpret_cast<const half*>(&wr);
#pragma unroll
            for (int j = 0; j < 8; j++) vh[j] = __float2half_rn(__half2float(vh[j]) * rinv * __half2float(wh[j]));
            x8[i] = v;
        }
        mine_x += g0 * kGroup;
    } else {
        const int first = g0 * (kGroup / 8), n8 = ng * (kGroup / 8);
        for (int i = tid; i < n8; i += kThreads) {
            uint4 v = xa[first + i];
            if (INPUT == kRowSilu) {
                const uint4 ur = xb[first + i];
                half* vh = reinterpret_cast<half*>(&v);
                const half* uh = reinterpret_cast<const half*>(&ur);
#pragma unroll
                for (int j = 0; j < 8; j++) vh[j] = __float2half_rn(silu_mul(__half2float(vh[j]), __half2float(uh[j])));
            }
            x8[i] = v;
        }
    }
    __syncthreads();

    float acc[R][2] = {};                                // rows gq, gq + 8
    for (int i0 = 0; i0 < mine; i0 += kOneAhead) {
#pragma unroll
        for (int d = 0; d < kOneAhead; d++) {
            const int i = i0 + d;
            if (i >= mine) break;
            const half* xr = mine_x + (i * KW + kw) * kGroup + 4 * t;
            float sum[R][2][4] = {};                     // two chains of MMAs
            uint32_t w[R][4];
#pragma unroll
            for (int r = 0; r < R; r++) {
                w[r][0] = prmt(cw[d][r].x, 0, 0x3120);
                w[r][1] = prmt(cw[d][r].y, 0, 0x3120);
                w[r][2] = prmt(cw[d][r].z, 0, 0x3120);
                w[r][3] = prmt(cw[d][r].w, 0, 0x3120);
            }
#pragma unroll
            for (int f = 0; f < 4; f++)
#pragma unroll
                for (int j2 = 0; j2 < 2; j2++) {
                    const uint2 b = *reinterpret_cast<const uint2*>(xr + 32 * f + 16 * j2);
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const uint32_t fr[4] = {code_f16<0>(w[r][j2], f), code_f16<0>(w[r][2 + j2], f), code_f16<8>(w[r][j2], f),
                                                code_f16<8>(w[r][2 + j2], f)};
                        mma_f16(sum[r][j2], fr, b.x, b.y);
                    }
                }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float2 sc = __half22float2(*reinterpret_cast<const half2*>(&sw[d][r]));
                acc[r][0] = fmaf(sc.x, sum[r][0][0] + sum[r][1][0], acc[r][0]);
                acc[r][1] = fmaf(sc.y, sum[r][0][2] + sum[r][1][2], acc[r][1]);
            }
            load(i + kOneAhead, cw[d], sw[d]);
        }
    }
    if (t == 0)
#pragma unroll
        for (int r = 0; r < R; r++) {
            red[kw][(rg * R + r) * kTileRows + gq] = acc[r][0];
            red[kw][(rg * R + r) * kTileRows + gq + 8] = acc[r][1];
        }
    __syncthreads();
    const int row0 = tile * kRows;
    auto first = [&](int z) { return (int)__umulhi(z * kRows + a.split - 1, a.over_split); };
    if (a.split > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");       // all of them run
    if (tid < kRows) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < KW; k++) v += red[k][tid];
        if (a.split == 1) {
            if (row0 + tid < a.rows) a.y[row0 + tid] = __float2half_rn(v);
        } else {
            const int to = tid * a.split / kRows;
            uint32_t peer;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(sm32(sent + rank * a.share + tid - first(to))), "r"(to));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer), "f"(v) : "memory");
        }
    }
    if (a.split > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int f0 = first(rank);
        if (tid < first(rank + 1) - f0 && row0 + f0 + tid < a.rows) {
            float v = 0.f;
            for (int z = 0; z < a.split; z++) v += sent[z * a.share + tid];
            a.y[row0 + f0 + tid] = __float2half_rn(v);
        }
    }
}


// How a product is cut: tiles, CTAs that share the scale groups of one, rounds of CTAs, and the groups that one of them walks in all rounds.
struct Cut {
    int tiles = 0, split = 0, rounds = 0, steps = 0;
};

// CTAs of a kernel that run at once in clusters of one to kMaxSplit: slots[cluster size], asked once per device.  Clusters come in
// GPCs, so fewer run at once the larger the cluster.
template <typename... KArgs>
int fill_slots(void (*kernel)(KArgs...), size_t smem, int (&slots)[64][kMaxSplit + 1], int* dev)
{
    if (cudaGetDevice(dev) != cudaSuccess || *dev < 0 || *dev >= 64) return fail(TLLM_ERR_LAUNCH, "gemm_rows: no current device");
    if (slots[*dev][1]) return TLLM_OK;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return fail(TLLM_ERR_LAUNCH, "gemm_rows: no current device");
    }
    prefer_max_shared(reinterpret_cast<const void*>(kernel));
    for (int split = kMaxSplit; split >= 1; split--) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = split;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(split * 1024);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            return fail(TLLM_ERR_LAUNCH, "gemm_rows: clusters of %d do not run", split);
        }
        slots[*dev][split] = n * split;
    }
    return TLLM_OK;
}

// A second round of clusters costs more than a split saves.  Among the splits that run at once, the fewest stages of kGroupWarps groups,
// of which the exchange in a cluster takes as long as one and a half (1024 x 1024: one CTA and two stages 2.3 us, two CTAs and one 2.7; 512 x
// 2048: two and two 3.1, four and one 2.6; 8192 x 2048: one and four 5.2, two and two 4.1), then the fewest CTAs.
constexpr int kCutRows = kRowWarps * 2 * kTileRows;      // features of a tile
void choose_cut(const int (&slots)[kMaxSplit + 1], int rows, int groups, Cut* c)
{
    const int tiles = (rows + kCutRows - 1) / kCutRows;
    int best = INT_MAX;
    for (int split = 1; split <= kMaxSplit; split++) {
        if (split > 1 && (tiles * split > slots[split] || groups < split * kGroupWarps)) continue;
        const int per = (groups + split - 1) / split, cost = 2 * ((per + kGroupWarps - 1) / kGroupWarps) + (split > 1 ? 3 : 0);
        if (cost >= best) continue;
        best = cost;
        c->tiles = tiles;
        c->split = split;
        c->rounds = (tiles * split + slots[split] - 1) / slots[split];
        c->steps = per * c->rounds;
    }
}

template <int NB>
int cut(int rows, int groups, Cut* c)
{
    using S = Shape<NB, kRowWarps, kGroupWarps>;
    static_assert(S::kRows == kCutRows, "one cut for all numbers of rows");
    static int slots[64][kMaxSplit + 1] = {};
    int dev = 0;
    const int st = fill_slots(gemm_rows_kernel<NB, kRowWarps, kGroupWarps>, S::kSmem, slots, &dev);
    if (!st) choose_cut(slots[dev], rows, groups, c);
    return st;
}
// Of the kernel for one vector, whatever part of its shared memory a launch takes.
template <int INPUT>
int cut_one(int rows, int groups, Cut* c)
{
    static int slots[64][kMaxSplit + 1] = {};
    int dev = 0;
    const int st = fill_slots(gemm_row_kernel<INPUT>, kOneSmem, slots, &dev);
    if (!st) choose_cut(slots[dev], rows, groups, c);
    return st;
}
int cut_for(int m, int rows, int groups, Cut* c)
{
    switch ((m + 7) / 8) {
        case 1: return cut<1>(rows, groups, c);
        case 2: return cut<2>(rows, groups, c);
        case 3: return cut<3>(rows, groups, c);
        default: return cut<4>(rows, groups, c);
    }
}

template <int NB>
int launch(RowsArgs a, cudaStream_t stream)
{
    using S = Shape<NB, kRowWarps, kGroupWarps>;
    Cut c;
    const int st = cut<NB>(a.nrb * kTileRows, a.groups, &c);
    if (st) return st;
    a.split = c.split;
    a.share = (S::kRows + a.split - 1) / a.split;
    a.over_split = (uint32_t)((0x100000000ull + a.split - 1) / a.split);         // of one CTA not used
    a.over_share = (uint32_t)((0x100000000ull + a.share - 1) / a.share);
    const int tiles = (a.nrb * kTileRows + S::kRows - 1) / S::kRows;
    return launch_pdl_cluster("gemm_rows", gemm_rows_kernel<NB, kRowWarps, kGroupWarps>, a.split, grid_of(a.split, tiles), dim3(kThreads),
                              S::kSmem, stream, a);
}

template <int INPUT>
int launch_one(OneArgs a, cudaStream_t stream)
{
    using S = Shape<1, kRowWarps, kGroupWarps>;
    Cut c;
    const int st = cut_one<INPUT>(a.rows, a.groups, &c);
    if (st) return st;
    a.split = c.split;
    a.share = (S::kRows + a.split - 1) / a.split;
    a.over_split = (uint32_t)((0x100000000ull + a.split - 1) / a.split);         // of one CTA not used
    const int per = (a.groups + a.split - 1) / a.split;
    const size_t smem = (size_t)(INPUT == kRowNorm ? a.cols : per * kGroup) * sizeof(half);
    if (smem > kOneSmem) return fail(TLLM_ERR_SHAPE, "gemm_row: %d columns", a.cols);
    const int tiles = (a.rows + S::kRows - 1) / S::kRows;
    return launch_pdl_cluster("gemm_row", gemm_row_kernel<INPUT>, a.split, grid_of(a.split, tiles), dim3(kThreads), smem, stream, a);
}

}  // namespace

// us in the chain of a step, streaming GEMV (SwiGLU's launch included) / here: plain 1024 x 1024 3.3 / 2.0, 2048 x 2048 4.1 / 3.0, 4096 x
// 4096 5.4 / 3.6, 8192 x 8192 11.2 / 9.0; SwiGLU 2048 x 8192 6.6 / 4.4, 4096 x 14336 11.8 / 9.2, 8192 x 28672 30.9 / 29.4; norm 3072 x 2048
// 5.5 / 3.9, 16384 x 2048 7.2 / 6.1, 12288 x 4096 (32 steps) 9.3 / 9.3, 10240 x 8192 (64) 16.1 / 16.5, 28672 x 4096 (64) 15.7 / 18.2.
bool row_supported(RowInput input, int rows, int cols)
{
    Cut c;
    const int groups = cols / kGroup;
    if (!groups) return false;
    if (input == kRowNorm ? cut_one<kRowNorm>(rows, groups, &c) : input == kRowSilu ? cut_one<kRowSilu>(rows, groups, &c) : cut_one<kRowPlain>(rows, groups, &c))
        return false;
    return (size_t)(input == kRowNorm ? cols : (groups + c.split - 1) / c.split * kGroup) * sizeof(half) <= kOneSmem &&
           (input != kRowNorm || c.steps <= 32);
}

int launch_gemm_row(const uint8_t* packed, RowInput input, const RowVector& x, half* y, int rows, int cols, cudaStream_t stream)
{
    OneArgs a = {};
    a.packed = packed;
    a.x = x;
    a.y = y;
    a.rows = rows;
    a.cols = cols;
    a.groups = cols / kGroup;
    a.nrb = (rows + kTileRows - 1) / kTileRows;
    switch (input) {
        case kRowNorm: return launch_one<kRowNorm>(a, stream);
        case kRowSilu: return launch_one<kRowSilu>(a, stream);
        default: return launch_one<kRowPlain>(a, stream);
    }
}

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

// Where the lines lie.  A CTA here walks its share of the scale groups in stages of four (0.9 us for 8 rows, 1.2 for 16, 1.8 for 24, two CTAs
// on an SM) beside 2.5 us a launch; the split falls from eight to one as the rows grow past 2112, 4544 and 9472.  The GEMV and the
// tcgen05 kernel divide their work more evenly.  us among launches of the same kind, weights larger than L2, other / here:
//   m = 1..3: one GEMV pass is as quick (14336 x 4096: 7.9 / 10), and its block fixed point answers a non-finite activation
//     with NaN in every output
//   m = 4, one GEMV pass: 4096 x 2048 5.7 / 3.0, 4096 x 14336 13.9 / 9.6, 6144 x 4096 7.0 / 6.0, 16384 x 2048 6.7 / 5.8, 16384 x 3072 (24
//     steps) 7.8 / 7.9, 14336 x 4096 (32) 8.4 / 10.2, 8192 x 14336 (56) 16.9 / 17.3; longer rows than 20480 leave the GEMV passes of two
//     vectors: 8192 x 24576 64 / 37 before these figures
//   m = 5..8, two GEMV passes: quicker everywhere, 512 x 2048 9.6 / 2.6, 28672 x 4096 22.1 / 19.8, 14336 x 14336 41 / 33
//   m = 9..16, tcgen05: 2048 x 14336 11.7 / 8.2, 8192 x 14336 (two CTAs, 56 steps) 25.1 / 22.8, 14336 x 4096 (one, 32) 13.7 / 13.1 - 13.4, 28672
//     x 4096 (one, 64) 24.0 / 24.1 - 25.3.  Of one CTA a tile one round of them: m = 10, 29209 x 256 (457 tiles) 4.4 / 5.5, m = 9, 26384 x 640 (413)
//     5.7 / 6.7, m = 11, 14672 x 512 (230) 4.3 / 3.5.  Above 12 up to 10 steps and up to 74 tiles, or more than one an SM: m = 16, 5648 x 640
//     (89) 3.8 / 4.4, m = 14, 8496 x 768 (133) 4.1 / 4.6, m = 16, 13744 x 512 (215) 4.2 / 3.8
//   m = 17..24: 2048 x 14336 12.0 / 10.3, 4096 x 14336 (four CTAs, 28 steps) 16.0 / 15.1 - 16.0, 8192 x 2048 (two, 8) 7.2 / 6.8, 6144 x 4096
//     (two, 16) 10.4 / 10.1 - 10.7, 4600 x 8192 (three, 22) 12.9 / 13.3 - 14.2.  One CTA a tile where tiles are few and no stage has a single
//     group: m = 20, 2769 x 1024 (44 tiles, 8 steps) 4.7 / 3.9, m = 19, 528 x 768 (6 steps) 4.0 / 3.8, m = 24, 603 x 640 (5) 3.7 / 4.0, m = 22, 464 x 256
//     (2) 2.8 / 3.2, m = 24, 5440 x 256 (85 tiles) 3.1 / 4.1
//   m = 25..32, up to 8 steps: 2048 x 8192 (eight CTAs) 9.3 / 8.6, 4096 x 4096 (four) 8.9 / 7.4 - 7.8, of three CTAs up to 34 tiles: m = 32, 1392 x 2432 (22)
//     6.1 / 6.0, m = 30, 2768 x 2176 (44) 6.6 / 7.5, m = 29, 5904 x 2560 (93) 8.5 / 11.3.  Up to 12 steps where tiles are few: m = 27, 362 x 10240 (6)
//     7.3 / 6.4, m = 28, 3511 x 6272 (55) 10.1 / 13.0
bool linear_takes_rows(int m, int rows, int cols)
{
    if (m < 4 || m > kRowsMax) return false;
    const int groups = cols / kGroup;
    Cut c;
    if (!groups || cut_for(m, rows, groups, &c)) return false;
    const int split = c.split, steps = c.steps;
    if (m == 4) return split >= 4 || steps <= 20 || cols > 20480;
    if (m <= 8) return true;
    if (m <= 12) return split > 1 || (c.rounds == 1 && steps <= 32);
    if (m <= 16) return split > 1 || (c.rounds == 1 && steps <= 10 && (c.tiles <= 74 || c.tiles > 148));
    if (m <= 24)
        return split >= 7 || (split >= 4 && steps <= 28) || (split > 1 && steps <= 8) ||
               (split == 1 && steps >= 3 && steps <= 8 && steps % kGroupWarps != 1 && c.tiles <= 60);
    return (steps <= 8 && (split >= 4 || (split == 3 && c.tiles <= 34))) || (steps <= 12 && split >= 3 && c.tiles <= 13);
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
