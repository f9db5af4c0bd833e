// Products of up to 32 activation rows with a dense FP16 matrix, y[M, rows] = x[M, cols] . W^T: the
// FP16 output head of a decode step, alone or for a batch of sequences.
//
// Bound: the stream of W from HBM.  On the CUDA cores eight rows already take more multiply-adds than
// the stream leaves time for; here W enters mma.sync.m16n8k16 as it lies in memory and the products
// cost a few per cent of the tensor pipe.
//
//   * A warp takes blocks of 16 rows of W, all columns, one block after the other.  Per window of 128 columns
//     a lane loads 16 bytes at four places of two rows (64 contiguous bytes a row and load); a contraction
//     may take its columns in any order, so the eight halves are slots of two MMAs as they come: MMA
//     (q, j) contracts, in lane t, the columns 32q + 8t + 4j .. + 3, and the B fragment is the 8-byte piece
//     of an activation row at the same place.
//   * Two windows per warp are in flight (8 KB, 128 KB per SM), across the ends of blocks; none is
//     requested before the wait on the previous kernel, which may be the one that makes W.  Loads in flight
//     need room in the L1 cache, so this kernel asks for no more shared memory than its activations need: with
//     the largest part, as its neighbours ask for it, about 25 KB of L1 remain and the stream stops at 3.7 TB/s
//     whatever else is done.
//   * The tensor cores cut their sums instead of rounding them, always towards zero: a window's sum is eight MMAs
//     long, and the windows are added in FP32 (one accumulator for 14336 columns of positive products was 2.17e-4
//     off in place of the CUDA cores' 1.96e-4, the rounding of the result included).
//   * All activations lie in shared memory, so that no warp waits for another one.  Rows are padded by 64
//     bytes: a fragment load touches every bank once.  Activations that do not fit are taken in as many
//     passes as they need.
//
// 128256 x 2048 (525 MB), us on the CUDA cores -> here: one row among launches of the same kind 107 -> 88 (6.0 TB/s); behind one layer of a
// decoder (26 of them): one row 134 -> 108, 8: 350 -> 112, 24: 982 -> 121.
#include "launch.cuh"
#include "layer.cuh"

namespace tllm {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBlock = 16;                           // rows of W per block
constexpr int kWin = 128;                            // columns per window
constexpr int kPad = 32;                             // halves behind a staged activation row
constexpr size_t kMaxSmem = 226 * 1024;

struct Args {
    const half* w;                                   // [rows, cols]
    const half* x;                                   // [m, cols]
    half* y;                                         // [m, rows]
    int m, rows, cols;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg_stream(const half* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <int NB>
__global__ void __launch_bounds__(kThreads, 1)
fp16_rows_kernel(const Args a)
{
    extern __shared__ __align__(16) half xs[];       // [NB * 8][cols + kPad]
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3;
    const int ld = a.cols + kPad, nwin = a.cols / kWin, nblk = (a.rows + kBlock - 1) / kBlock;
    const int nw = gridDim.x * kWarps;
    // place of the next load: window lw of block lb; rows past the matrix repeat the last one and are not stored
    int lb = blockIdx.x + gridDim.x * warp, lw = 0;
    const half *w0 = nullptr, *w1 = nullptr;
    auto at_block = [&]() {
        w0 = a.w + (size_t)min(lb * kBlock + gq, a.rows - 1) * a.cols + 8 * t;
        w1 = a.w + (size_t)min(lb * kBlock + gq + 8, a.rows - 1) * a.cols + 8 * t;
    };
    uint4 wr[2][2][4];
    auto load = [&](uint4 (&v)[2][4]) {
        if (lb < nblk) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                v[0][q] = ldg_stream(w0 + lw * kWin + 32 * q);
                v[1][q] = ldg_stream(w1 + lw * kWin + 32 * q);
            }
            if (++lw == nwin) {
                lw = 0;
                lb += nw;
                at_block();
            }
        }
    };
    int cb = lb, cw = 0;                             // the window whose turn it is
    at_block();
    pdl_wait();
    load(wr[0]);
    load(wr[1]);

    const int pieces = a.cols / 8;
    for (int n = 0; n < NB * 8; n++)
        for (int c = tid; c < pieces; c += kThreads) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs + (size_t)n * ld + c * 8);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         ::"r"(dst), "l"(n < a.m ? a.x + (size_t)n * a.cols + c * 8 : a.x), "r"(n < a.m ? 16 : 0) : "memory");
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    float acc[NB][4] = {};
    const half* xl = xs + (size_t)gq * ld + 8 * t;
    while (cb < nblk) {
#pragma unroll
        for (int d = 0; d < 2; d++) {
            if (cb >= nblk) break;
            const half* xr = xl + cw * kWin;
            float sum[NB][4] = {};                       // of the window
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint4 u = wr[d][0][q], v = wr[d][1][q];
#pragma unroll
                for (int n = 0; n < NB; n++) {
                    const uint4 b = *reinterpret_cast<const uint4*>(xr + (size_t)n * 8 * ld + 32 * q);
                    mma_f16(sum[n], u.x, v.x, u.y, v.y, b.x, b.y);
                    mma_f16(sum[n], u.z, v.z, u.w, v.w, b.z, b.w);
                }
            }
            load(wr[d]);
#pragma unroll
            for (int n = 0; n < NB; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[n][e] += sum[n][e];
            if (++cw == nwin) {
                const int r = cb * kBlock + gq;
#pragma unroll
                for (int n = 0; n < NB; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int vec = n * 8 + 2 * t + (e & 1), row = r + 8 * (e >> 1);
                        if (vec < a.m && row < a.rows) a.y[(size_t)vec * a.rows + row] = __float2half_rn(acc[n][e]);
                        acc[n][e] = 0.f;
                    }
                cw = 0;
                cb += nw;
            }
        }
    }
}

template <int NB>
int launch(const Args& a, cudaStream_t stream)
{
    static bool attr[64] = {};
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return fail(TLLM_ERR_LAUNCH, "fp16_rows: no current device");
    if (!attr[dev]) {
        cudaFuncSetAttribute(fp16_rows_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        attr[dev] = true;
    }
    const int nblk = (a.rows + kBlock - 1) / kBlock;
    const int grid = nblk < sms[dev] ? nblk : sms[dev];
    const size_t smem = (size_t)NB * 8 * (a.cols + kPad) * sizeof(half);
    const int carveout = (int)((smem + 1024) * 100 / (228 * 1024)) + 1;       // just what the activations need
    return launch_pdl_split("fp16_rows", fp16_rows_kernel<NB>, 1, carveout, dim3((unsigned)grid), dim3(kThreads), smem, stream, a);
}

// Vectors (a multiple of 8) whose activations fit in shared memory.
int vectors_per_pass(int cols)
{
    const size_t n = kMaxSmem / ((size_t)8 * (cols + kPad) * sizeof(half));
    return n >= 4 ? 32 : (int)n * 8;
}

}  // namespace

// Whole windows and 16-byte loads; the CUDA-core kernels (layer_ops.cu) take every other shape.
bool fp16_rows_supported(const half* w, const half* x, int cols)
{
    return cols >= kWin && cols % kWin == 0 && vectors_per_pass(cols) > 0 &&
           ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
}

int launch_fp16_rows(const half* w, const half* x, half* y, int m, int rows, int cols, cudaStream_t stream)
{
    const int per = vectors_per_pass(cols);
    for (int b = 0; b < m; b += per) {
        const Args a = {w, x + (size_t)b * cols, y + (size_t)b * rows, m - b < per ? m - b : per, rows, cols};
        int st;
        switch ((a.m + 7) / 8) {
            case 1: st = launch<1>(a, stream); break;
            case 2: st = launch<2>(a, stream); break;
            case 3: st = launch<3>(a, stream); break;
            default: st = launch<4>(a, stream); break;
        }
        if (st) return st;
    }
    return TLLM_OK;
}

}  // namespace tllm
