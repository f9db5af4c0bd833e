// Grouped-query attention over prompts on the 5th-generation tensor cores (head sizes 64 and 128):
// BF16 for the models of mixer layers (their other sizes run on mma.sync, grouped_attention.cu), FP16
// for the LLaMA design (its other sizes run on attention.cu).
//
// A CTA takes 128 queries of one head and walks over tiles of 128 positions that some of its queries
// sees; two CTAs share an SM, so that one's softmax runs beside the other's products.  Roles: a warp
// for the TMA copies and one for tcgen05.mma, an elected lane of each issuing, four warps with a query row per thread.
//   S = Q K^T      both operands in shared memory, 128 FP32 columns of tensor memory
//   softmax        a thread reads its row; the weights go back over S as two BF16 numbers each
//   O += P V       weights from tensor memory, values as they lie in the cache (feature-major
//                  operand); the high and the low parts are two products
// The running maximum moves only when it grows by more than 2^8 (FP16: 2^4): the sums stay far inside
// FP32, and the output in tensor memory is rescaled a few times per row at most.  FP16 weights carry a
// factor of 2^10, which the division by their sum takes out again: the largest is then between 2^10 and
// 2^14, and a weight keeps 22 bits in its two parts down to 2^-13 of the largest (below that the parts
// hold it to 2^-35 of the largest).  A position that a query does not see enters its product with the
// weight 0, which turns a NaN or an infinity among the values of such a position in the query's last tile
// into a NaN of the query.  FP16 rows that are not finite at the end are therefore computed once more, over the
// positions that they see alone (visible_row); with finite values this costs a comparison per output.
//
// FP16, 32 heads over 8 key/value heads, one launch among others, against the form with a CTA per query
// and key/value head on the CUDA cores (attention.cu), which read every position once per query: 2000
// queries 2210 -> 76 us (head size 64), 6733 -> 90 us (128); 300 queries 82 -> 12.6 and 256 -> 15.7 us.  few_queries has the calls
// that stay there.  Bound by the chain of a tile (product, softmax, product, 3.5 us), which two CTAs an SM hide in part.  Its
// longest link is the softmax, a row per thread: two scores per instruction where there is one for it and no mask but in the tiles that
// need one; with a mask in every tile and one score at a time 2000 queries took 117 and 130 us, 300 16.1 and 17.9.  The MMAs and
// copies are issued by an elected lane of a warp that runs the loop together (2000 queries 85 -> 76, 96 -> 90).
//
// Latent attention over expanded keys and values (BF16, key parts and values in pieces of 64) is the same walk with a key of two
// parts; its operands leave room for one CTA an SM.  16 heads of 128 + 64, 2000 tokens: 192 -> 75 us a launch against
// mma.sync on 64 queries (latent_attention.cu, which keeps the other sizes and up to 64 positions).  Tried: the scores read from tensor memory twice, 64 at a time,
// which leaves no spills: 75 -> 85, 90 -> 100 (FP16, 128).
// All mbarrier waits are bounded (see dense_gemm.cu).
#include <cfloat>
#include <climits>
#include <type_traits>

#include "f32x2.cuh"
#include "launch.cuh"
#include "layer.cuh"
#include "mixers.cuh"
#include "tcgen05.cuh"

namespace tllm {

namespace {

using namespace gemm;

constexpr int kTile = 128, kThreads = 192;
constexpr int kBlock = kTile * 128;                 // bytes of 64 columns of a tile: 128-byte rows
constexpr uint32_t kTmemCols = 256;                 // S and the weights: 128, O: 128
constexpr float kLog2e = 1.4426950408889634f;

template <typename T> struct Operand;
template <> struct Operand<bf16> {
    using Pair = __nv_bfloat162;
    static constexpr uint32_t kFormats = (1u << 7) | (1u << 10);
    static constexpr float kSlack = 8.f, kLift = 0.f;
    static constexpr CUtensorMapDataType kMap = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    static __device__ __forceinline__ Pair pair(float x, float y) { return __floats2bfloat162_rn(x, y); }
    static __device__ __forceinline__ float2 floats(Pair p) { return __bfloat1622float2(p); }
};
template <> struct Operand<half> {
    using Pair = half2;
    static constexpr uint32_t kFormats = 0;
    static constexpr float kSlack = 4.f, kLift = 10.f;
    static constexpr CUtensorMapDataType kMap = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    static __device__ __forceinline__ Pair pair(float x, float y) { return __floats2half2_rn(x, y); }
    static __device__ __forceinline__ float2 floats(Pair p) { return __half22float2(p); }
};

// Keys of sequence b and key/value head g lie in rows (b * kv_heads + g) * head_rows + position and
// columns g * k_cols .. of their map, values alike.
template <typename T>
struct PromptArgs {
    T* out;
    const T *q, *k, *v;                 // FP16: what the maps show, for rows that are computed once more
    int ld_out, per_kv, kv_heads, dim, vdim, n, pos0, chunk, cache_rows;
    int head_rows, k_cols, v_cols;
    float scale2, out_scale;
    int* err;
};

// Latent attention: a head's keys are dim columns of its own and rot columns that all heads share (columns shared_col .. of rows of
// ld_shared); q has rows of ld_q with dim + rot columns a head, k and v of heads * dim and heads * vdim.  The other kernels take the
// empty one, so that nothing of it is in their parameters.
template <bool LATENT> struct LatentPart {};
template <> struct LatentPart<true> {
    CUtensorMap map_r;                  // the shared columns
    const bf16* shared;
    const float* sink;                  // [heads] or null: exp(sink) joins the sum of the weights
    const bf16* gate;                   // out *= sigmoid(gate[row * gate_ld + head]), or null
    int rot, ld_q, ld_shared, shared_col, gate_ld;
};

__device__ __forceinline__ int chunk_start(int pos, int chunk) { return chunk > 0 ? pos / chunk * chunk : 0; }

template <typename T>
__device__ __forceinline__ uint32_t idesc(int n, bool feature_major)
{
    return (1u << 4) | Operand<T>::kFormats | ((feature_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);
}
// operand whose rows are the contracted index: blocks of 64 features kBlock apart, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t feature_major_desc(uint32_t addr)
{
    return (make_sw128_desc(addr) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(kBlock >> 4) << 16);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, bool acc)
{
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
        ::"r"(d), "l"(a), "l"(b), "r"(id), "r"((uint32_t)acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, bool acc)
{
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
        ::"r"(d), "r"(a), "l"(b), "r"(id), "r"((uint32_t)acc) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                 "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                 "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// One query by one warp over the positions that it sees, as attention.cu computes it.
__device__ __forceinline__ void visible_row(const PromptArgs<half>& a, int h, int g, int seq, int qi, int lane)
{
    const size_t qo = ((size_t)seq * a.n + qi) * a.ld_out + (size_t)h * a.dim, head = (size_t)(seq * a.kv_heads + g) * a.head_rows * a.dim;
    const half *kb = a.k + head, *vb = a.v + head;
    const int len = a.pos0 + qi + 1, pairs = a.dim / 64;          // channel pairs lane, lane + 32 of the output
    float m = -FLT_MAX, l = 0.f;
    float2 o[2] = {};
#pragma unroll 1
    for (int p0 = 0; p0 < len; p0 += 32) {
        const bool sees = p0 + lane < len;
        float s = 0.f;
#pragma unroll 1
        for (int d = 0; sees && d < a.dim; d += 8) {
            const uint4 x = *reinterpret_cast<const uint4*>(a.q + qo + d), y = *reinterpret_cast<const uint4*>(kb + (size_t)(p0 + lane) * a.dim + d);
            const half2 *xh = reinterpret_cast<const half2*>(&x), *yh = reinterpret_cast<const half2*>(&y);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 u = __half22float2(xh[i]), w = __half22float2(yh[i]);
                s = fmaf(u.x, w.x, fmaf(u.y, w.y, s));
            }
        }
        s *= a.scale2;
        const float m_new = fmaxf(m, warp_max(sees ? s : -FLT_MAX)), c = exp2_neg(m - m_new), p = sees ? exp2_neg(s - m_new) : 0.f;
        l = l * c + p;
        for (int i = 0; i < pairs; i++) o[i] = make_float2(o[i].x * c, o[i].y * c);
#pragma unroll 1
        for (int j = 0; j < min(32, len - p0); j++) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const half2* vr = reinterpret_cast<const half2*>(vb + (size_t)(p0 + j) * a.dim) + lane;
#pragma unroll
            for (int i = 0; i < 2; i++)
                if (i < pairs) {
                    const float2 w = __half22float2(vr[32 * i]);
                    o[i].x = fmaf(pj, w.x, o[i].x);
                    o[i].y = fmaf(pj, w.y, o[i].y);
                }
        }
        m = m_new;
    }
    l = warp_sum(l);
    half2* out = reinterpret_cast<half2*>(a.out + qo) + lane;
#pragma unroll
    for (int i = 0; i < 2; i++)
        if (i < pairs) out[32 * i] = l > 0.f ? __floats2half2_rn(o[i].x / l, o[i].y / l) : __floats2half2_rn(0.f, 0.f);
}

// The same for latent attention in BF16: a lane has vdim / 32 neighbouring outputs (two or four).
__device__ __forceinline__ void visible_row(const PromptArgs<bf16>& a, const LatentPart<true>& x, int h, int qi, int lane)
{
    const int dq = a.dim + x.rot, heads = gridDim.y, len = a.pos0 + qi + 1, per = a.vdim / 32;
    const bf16 *q = a.q + (size_t)qi * x.ld_q + (size_t)h * dq, *vb = a.v + (size_t)h * a.vdim + lane * per;
    float m = -FLT_MAX, l = 0.f, o[4] = {};
#pragma unroll 1
    for (int p0 = 0; p0 < len; p0 += 32) {
        const int p = p0 + lane;
        const bool sees = p < len;
        float s = 0.f;
#pragma unroll 1
        for (int d = 0; sees && d < dq; d += 8) {
            const bf16* k = d < a.dim ? a.k + ((size_t)p * heads + h) * a.dim + d : x.shared + (size_t)p * x.ld_shared + x.shared_col + d - a.dim;
            float u[8], w8[8];
            Vec16<bf16>::unpack(*reinterpret_cast<const uint4*>(q + d), u);
            Vec16<bf16>::unpack(*reinterpret_cast<const uint4*>(k), w8);
#pragma unroll
            for (int i = 0; i < 8; i++) s = fmaf(u[i], w8[i], s);
        }
        s *= a.scale2;
        const float m_new = fmaxf(m, warp_max(sees ? s : -FLT_MAX)), c = exp2_neg(m - m_new), w = sees ? exp2_neg(s - m_new) : 0.f;
        l = l * c + w;
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] *= c;
#pragma unroll 1
        for (int j = 0; j < min(32, len - p0); j++) {
            const float wj = __shfl_sync(0xffffffffu, w, j);
            const bf16* v = vb + (size_t)(p0 + j) * heads * a.vdim;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i < per) o[i] = fmaf(wj, to_f<bf16>(v[i]), o[i]);
        }
        m = m_new;
    }
    l = warp_sum(l);
    if (x.sink) l += exp2f(x.sink[h] * kLog2e - m);
    float f = a.out_scale / l;
    if (x.gate) f *= sigmoid_f(to_f<bf16>(x.gate[(size_t)qi * x.gate_ld + h]));
    bf16* out = a.out + (size_t)qi * a.ld_out + (size_t)h * a.vdim + lane * per;
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (i < per) out[i] = from_f<bf16>(o[i] * f);
}

enum Bar { kQFull, kKFull, kKEmpty, kVFull, kVEmpty, kSFull, kPReady, kPvDone, kBars };

// LATENT: keys of two parts, a sink and a gate per head
template <typename T, bool LATENT>
__global__ void __launch_bounds__(kThreads, LATENT ? 1 : 2)
grouped_prompt_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const PromptArgs<T> a, const __grid_constant__ LatentPart<LATENT> x)
{
    using Op = Operand<T>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[kBars];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.y, g = h / a.per_kv, seq = blockIdx.z, q0 = (gridDim.x - 1 - blockIdx.x) * kTile;       // longest first
    const int nq = min(kTile, a.n - q0), first = a.pos0 + q0, hi = first + nq;                    // positions of the queries
    const int lo = chunk_start(first, a.chunk) & ~(kTile - 1), lo_last = chunk_start(hi - 1, a.chunk);
    const int tiles = (hi - lo + kTile - 1) / kTile, ne = a.vdim / 64;
    int nd = a.dim / 64;
    if constexpr (LATENT) nd += x.rot / 64;
    const uint32_t qs = smem_u32(smem), ks = qs + nd * kBlock, vs = ks + nd * kBlock, bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * i; };
    volatile int* abortp = &abort_flag;
    int never = 0;

    if (tid == 0) {
        prefetch_map(&map_q);
        prefetch_map(&map_k);
        prefetch_map(&map_v);
        if constexpr (LATENT) prefetch_map(&x.map_r);
        for (int i = 0; i < kBars; i++) mbar_init(bar(i), i == kPReady ? kTile : 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot, tmem_o = tmem + kTile;
    pdl_wait();

    if (warp == 4) {
        // ---------------- TMA producer ----------------
        const bool leader = elect_one();
        int issued = 0;                                         // tiles whose copies were issued: keys, then values
        bool ok = true;
        const int head_row = (seq * a.kv_heads + g) * a.head_rows;
        if (leader) {
            mbar_expect_tx(bar(kQFull), nd * kBlock);
            for (int j = 0; j < nd; j++) tma_load_2d(qs + j * kBlock, &map_q, h * (LATENT ? nd * 64 : a.dim) + j * 64, seq * a.n + q0, bar(kQFull));
        }
        for (int i = 0; i < 2 * tiles; i++, issued++) {
            const int t = i >> 1, row = head_row + (lo + t * kTile) % a.cache_rows;
            const bool v = i & 1;
            if (!(ok = mbar_wait(bar(v ? kVEmpty : kKEmpty), (t & 1) ^ 1, abortp))) break;
            if (leader) {
                const int blocks = v ? ne : nd;
                mbar_expect_tx(bar(v ? kVFull : kKFull), blocks * kBlock);
                for (int j = 0; j < blocks; j++) {
                    if (v) tma_load_2d(vs + j * kBlock, &map_v, g * a.v_cols + j * 64, row, bar(kVFull));
                    else {
                        if constexpr (LATENT)
                            if (j * 64 >= a.dim) {
                                tma_load_2d(ks + j * kBlock, &x.map_r, x.shared_col + j * 64 - a.dim, row, bar(kKFull));
                                continue;
                            }
                        tma_load_2d(ks + j * kBlock, &map_k, g * a.k_cols + j * 64, row, bar(kKFull));
                    }
                }
            }
        }
        if (!ok) abort_flag = 1;
        __syncwarp();
        // after an abort the copies still in flight must land before the shared memory goes away
        if (*abortp) {
            mbar_wait(bar(kQFull), 0, &never);
            if (issued > 0) mbar_wait(bar(kKFull), ((issued - 1) >> 1) & 1, &never);
            if (issued > 1) mbar_wait(bar(kVFull), ((issued - 2) >> 1) & 1, &never);
        }
    } else if (warp == 5) {
        // ---------------- MMA issuer ----------------
        const bool leader = elect_one();
        const uint32_t id_s = idesc<T>(kTile, false), id_o = idesc<T>(a.vdim, true);
        const uint64_t qd = make_sw128_desc(qs), kd = make_sw128_desc(ks), vd = feature_major_desc(vs);
        bool ok = mbar_wait(bar(kQFull), 0, abortp);
        int done = 0;                                           // tiles whose last product was issued
        for (int t = 0; ok && t < tiles; t++) {
            // the weights of the tile before lie where S goes
            ok = (t == 0 || mbar_wait(bar(kPvDone), (t - 1) & 1, abortp)) && mbar_wait(bar(kKFull), t & 1, abortp);
            if (!ok) break;
            fence_after();
            if (leader) {
                for (int j = 0; j < nd; j++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {               // 32 bytes (2 in the descriptor) inside the swizzled row
                        const uint32_t o = j * (kBlock >> 4) + k * 2;
                        mma_ss(tmem, qd + o, kd + o, id_s, j > 0 || k > 0);
                    }
                mma_commit(bar(kKEmpty));
                mma_commit(bar(kSFull));
            }
            ok = mbar_wait(bar(kVFull), t & 1, abortp) && mbar_wait(bar(kPReady), t & 1, abortp);
            if (!ok) break;
            fence_after();
            if (leader) {
#pragma unroll
                for (int part = 0; part < 2; part++)
#pragma unroll
                    for (int k = 0; k < kTile / 16; k++)
                        mma_ts(tmem_o, tmem + part * 64 + k * 8, vd + k * (2048 >> 4), id_o, t > 0 || part > 0 || k > 0);
                mma_commit(bar(kVEmpty));
                mma_commit(bar(kPvDone));
            }
            done++;
        }
        if (!ok) {
            abort_flag = 1;
            // what was issued completes before the memory is given up
            if (leader) mma_commit(bar(kPvDone));
            __syncwarp();
            mbar_wait(bar(kPvDone), done & 1, &never);
        }
    } else if (warp < 4) {
        // ---------------- softmax: a row per thread ----------------
        const uint32_t row_s = tmem + ((uint32_t)(warp * 32) << 16), row_o = row_s + kTile;
        const int pos = first + tid, from = chunk_start(pos, a.chunk);
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int t = 0; t < tiles; t++) {
            const int k0 = lo + t * kTile;
            ok = __all_sync(0xffffffffu, mbar_wait(bar(kSFull), t & 1, abortp));
            if (!ok) break;
            fence_after();
            uint32_t raw[4][32];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) tmem_ld32(row_s + i * 32, raw[i]);
            wait_ld();
            f32x2 s[64];                                                      // scores of two positions each
            const f32x2 scale = pair_f32(a.scale2, a.scale2);
#pragma unroll
            for (int i = 0; i < 64; i++) s[i] = mul_pair(pair_f32(raw[i >> 4][2 * (i & 15)], raw[i >> 4][2 * (i & 15) + 1]), scale);
            if (k0 + kTile > first + 1 || k0 < lo_last) {                     // some (query, position) pair of the tile is masked
                const int seen = pos - k0, unseen = from - k0;                // the last and the first that this row sees
#pragma unroll
                for (int i = 0; i < 64; i++) {
                    const float2 v = split_f32(s[i]);
                    s[i] = pair_f32(2 * i > seen || 2 * i < unseen ? -INFINITY : v.x, 2 * i + 1 > seen || 2 * i + 1 < unseen ? -INFINITY : v.y);
                }
            }
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 64; i++) {
                const float2 v = split_f32(s[i]);
                top[i & 3] = fmaxf(top[i & 3], fmaxf(v.x, v.y));
            }
            const float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            const bool grows = mx > m + Op::kSlack || (m == -INFINITY && mx > m);
            if (__any_sync(0xffffffffu, grows)) {
                const float f = grows ? exp2_neg(m - mx) : 1.f;               // 0 where nothing was seen before
                if (grows) {
                    m = mx;
                    l *= f;
                }
                if (t > 0) {
#pragma unroll 1
                    for (int c = 0; c < a.vdim; c += 32) {
                        uint32_t o[32];
                        tmem_ld32(row_o + c, o);
                        wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                        tmem_st32(row_o + c, o);
                    }
                }
            }
            const float ref = Op::kLift - (m == -INFINITY ? 0.f : m);
            const f32x2 off = pair_f32(ref, ref);
            f32x2 sum[2] = {0ull, 0ull};
#pragma unroll
            for (int part = 0; part < 4; part++) {                            // 32 positions: 16 words of high, 16 of low parts
                uint32_t ph[16], pl[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float2 e = split_f32(add_pair(s[part * 16 + j], off));
                    const f32x2 p = pair_f32(exp2_neg(e.x), exp2_neg(e.y));
                    sum[j & 1] = add_pair(sum[j & 1], p);
                    const float2 pf = split_f32(p);
                    const typename Op::Pair b = Op::pair(pf.x, pf.y);
                    const float2 r = Op::floats(b);
                    const float2 low = split_f32(add_pair(p, pair_f32(-r.x, -r.y)));
                    const typename Op::Pair c = Op::pair(low.x, low.y);
                    ph[j] = *reinterpret_cast<const uint32_t*>(&b);
                    pl[j] = *reinterpret_cast<const uint32_t*>(&c);
                }
                tmem_st16(row_s + part * 16, ph);
                tmem_st16(row_s + 64 + part * 16, pl);
            }
            l += sum_pair(add_pair(sum[0], sum[1]));
            if (k0 + kTile > hi) {
                // rows of the cache behind the last query hold anything: their weights are 0, their values become 0
                ok = __all_sync(0xffffffffu, mbar_wait(bar(kVFull), t & 1, abortp));
                if (!ok) break;
                if (k0 + tid >= hi)
                    for (int j = 0; j < ne * 8; j++)
                        *reinterpret_cast<uint4*>(smem + (size_t)(2 * nd + (j >> 3)) * kBlock + tid * 128 + (j & 7) * 16) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            wait_st();
            fence_before();
            mbar_arrive(bar(kPReady));
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(kPvDone), (tiles - 1) & 1, abortp));
        if (ok) {
            fence_after();
            // a row without a positive sum: zeros from the FP16 operator, as from its decode form
            const bool zeros = std::is_same<T, half>::value && !(l > 0.f);
            float f;
            if constexpr (LATENT) {
                if (x.sink) l += exp2f(x.sink[h] * kLog2e - m);
                f = a.out_scale / l;
                if (x.gate && tid < nq) f *= sigmoid_f(to_f<T>(x.gate[(size_t)(q0 + tid) * x.gate_ld + h]));
            } else {
                f = zeros ? 1.f : a.out_scale / l;
            }
            T* op = a.out + ((size_t)seq * a.n + q0 + tid) * a.ld_out + (size_t)h * a.vdim;
            uint32_t largest = 0;                                             // exponents order infinities and NaN last
#pragma unroll 1
            for (int c = 0; c < a.vdim; c += 32) {
                uint32_t o[32];
                tmem_ld32(row_o + c, o);
                wait_ld();
                if (zeros) {
#pragma unroll
                    for (int j = 0; j < 32; j++) o[j] = 0;
                }
                if (tid < nq) {
#pragma unroll
                    for (int j = 0; (std::is_same<T, half>::value || LATENT) && j < 32; j++) largest = max(largest, o[j] & 0x7fffffffu);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        typename Op::Pair w[4];
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            w[i] = Op::pair(__uint_as_float(o[8 * j + 2 * i]) * f, __uint_as_float(o[8 * j + 2 * i + 1]) * f);
                        *reinterpret_cast<uint4*>(op + c + 8 * j) = *reinterpret_cast<const uint4*>(w);
                    }
                }
            }
            if constexpr (std::is_same<T, half>::value || LATENT) {
                __syncwarp();                                                 // the rows' first outputs lie before their second
                for (uint32_t again = __ballot_sync(0xffffffffu, largest >= 0x7f800000u); again; again &= again - 1) {
                    const int qi = q0 + warp * 32 + __ffs(again) - 1;
                    if constexpr (LATENT) visible_row(a, x, h, qi, lane);
                    else visible_row(a, h, g, seq, qi, lane);
                }
            }
        } else {
            abort_flag = 1;
        }
    }
    fence_before();
    __syncthreads();
    if (abort_flag && tid == 0) atomicExch(a.err, TLLM_ERR_TIMEOUT);
    if (warp == 5) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

constexpr size_t kLatentSmem = 220 * 1024;
size_t smem_bytes(int dim, int vdim) { return (size_t)(2 * (dim / 64) + vdim / 64) * kBlock + 1024; }

template <typename T>
int encode(EncodeTiledFn enc, CUtensorMap* map, const T* p, int cols, size_t rows, size_t ld)
{
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(T)};
    const cuuint32_t box[2] = {64, (cuuint32_t)kTile};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, Operand<T>::kMap, 2, const_cast<T*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TLLM_ERR_LAUNCH, "grouped_prompt: cuTensorMapEncodeTiled failed with %d", (int)r);
    return TLLM_OK;
}

template <typename T, bool LATENT = false>
int launch(PromptArgs<T>& p, const LatentPart<LATENT>& x, int columns, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, int heads,
           int batch, cudaStream_t stream)
{
    p.err = device_error_flag();
    if (!p.err) return fail(TLLM_ERR_LAUNCH, "device scratch unavailable");
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return fail(TLLM_ERR_LAUNCH, "grouped_prompt: no current device");
    const auto kernel = grouped_prompt_tc_kernel<T, LATENT>;
    if (!attr[dev]) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(LATENT ? kLatentSmem : smem_bytes(128, 128)));
        attr[dev] = true;
    }
    return launch_pdl("grouped_prompt", kernel, dim3((p.n + kTile - 1) / kTile, heads, batch), dim3(kThreads),
                      smem_bytes(columns, p.vdim), stream, mq, mk, mv, p, x);
}

}  // namespace

bool grouped_prompt_tcgen05_supported(const GroupedArgs<bf16>& a)
{
    // the tiles of a ring do not wrap when its rows are a multiple of a tile
    return (a.dim == 64 || a.dim == 128) && (a.vdim == 64 || a.vdim == 128) && a.g.n_seq == 1 && !a.g.pos_dev && a.g.seq_len >= kTile &&
           (a.cache_rows >= a.max_seq || a.cache_rows % kTile == 0) && a.ld_out % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.proj + a.q_off) | reinterpret_cast<uintptr_t>(a.kc) |
             reinterpret_cast<uintptr_t>(a.vc)) & 15) == 0;
}

int launch_grouped_prompt_tcgen05(const GroupedArgs<bf16>& a, cudaStream_t stream)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from this driver");
    const bf16 *kc = a.kc + (size_t)a.g.first_slot * a.k_slot, *vc = a.vc + (size_t)a.g.first_slot * a.v_slot;
    CUtensorMap mq, mk, mv;
    int st;
    if ((st = encode(enc, &mq, a.proj + a.q_off, a.heads * a.dim, a.g.seq_len, a.ld))) return st;
    if ((st = encode(enc, &mk, kc, a.kv_heads * a.dim, a.cache_rows, (size_t)a.kv_heads * a.dim))) return st;
    if ((st = encode(enc, &mv, vc, a.kv_heads * a.vdim, a.cache_rows, (size_t)a.kv_heads * a.vdim))) return st;
    PromptArgs<bf16> p = {};
    p.out = a.out;
    p.ld_out = a.ld_out;
    p.per_kv = a.heads / a.kv_heads;
    p.kv_heads = a.kv_heads;
    p.dim = a.dim;
    p.vdim = a.vdim;
    p.n = a.g.seq_len;
    p.pos0 = a.g.start_pos;
    p.chunk = a.chunk;
    p.cache_rows = a.cache_rows;
    p.head_rows = 0;
    p.k_cols = a.dim;
    p.v_cols = a.vdim;
    p.scale2 = a.scale * kLog2e;
    p.out_scale = a.out_scale;
    return launch(p, LatentPart<false>(), p.dim, mq, mk, mv, a.heads, 1, stream);
}

bool latent_prompt_tcgen05_supported(const LatentArgs<bf16>& a)
{
    return a.dim > 0 && a.dim % 64 == 0 && a.rot % 64 == 0 && (a.vdim == 64 || a.vdim == 128) && smem_bytes(a.dim + a.rot, a.vdim) <= kLatentSmem &&
           a.g.n_seq == 1 && !a.g.pos_dev && a.q_off % 8 == 0 && a.ld % 8 == 0 && a.rank % 8 == 0 && a.slot_stride % 8 == 0 && a.heads <= 65535 &&
           ((reinterpret_cast<uintptr_t>(a.proj) | reinterpret_cast<uintptr_t>(a.cache)) & 15) == 0;
}

// kx [context][heads][dim], vx [context][heads][vdim], out [rows][heads][vdim], all on 16-byte boundaries
int launch_latent_prompt_tcgen05(const LatentArgs<bf16>& a, const bf16* kx, const bf16* vx, bf16* out, cudaStream_t stream)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from this driver");
    const int ctx = a.g.start_pos + a.g.seq_len, dq = a.dim + a.rot, ldc = a.rank + a.rot;
    const bf16* cache = a.cache + (size_t)a.g.first_slot * a.slot_stride;
    CUtensorMap mq, mk, mv;
    LatentPart<true> x = {};
    int st;
    if ((st = encode(enc, &mq, a.proj + a.q_off, a.heads * dq, a.g.seq_len, a.ld))) return st;
    if ((st = encode(enc, &mk, kx, a.heads * a.dim, ctx, (size_t)a.heads * a.dim))) return st;
    if ((st = encode(enc, &mv, vx, a.heads * a.vdim, ctx, (size_t)a.heads * a.vdim))) return st;
    if ((st = encode(enc, &x.map_r, cache, ldc, ctx, ldc))) return st;
    PromptArgs<bf16> p = {};
    p.out = out;
    p.ld_out = a.heads * a.vdim;
    p.q = a.proj + a.q_off;
    p.k = kx;
    p.v = vx;
    p.per_kv = 1;
    p.kv_heads = a.heads;
    p.dim = a.dim;
    p.vdim = a.vdim;
    p.n = a.g.seq_len;
    p.pos0 = a.g.start_pos;
    p.cache_rows = INT_MAX;
    p.k_cols = a.dim;
    p.v_cols = a.vdim;
    p.scale2 = a.scale * kLog2e;
    p.out_scale = 1.f;
    x.rot = a.rot;
    x.ld_q = a.ld;
    x.ld_shared = ldc;
    x.shared_col = a.rank;
    x.shared = cache;
    x.sink = a.sink;
    x.gate = a.gate;
    x.gate_ld = a.gate_ld;
    return launch<bf16, true>(p, x, dq, mq, mk, mv, a.heads, 1, stream);
}

// Few queries over few channels: a CTA per query and key/value head on the CUDA cores (attention.cu) has the shorter launch, and one
// chunk of 256 positions there is two tiles here.  us there / here, heads of 64 without groups unless said:
//   * up to 32 positions, while all CTAs run at once: one head of two sequences, 6 queries of 11 5.5 / 6.0, 4 heads of two, 2 of 2 5.3 / 6.1,
//     32 heads of two, 5 of 10 6.9 / 6.9, 8 heads, 16 of 21 6.4 / 6.1; groups of two, 4 heads, 4 of 4 5.8 / 6.2, of 8 sequences, 8 of 13 7.1 / 6.9;
//     heads of 128, 8 heads, 6 of 11 7.2 / 7.5; groups of four only where the tiles here share SMs: 8 heads of 8 sequences, 3 of 13
//     7.8 / 8.5, 4 heads of one, 2 of 22 7.4 / 6.3;
//   * up to 48 positions for two or three queries: 32 heads, 3 of 33 6.2 / 6.5; of 63 6.2 / 5.9 (8 heads);
//   * up to 128 positions, one tile here, never;
//   * one chunk there behind them, while few CTAs share an SM: 4 heads, 3 of 153 7.2 / 8.1; 8 heads, 5 of 205 7.8 / 8.0; 4 heads, 8 of 248
//     8.2 / 7.7; 2 heads of 8 sequences, 8 of 208 9.3 / 8.3; heads of 128, 2 heads, 8 of 158 9.3 / 9.7, 8 sequences of one, 3 of 203 9.9 / 9.5;
//   * behind more never: 8 queries of one head behind 1000 25.4 / 19.8; 32 heads over 8, 2 queries behind 400 13.6 / 12.0.
static bool few_queries(int batch, int group, int n_kv_heads, int head_dim, int seq_len, int kv_len)
{
    const long long ctas = (long long)batch * n_kv_heads * seq_len;
    const int channels = group * head_dim;
    if (seq_len > 12 && seq_len * group > 16) return false;
    if (kv_len <= 32) {
        if (channels <= 128) return ctas <= (channels == 64 ? 444 : head_dim == 64 ? 192 : 148);
        return head_dim == 64 && channels <= 256 && seq_len <= 8 && ctas >= 64 && ctas <= 192;
    }
    if (kv_len <= 128) return channels == 64 && seq_len <= 3 && kv_len <= 48 && ctas <= 444;
    return channels <= 128 && ctas <= 64 && kv_len <= (channels == 64 ? 208 : 160);
}

bool attention_prompt_supported(const half* q, const half* k_cache, const half* v_cache, const half* out, int batch, int n_heads, int n_kv_heads,
                                int head_dim, int seq_len, int kv_len, int kv_len_max)
{
    // rows of a map are addressed with 32-bit coordinates; one query splits the positions (attention.cu)
    return (head_dim == 64 || head_dim == 128) && seq_len >= 2 && !few_queries(batch, n_heads / n_kv_heads, n_kv_heads, head_dim, seq_len, kv_len) &&
           (long long)batch * n_kv_heads * kv_len_max < (1ll << 30) &&
           (long long)batch * seq_len < (1ll << 30) && batch <= 65535 &&
           ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
             reinterpret_cast<uintptr_t>(out)) & 15) == 0;
}

int launch_attention_prompt(const half* q, const half* k_cache, const half* v_cache, half* out, int batch, int n_heads, int n_kv_heads,
                            int head_dim, int seq_len, int kv_len, int kv_len_max, cudaStream_t stream)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(TLLM_ERR_LAUNCH, "cuTensorMapEncodeTiled is not available from this driver");
    const size_t rows = (size_t)batch * n_kv_heads * kv_len_max;
    CUtensorMap mq, mk, mv;
    int st;
    if ((st = encode(enc, &mq, q, n_heads * head_dim, (size_t)batch * seq_len, (size_t)n_heads * head_dim))) return st;
    if ((st = encode(enc, &mk, k_cache, head_dim, rows, head_dim))) return st;
    if ((st = encode(enc, &mv, v_cache, head_dim, rows, head_dim))) return st;
    PromptArgs<half> p = {};
    p.out = out;
    p.q = q;
    p.k = k_cache;
    p.v = v_cache;
    p.ld_out = n_heads * head_dim;
    p.per_kv = n_heads / n_kv_heads;
    p.kv_heads = n_kv_heads;
    p.dim = p.vdim = head_dim;
    p.n = seq_len;
    p.pos0 = kv_len - seq_len;
    p.cache_rows = p.head_rows = kv_len_max;
    p.scale2 = kLog2e / sqrtf((float)head_dim);
    p.out_scale = 1.f;
    return launch(p, LatentPart<false>(), p.dim, mq, mk, mv, n_heads, batch, stream);
}

}  // namespace tllm
