// One new token of each sequence against its FP16 KV cache: rotation, cache append and attention in one
// launch, for head sizes 64 and 128 with 1, 2, 4 or 8 query heads to a key/value head.
//
// A launch is a chain of latencies (a few hundred KB of cache a head), so it is built around having few
// steps that wait:
//   - a cluster of up to eight CTAs shares a key/value head and splits its positions; the parts meet in
//     shared memory of the cluster, every CTA finishing its share of the outputs, so there are no records
//     in global memory, no counter and no last arriver;
//   - a thread copies its own 16-byte pieces of K and V (cp.async, read back by the same thread: no
//     barrier) and a warp walks its own positions with its own running maximum, so scores, softmax and
//     P.V follow one another without a barrier of the CTA; the warps meet once, at the end;
//   - a piece of K or V is converted once for all query heads of the group, and two channels go into one
//     multiplication;
//   - rotation angles and, into L2, the cache lines are requested before the wait on the launch before.
// All sums are FP32.
// Bound by those latencies: a launch in the chain of a step takes 6.0 us behind 1500 positions of the 1B model (8 heads x 8
// CTAs), 6.4 behind 300 of the 8B shape, 9.7 for 24 sequences behind 300 (14.7 MB of cache, 2.3 us); the kernel with 64 positions a
// CTA and records in global memory took 12.4 and 11.9, rotation and ranges of 256 positions 26.
#include <cfloat>

#include <cooperative_groups.h>

#include "f32x2.cuh"
#include "launch.cuh"
#include "layer.cuh"

namespace tllm {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kPasses = 8;             // passes over a warp's positions between two softmax updates
constexpr int kMaxCluster = 8;
// A cluster grows while all CTAs run at once and a CTA keeps more than 32 positions, or 64 where an SM has more than two of them.  How
// many run at once is asked of each instantiation and cluster size: a group of eight has one CTA an SM (registers), of four two, of two
// and one three, and clusters leave some SMs out (264 CTAs of a group of four in clusters of eight).  A launch among others, us, CTAs
// to 296 for all / so: heads of 128 in groups of eight, 32 key/value heads, behind 400 22.9 / 9.2, behind 2000 39.6 / 22.0, 64 heads behind
// 2000 43.3 / 37.9; groups of four, 37 heads behind 400 13.4 / 8.2; groups of one, 80 heads behind 2000 30.6 / 19.8; with 32 positions in three
// CTAs an SM 48 heads of 64 in groups of two, behind 400, 8.5 instead of 6.3.  A step: 8 sequences of the 1B model (64 heads) behind 1800
// positions 4 parts 762, 2 parts 871; behind 500 666 / 696; 24 sequences (192) behind 300 one part 869, two 952; 8 of four 8B layers
// behind 200 4 parts 455, 8 parts 504.
constexpr int kLeast = 64;

struct StepArgs {
    const half *q, *k, *v;             // [batch, heads, hd] of the new token, not rotated
    half *k_cache, *v_cache;           // [batch, n_kv_heads, kv_len_max, hd]
    half* out;                         // [batch, n_heads, hd]
    int n_kv_heads, kv_len_max, pos;
    const int* pos_dev;                // not null: the position
    float theta;
};

template <int HD, int G>
struct Shared {
    uint4 k[kPasses][kThreads], v[kPasses][kThreads];
    float q[G * HD];
    half new_k[HD], new_v[HD];
    float rec[kWarps][G * HD];                      // the warps' outputs
    float ml[kWarps][2 * G];                        // their maxima and sums
    float cluster_o[G * HD];                        // the cluster's parts of this CTA's outputs
    float cluster_ml[kMaxCluster][2 * G];
};

__device__ __forceinline__ void copy16(uint4* dst, const half* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void unpack_half(const uint4& r, f32x2 (&f)[4])
{
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 t = __half22float2(*reinterpret_cast<const half2*>(&w[i]));
        f[i] = pair_f32(t.x, t.y);
    }
}

// Sums v[0..N) over the LANES lanes that differ in bits below LANES; on return v[0..N/LANES) (at least
// one) are the sums of entries first * .. of this lane, `first` rising with the lane.
template <int N, int LANES>
__device__ __forceinline__ void halve_sum(float* v, int lane)
{
    if constexpr (LANES > 1) {
        constexpr int O = LANES / 2;
        if constexpr (N > 1) {
            const bool up = lane & O;
#pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const float send = up ? v[i] : v[i + N / 2], keep = up ? v[i + N / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
            }
            halve_sum<N / 2, O>(v, lane);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            halve_sum<1, O>(v, lane);
        }
    }
}

template <int HD, int G>
__global__ void __launch_bounds__(kThreads)
attention_step_kernel(StepArgs a)
{
    constexpr int LP = HD / 8, PW = 32 / LP, PP = kWarps * PW;        // lanes per position; positions of a warp's and of the CTA's pass
    constexpr int HP = HD / 2, kItems = (G + 1) * HP, kRot = (kItems + kThreads - 1) / kThreads;
    constexpr int LH = LP / G;                                        // lanes that end up with the same head's score
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Shared<HD, G>& S = *reinterpret_cast<Shared<HD, G>*>(smem_raw);
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = lane % LP, sub = lane / LP;
    const int parts = gridDim.x, rank = blockIdx.x, kvh = blockIdx.y;
    const size_t row = (size_t)blockIdx.z * a.n_kv_heads + kvh;       // key/value head over all sequences
    cg::cluster_group cluster = cg::this_cluster();
    if (parts > 1) cluster.barrier_arrive();

    half* kb = a.k_cache + row * a.kv_len_max * HD;
    half* vb = a.v_cache + row * a.kv_len_max * HD;
    float freq[kRot];
#pragma unroll
    for (int u = 0; u < kRot; u++) freq[u] = 1.0f / powf(a.theta, (2.0f * (float)((tid + u * kThreads) % HP)) / (float)HD);
    if (!a.pos_dev && (lane & 7) == 0) {                              // L2 holds what the launches before write
        const int per = ((a.pos + parts) / parts + PP - 1) / PP * PP, hi = min(a.pos, (rank + 1) * per);
        for (int j = rank * per + warp * PW + sub, p = 0; p < kPasses && j < hi; p++, j += PP) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(kb + (size_t)j * HD + c * 8));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(vb + (size_t)j * HD + c * 8));
        }
    }

    pdl_wait();
    const int pos = a.pos_dev ? *a.pos_dev : a.pos, limit = pos + 1;
    const int per = ((limit + parts - 1) / parts + PP - 1) / PP * PP;
    const int lo = rank * per, hi = min(limit, lo + per);             // this CTA's positions (none: lo >= hi)
    const int cached = min(pos, a.kv_len_max);                        // positions that come from the cache
    auto request = [&](uint4 (*dst)[kThreads], const half* src, int j0) {
#pragma unroll
        for (int p = 0; p < kPasses; p++) {
            const int j = j0 + p * PP + warp * PW + sub;
            const bool in = j < hi && j < cached;
            if (j0 + p * PP < hi) copy16(&dst[p][tid], in ? src + (size_t)j * HD + c * 8 : src, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    request(S.k, kb, lo);
    request(S.v, vb, lo);

    const bool owner = lo <= pos && pos < hi;
    const float scale = rsqrtf((float)HD);
#pragma unroll
    for (int u = 0; u < kRot; u++) {
        const int i = tid + u * kThreads, pr = i % HP, g = i / HP;
        if (i >= kItems || (g == G && !owner)) continue;
        const half2 raw = *(reinterpret_cast<const half2*>(g < G ? a.q + (row * G + g) * HD : a.k + row * HD) + pr);
        const float2 x = __half22float2(raw);
        float sn, cs;
        sincosf((float)pos * freq[u], &sn, &cs);
        const half r0 = __float2half_rn(x.x * cs - x.y * sn), r1 = __float2half_rn(x.x * sn + x.y * cs);
        if (g < G) {
            // rounded to FP16 like the rotated q the reference stores, then scaled
            *reinterpret_cast<float2*>(&S.q[g * HD + 2 * pr]) = make_float2(__half2float(r0) * scale, __half2float(r1) * scale);
        } else {
            const half2 kr = __halves2half2(r0, r1), vr = *(reinterpret_cast<const half2*>(a.v + row * HD) + pr);
            reinterpret_cast<half2*>(S.new_k)[pr] = kr;
            reinterpret_cast<half2*>(S.new_v)[pr] = vr;
            if (pos < a.kv_len_max) {
                *(reinterpret_cast<half2*>(kb + (size_t)pos * HD) + pr) = kr;
                *(reinterpret_cast<half2*>(vb + (size_t)pos * HD) + pr) = vr;
            }
        }
    }
    __syncthreads();

    f32x2 q[G][4];
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float4 q0 = *reinterpret_cast<const float4*>(&S.q[g * HD + c * 8]), q1 = *reinterpret_cast<const float4*>(&S.q[g * HD + c * 8 + 4]);
        q[g][0] = pair_f32(q0.x, q0.y);
        q[g][1] = pair_f32(q0.z, q0.w);
        q[g][2] = pair_f32(q1.x, q1.y);
        q[g][3] = pair_f32(q1.z, q1.w);
    }
    f32x2 o[G][4];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < 4; i++) o[g][i] = 0ull;
    float m = -FLT_MAX, l = 0.f;                   // of head (c / LH): the same maximum in the warp, this lane's positions in the sum
    for (int j0 = lo; j0 < hi; j0 += kPasses * PP) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        float s[kPasses], mx = -FLT_MAX;
#pragma unroll
        for (int p = 0; p < kPasses; p++) {
            const int j = j0 + p * PP + warp * PW + sub;
            s[p] = -INFINITY;
            if (j0 + p * PP >= hi) continue;
            uint4 raw = S.k[p][tid];
            if (j == pos) raw = *reinterpret_cast<const uint4*>(&S.new_k[c * 8]);
            f32x2 kf[4];
            unpack_half(raw, kf);
            float d[G];
#pragma unroll
            for (int g = 0; g < G; g++) {
                f32x2 t = mul_pair(kf[0], q[g][0]), t1 = mul_pair(kf[1], q[g][1]);
                fma_pair(t, kf[2], q[g][2]);
                fma_pair(t1, kf[3], q[g][3]);
                d[g] = sum_pair(t) + sum_pair(t1);
            }
            halve_sum<G, LP>(d, lane);
            if (j < hi) s[p] = d[0];
            mx = fmaxf(mx, s[p]);
        }
        request(S.k, kb, j0 + kPasses * PP);
#pragma unroll
        for (int w = LP; w < 32; w *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
        const float m_new = fmaxf(m, mx), corr = __expf(m - m_new);
        m = m_new;
        l *= corr;
#pragma unroll
        for (int p = 0; p < kPasses; p++) {
            s[p] = __expf(s[p] - m_new);
            l += s[p];
        }
        if (j0 != lo) {
#pragma unroll
            for (int g = 0; g < G; g++) {
                const float cg_ = __shfl_sync(0xffffffffu, corr, (lane & ~(LP - 1)) + g * LH);
                const f32x2 cc = pair_f32(cg_, cg_);
#pragma unroll
                for (int i = 0; i < 4; i++) o[g][i] = mul_pair(o[g][i], cc);
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
        for (int p = 0; p < kPasses; p++) {
            if (j0 + p * PP >= hi) continue;
            const int j = j0 + p * PP + warp * PW + sub;
            uint4 raw = S.v[p][tid];
            if (j == pos) raw = *reinterpret_cast<const uint4*>(&S.new_v[c * 8]);
            f32x2 vf[4];
            unpack_half(raw, vf);
#pragma unroll
            for (int g = 0; g < G; g++) {
                const float w = __shfl_sync(0xffffffffu, s[p], (lane & ~(LP - 1)) + g * LH);
                const f32x2 ww = pair_f32(w, w);
#pragma unroll
                for (int i = 0; i < 4; i++) fma_pair(o[g][i], vf[i], ww);
            }
        }
        request(S.v, vb, j0 + kPasses * PP);
    }

    // ---- the warps' parts -------------------------------------------------------------------------
#pragma unroll
    for (int w = LP; w < 32; w *= 2) l += __shfl_xor_sync(0xffffffffu, l, w);
    float t[8 * G];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 f = split_f32(o[g][i]);
            t[g * 8 + 2 * i] = f.x;
            t[g * 8 + 2 * i + 1] = f.y;
        }
    {
        // over the position groups of the warp: lane bits LP .. 16
        constexpr int N1 = 8 * G / 2;
        const bool up = lane & 16;
#pragma unroll
        for (int i = 0; i < N1; i++) {
            const float send = up ? t[i] : t[i + N1], keep = up ? t[i + N1] : t[i];
            t[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
        int first = up ? N1 : 0, n = N1;
        if constexpr (PW == 4) {
            constexpr int N2 = N1 / 2;
            const bool up2 = lane & 8;
#pragma unroll
            for (int i = 0; i < N2; i++) {
                const float send = up2 ? t[i] : t[i + N2], keep = up2 ? t[i + N2] : t[i];
                t[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
            }
            first += up2 ? N2 : 0;
            n = N2;
        }
#pragma unroll
        for (int i = 0; i < N1; i++)
            if (i < n) S.rec[warp][(first + i) / 8 * HD + c * 8 + (first + i) % 8] = t[i];
        if (sub == 0 && c % LH == 0) {
            S.ml[warp][c / LH] = m;
            S.ml[warp][G + c / LH] = l;
        }
    }
    __syncthreads();
    constexpr int kOut = (G * HD + kThreads - 1) / kThreads;
    const int slice = G * HD / parts;
    half* out = a.out + row * G * HD;
    auto finish = [](float num, float den) { return den > 0.f ? __float2half_rn(num / den) : __ushort_as_half(0); };
    if (parts > 1) cluster.barrier_wait();                            // the others run: their shared memory is there
#pragma unroll
    for (int u = 0; u < kOut; u++) {
        const int i = tid + u * kThreads, g = i / HD;
        if (i >= G * HD) break;
        float M = -FLT_MAX, num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) M = fmaxf(M, S.ml[w][g]);
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const float e = __expf(S.ml[w][g] - M);
            num = fmaf(e, S.rec[w][i], num);
            den = fmaf(e, S.ml[w][G + g], den);
        }
        if (parts == 1) {
            out[i] = finish(num, den);
            continue;
        }
        *cluster.map_shared_rank(&S.cluster_o[rank * slice + i % slice], i / slice) = num;
        if (i % HD < parts) {
            float* ml = cluster.map_shared_rank(&S.cluster_ml[rank][0], i % HD);
            ml[g] = M;
            ml[G + g] = den;
        }
    }
    if (parts == 1) return;
    cluster.sync();
    for (int i = tid; i < slice; i += kThreads) {
        const int g = (rank * slice + i) / HD;
        float M = -FLT_MAX, num = 0.f, den = 0.f;
        for (int r = 0; r < parts; r++) M = fmaxf(M, S.cluster_ml[r][g]);
        for (int r = 0; r < parts; r++) {
            const float e = __expf(S.cluster_ml[r][g] - M);
            num = fmaf(e, S.cluster_o[r * slice + i], num);
            den = fmaf(e, S.cluster_ml[r][G + g], den);
        }
        out[rank * slice + i] = finish(num, den);
    }
}

struct Plan {
    int parts, at_once;                // CTAs of a head; CTAs of such clusters that run at once
};

template <int HD, int G>
int plan(int heads, int longest, Plan* p)
{
    const auto kernel = attention_step_kernel<HD, G>;
    static int slots[64][kMaxCluster + 1] = {};          // CTAs that run at once in clusters of 1, 2, 4, 8
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(TLLM_ERR_LAUNCH, "attention_step: no current device");
    if (!slots[dev][1]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared<HD, G>)) != cudaSuccess) {
            cudaGetLastError();
            return fail(TLLM_ERR_LAUNCH, "attention_step: no current device");
        }
        prefer_max_shared(reinterpret_cast<const void*>(kernel));
        for (int c = kMaxCluster; c >= 1; c /= 2) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at = {};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = c;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.gridDim = dim3(c * 1024);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = sizeof(Shared<HD, G>);
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            slots[dev][c] = c == 1 && n < 1 ? 1 : n * c;
        }
    }
    p->parts = 1;
    while (p->parts < kMaxCluster && heads * p->parts * 2 <= slots[dev][2 * p->parts] &&
           longest > p->parts * (heads * p->parts * 2 > 2 * 148 ? 2 * kLeast : kLeast))
        p->parts *= 2;
    p->at_once = slots[dev][p->parts];
    return TLLM_OK;
}

// batch 0: the plan alone
template <int HD, int G>
int launch(const StepArgs& a, int heads, int longest, int batch, cudaStream_t stream, Plan* p)
{
    const int st = plan<HD, G>(heads, longest, p);
    if (st || !batch) return st;
    return launch_pdl_cluster("attention_step", attention_step_kernel<HD, G>, p->parts, dim3(p->parts, a.n_kv_heads, batch), dim3(kThreads),
                              sizeof(Shared<HD, G>), stream, a);
}

template <int HD>
int launch_group(const StepArgs& a, int group, int heads, int longest, int batch, cudaStream_t stream, Plan* p)
{
    switch (group) {
        case 8: return launch<HD, 8>(a, heads, longest, batch, stream, p);
        case 4: return launch<HD, 4>(a, heads, longest, batch, stream, p);
        case 2: return launch<HD, 2>(a, heads, longest, batch, stream, p);
        default: return launch<HD, 1>(a, heads, longest, batch, stream, p);
    }
}

}  // namespace

bool attention_step_supported(const half* q, const half* k, const half* v, const half* k_cache, const half* v_cache, int n_heads, int n_kv_heads,
                              int head_dim)
{
    const int group = n_kv_heads > 0 && n_heads % n_kv_heads == 0 ? n_heads / n_kv_heads : 0;
    const uintptr_t p = reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache);
    const uintptr_t n = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v);
    return (head_dim == 64 || head_dim == 128) && (group == 1 || group == 2 || group == 4 || group == 8) && p % 16 == 0 && n % 4 == 0;
}

int launch_attention_step(const half* q, const half* k, const half* v, half* k_cache, half* v_cache, half* out, int batch, int n_heads, int n_kv_heads,
                          int head_dim, int kv_len_max, int pos, const int* pos_dev, float theta, cudaStream_t stream)
{
    const StepArgs a = {q, k, v, k_cache, v_cache, out, n_kv_heads, kv_len_max, pos, pos_dev, theta};
    const int heads = batch * n_kv_heads, longest = pos_dev ? kv_len_max : pos + 1;
    Plan p;
    return head_dim == 64 ? launch_group<64>(a, n_heads / n_kv_heads, heads, longest, batch, stream, &p)
                          : launch_group<128>(a, n_heads / n_kv_heads, heads, longest, batch, stream, &p);
}

int attention_step_plan(int n_heads, int n_kv_heads, int head_dim, int heads, int longest, int* parts, int* at_once)
{
    const StepArgs a = {};
    Plan p = {};
    const int st = head_dim == 64 ? launch_group<64>(a, n_heads / n_kv_heads, heads, longest, 0, nullptr, &p)
                                  : launch_group<128>(a, n_heads / n_kv_heads, heads, longest, 0, nullptr, &p);
    *parts = p.parts;
    *at_once = p.at_once;
    return st;
}

}  // namespace tllm
