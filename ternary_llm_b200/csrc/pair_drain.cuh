// What two CTAs that share a ring of stages may have in flight when they give up (dense_gemm.cu, pairs).
//
// Each CTA fills a stage with its own half of the bytes, and both halves count on the barrier of the first CTA, which expects them
// once the first CTA's producer has reached the stage.  A producer fills a stage again only when the first CTA's MMAs
// have consumed it, so of every stage no more than the last filling can be under way; but the two producers need not have stopped
// at the same filling.  Plain C++, so that the rule can be checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define TLLM_HD __host__ __device__ __forceinline__
#else
#define TLLM_HD inline
#endif

namespace tllm {

struct PairFill {
    int stage, parity;       // barrier, and parity of the phase that ends when all of it is there
    bool unarmed;            // the second CTA alone: the barrier expects nothing yet
    bool lacks;              // the first CTA alone: the barrier expects the other half too, which will not come
};

// fillings begin .. end may be under way after `first` of the first CTA's producer and `second` of the other's
TLLM_HD int pair_fills_end(int first, int second) { return first > second ? first : second; }
TLLM_HD int pair_fills_begin(int first, int second, int stages)
{
    const int end = pair_fills_end(first, second);
    return end > stages ? end - stages : 0;
}
TLLM_HD PairFill pair_fill(int f, int first, int second, int stages) { return {f % stages, (f / stages) & 1, f >= first, f >= second}; }

}  // namespace tllm
