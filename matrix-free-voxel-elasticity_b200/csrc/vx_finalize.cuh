// Scalar slots of the Krylov loops and the reductions that end in them: the sum of one partial per CTA in a
// fixed order, then the scalar recurrence.  It runs in a kernel of its own (finalize_kernel) or in the last
// CTA of the kernel that wrote the partials (finalize_last), with the same threads, order and result.
#pragma once
#include "vx_common.cuh"

namespace vx {

constexpr int FT = 256;

enum Slot {
    S_RZ = 0, S_PQ = 1, S_ALPHA = 2, S_RR = 3, S_REL = 4, S_NB = 5, S_BETA = 6, S_RZN = 7, S_RZD = 8,
    S_TOL = 9, S_DONE = 10, S_IT = 11, S_MAXIT = 12, S_MV = 13, S_BREAK = 14, S_CHECK = 15, S_COUNT = 16
};

enum FinOp {
    FIN_PQ = 0,        // S[PQ] = sum; alpha = rz / pq (breakdown if pq == 0); it += 1; mv += 1
    FIN_TRUE = 1,      // S[RR] = sum; rel = sqrt(rr) / nb; mv += 1; done if rel <= tol
    FIN_BETA_PR = 2,   // rzn = sum0, rzd = sum1; beta = rzd / rz; rz = rzn      (flexible / Polak-Ribiere)
    FIN_BETA_FR = 3,   // rzn = sum0; beta = rzn / rz; rz = rzn                  (Fletcher-Reeves)
    FIN_NB = 4,        // nb = sqrt(sum)
    FIN_RZ = 5,        // rz = sum0
    FIN_RR_ONLY = 6    // rr = sum; rel = sqrt(rr) / nb (no counters, no flag)
};

__device__ __forceinline__ double fin_warp_sum(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double block_sum_ft(double v) {
    __shared__ double red[FT / 32];
    v = fin_warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) s = fin_warp_sum(threadIdx.x < FT / 32 ? red[threadIdx.x] : 0.0);
    return s;
}

// The scalar recurrence of `op` from the sums (one thread).
__device__ __forceinline__ void fin_scalars(int op, double s0, double s1, double* S) {
    switch (op) {
        case FIN_PQ:
            if (S[S_DONE] != 0.0) break;            // a converged warm start: the body is a no-op
            S[S_PQ] = s0;
            S[S_MV] += 1.0;
            if (s0 == 0.0 || !isfinite(s0)) { S[S_BREAK] = 1.0; S[S_ALPHA] = 0.0; }   // no step is taken
            else { S[S_ALPHA] = S[S_RZ] / s0; S[S_IT] += 1.0; }
            break;
        case FIN_TRUE:
            if (S[S_DONE] != 0.0) break;
            S[S_RR] = s0;
            S[S_REL] = sqrt(s0) / S[S_NB];
            S[S_MV] += 1.0;
            if (S[S_REL] <= S[S_TOL]) S[S_DONE] = 1.0;
            if (!isfinite(S[S_REL])) S[S_BREAK] = 1.0;
            break;
        case FIN_BETA_PR:
            S[S_RZN] = s0;
            S[S_RZD] = s1;
            S[S_BETA] = s1 / S[S_RZ];
            S[S_RZ] = s0;
            break;
        case FIN_BETA_FR:
            S[S_RZN] = s0;
            S[S_BETA] = s0 / S[S_RZ];
            S[S_RZ] = s0;
            break;
        case FIN_NB: S[S_NB] = sqrt(s0); break;
        case FIN_RZ: S[S_RZ] = S[S_RZN] = s0; break;
        case FIN_RR_ONLY:
            S[S_RR] = s0;
            S[S_REL] = sqrt(s0) / S[S_NB];
            break;
    }
}

// Sums of the G partials (and, for FIN_BETA_PR, the G after them) by FT threads, then the recurrence.  The
// scalars are read together with the partials: one by one they would be a chain of L2 round trips.
__device__ __forceinline__ void fin_reduce(int op, int64_t G, const double* partials, double* S) {
    __shared__ double sv[S_COUNT];
    if (threadIdx.x < S_COUNT) sv[threadIdx.x] = __ldcg(S + threadIdx.x);
    double s0 = 0.0, s1 = 0.0;
    #pragma unroll 4
    for (int64_t j = threadIdx.x; j < G; j += FT) s0 += __ldcg(partials + j);
    if (op == FIN_BETA_PR) {
        #pragma unroll 4
        for (int64_t j = threadIdx.x; j < G; j += FT) s1 += __ldcg(partials + G + j);
    }
    s0 = block_sum_ft(s0);
    if (op == FIN_BETA_PR) s1 = block_sum_ft(s1);
    if (threadIdx.x == 0) fin_scalars(op, s0, s1, sv);
    __syncthreads();
    if (threadIdx.x < S_COUNT) S[threadIdx.x] = sv[threadIdx.x];
}

// Called by every CTA (FT threads) after its thread 0 has written its partials: the CTA that arrives last
// finishes the reduction.  *counter is 0 before the launch and again after it.  One launch less than a
// finalize kernel, which costs 2 to 3 us in a loop of short kernels.
__device__ __forceinline__ void finalize_last(int op, int64_t G, const double* partials, double* S, unsigned* counter) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();                                     // this CTA's partials before its arrival
        last = atomicInc(counter, unsigned(G - 1)) == unsigned(G - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    fin_reduce(op, G, partials, S);
}

}  // namespace vx
