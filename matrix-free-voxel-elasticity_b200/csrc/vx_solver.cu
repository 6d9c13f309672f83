// Solver kernels with device-resident scalars, and a CUDA-graph WHILE loop.
//
// The outer Krylov loops keep every scalar (r.z, p.q, alpha, beta, |b - A x|, the iteration and
// matvec counters, the converged flag) in a small FP64 array S on the device.  Each reduction is
// two-stage and deterministic: the producing kernel writes one partial per CTA, a one-CTA
// "finalize" kernel sums them in a fixed order and applies the scalar recurrence.  With the loop
// body captured as the body of a conditional WHILE graph node, a complete solve is a single graph
// launch with no host round trip per iteration; the condition kernel stops the loop on
// convergence, on breakdown or at maxiter.
#include "vx_finalize.cuh"
#include <algorithm>
#include <type_traits>

namespace vx {

// Slot blockIdx.y (a batch of independent systems solved in lockstep) uses S + 16 slot and
// partials + slot * pstride; unbatched launches have one slot.
__global__ void __launch_bounds__(FT) finalize_kernel(int op, int64_t G, const double* __restrict__ partials,
                                                      double* __restrict__ S, int64_t pstride) {
    vx::pdl_begin();
    fin_reduce(op, G, partials + pstride * int64_t(blockIdx.y), S + S_COUNT * int64_t(blockIdx.y));
}

// The vector kernels move W consecutive entries per thread: 4 (16-byte accesses, two for doubles) on long
// aligned vectors, where one entry per thread left HBM at 84 to 88% for want of bytes in flight, else 1.
// The same operations either way.  576x288x288 (us, W = 1 -> 4, FP32 z): direction with
// the x update 1006 -> 850 (6.8 TB/s), V-cycle entry with the r update 920 -> 762, direction 600 -> 506, entry
// 590 -> 424, x and r update 1077 -> 988.
constexpr int64_t WIDE_MIN = 1 << 20;      // below this, 4 entries a thread leave SMs without CTAs
template <int W, typename T>
__device__ __forceinline__ void ldv(const T* p, T (&v)[W]) {
    if constexpr (W == 1) v[0] = p[0];
    else if constexpr (sizeof(T) == 8) {
        const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else if constexpr (sizeof(T) == 4) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
        union { uint2 u; T t[4]; } a;
        a.u = *reinterpret_cast<const uint2*>(p);
        for (int k = 0; k < 4; ++k) v[k] = a.t[k];
    }
}
template <int W, typename T>
__device__ __forceinline__ void stv(T* p, const T (&v)[W]) {
    if constexpr (W == 1) p[0] = v[0];
    else if constexpr (sizeof(T) == 8) {
        reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
    } else if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        union { uint2 u; T t[4]; } a;
        for (int k = 0; k < 4; ++k) a.t[k] = v[k];
        *reinterpret_cast<uint2*>(p) = a.u;
    }
}
// Runs f(i, integral_constant<W>) for this thread's entries: the W at i, or the last few one by one.
template <int W, typename F>
__device__ __forceinline__ void for_entries(int64_t n, F&& f) {
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * W;
    if (i + W <= n) f(i, std::integral_constant<int, W>{});
    else if constexpr (W > 1)
        for (int64_t k = i; k < n; ++k) f(k, std::integral_constant<int, 1>{});
}
template <typename... T> bool wide(int64_t n, const T*... p) {
    return n >= WIDE_MIN && ((p == nullptr || aligned(p, 4 * sizeof(T) > 16 ? 16 : 4 * sizeof(T))) && ...);
}

// x += alpha p; r -= alpha q (r update skipped when it is about to be replaced by b - A x).
// Nothing moves once the loop has converged or broken down.
// Vector kernels of a batch: slot blockIdx.y works on its n entries at slot * vs and on S + 16 slot.
template <int W, typename T>
__global__ void cg_update_kernel(int64_t n, const double* __restrict__ S, T* __restrict__ x, const T* __restrict__ p,
                                 T* __restrict__ r, const T* __restrict__ q, int update_r, int64_t vs) {
    vx::pdl_begin();
    const int64_t o = vs * int64_t(blockIdx.y);
    S += S_COUNT * int64_t(blockIdx.y);
    x += o;
    p += o;
    if (update_r) { r += o; q += o; }
    if (S[S_DONE] != 0.0 || S[S_BREAK] != 0.0) return;
    const T a = T(S[S_ALPHA]);
    for_entries<W>(n, [&](int64_t i, auto wc) {
        constexpr int V = decltype(wc)::value;
        T xv[V], pv[V], rv[V], qv[V];
        ldv<V>(x + i, xv);
        ldv<V>(p + i, pv);
        if (update_r) { ldv<V>(r + i, rv); ldv<V>(q + i, qv); }
        #pragma unroll
        for (int k = 0; k < V; ++k) {
            xv[k] = xv[k] + a * pv[k];
            if (update_r) rv[k] = rv[k] - a * qv[k];
        }
        stv<V>(x + i, xv);
        if (update_r) stv<V>(r + i, rv);
    });
}

// p = z + beta p and, when z_old is given, z_old = z; z and z_old in the preconditioner's storage TZ
// (a copy in z's own type is exact and moves half the bytes of an FP64 copy of an FP32 z)
template <int W, typename T, typename TZ>
__global__ void cg_direction_kernel(int64_t n, const double* __restrict__ S, const TZ* __restrict__ z, T* __restrict__ p,
                                    TZ* __restrict__ z_old, int64_t vs) {
    vx::pdl_begin();
    const int64_t o = vs * int64_t(blockIdx.y);
    S += S_COUNT * int64_t(blockIdx.y);
    z += o;
    p += o;
    if (z_old) z_old += o;
    const T beta = T(S[S_BETA]);
    for_entries<W>(n, [&](int64_t i, auto wc) {
        constexpr int V = decltype(wc)::value;
        TZ zr[V];
        T pv[V];
        ldv<V>(z + i, zr);
        ldv<V>(p + i, pv);
        #pragma unroll
        for (int k = 0; k < V; ++k) pv[k] = T(Storage<TZ>::cvt(zr[k])) + beta * pv[k];
        stv<V>(p + i, pv);
        if (z_old) stv<V>(z_old + i, zr);
    });
}

// The same direction update preceded by the deferred x += alpha p of this iteration (p still the old
// direction), skipped once the loop has converged or broken down: one read of p serves both.
template <int W, typename T, typename TZ>
__global__ void cg_direction_update_kernel(int64_t n, const double* __restrict__ S, const TZ* __restrict__ z,
                                           T* __restrict__ p, TZ* __restrict__ z_old, T* __restrict__ x) {
    vx::pdl_begin();
    const bool move = S[S_DONE] == 0.0 && S[S_BREAK] == 0.0;
    const T alpha = T(S[S_ALPHA]), beta = T(S[S_BETA]);
    for_entries<W>(n, [&](int64_t i, auto wc) {
        constexpr int V = decltype(wc)::value;
        T pv[V], xv[V];
        TZ zr[V];
        ldv<V>(p + i, pv);
        if (move) ldv<V>(x + i, xv);
        ldv<V>(z + i, zr);
        #pragma unroll
        for (int k = 0; k < V; ++k) {
            xv[k] = xv[k] + alpha * pv[k];
            pv[k] = T(Storage<TZ>::cvt(zr[k])) + beta * pv[k];
        }
        if (move) stv<V>(x + i, xv);
        stv<V>(p + i, pv);
        if (z_old) stv<V>(z_old + i, zr);
    });
}

// partials for r . zn and r . (zn - zo), fixed grid G (a function of n), fixed order
// (slot blockIdx.y: vectors at slot * vs, partials at slot * 2G)
template <typename T, typename TZ>
__global__ void __launch_bounds__(FT) dots_pr_kernel(int64_t n, const T* __restrict__ r, const TZ* __restrict__ zn,
                                                     const TZ* __restrict__ zo, double* partials, int64_t vs,
                                                     int fin, double* S, unsigned* counter) {
    vx::pdl_begin();
    const int64_t G = gridDim.x;
    {
        const int64_t o = vs * int64_t(blockIdx.y);
        r += o;
        zn += o;
        if (zo) zo += o;
        partials += 2 * G * int64_t(blockIdx.y);
    }
    double a = 0.0, b = 0.0;
    #pragma unroll 4
    for (int64_t i = int64_t(blockIdx.x) * FT + threadIdx.x; i < n; i += G * FT) {
        const double ri = double(r[i]), zi = double(Storage<TZ>::load(zn + i));
        a = fma(ri, zi, a);
        if (zo) b = fma(ri, zi - double(Storage<TZ>::load(zo + i)), b);
    }
    a = block_sum_ft(a);
    if (threadIdx.x == 0) partials[blockIdx.x] = a;
    if (zo) {
        b = block_sum_ft(b);
        if (threadIdx.x == 0) partials[G + blockIdx.x] = b;
    }
    if (counter) finalize_last(fin, G, partials, S, counter);
}

// One Jacobi-preconditioned CG step between two operator applications: x += alpha p, r -= alpha q (skipped
// when update is 0 or once the loop has converged or broken down), z = d r over the previous z, the partials
// of r . z and r . (z - z_old) and, in the last CTA, beta.  One pass over each vector where the separate
// update, product, dots and finalize kernels read r three times and z twice; on small grids, where every
// launch costs 2 to 3 us, three launches less an iteration.
__global__ void __launch_bounds__(FT) jacobi_step_kernel(int64_t n, double* S, double* __restrict__ x,
                                                         const double* __restrict__ p, double* __restrict__ r,
                                                         const double* __restrict__ q, const double* __restrict__ d,
                                                         double* __restrict__ z, int update, double* partials,
                                                         unsigned* counter) {
    vx::pdl_begin();
    const int64_t G = gridDim.x;
    const bool move = update && S[S_DONE] == 0.0 && S[S_BREAK] == 0.0;
    const double alpha = S[S_ALPHA];
    double a = 0.0, b = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * FT + threadIdx.x; i < n; i += G * FT) {
        double ri = r[i];
        if (move) {
            x[i] = x[i] + alpha * p[i];
            ri = ri - alpha * q[i];
            r[i] = ri;
        }
        const double zo = z[i], zi = d[i] * ri;
        z[i] = zi;
        a = fma(ri, zi, a);
        b = fma(ri, zi - zo, b);
    }
    a = block_sum_ft(a);
    b = block_sum_ft(b);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = a;
        partials[G + blockIdx.x] = b;
    }
    finalize_last(FIN_BETA_PR, G, partials, S, counter);
}

// The same iteration for small grids (at most SMALL_CTAS CTAs of one entry per thread), where the hand-over of
// a sum through the last CTA (a fence, an atomic, the partials' and scalars' round trips: 2 to 3 us) costs
// more than the work: every CTA of the kernel that needs a sum adds up the partials itself, in the same
// order, and CTA 0 alone writes the scalars.  No CTA depends on a slot that CTA 0 may have written already: the step
// takes rz from S_RZN and leaves it in S_RZ, the direction takes S_RZ and leaves the new one in S_RZN.  S_BREAK
// is read and may be set in the step, but only where every CTA finds `stop` from the same sum and takes no step anyway.
// 32x16x16, 700 iterations: 12.8 -> 9.0 us an iteration (separate update, product, dots and
// finalize kernels: 16.8).
constexpr int64_t SMALL_CTAS = 1184;
__device__ __forceinline__ double sum_partials(int64_t G, const double* __restrict__ partials) {
    __shared__ double total;
    double s = 0.0;
    #pragma unroll 4
    for (int64_t j = threadIdx.x; j < G; j += FT) s += partials[j];
    s = block_sum_ft(s);
    if (threadIdx.x == 0) total = s;
    __syncthreads();
    s = total;
    __syncthreads();
    return s;
}

// alpha = rz / (p . q) from the G partials pq (FIN_PQ), then x += alpha p and, with step, r -= alpha q, z = d r
// and the partials of r . z and r . (z - z_old); fin 0 (after a true residual) skips alpha and the updates.
__global__ void __launch_bounds__(FT) small_step_kernel(int64_t n, int64_t G, const double* __restrict__ pq, double* S,
                                                        double* __restrict__ x, const double* __restrict__ p,
                                                        double* __restrict__ r, const double* __restrict__ q,
                                                        const double* __restrict__ d, double* __restrict__ z,
                                                        int fin, int step, double* __restrict__ partials) {
    vx::pdl_begin();
    const int64_t i = int64_t(blockIdx.x) * FT + threadIdx.x;
    const bool in = i < n;
    double xi = 0.0, pi = 0.0, ri = 0.0, qi = 0.0, di = 0.0, zo = 0.0;
    if (in) {
        if (fin) { xi = x[i]; pi = p[i]; }
        if (step) { ri = r[i]; di = d[i]; zo = z[i]; if (fin) qi = q[i]; }
    }
    if (fin) {
        const double rz = S[S_RZN];
        const bool done = S[S_DONE] != 0.0, broken = S[S_BREAK] != 0.0;
        const double s = sum_partials(G, pq);
        const bool stop = s == 0.0 || !isfinite(s);
        const double alpha = stop ? 0.0 : rz / s;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            S[S_RZ] = rz;
            if (!done) {
                S[S_PQ] = s;
                S[S_MV] += 1.0;
                S[S_ALPHA] = alpha;
                if (stop) S[S_BREAK] = 1.0;
                else S[S_IT] += 1.0;
            }
        }
        if (in && !done && !broken && !stop) {
            x[i] = xi + alpha * pi;
            if (step) {
                ri = ri - alpha * qi;
                r[i] = ri;
            }
        }
    }
    if (!step) return;
    const double zi = di * ri;
    if (in) z[i] = zi;
    const double a = block_sum_ft(ri * zi), b = block_sum_ft(ri * (zi - zo));
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = a;
        partials[gridDim.x + blockIdx.x] = b;
    }
}

// beta from the step's partials (FIN_BETA_PR), p = z + beta p
__global__ void __launch_bounds__(FT) small_direction_kernel(int64_t n, const double* __restrict__ partials, double* S,
                                                             const double* __restrict__ z, double* __restrict__ p) {
    vx::pdl_begin();
    const int64_t i = int64_t(blockIdx.x) * FT + threadIdx.x, G = gridDim.x;
    const bool in = i < n;
    const double zi = in ? z[i] : 0.0, pi = in ? p[i] : 0.0, rz = S[S_RZ];
    double s0 = 0.0, s1 = 0.0;
    #pragma unroll 4
    for (int64_t j = threadIdx.x; j < G; j += FT) { s0 += partials[j]; s1 += partials[G + j]; }
    __shared__ double beta_s;
    s0 = block_sum_ft(s0);
    s1 = block_sum_ft(s1);
    if (threadIdx.x == 0) {
        beta_s = s1 / rz;
        if (blockIdx.x == 0) {
            S[S_RZN] = s0;
            S[S_RZD] = s1;
            S[S_BETA] = beta_s;
        }
    }
    __syncthreads();
    if (in) p[i] = zi + beta_s * pi;
}

// z = d * r (Jacobi) with partial r . z
template <typename T>
__global__ void __launch_bounds__(FT) jacobi_precond_dot_kernel(int64_t n, const T* __restrict__ d, const T* __restrict__ r,
                                                                T* __restrict__ z, double* __restrict__ partials) {
    vx::pdl_begin();
    const int64_t G = gridDim.x;
    double a = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * FT + threadIdx.x; i < n; i += G * FT) {
        const T zi = d[i] * r[i];
        z[i] = zi;
        a = fma(double(r[i]), double(zi), a);
    }
    a = block_sum_ft(a);
    if (threadIdx.x == 0) partials[blockIdx.x] = a;
}

// V-cycle entry: r_mg = r64 in auxiliary storage (skipped when r_mg is NULL), x = omega * invd * r_mg (the first
// pre-sweep from x = 0).  With UPDATE it is preceded by the CG residual update r64 -= alpha q (alpha =
// S[S_ALPHA]), which is skipped, like vx_cg_update's, once the loop has converged or broken down.
template <int W, bool UPDATE, typename TX, typename TR>
__global__ void vcycle_entry_kernel(int64_t n, const double* __restrict__ S, const double* __restrict__ r_in,
                                    double* __restrict__ r_out, const double* __restrict__ q, TR* __restrict__ rmg,
                                    const TR* __restrict__ invd, double omega, TX* __restrict__ x) {
    vx::pdl_begin();
    using A = arith_t<TX>;
    const bool move = UPDATE && S[S_DONE] == 0.0 && S[S_BREAK] == 0.0;
    const double alpha = UPDATE ? S[S_ALPHA] : 0.0;
    const double* const rp = UPDATE ? r_out : r_in;
    for_entries<W>(n, [&](int64_t i, auto wc) {
        constexpr int V = decltype(wc)::value;
        double rv[V], qv[V];
        TR dv[V], mv[V];
        TX xv[V];
        ldv<V>(rp + i, rv);
        if (move) ldv<V>(q + i, qv);
        ldv<V>(invd + i, dv);
        #pragma unroll
        for (int k = 0; k < V; ++k) {
            if (move) rv[k] = rv[k] - alpha * qv[k];
            const A r = A(Storage<TR>::round(arith_t<TR>(rv[k])));   // the level residual as stored
            Storage<TR>::store(&mv[k], r);
            Storage<TX>::store(&xv[k], A(omega) * A(Storage<TR>::cvt(dv[k])) * r);
        }
        if (move) stv<V>(r_out + i, rv);
        if (rmg) stv<V>(rmg + i, mv);
        stv<V>(x + i, xv);
    });
}

// out = omega * a * b: a, b auxiliary, out an iterate
template <typename TX, typename TR>
__global__ void scaled_product_kernel(int64_t n, double omega, const TR* __restrict__ a, const TR* __restrict__ b,
                                      TX* __restrict__ out) {
    vx::pdl_begin();
    using A = arith_t<TX>;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Storage<TX>::store(out + i, A(omega) * A(Storage<TR>::load(a + i)) * A(Storage<TR>::load(b + i)));
}

__global__ void set_scalars_kernel(double* S, int first, int count, double value) {
    vx::pdl_begin();
    const int i = threadIdx.x;
    if (i < count) S[first + i] = value;
}

// Another loop body runs while any of the `slots` systems is still running.
__global__ void condition_kernel(cudaGraphConditionalHandle h, const double* __restrict__ S, int slots) {
    vx::pdl_begin();
    if (threadIdx.x == 0) {
        bool go = false;
        for (int k = 0; k < slots; ++k) {
            const double* s = S + S_COUNT * k;
            // S[S_CHECK] = iterations per loop body: the next body must not pass maxiter
            go = go || (s[S_DONE] == 0.0 && s[S_BREAK] == 0.0 && s[S_IT] + s[S_CHECK] <= s[S_MAXIT]);
        }
        cudaGraphSetConditional(h, go ? 1u : 0u);
    }
}

// one entry per thread while the partials stay few: on small grids the step is one memory round trip
int64_t step_ctas(int64_t n) { return std::min<int64_t>((n + FT - 1) / FT, 1184); }

int64_t fixed_ctas(int64_t n) {
    int64_t g = (n + FT * 8 - 1) / (FT * 8);
    return g < 1 ? 1 : (g > 1184 ? 1184 : g);
}

inline unsigned nb(int64_t n, int t) { return unsigned((n + t - 1) / t); }

struct WhileGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraphConditionalHandle handle = 0;
    cudaGraph_t body = nullptr;
};

}  // namespace vx

using namespace vx;

extern "C" int vx_solver_slots(void) { return S_COUNT; }

extern "C" int64_t vx_solver_partials(int64_t n) { return fixed_ctas(n); }

extern "C" int vx_solver_finalize(int op, int64_t G, const double* partials, double* S, cudaStream_t stream) {
    VX_CHECK_ARG(op >= 0 && op <= FIN_RR_ONLY && G > 0, VX_ERR_INVALID_ARGUMENT, "vx_solver_finalize: bad op/G");
    VX_CHECK_ARG(partials && S, VX_ERR_NULL_POINTER, "vx_solver_finalize: NULL pointer");
    vx::launch(finalize_kernel, 1, FT, 0, stream, op, G, partials, S, int64_t(0));
    VX_CHECK_LAUNCH("vx_solver_finalize");
    return VX_OK;
}

extern "C" int vx_cg_update(int prec, int64_t n, const double* S, void* x, const void* p, void* r, const void* q,
                            int update_r, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_cg_update: n must be positive");
    VX_CHECK_ARG(S && x && p && (!update_r || (r && q)), VX_ERR_NULL_POINTER, "vx_cg_update: NULL pointer");
    auto go = [&](auto t) {
        using T = decltype(t);
        const bool w = wide(n, (const T*)x, (const T*)p, update_r ? (const T*)r : nullptr, update_r ? (const T*)q : nullptr);
        vx::launch(w ? cg_update_kernel<4, T> : cg_update_kernel<1, T>, nb(n, w ? 1024 : 256), 256, 0, stream, n, S, (T*)x,
                   (const T*)p, (T*)r, (const T*)q, update_r, int64_t(0));
    };
    if (prec == VX_F64) go(double());
    else if (prec == VX_F32) go(float());
    else { set_error("vx_cg_update: unsupported precision %d", prec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH("vx_cg_update");
    return VX_OK;
}

extern "C" int vx_cg_direction(int prec, int zprec, int64_t n, const double* S, const void* z, void* p, void* z_old,
                               cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_cg_direction: n must be positive");
    VX_CHECK_ARG(S && z && p, VX_ERR_NULL_POINTER, "vx_cg_direction: NULL pointer");
    auto go = [&](auto t, auto tz) {
        using T = decltype(t);
        using TZ = decltype(tz);
        const bool w = wide(n, (const TZ*)z, (const T*)p, (const TZ*)z_old);
        vx::launch(w ? cg_direction_kernel<4, T, TZ> : cg_direction_kernel<1, T, TZ>, nb(n, w ? 1024 : 256), 256, 0, stream, n,
                   S, (const TZ*)z, (T*)p, (TZ*)z_old, int64_t(0));
    };
    if (prec == VX_F64 && zprec == VX_F64) go(double(), double());
    else if (prec == VX_F64 && zprec == VX_F32) go(double(), float());
    else if (prec == VX_F64 && zprec == VX_BF16_F32) go(double(), __nv_bfloat16());
    else if (prec == VX_F32 && zprec == VX_F32) go(float(), float());
    else { set_error("vx_cg_direction: unsupported precisions %d/%d", prec, zprec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH("vx_cg_direction");
    return VX_OK;
}

extern "C" int vx_cg_direction_update(int zprec, int64_t n, const double* S, const void* z, double* p, void* z_old,
                                      double* x, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_cg_direction_update: n must be positive");
    VX_CHECK_ARG(S && z && p && x, VX_ERR_NULL_POINTER, "vx_cg_direction_update: NULL pointer");
    const bool ok = dispatch_prec(zprec, [&](auto t) {
        using X = typename decltype(t)::X;
        const bool w = wide(n, (const X*)z, (const double*)p, (const X*)z_old, (const double*)x);
        vx::launch(w ? cg_direction_update_kernel<4, double, X> : cg_direction_update_kernel<1, double, X>,
                   nb(n, w ? 1024 : 256), 256, 0, stream, n, S, (const X*)z, p, (X*)z_old, x);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_cg_direction_update: unsupported precision %d", zprec);
    VX_CHECK_LAUNCH("vx_cg_direction_update");
    return VX_OK;
}

namespace {
int launch_dots_pr(const char* what, int prec, int zprec, int64_t n, const void* r, const void* zn, const void* zo,
                   double* partials, int fin, double* S, unsigned* counter, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "%s: n must be positive", what);
    VX_CHECK_ARG(r && zn && partials, VX_ERR_NULL_POINTER, "%s: NULL pointer", what);
    const unsigned G = unsigned(fixed_ctas(n));
    auto go = [&](auto rt, auto zt) {
        using T = decltype(rt);
        using TZ = decltype(zt);
        vx::launch(dots_pr_kernel<T, TZ>, G, FT, 0, stream, n, (const T*)r, (const TZ*)zn, (const TZ*)zo, partials,
                   int64_t(0), fin, S, counter);
    };
    if (prec == VX_F64 && zprec == VX_F64) go(double(), double());
    else if (prec == VX_F64 && zprec == VX_F32) go(double(), float());
    else if (prec == VX_F64 && zprec == VX_BF16_F32) go(double(), __nv_bfloat16());
    else if (prec == VX_F32 && zprec == VX_F32) go(float(), float());
    else { set_error("%s: unsupported precisions %d/%d", what, prec, zprec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH(what);
    return VX_OK;
}
}  // namespace

extern "C" int vx_dots_pr(int prec, int zprec, int64_t n, const void* r, const void* zn, const void* zo,
                          double* partials, cudaStream_t stream) {
    return launch_dots_pr("vx_dots_pr", prec, zprec, n, r, zn, zo, partials, 0, nullptr, nullptr, stream);
}

extern "C" int vx_dots_pr_fin(int op, int prec, int zprec, int64_t n, const void* r, const void* zn, const void* zo,
                              double* partials, double* S, unsigned* counter, cudaStream_t stream) {
    VX_CHECK_ARG(op >= 0 && op <= FIN_RR_ONLY && (op != FIN_BETA_PR || zo), VX_ERR_INVALID_ARGUMENT, "vx_dots_pr_fin: bad op");
    VX_CHECK_ARG(S && counter, VX_ERR_NULL_POINTER, "vx_dots_pr_fin: NULL pointer");
    return launch_dots_pr("vx_dots_pr_fin", prec, zprec, n, r, zn, zo, partials, op, S, counter, stream);
}

extern "C" int64_t vx_jacobi_step_partials(int64_t n) { return n > 0 ? 2 * step_ctas(n) : 2; }

extern "C" int vx_jacobi_step(int64_t n, double* S, double* x, const double* p, double* r, const double* q,
                              const double* inv_diag, double* z, int update, double* partials, unsigned* counter,
                              cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_jacobi_step: n must be positive");
    VX_CHECK_ARG(S && r && inv_diag && z && partials && counter && (!update || (x && p && q)), VX_ERR_NULL_POINTER,
                 "vx_jacobi_step: NULL pointer");
    vx::launch(jacobi_step_kernel, unsigned(step_ctas(n)), FT, 0, stream, n, S, x, p, r, q, inv_diag, z, update, partials,
               counter);
    VX_CHECK_LAUNCH("vx_jacobi_step");
    return VX_OK;
}

extern "C" int64_t vx_small_cg_limit(void) { return SMALL_CTAS * FT; }

extern "C" int vx_small_step(int64_t n, int64_t G, const double* pq, double* S, double* x, const double* p, double* r,
                             const double* q, const double* inv_diag, double* z, int fin, int step, double* partials,
                             cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && n <= SMALL_CTAS * FT && (fin || step) && (!fin || G > 0), VX_ERR_INVALID_ARGUMENT,
                 "vx_small_step: bad sizes");
    VX_CHECK_ARG(S && (!fin || (pq && x && p)) && (!step || (r && inv_diag && z && partials)) && (!(fin && step) || q),
                 VX_ERR_NULL_POINTER, "vx_small_step: NULL pointer");
    vx::launch(small_step_kernel, unsigned(step_ctas(n)), FT, 0, stream, n, G, pq, S, x, p, r, q, inv_diag, z, fin, step,
               partials);
    VX_CHECK_LAUNCH("vx_small_step");
    return VX_OK;
}

extern "C" int vx_small_direction(int64_t n, const double* partials, double* S, const double* z, double* p,
                                  cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && n <= SMALL_CTAS * FT, VX_ERR_INVALID_ARGUMENT, "vx_small_direction: bad size");
    VX_CHECK_ARG(partials && S && z && p, VX_ERR_NULL_POINTER, "vx_small_direction: NULL pointer");
    vx::launch(small_direction_kernel, unsigned(step_ctas(n)), FT, 0, stream, n, partials, S, z, p);
    VX_CHECK_LAUNCH("vx_small_direction");
    return VX_OK;
}

extern "C" int vx_jacobi_precond_dot(int prec, int64_t n, const void* d, const void* r, void* z, double* partials,
                                     cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_jacobi_precond_dot: n must be positive");
    VX_CHECK_ARG(d && r && z && partials, VX_ERR_NULL_POINTER, "vx_jacobi_precond_dot: NULL pointer");
    const unsigned G = unsigned(fixed_ctas(n));
    if (prec == VX_F64)
        vx::launch(jacobi_precond_dot_kernel<double>, G, FT, 0, stream, n, (const double*)d, (const double*)r, (double*)z, partials);
    else if (prec == VX_F32)
        vx::launch(jacobi_precond_dot_kernel<float>, G, FT, 0, stream, n, (const float*)d, (const float*)r, (float*)z, partials);
    else { set_error("vx_jacobi_precond_dot: unsupported precision %d", prec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH("vx_jacobi_precond_dot");
    return VX_OK;
}

extern "C" int vx_vcycle_entry(int prec, int64_t n, const double* r64, void* r_mg, const void* inv_diag, double omega,
                               void* x, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_vcycle_entry: n must be positive");
    VX_CHECK_ARG(r64 && inv_diag && x, VX_ERR_NULL_POINTER, "vx_vcycle_entry: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {
        using X = typename decltype(t)::X;
        using R = typename decltype(t)::R;
        const bool w = wide(n, r64, (const R*)r_mg, (const R*)inv_diag, (const X*)x);
        vx::launch(w ? vcycle_entry_kernel<4, false, X, R> : vcycle_entry_kernel<1, false, X, R>, nb(n, w ? 1024 : 256), 256, 0,
                   stream, n, (const double*)nullptr, r64, (double*)nullptr, (const double*)nullptr, (R*)r_mg,
                   (const R*)inv_diag, omega, (X*)x);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_vcycle_entry: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_vcycle_entry");
    return VX_OK;
}

extern "C" int vx_vcycle_entry_update(int prec, int64_t n, const double* S, double* r64, const double* q, void* r_mg,
                                      const void* inv_diag, double omega, void* x, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_vcycle_entry_update: n must be positive");
    VX_CHECK_ARG(S && r64 && q && inv_diag && x, VX_ERR_NULL_POINTER, "vx_vcycle_entry_update: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {
        using X = typename decltype(t)::X;
        using R = typename decltype(t)::R;
        const bool w = wide(n, (const double*)r64, q, (const R*)r_mg, (const R*)inv_diag, (const X*)x);
        vx::launch(w ? vcycle_entry_kernel<4, true, X, R> : vcycle_entry_kernel<1, true, X, R>, nb(n, w ? 1024 : 256), 256, 0,
                   stream, n, S, (const double*)nullptr, r64, q, (R*)r_mg, (const R*)inv_diag, omega, (X*)x);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_vcycle_entry_update: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_vcycle_entry_update");
    return VX_OK;
}

extern "C" int vx_scaled_product(int prec, int64_t n, double omega, const void* a, const void* b, void* out,
                                 cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_scaled_product: n must be positive");
    VX_CHECK_ARG(a && b && out, VX_ERR_NULL_POINTER, "vx_scaled_product: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {
        using X = typename decltype(t)::X;
        using R = typename decltype(t)::R;
        vx::launch(scaled_product_kernel<X, R>, nb(n, 256), 256, 0, stream, n, omega, (const R*)a, (const R*)b, (X*)out);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_scaled_product: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_scaled_product");
    return VX_OK;
}

extern "C" int vx_set_scalars(double* S, int first, int count, double value, cudaStream_t stream) {
    VX_CHECK_ARG(S, VX_ERR_NULL_POINTER, "vx_set_scalars: NULL S");
    VX_CHECK_ARG(first >= 0 && count >= 1 && first + count <= S_COUNT, VX_ERR_INVALID_ARGUMENT,
                 "vx_set_scalars: slots out of range");
    vx::launch(set_scalars_kernel, 1, 32, 0, stream, S, first, count, value);
    VX_CHECK_LAUNCH("vx_set_scalars");
    return VX_OK;
}

// ----------------------------------------------------------------------------- WHILE graphs
extern "C" int vx_graph_while_begin(cudaStream_t stream, void** handle) {
    VX_CHECK_ARG(handle, VX_ERR_NULL_POINTER, "vx_graph_while_begin: NULL handle");
    VX_CHECK_ARG(stream != nullptr, VX_ERR_INVALID_ARGUMENT, "vx_graph_while_begin: capture needs a non-default stream");
    // load the condition kernel now: with lazy module loading its first launch would otherwise
    // happen inside the capture
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, condition_kernel);
    if (e != cudaSuccess) {
        set_error("vx_graph_while_begin: %s", cudaGetErrorString(e));
        return VX_ERR_CUDA;
    }
    auto* w = new WhileGraph();
    e = cudaGraphCreate(&w->graph, 0);
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&w->handle, w->graph, 1, cudaGraphCondAssignDefault);
    cudaGraphNode_t node;
    cudaGraphNodeParams p = {};
    if (e == cudaSuccess) {
        p.type = cudaGraphNodeTypeConditional;
        p.conditional.handle = w->handle;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        e = cudaGraphAddNode(&node, w->graph, nullptr, 0, &p);
    }
    if (e == cudaSuccess) {
        w->body = p.conditional.phGraph_out[0];
        e = cudaStreamBeginCaptureToGraph(stream, w->body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    }
    if (e != cudaSuccess) {
        if (w->graph) cudaGraphDestroy(w->graph);
        delete w;
        set_error("vx_graph_while_begin: %s", cudaGetErrorString(e));
        return VX_ERR_CUDA;
    }
    *handle = w;
    return VX_OK;
}

static int graph_while_end(void* handle, const double* S, int slots, cudaStream_t stream) {
    VX_CHECK_ARG(handle && S, VX_ERR_NULL_POINTER, "vx_graph_while_end: NULL pointer");
    VX_CHECK_ARG(slots >= 1, VX_ERR_INVALID_ARGUMENT, "vx_graph_while_end: slots must be positive");
    auto* w = static_cast<WhileGraph*>(handle);
    vx::launch(condition_kernel, 1, 32, 0, stream, w->handle, S, slots);
    cudaError_t e = cudaGetLastError();
    cudaGraph_t captured = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(stream, &captured);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&w->exec, w->graph, 0);
    if (e != cudaSuccess) {
        set_error("vx_graph_while_end: %s", cudaGetErrorString(e));
        return VX_ERR_CUDA;
    }
    return VX_OK;
}

extern "C" int vx_graph_while_end(void* handle, const double* S, cudaStream_t stream) {
    return graph_while_end(handle, S, 1, stream);
}

// The batch form: the loop runs while any of `slots` systems (scalars S + 16 k) is running.
extern "C" int vx_batch_graph_while_end(void* handle, const double* S, int slots, cudaStream_t stream) {
    return graph_while_end(handle, S, slots, stream);
}

// ----------------------------------------------------------------------------- batches
// `slots` independent systems of n unknowns, slot k's vectors at k * stride, scalars at S + 16 k:
// the kernels above with the slot in blockIdx.y (one launch for the whole batch).
extern "C" int vx_batch_finalize(int op, int64_t G, int slots, const double* partials, int64_t pstride, double* S,
                                 cudaStream_t stream) {
    VX_CHECK_ARG(op >= 0 && op <= FIN_RR_ONLY && G > 0 && slots >= 1 && slots <= 65535, VX_ERR_INVALID_ARGUMENT,
                 "vx_batch_finalize: bad op/G/slots");
    VX_CHECK_ARG(partials && S, VX_ERR_NULL_POINTER, "vx_batch_finalize: NULL pointer");
    vx::launch(finalize_kernel, dim3(1, slots), FT, 0, stream, op, G, partials, S, pstride);
    VX_CHECK_LAUNCH("vx_batch_finalize");
    return VX_OK;
}

extern "C" int vx_batch_cg_update(int prec, int64_t n, int slots, int64_t stride, const double* S, void* x,
                                  const void* p, void* r, const void* q, int update_r, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && slots >= 1 && slots <= 65535, VX_ERR_INVALID_ARGUMENT, "vx_batch_cg_update: bad n/slots");
    VX_CHECK_ARG(S && x && p && (!update_r || (r && q)), VX_ERR_NULL_POINTER, "vx_batch_cg_update: NULL pointer");
    VX_CHECK_ARG(prec == VX_F64, VX_ERR_INVALID_ARGUMENT, "vx_batch_cg_update: unsupported precision %d", prec);
    vx::launch(cg_update_kernel<1, double>, dim3(nb(n, 256), slots), 256, 0, stream, n, S, (double*)x, (const double*)p,
               (double*)r, (const double*)q, update_r, stride);
    VX_CHECK_LAUNCH("vx_batch_cg_update");
    return VX_OK;
}

extern "C" int vx_batch_cg_direction(int zprec, int64_t n, int slots, int64_t stride, const double* S, const void* z,
                                     double* p, void* z_old, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && slots >= 1 && slots <= 65535, VX_ERR_INVALID_ARGUMENT, "vx_batch_cg_direction: bad n/slots");
    VX_CHECK_ARG(S && z && p, VX_ERR_NULL_POINTER, "vx_batch_cg_direction: NULL pointer");
    if (zprec == VX_F64)
        vx::launch(cg_direction_kernel<1, double, double>, dim3(nb(n, 256), slots), 256, 0, stream, n, S, (const double*)z, p,
                   (double*)z_old, stride);
    else if (zprec == VX_F32)
        vx::launch(cg_direction_kernel<1, double, float>, dim3(nb(n, 256), slots), 256, 0, stream, n, S, (const float*)z, p,
                   (float*)z_old, stride);
    else { set_error("vx_batch_cg_direction: unsupported precision %d", zprec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH("vx_batch_cg_direction");
    return VX_OK;
}

// per-slot partials of r . zn (and r . (zn - zo)) at slot * 2 vx_solver_partials(n)
extern "C" int vx_batch_dots_pr(int zprec, int64_t n, int slots, int64_t stride, const double* r, const void* zn,
                                const void* zo, double* partials, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && slots >= 1 && slots <= 65535, VX_ERR_INVALID_ARGUMENT, "vx_batch_dots_pr: bad n/slots");
    VX_CHECK_ARG(r && zn && partials, VX_ERR_NULL_POINTER, "vx_batch_dots_pr: NULL pointer");
    const unsigned G = unsigned(fixed_ctas(n));
    if (zprec == VX_F64)
        vx::launch(dots_pr_kernel<double, double>, dim3(G, slots), FT, 0, stream, n, r, (const double*)zn,
                   (const double*)zo, partials, stride, 0, (double*)nullptr, (unsigned*)nullptr);
    else if (zprec == VX_F32)
        vx::launch(dots_pr_kernel<double, float>, dim3(G, slots), FT, 0, stream, n, r, (const float*)zn,
                   (const float*)zo, partials, stride, 0, (double*)nullptr, (unsigned*)nullptr);
    else { set_error("vx_batch_dots_pr: unsupported precision %d", zprec); return VX_ERR_INVALID_ARGUMENT; }
    VX_CHECK_LAUNCH("vx_batch_dots_pr");
    return VX_OK;
}

// 0: not capturing, 1: capture active, 2: capture invalidated, -1: query failed
extern "C" int vx_capture_status(cudaStream_t stream) {
    cudaStreamCaptureStatus st;
    if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) return -1;
    return st == cudaStreamCaptureStatusNone ? 0 : (st == cudaStreamCaptureStatusActive ? 1 : 2);
}

extern "C" int vx_graph_launch(void* handle, cudaStream_t stream) {
    VX_CHECK_ARG(handle, VX_ERR_NULL_POINTER, "vx_graph_launch: NULL handle");
    auto* w = static_cast<WhileGraph*>(handle);
    VX_CHECK_ARG(w->exec, VX_ERR_INVALID_ARGUMENT, "vx_graph_launch: graph was not instantiated");
    cudaError_t e = cudaGraphLaunch(w->exec, stream);
    if (e != cudaSuccess) {
        set_error("vx_graph_launch: %s", cudaGetErrorString(e));
        return VX_ERR_CUDA;
    }
    return VX_OK;
}

// Number of nodes in the captured loop body (introspection for tests).
extern "C" int64_t vx_graph_body_nodes(void* handle) {
    if (!handle) return -1;
    auto* w = static_cast<WhileGraph*>(handle);
    size_t n = 0;
    if (cudaGraphGetNodes(w->body, nullptr, &n) != cudaSuccess) return -1;
    return int64_t(n);
}

extern "C" int vx_graph_destroy(void* handle) {
    if (!handle) return VX_OK;
    auto* w = static_cast<WhileGraph*>(handle);
    if (w->exec) cudaGraphExecDestroy(w->exec);
    if (w->graph) cudaGraphDestroy(w->graph);
    delete w;
    return VX_OK;
}
