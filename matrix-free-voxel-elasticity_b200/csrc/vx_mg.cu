// Multigrid kernels of the rediscretised voxel hierarchy: trilinear restriction / prolongation,
// modulus and mask coarsening, dense coarse assembly and the dense coarse solve.
// The transfers evaluate the separable per-axis passes in the reference's order (x, then y,
// then z; restriction adds the right neighbour before the left), so FP64 results agree with the
// reference's NumPy transfers to the last bit or within an ulp.
#include "vx_common.cuh"

namespace vx {

__device__ __forceinline__ void node_coords(const Grid& g, int64_t n, int& ix, int& iy, int& iz) {
    iz = int(n % (g.nz + 1));
    iy = int((n / (g.nz + 1)) % (g.ny + 1));
    ix = int(n / (int64_t(g.nz + 1) * (g.ny + 1)));
}

__device__ __forceinline__ int node32(const Grid& g, int ix, int iy, int iz) { return (ix * (g.ny + 1) + iy) * (g.nz + 1) + iz; }

// Restriction: coarse node (I,J,K) of fine grid f: rc = sum w(a) w(b) w(d) f(2I+a, 2J+b, 2K+d), w(0)=1,
// w(+-1)=1/2; arithmetic in arith_t<T> (bf16 storage: FP32).
// A thread owns one word of a fine row span and forms the x and y passes from the nine rows around its
// coarse row (independent, fully coalesced loads; the row shared with the next coarse row is carried over,
// the next rows' loads are in flight over the barrier), the CTA does the z pass through shared memory.  A
// CTA takes rj coarse rows of one coarse plane.  With x != NULL the first sweep of the coarse level from
// zero, x = omega invd r, rides on the store.  The gather of one coarse node per thread that this replaces
// read 27 words with a stride of two nodes and was bound by its load latency.
// Measured (us, L2 flushed, FP32 / bf16 / FP64, before -> now): 576x288x288 276 / 207 / 549 -> 209 / 195 /
// 280 (3.1 TB/s in FP32), 256x128x128 37 / 31 / 63 -> 31 / 27 / 40.
constexpr int RT_MAX = 256, RK_MAX = (RT_MAX / 3 - 1) / 2;       // 42 coarse nodes of a span
template <typename T, typename X>
__global__ void __launch_bounds__(RT_MAX) restrict_kernel(Grid f, Grid c, int rk, int rj, const T* __restrict__ fine,
                                                          const uint8_t* __restrict__ cmask, T* __restrict__ coarse,
                                                          const T* __restrict__ invd, double omega, X* __restrict__ x) {
    vx::pdl_begin();
    using A = arith_t<T>;
    using Raw = typename Storage<T>::raw_t;
    __shared__ A tz[2][RT_MAX];
    const int t = threadIdx.x, I = blockIdx.z, K0 = blockIdx.x * rk;
    const int nk = min(rk, c.nz + 1 - K0);                       // coarse nodes of this CTA's span
    const bool right = 2 * I + 1 <= f.nx, left = I >= 1;
    const int row = 3 * (f.nz + 1), plane = row * (f.ny + 1);
    const int fw = 3 * (2 * K0 - 1) + t;                         // this thread's word of the fine row
    const bool in = t < 3 * (2 * nk + 1) && fw >= 0 && fw < row;
    const T* const base = fine + 2 * I * plane + (in ? fw : 0);
    struct Row { Raw v, r, l; };                                 // unconverted: a conversion would wait for the load
    auto load = [&](int fy) -> Row {                             // the three planes' words of fine row fy
        Row o{Raw(0.0f), Raw(0.0f), Raw(0.0f)};
        if (in && fy >= 0 && fy <= f.ny) {
            const T* p = base + fy * row;
            o.v = Storage<T>::raw(p);
            if (right) o.r = Storage<T>::raw(p + plane);
            if (left) o.l = Storage<T>::raw(p - plane);
        }
        return o;
    };
    auto xpass = [&](const Row& o) -> A {
        A v = Storage<T>::cvt(o.v);
        if (right) v = v + A(0.5) * A(Storage<T>::cvt(o.r));
        if (left) v = v + A(0.5) * A(Storage<T>::cvt(o.l));
        return v;
    };
    const int J0 = blockIdx.y * rj, J1 = min(J0 + rj, c.ny + 1);
    const Row lo = load(2 * J0 - 1);
    Row mi = load(2 * J0), up = load(2 * J0 + 1);
    A below = xpass(lo);
    const bool out = t < 3 * nk;
    const int kk = t / 3, comp = t - 3 * kk, K = K0 + kk, w = t + 3 * kk + 3;      // coarse word t, fine word 2K
    for (int J = J0; J < J1; ++J) {
        A* const buf = tz[J & 1];
        A v = xpass(mi);
        const A above = xpass(up);
        if (2 * J + 1 <= f.ny) v = v + A(0.5) * above;
        if (J >= 1) v = v + A(0.5) * below;
        below = above;
        buf[t] = v;
        if (J + 1 < J1) {
            mi = load(2 * J + 2);
            up = load(2 * J + 3);
        }
        __syncthreads();
        if (out) {
            A s = buf[w];
            if (2 * K + 1 <= f.nz) s = s + A(0.5) * buf[w + 3];
            if (K >= 1) s = s + A(0.5) * buf[w - 3];
            const int n = node32(c, I, J, K);
            const unsigned bits = cmask ? unsigned(cmask[n]) : 7u;
            s = ((bits >> comp) & 1u) ? s : A(0);
            Storage<T>::store(coarse + 3 * n + comp, s);
            if (x) {
                using B = arith_t<X>;
                Storage<X>::store(x + 3 * n + comp, B(omega) * B(Storage<T>::load(invd + 3 * n + comp)) * B(Storage<T>::round(s)));
            }
        }
    }
}
struct RestrictShape { dim3 grid; unsigned threads; int rk, rj; };
// Rows per CTA: the more, the fewer loads are repeated (9 a word at one row, 6.4 at eight) but the longer a
// CTA's chain of dependent rows; eight while about 1000 CTAs are left, fewer on small grids (FP32, 1 / 2 / 4 / 8 rows: 576x288x288
// 373 / 279 / 232 / 209 us, 128x64x64 12.3 / 10.3 / 10.2 / 12.4, 64x32x32 8.2 / 8.2 / 10.2 / 12.3).
inline RestrictShape restrict_shape(const Grid& c) {
    RestrictShape r;
    const int chunks = (c.nz + 1 + RK_MAX - 1) / RK_MAX;
    r.rk = (c.nz + 1 + chunks - 1) / chunks;
    r.rj = 8;
    while (r.rj > 1 && int64_t(chunks) * ((c.ny + r.rj) / r.rj) * (c.nx + 1) < 1000) r.rj /= 2;
    r.grid = dim3(unsigned(chunks), unsigned((c.ny + r.rj) / r.rj), unsigned(c.nx + 1));
    r.threads = unsigned((3 * (2 * r.rk + 1) + 31) / 32 * 32);
    return r;
}

// Prolongation: x(i,j,k) += (P ec)(i,j,k) * mask; P is the separable trilinear interpolation.
// A thread owns one fine word (z, component) of the four fine rows (2I, 2I+1) x (2J, 2J+1), which
// interpolate from the same four coarse rows: at most eight coarse loads feed four updates, and every
// access is a run of consecutive words.  3-D launch, so no thread divides by a grid extent.
// Bound by HBM (4.1 TB/s in FP32); measured (us, L2 flushed, FP32 / bf16 / FP64, one fine node per thread
// -> now): 576x288x288 463 / 557 / 580 -> 309 / 330 / 549, 256x128x128 49 / 59 / 57 -> 41 / 41 / 52.
// SHORT: rows of at most half a CTA; it takes several coarse rows, each on the least power of two of threads that
// holds one (us, FP32, one row a CTA -> now: 74x156x4 4.1 -> 2.6, 102x352x20 10.7 -> 6.2, 576x288x16 44.6 -> 23.1).
constexpr int PT = 128;
template <typename T, bool SHORT>
__global__ void __launch_bounds__(PT) prolong_add_kernel(Grid f, Grid c, const T* __restrict__ coarse,
                                                         const uint8_t* __restrict__ fmask, T* __restrict__ x) {
    vx::pdl_begin();
    using A = arith_t<T>;
    const int w = SHORT ? threadIdx.x : blockIdx.x * PT + threadIdx.x, I = blockIdx.z;
    const int J = SHORT ? blockIdx.y * blockDim.y + threadIdx.y : blockIdx.y;
    if (w >= 3 * (f.nz + 1) || (SHORT && J > c.ny)) return;
    const int k = w / 3, comp = w - 3 * k;
    const bool oz = k & 1, ox = 2 * I + 1 <= f.nx, oy = 2 * J + 1 <= f.ny;
    const int crow = 3 * (c.nz + 1), cplane = crow * (c.ny + 1);
    const T* p = coarse + I * cplane + J * crow + 3 * (k >> 1) + comp;
    const int frow = 3 * (f.nz + 1), fplane = frow * (f.ny + 1);
    T* px = x + 2 * I * fplane + 2 * J * frow + w;
    const uint8_t* pm = fmask ? fmask + (2 * I * (f.ny + 1) + 2 * J) * (f.nz + 1) + k : nullptr;
    A xo[4];
    unsigned bits[4] = {7u, 7u, 7u, 7u};
    #pragma unroll
    for (int q = 0; q < 4; ++q) {                                // (x parity, y parity) = (q & 1, q >> 1)
        if ((q & 1 && !ox) || (q >> 1 && !oy)) continue;
        xo[q] = Storage<T>::load(px + (q & 1) * fplane + (q >> 1) * frow);
        if (fmask) bits[q] = pm[((q & 1) * (f.ny + 1) + (q >> 1)) * (f.nz + 1)];
    }
    A r[2][4];                                                   // the four rows at K and K + 1
    #pragma unroll
    for (int d = 0; d < 2; ++d) {
        if (d && !oz) break;
        const A a = Storage<T>::load(p + 3 * d);
        const A b = ox ? A(Storage<T>::load(p + 3 * d + cplane)) : a;
        const A e = oy ? A(Storage<T>::load(p + 3 * d + crow)) : a;
        const A g = ox && oy ? A(Storage<T>::load(p + 3 * d + cplane + crow)) : a;
        const A ab = A(0.5) * (a + b), eg = A(0.5) * (e + g);
        r[d][0] = a;
        r[d][1] = ab;
        r[d][2] = A(0.5) * (a + e);
        r[d][3] = A(0.5) * (ab + eg);
    }
    #pragma unroll
    for (int q = 0; q < 4; ++q) {
        if ((q & 1 && !ox) || (q >> 1 && !oy)) continue;
        const A v = oz ? A(0.5) * (r[0][q] + r[1][q]) : r[0][q];
        if ((bits[q] >> comp) & 1u) Storage<T>::store(px + (q & 1) * fplane + (q >> 1) * frow, xo[q] + v);
    }
}

template <typename S>
__global__ void coarsen_modulus_kernel(Grid f, Grid c, const S* __restrict__ Ef, S* __restrict__ Ec) {
    vx::pdl_begin();
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= c.elems()) return;
    const int ez = int(e % c.nz), ey = int((e / c.nz) % c.ny), ex = int(e / (int64_t(c.nz) * c.ny));
    double s = 0.0;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            for (int d = 0; d < 2; ++d) s += double(Storage<S>::load(Ef + f.elem(2 * ex + a, 2 * ey + b, 2 * ez + d)));
    Storage<S>::store(Ec + e, decltype(Storage<S>::load(Ef))(s * 0.125));
}

__global__ void coarsen_mask_kernel(Grid f, Grid c, const uint8_t* __restrict__ mf, uint8_t* __restrict__ mc) {
    vx::pdl_begin();
    const int64_t n = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (n >= c.nodes()) return;
    int I, J, K;
    node_coords(c, n, I, J, K);
    mc[n] = mf[f.node(2 * I, 2 * J, 2 * K)];
}

struct Ke576 { double k[576]; };

// one thread per (row DOF, neighbour offset, column component); A is zeroed beforehand
__global__ void assemble_dense_kernel(Grid g, const __grid_constant__ Ke576 ke, const double* __restrict__ E,
                                      const uint8_t* __restrict__ mask, double* __restrict__ A) {
    vx::pdl_begin();
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t nn = g.nodes();
    if (t >= nn * 3 * 81) return;
    const int64_t row = t / 81;
    const int rem = int(t % 81);
    const int off = rem / 3, cd = rem % 3;
    const int64_t nr = row / 3;
    const int cr = int(row % 3);
    int ix, iy, iz;
    node_coords(g, nr, ix, iy, iz);
    const int ox = off % 3 - 1, oy = (off / 3) % 3 - 1, oz = off / 9 - 1;
    const int mx = ix + ox, my = iy + oy, mz = iz + oz;
    if (mx < 0 || mx > g.nx || my < 0 || my > g.ny || mz < 0 || mz > g.nz) return;
    constexpr int nat[8] = {0, 1, 3, 2, 4, 5, 7, 6};
    double v = 0.0;
    for (int bx = 0; bx < 2; ++bx) for (int by = 0; by < 2; ++by) for (int bz = 0; bz < 2; ++bz) {
        const int ex = ix - 1 + bx, ey = iy - 1 + by, ez = iz - 1 + bz;   // element containing the row node
        if (ex < 0 || ex >= g.nx || ey < 0 || ey >= g.ny || ez < 0 || ez >= g.nz) continue;
        const int qx = mx - ex, qy = my - ey, qz = mz - ez;              // column node's offset in it
        if (qx < 0 || qx > 1 || qy < 0 || qy > 1 || qz < 0 || qz > 1) continue;
        const int li = nat[(1 - bx) + 2 * (1 - by) + 4 * (1 - bz)];
        const int lj = nat[qx + 2 * qy + 4 * qz];
        v += E[g.elem(ex, ey, ez)] * ke.k[(3 * li + cr) * 24 + 3 * lj + cd];
    }
    const int64_t col = 3 * g.node(mx, my, mz) + cd;
    const double mr = mask ? double((mask[nr] >> cr) & 1u) : 1.0;
    const double mcv = mask ? double((mask[col / 3] >> cd) & 1u) : 1.0;
    double out = mr * v * mcv;
    if (col == row) out += 1.0 - mr;
    A[row * (nn * 3) + col] = out;
}

// sum over j in [j0, j1) of row[j] * v(j) by one CTA of CT threads (stride CT), reduced in a fixed
// order.  A CTA per row keeps each thread's dependent chain short: with a warp per row, every warp
// is resident at once and the launch lasts as long as one warp's walk along a full row.
constexpr int CT = 256;
template <typename V>
__device__ __forceinline__ double block_row_dot(const double* __restrict__ row, int j0, int j1, V v) {
    __shared__ double red[CT / 32];
    double s = 0.0;
    for (int j = j0 + int(threadIdx.x); j < j1; j += CT) s = fma(row[j], v(j), s);
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < CT / 32; ++k) t += red[k];
    return t;                                                   // valid in thread 0
}

// z = (Ainv r) * mask, one CTA per row, FP64 accumulation
template <typename TR, typename T>
__global__ void __launch_bounds__(CT) coarse_apply_kernel(int n, const double* __restrict__ Ainv,
                                                          const TR* __restrict__ r, const uint8_t* __restrict__ mask,
                                                          T* __restrict__ z) {
    vx::pdl_begin();
    using A = arith_t<T>;
    const int row = blockIdx.x;
    const double s = block_row_dot(Ainv + int64_t(row) * n, 0, n, [&](int j) { return double(Storage<TR>::load(r + j)); });
    if (threadIdx.x == 0) {
        const bool fr = mask ? ((mask[row / 3] >> (row % 3)) & 1u) : true;
        Storage<T>::store(z + row, fr ? A(s) : A(0));
    }
}

// Packed inverse factor: M = tril(Linv) + triu(Linv^T, 1), Linv = L^-1 of A = L L^T, so
// A^-1 r = Linv^T (Linv r) reads row i of M left of the diagonal (pass 1) and right of it (pass 2).
// 32x32 tiles through shared memory keep the transposed reads coalesced.
__global__ void coarse_pack_kernel(int n, const double* __restrict__ linv, double* __restrict__ m) {
    vx::pdl_begin();
    __shared__ double tile[32][33];
    const int bi = blockIdx.y * 32, bj = blockIdx.x * 32;      // output tile rows bi.., cols bj..
    const int tx = threadIdx.x, ty = threadIdx.y;              // 32 x 8 threads
    if (bj > bi) {                                             // strictly-upper tile: read Linv^T
        for (int k = ty; k < 32; k += 8) {
            const int r = bj + k, c = bi + tx;                 // source element Linv[r][c]
            tile[k][tx] = (r < n && c < n) ? linv[int64_t(r) * n + c] : 0.0;
        }
        __syncthreads();
        for (int k = ty; k < 32; k += 8) {
            const int i = bi + k, j = bj + tx;
            if (i < n && j < n) m[int64_t(i) * n + j] = tile[tx][k];
        }
    } else {                                                   // lower or diagonal tile
        for (int k = ty; k < 32; k += 8) {
            const int i = bi + k, j = bj + tx;
            if (i < n && j < n) {
                if (j <= i) m[int64_t(i) * n + j] = linv[int64_t(i) * n + j];
                else m[int64_t(i) * n + j] = linv[int64_t(j) * n + i];    // diagonal tile, upper part
            }
        }
    }
}

// pass 1: y = Linv r (row i, columns 0..i of M), one CTA per row, FP64 accumulation.
// Batches: system blockIdx.y has its factor at m + slot * n^2, its vectors at slot * vs, y at slot * n.
template <typename TR>
__global__ void __launch_bounds__(CT) coarse_lower_kernel(int n, const double* __restrict__ m,
                                                          const TR* __restrict__ r, double* __restrict__ y, int64_t vs) {
    vx::pdl_begin();
    const int row = blockIdx.x;
    m += int64_t(n) * n * blockIdx.y;
    r += vs * blockIdx.y;
    y += int64_t(n) * blockIdx.y;
    const double s = block_row_dot(m + int64_t(row) * n, 0, row + 1, [&](int j) { return double(Storage<TR>::load(r + j)); });
    if (threadIdx.x == 0) y[row] = s;
}

// pass 2: z = Linv^T y (row i: the diagonal Linv[i][i] and columns i+1.. of M), masked
template <typename T>
__global__ void __launch_bounds__(CT) coarse_upper_kernel(int n, const double* __restrict__ m,
                                                          const double* __restrict__ y,
                                                          const uint8_t* __restrict__ mask, T* __restrict__ z, int64_t vs) {
    vx::pdl_begin();
    using A = arith_t<T>;
    const int row = blockIdx.x;
    m += int64_t(n) * n * blockIdx.y;
    y += int64_t(n) * blockIdx.y;
    z += vs * blockIdx.y;
    if (mask) mask += (vs / 3) * blockIdx.y;
    const double s = block_row_dot(m + int64_t(row) * n, row, n, [&](int j) { return y[j]; });
    if (threadIdx.x == 0) {
        const bool fr = mask ? ((mask[row / 3] >> (row % 3)) & 1u) : true;
        Storage<T>::store(z + row, fr ? A(s) : A(0));
    }
}

__global__ void mask_from_dofs_kernel(int64_t nodes, const double* __restrict__ m, uint8_t* __restrict__ out) {
    vx::pdl_begin();
    const int64_t n = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (n >= nodes) return;
    out[n] = uint8_t((m[3 * n] != 0.0) | ((m[3 * n + 1] != 0.0) << 1) | ((m[3 * n + 2] != 0.0) << 2));
}

inline unsigned blocks_for(int64_t n, int t) { return unsigned((n + t - 1) / t); }

int check_even(int nx, int ny, int nz, const char* what) {
    int st = check_grid(nx, ny, nz);
    if (st) return st;
    if (nx + 1 > 65535 || (ny + 2) / 2 > 65535) {                    // grid dimensions of the transfer launches
        set_error("%s: fine grid (%d, %d, %d) is too long in x or y for one launch", what, nx, ny, nz);
        return VX_ERR_INVALID_ARGUMENT;
    }
    if ((nx | ny | nz) & 1) {
        set_error("%s: fine grid (%d, %d, %d) must have even extents", what, nx, ny, nz);
        return VX_ERR_INVALID_ARGUMENT;
    }
    return VX_OK;
}

}  // namespace vx

using namespace vx;

namespace {
int launch_restrict(const char* what, int prec, int nx, int ny, int nz, const void* fine, const uint8_t* coarse_mask,
                    void* coarse, const void* invd, double omega, void* x, cudaStream_t stream) {
    int st = check_even(nx, ny, nz, what);
    if (st) return st;
    VX_CHECK_ARG(fine && coarse, VX_ERR_NULL_POINTER, "%s: NULL pointer", what);
    Grid f{nx, ny, nz}, c{nx / 2, ny / 2, nz / 2};
    const RestrictShape r = restrict_shape(c);
    const bool ok = dispatch_prec(prec, [&](auto t) {             // auxiliary vectors on both sides
        using R = typename decltype(t)::R;
        using X = typename decltype(t)::X;
        vx::launch(restrict_kernel<R, X>, r.grid, r.threads, 0, stream, f, c, r.rk, r.rj, (const R*)fine, coarse_mask, (R*)coarse,
                   (const R*)invd, omega, (X*)x);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "%s: unsupported precision %d", what, prec);
    VX_CHECK_LAUNCH(what);
    return VX_OK;
}
}  // namespace

extern "C" int vx_restrict(int prec, int nx, int ny, int nz, const void* fine, const uint8_t* coarse_mask,
                           void* coarse, cudaStream_t stream) {
    return launch_restrict("vx_restrict", prec, nx, ny, nz, fine, coarse_mask, coarse, nullptr, 0.0, nullptr, stream);
}

extern "C" int vx_restrict_sweep(int prec, int nx, int ny, int nz, const void* fine, const uint8_t* coarse_mask,
                                 void* coarse, const void* inv_diag, double omega, void* x, cudaStream_t stream) {
    VX_CHECK_ARG(inv_diag && x, VX_ERR_NULL_POINTER, "vx_restrict_sweep: NULL pointer");
    return launch_restrict("vx_restrict_sweep", prec, nx, ny, nz, fine, coarse_mask, coarse, inv_diag, omega, x, stream);
}

extern "C" int vx_prolong_add(int prec, int nx, int ny, int nz, const void* coarse, const uint8_t* fine_mask,
                              void* x, cudaStream_t stream) {
    int st = check_even(nx, ny, nz, "vx_prolong_add");
    if (st) return st;
    VX_CHECK_ARG(coarse && x, VX_ERR_NULL_POINTER, "vx_prolong_add: NULL pointer");
    Grid f{nx, ny, nz}, c{nx / 2, ny / 2, nz / 2};
    const bool ok = dispatch_prec(prec, [&](auto t) {             // iterates on both sides
        using X = typename decltype(t)::X;
        unsigned tx = PT;
        while (tx > 16 && tx / 2 >= 3 * (unsigned(nz) + 1)) tx /= 2;
        const dim3 grid(blocks_for(3 * (int64_t(nz) + 1), tx), blocks_for(c.ny + 1, PT / tx), unsigned(c.nx + 1));
        vx::launch(tx < PT ? prolong_add_kernel<X, true> : prolong_add_kernel<X, false>, grid, dim3(tx, PT / tx), 0, stream, f, c,
                   (const X*)coarse, fine_mask, (X*)x);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_prolong_add: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_prolong_add");
    return VX_OK;
}

extern "C" int vx_coarsen_modulus(int prec, int nx, int ny, int nz, const void* E_fine, void* E_coarse,
                                  cudaStream_t stream) {
    int st = check_even(nx, ny, nz, "vx_coarsen_modulus");
    if (st) return st;
    VX_CHECK_ARG(E_fine && E_coarse, VX_ERR_NULL_POINTER, "vx_coarsen_modulus: NULL pointer");
    Grid f{nx, ny, nz}, c{nx / 2, ny / 2, nz / 2};
    const unsigned gb = blocks_for(c.elems(), 256);
    const bool ok = dispatch_prec(prec, [&](auto t) {
        using M = typename decltype(t)::M;
        vx::launch(coarsen_modulus_kernel<M>, gb, 256, 0, stream, f, c, (const M*)E_fine, (M*)E_coarse);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_coarsen_modulus: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_coarsen_modulus");
    return VX_OK;
}

extern "C" int vx_coarsen_mask(int nx, int ny, int nz, const uint8_t* mask_fine, uint8_t* mask_coarse,
                               cudaStream_t stream) {
    int st = check_even(nx, ny, nz, "vx_coarsen_mask");
    if (st) return st;
    VX_CHECK_ARG(mask_fine && mask_coarse, VX_ERR_NULL_POINTER, "vx_coarsen_mask: NULL pointer");
    Grid f{nx, ny, nz}, c{nx / 2, ny / 2, nz / 2};
    vx::launch(coarsen_mask_kernel, blocks_for(c.nodes(), 256), 256, 0, stream, f, c, mask_fine, mask_coarse);
    VX_CHECK_LAUNCH("vx_coarsen_mask");
    return VX_OK;
}

extern "C" int vx_assemble_dense(int nx, int ny, int nz, const double* ke, const double* E,
                                 const uint8_t* node_mask, double* A, cudaStream_t stream) {
    int st = check_grid(nx, ny, nz);
    if (st) return st;
    VX_CHECK_ARG(ke && E && A, VX_ERR_NULL_POINTER, "vx_assemble_dense: NULL pointer");
    Grid g{nx, ny, nz};
    const int64_t n = 3 * g.nodes();
    VX_CHECK_ARG(n <= 65536, VX_ERR_INVALID_ARGUMENT, "vx_assemble_dense: %lld DOFs is too many for a dense matrix",
                 (long long)n);
    Ke576 k;
    for (int i = 0; i < 576; ++i) k.k[i] = ke[i];
    cudaError_t e = cudaMemsetAsync(A, 0, size_t(n) * size_t(n) * sizeof(double), stream);
    if (e != cudaSuccess) { set_error("vx_assemble_dense: memset: %s", cudaGetErrorString(e)); return VX_ERR_CUDA; }
    vx::launch(assemble_dense_kernel, blocks_for(g.nodes() * 243, 256), 256, 0, stream, g, k, E, node_mask, A);
    VX_CHECK_LAUNCH("vx_assemble_dense");
    return VX_OK;
}

extern "C" int vx_coarse_apply(int prec, int n, const double* Ainv, const void* r, const uint8_t* node_mask,
                               void* z, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_coarse_apply: n must be positive");
    VX_CHECK_ARG(Ainv && r && z, VX_ERR_NULL_POINTER, "vx_coarse_apply: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {             // r auxiliary, z an iterate
        using R = typename decltype(t)::R;
        using X = typename decltype(t)::X;
        vx::launch(coarse_apply_kernel<R, X>, unsigned(n), CT, 0, stream, n, Ainv, (const R*)r, node_mask, (X*)z);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_coarse_apply: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_coarse_apply");
    return VX_OK;
}

extern "C" int vx_mask_from_dofs(int64_t nodes, const double* dof_mask, uint8_t* node_mask, cudaStream_t stream) {
    VX_CHECK_ARG(nodes > 0, VX_ERR_INVALID_ARGUMENT, "vx_mask_from_dofs: nodes must be positive");
    VX_CHECK_ARG(dof_mask && node_mask, VX_ERR_NULL_POINTER, "vx_mask_from_dofs: NULL pointer");
    vx::launch(mask_from_dofs_kernel, blocks_for(nodes, 256), 256, 0, stream, nodes, dof_mask, node_mask);
    VX_CHECK_LAUNCH("vx_mask_from_dofs");
    return VX_OK;
}

extern "C" int vx_coarse_pack(int n, const double* linv, double* m, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_coarse_pack: n must be positive");
    VX_CHECK_ARG(linv && m, VX_ERR_NULL_POINTER, "vx_coarse_pack: NULL pointer");
    VX_CHECK_ARG(linv != m, VX_ERR_INVALID_ARGUMENT, "vx_coarse_pack: m may not alias linv");
    const unsigned t = unsigned((n + 31) / 32);
    vx::launch(coarse_pack_kernel, dim3(t, t), dim3(32, 8), 0, stream, n, linv, m);
    VX_CHECK_LAUNCH("vx_coarse_pack");
    return VX_OK;
}

extern "C" int vx_coarse_apply_factor(int prec, int n, const double* m, const void* r, const uint8_t* node_mask,
                                      double* y, void* z, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0, VX_ERR_INVALID_ARGUMENT, "vx_coarse_apply_factor: n must be positive");
    VX_CHECK_ARG(m && r && y && z, VX_ERR_NULL_POINTER, "vx_coarse_apply_factor: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {             // r auxiliary, z an iterate
        using R = typename decltype(t)::R;
        using X = typename decltype(t)::X;
        vx::launch(coarse_lower_kernel<R>, unsigned(n), CT, 0, stream, n, m, (const R*)r, y, int64_t(0));
        vx::launch(coarse_upper_kernel<X>, unsigned(n), CT, 0, stream, n, m, y, node_mask, (X*)z, int64_t(0));
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_coarse_apply_factor: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_coarse_apply_factor");
    return VX_OK;
}

// The same for `slots` independent coarse systems: factors back to back (slot k at m + k n^2), the
// right-hand side, mask and solution of slot k at k * vs DOFs (vs a multiple of 3), y holding
// slots * n doubles.
extern "C" int vx_batch_coarse_apply_factor(int prec, int n, int slots, int64_t vs, const double* m, const void* r,
                                            const uint8_t* node_mask, double* y, void* z, cudaStream_t stream) {
    VX_CHECK_ARG(n > 0 && slots >= 1 && slots <= 65535 && vs >= n && vs % 3 == 0, VX_ERR_INVALID_ARGUMENT,
                 "vx_batch_coarse_apply_factor: bad n/slots/stride");
    VX_CHECK_ARG(m && r && y && z, VX_ERR_NULL_POINTER, "vx_batch_coarse_apply_factor: NULL pointer");
    const bool ok = dispatch_prec(prec, [&](auto t) {
        using R = typename decltype(t)::R;
        using X = typename decltype(t)::X;
        vx::launch(coarse_lower_kernel<R>, dim3(n, slots), CT, 0, stream, n, m, (const R*)r, y, vs);
        vx::launch(coarse_upper_kernel<X>, dim3(n, slots), CT, 0, stream, n, m, y, node_mask, (X*)z, vs);
    });
    VX_CHECK_ARG(ok, VX_ERR_INVALID_ARGUMENT, "vx_batch_coarse_apply_factor: unsupported precision %d", prec);
    VX_CHECK_LAUNCH("vx_batch_coarse_apply_factor");
    return VX_OK;
}
