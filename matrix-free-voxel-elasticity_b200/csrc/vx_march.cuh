// parity_march: the streaming operator with the stages in the order y, z, x.
//
// The separable 2x2x2 transform hands 3 values per node to its first stage, 6 to its second and 12 to
// its third, so the dearest exchange belongs in the direction that costs nothing: a CTA marches along
// x and keeps the twelve y-z transformed values of the previous node plane (and the twelve pending
// contributions to the next one) in registers.  The y stage exchanges 3 values with the next node row
// through shared memory, the z stage 6 with the next lane by shuffles; the inverse runs z, y the same
// way back.  Per element that is half the shuffles' and half the shared-memory traffic of the order
// x, y, z (parity_stream_xp: 6 through shared memory, 12 by shuffles each way).
//
// A thread owns one z column of one node row in FP64, and of two node rows half a tile apart in FP32, whose
// values travel as packed f32x2 pairs that are never taken apart: only the rows at the seam between the two
// halves swap a half when they read a neighbour row.  A tile's outer rows and columns are halo.
//
// The parity blocks couple the x, y and z components of one (py, pz) class only with their own px = 0, 1
// values, so each class is finished before the next one starts: six block inputs are live, not 24.
//
// One CTA barrier per node plane: the masked operand of plane e + 2 and the inverse-y contributions of
// plane e are written before it; their readers (rows above and below) come after it.  The operand ring
// has three planes (own read of plane e, neighbour read of e + 1, write of e + 2), the contributions two.
//
// What bounds it: the FP64 forms the double-precision pipe (150 of about 296 issued instructions an element
// row, half busy) together with the latency between its barriers, the FP32 sweep HBM, issue and registers.
// Eight warps and two CTAs an SM (128 registers) let one CTA compute while the other waits at its barrier;
// measured at 576x288x288 (us, matvec FP64 / FP32, Jacobi FP64 / FP32) before the changes noted below: 2 x 8
// warps 1053 / 513 / 1193 / 606, 1 x 12 warps 1137 / 562 / 1242 / 685, 1 x 16 warps 1193 / 550 / 1250 / 610, named
// barriers between neighbouring rows 1102 / 551 (matvecs).  As it is now: 960 / 484 / 1081 / 609 (2.9, 3.3, 4.2
// and 4.2 TB/s); parity_stream_xp: 1405 / 638 / 1615 / 732.
#pragma once

namespace vx {

// one FP64 value in the interface of the pairs of vx_pair.cuh
struct V1 { double x; };
__device__ __forceinline__ V1 add2(V1 a, V1 b) { return {a.x + b.x}; }
__device__ __forceinline__ V1 sub2(V1 a, V1 b) { return {a.x - b.x}; }
__device__ __forceinline__ V1 mul2(V1 a, V1 b) { return {a.x * b.x}; }
__device__ __forceinline__ V1 fma2(V1 a, V1 b, V1 c) { return {fma(a.x, b.x, c.x)}; }
__device__ __forceinline__ V1 cmul2(double c, V1 a) { return {c * a.x}; }
__device__ __forceinline__ V1 cfma2(double c, V1 a, V1 acc) { return {fma(c, a.x, acc.x)}; }
// exchange with the next / previous lane of a row of LZ lanes (its last / first lane keeps its own value)
template <int LZ> __device__ __forceinline__ V1 next_lane(V1 a) { return {__shfl_down_sync(0xffffffffu, a.x, 1, LZ)}; }
template <int LZ> __device__ __forceinline__ V1 prev_lane(V1 a) { return {__shfl_up_sync(0xffffffffu, a.x, 1, LZ)}; }
template <int LZ> __device__ __forceinline__ V2<float> next_lane(V2<float> a) {
    const unsigned long long b = __shfl_down_sync(0xffffffffu, *reinterpret_cast<const unsigned long long*>(&a.v), 1, LZ);
    return {*reinterpret_cast<const float2*>(&b)};
}
template <int LZ> __device__ __forceinline__ V2<float> prev_lane(V2<float> a) {
    const unsigned long long b = __shfl_up_sync(0xffffffffu, *reinterpret_cast<const unsigned long long*>(&a.v), 1, LZ);
    return {*reinterpret_cast<const float2*>(&b)};
}

template <typename TC, int N> struct MarchPack;
template <typename TC> struct MarchPack<TC, 1> {
    using P = V1;
    __device__ static __forceinline__ P make(const TC* v) { return {v[0]}; }
    __device__ static __forceinline__ TC get(P p, int) { return p.x; }
};
template <typename TC> struct MarchPack<TC, 2> {
    using P = V2<TC>;
    __device__ static __forceinline__ P make(const TC* v) { return mk2(v[0], v[1]); }
    __device__ static __forceinline__ TC get(P p, int c) { return c ? p.hi() : p.lo(); }
};
template <typename TC> struct March;
// Lanes per node row.  A row of 32 lanes owns 30 columns; in FP64, where a CTA has only eight warps of single
// rows, rows of 16 lanes (two a warp) make the tile 14 x 14 of 16 x 16 nodes instead of 6 x 30 of 8 x 32: 77%
// of the lanes own a node instead of 70%, and the node counts 2^k + 1 waste less of the last tile (128x64x64
// 21.5 -> 16.1 us, 192x96x96 57 -> 38, 576x288x288 1017 -> 898; rows of 8 lanes 23.5, 62, 1068).  The FP32 tile
// is 14 x 30 of 16 x 32 either way round; 32 lanes coalesce better (484 us against 508).
template <> struct March<double> : MarchPack<double, 1> { static constexpr int N = 1, NW = 8, MINB = 2, LZ = 16; };
template <> struct March<float> : MarchPack<float, 2> { static constexpr int N = 2, NW = 8, MINB = 2, LZ = 32; };
template <typename TC> constexpr int march_rows() { return March<TC>::N * March<TC>::NW * 32 / March<TC>::LZ; }
template <typename TC> constexpr size_t march_smem() { return size_t(5) * 3 * March<TC>::NW * 32 * sizeof(typename March<TC>::P); }

// The block products of class (py, pz): s[c], d[c] are the px = 0 and px = 1 inputs of component c (at the
// class's parities), replaced by the outputs.  The component whose (py, pz) is (0, 0) has no px = 0 value
// (a translation); its s is left alone.
template <typename TC, bool CUBIC, int PY, int PZ, typename P, typename Args>
__device__ __forceinline__ void march_blocks(const Args& args, P (&s)[3], P (&d)[3]) {
    if constexpr (CUBIC) {
        const auto& K = args.M;
        auto cd = [&](P other, P self) { return cfma2(K.d, other, cmul2(K.c, self)); };      // a row of [c d; d c]
        if constexpr (PY == 0 && PZ == 0) {
            const P bs = cmul2(K.b0, add2(add2(d[0], s[1]), s[2]));          // g0: x@1 y@2 z@4
            d[0] = cfma2(K.amb0, d[0], bs);
            s[1] = cfma2(K.amb0, s[1], bs);
            s[2] = cfma2(K.amb0, s[2], bs);
            const P a1 = d[1], a2 = d[2];                                    // g1: y@3 z@5
            d[1] = cd(a2, a1);
            d[2] = cd(a1, a2);
        } else if constexpr (PY == 1 && PZ == 0) {
            const P a0 = d[0], a2 = s[2];                                    // g2: x@3 z@6
            d[0] = cd(a2, a0);
            s[2] = cd(a0, a2);
            const P t = cmul2(K.e, add2(s[0], d[1]));                        // g3: x@2 y@1, z@7
            s[0] = t;
            d[1] = t;
            d[2] = cmul2(K.f, d[2]);
        } else if constexpr (PY == 0 && PZ == 1) {
            const P a0 = d[0], a1 = s[1];                                    // g4: x@5 y@6
            d[0] = cd(a1, a0);
            s[1] = cd(a0, a1);
            const P t = cmul2(K.e, add2(s[0], d[2]));                        // g5: x@4 z@1, y@7
            s[0] = t;
            d[2] = t;
            d[1] = cmul2(K.f, d[1]);
        } else {
            const P t = cmul2(K.e, add2(s[1], s[2]));                        // g6: y@4 z@2, x@7
            s[1] = t;
            s[2] = t;
            d[0] = cmul2(K.f, d[0]);
            const P ks = cmul2(K.k7, add2(add2(s[0], d[1]), d[2]));          // g7: x@6 y@5 z@3
            s[0] = cfma2(K.hmk7, s[0], ks);
            d[1] = cfma2(K.hmk7, d[1], ks);
            d[2] = cfma2(K.hmk7, d[2], ks);
        }
    } else {
        constexpr int g0 = 2 * PY + 4 * PZ;
        #pragma unroll
        for (int h = 0; h < 2; ++h) {                        // group g0: x@px=1, y, z@px=0; g0 + 1: the others
            const int g = g0 + h;
            const P in[3] = {h ? s[0] : d[0], h ? d[1] : s[1], h ? d[2] : s[2]};
            #pragma unroll
            for (int r = 0; r < 3; ++r) {
                if ((g ^ (1 << r)) == 0) continue;
                P acc = in[0];
                bool first = true;
                #pragma unroll
                for (int cc = 0; cc < 3; ++cc) {
                    if (!parity_nonzero(g, r, cc)) continue;
                    const auto coef = args.C2.c[9 * g + 3 * r + cc];
                    acc = first ? cmul2(coef, in[cc]) : cfma2(coef, in[cc], acc);
                    first = false;
                }
                if ((r == 0) == (h == 0)) d[r] = acc;
                else s[r] = acc;
            }
        }
    }
}

template <typename TC, typename TU, typename TE, typename TY, typename TR, int EPI, int MASK, bool CUBIC>
__global__ void __launch_bounds__(March<TC>::NW * 32, March<TC>::MINB)
parity_march(const __grid_constant__ OpArgs2<TC, TU, TE, TY, TR> args) {
    vx::pdl_begin();
    using C = March<TC>;
    using P = typename C::P;
    constexpr int N = C::N, LZ = C::LZ, ROWS = C::NW * 32 / LZ, OWN = N * ROWS - 2, OWNZ = LZ - 2;
    constexpr bool HAS_R = EPI == EPI_JACOBI || EPI == EPI_RESIDUAL || EPI == EPI_TRUE_RES;
    constexpr bool HAS_D = EPI == EPI_JACOBI;
    // does the epilogue read the operand at the output node?
    constexpr bool USES_X = EPI == EPI_JACOBI || EPI == EPI_APPLY_DOT;
    // Most forms run the planes inside the grid in a loop without tests (FP32 matvec 513 -> 483 us at
    // 576x288x288) and, in FP32, test a warp's masks by a vote.  The forms that have no registers left for a
    // second step loop keep one (FP32 sweep 603 us, with it 701; FP64 apply 976, with it 1000).
    constexpr bool LEAN = N == 2 ? EPI == EPI_JACOBI || EPI == EPI_TRUE_RES : EPI == EPI_APPLY_DOT;
    constexpr bool VOTE = N == 2 && !LEAN;
    // The x stage's E (p +- c) is E p +- E c by multiply-adds, or the sum times E: one FP64 operation more a value, yet
    // the faster schedule in all FP64 forms but one (576x288x288, multiply-adds -> sums: matvec 1043 -> 960 us, sweep
    // 1138 -> 1081, true residual 1027 -> 1008, apply 1029 -> 1031, residual 1000 -> 1154; FP32 matvec 483 -> 494).
    constexpr bool SUM_FIRST = N == 1 && EPI != EPI_RESIDUAL;
    const auto& a = args.a;
    const int lane = threadIdx.x % LZ;                       // node column of the row
    const int row = threadIdx.x / LZ;
    const Grid g = a.g;
    const int iz = blockIdx.x * OWNZ - 1 + lane;
    const int x0 = blockIdx.z * a.cx;
    const int x1 = min(x0 + a.cx, g.nx + 1);                 // owned node planes [x0, x1)
    const int plane_nodes = (g.ny + 1) * (g.nz + 1);
    const int plane_elems = g.ny * g.nz;

    // Clamped (always in-bounds) offsets: a node outside the grid only meets elements outside the grid,
    // whose modulus is 0.  They fit in 32 bits (fewer than 2^31 DOFs).  n_in / e_in / n_out: this thread's
    // node of the plane in flight, element of the next element plane, node of the output plane.
    int n_in[N], e_in[N], n_out[N];
    bool owner[N], elem_ok[N];
    const int pl0 = max(x0 - 1, 0);
    #pragma unroll
    for (int c = 0; c < N; ++c) {
        const int rr = row + c * ROWS, iy = blockIdx.y * OWN - 1 + rr;
        owner[c] = iy >= 0 && iy <= g.ny && iz >= 0 && iz <= g.nz && lane >= 1 && lane <= OWNZ && rr >= 1 && rr <= OWN;
        elem_ok[c] = iy >= 0 && iy < g.ny && iz >= 0 && iz < g.nz && lane < LZ - 1 && rr < N * ROWS - 1;
        const int cn = min(max(iy, 0), g.ny) * (g.nz + 1) + min(max(iz, 0), g.nz);
        n_in[c] = pl0 * plane_nodes + cn;
        n_out[c] = (x0 - 1) * plane_nodes + cn;              // plane x0 - 1 is never stored
        e_in[c] = (x0 - 1) * plane_elems + min(max(iy, 0), g.ny - 1) * g.nz + min(max(iz, 0), g.nz - 1);
    }

    extern __shared__ __align__(16) unsigned char smem_raw[];
    P* const us = reinterpret_cast<P*>(smem_raw);            // operand ring: 3 planes x ROWS x 3 x LZ
    P* const hs = us + 3 * ROWS * 3 * LZ;                         // inverse-y contributions: 2 planes
    const int own_at = row * 3 * LZ + lane;
    const int up_at = (row + 1 < ROWS ? row + 1 : (N == 2 ? 0 : row)) * 3 * LZ + lane;
    const int dn_at = (row > 0 ? row - 1 : (N == 2 ? ROWS - 1 : 0)) * 3 * LZ + lane;

    typename Storage<TU>::raw_t ur[N][3];                    // operand of the plane in flight
    uint8_t um[N];
    typename Storage<TE>::raw_t er[N];                       // modulus of the next element plane
    // loads of node plane ix (then moves on to ix + 1) and of element plane ex (then ex + 1)
    auto load_u = [&](int ix, bool inside = false) {
        const int step = inside || (ix >= 0 && ix < g.nx) ? plane_nodes : 0;
        #pragma unroll
        for (int c = 0; c < N; ++c) {
            const TU* p = a.u + 3 * n_in[c];
            #pragma unroll
            for (int k = 0; k < 3; ++k) ur[c][k] = Storage<TU>::raw(p + k);
            if constexpr (MASK == MASK_NODE) um[c] = a.node_mask[n_in[c]];
            n_in[c] += step;
        }
    };
    auto load_e = [&](int ex, bool inside = false) {
        const bool in = inside || (ex >= 0 && ex < g.nx);
        #pragma unroll
        for (int c = 0; c < N; ++c) {
            er[c] = typename Storage<TE>::raw_t(0.0f);
            if (in && elem_ok[c]) er[c] = Storage<TE>::raw(a.E + e_in[c]);
            e_in[c] += plane_elems;
        }
    };
    // the plane in flight: masked operand to ring slot `at`; returns its mask bits (8 per column)
    auto put_u = [&](int at) -> unsigned {
        unsigned bits = 0x0707;
        TC v[3][N];
        #pragma unroll
        for (int k = 0; k < 3; ++k)
            #pragma unroll
            for (int c = 0; c < N; ++c) v[k][c] = TC(Storage<TU>::cvt(ur[c][k]));
        if constexpr (MASK == MASK_NODE) {
            bits = N == 2 ? unsigned(um[0]) | unsigned(um[N - 1]) << 8 : unsigned(um[0]) | 0x0700u;
            if (!VOTE ? (bits & 0x0707u) != 0x0707u : !__all_sync(0xffffffffu, (bits & 0x0707u) == 0x0707u)) {   // a fixed DOF
                #pragma unroll
                for (int k = 0; k < 3; ++k)
                    #pragma unroll
                    for (int c = 0; c < N; ++c)
                        if (!((um[c] >> k) & 1u)) v[k][c] = TC(0);
            }
        }
        #pragma unroll
        for (int k = 0; k < 3; ++k) us[at + own_at + LZ * k] = C::make(v[k]);
        return bits;
    };
    // y stage of a ring plane: ya[c][py] at this row's face
    auto y_stage = [&](int at, P (&ya)[3][2]) {
        #pragma unroll
        for (int k = 0; k < 3; ++k) {
            const P o = us[at + own_at + LZ * k];
            P n = us[at + up_at + LZ * k];
            if constexpr (N == 2) { if (row == ROWS - 1) n = mk2(n.hi(), n.hi()); }   // row ROWS is the other half's row 0
            ya[k][0] = add2(o, n);
            ya[k][1] = sub2(o, n);
        }
    };

    constexpr int RING = ROWS * 3 * LZ;
    P pp[3][2][2];                                           // y-z transformed operand of node plane e
    P gg[3][2][2];                                           // element plane e-1's contributions to node plane e
    unsigned bits0, bits1, bits2 = 0;                        // mask bits of node planes e, e+1, e+2
    load_u(x0 - 1);
    load_e(x0 - 1);
    bits0 = put_u(0);
    load_u(x0);
    bits1 = put_u(RING);
    load_u(x0 + 1);
    __syncthreads();
    {
        P ya[3][2];
        y_stage(0, ya);
        #pragma unroll
        for (int k = 0; k < 3; ++k)
            #pragma unroll
            for (int py = 0; py < 2; ++py) {
                const P yb = next_lane<LZ>(ya[k][py]);
                pp[k][py][0] = add2(ya[k][py], yb);
                pp[k][py][1] = sub2(ya[k][py], yb);
                const TC z[2] = {TC(0), TC(0)};
                gg[k][py][0] = gg[k][py][1] = C::make(z);
            }
    }
    int at0 = 0, at1 = RING, at2 = 2 * RING, hat = 0;        // ring offsets of planes e, e+1, e+2
    double acc = 0.0;

    // element plane e, output node plane e (the first element plane only feeds node plane x0)
    // BULK: planes e + 3 and e + 1 are inside the grid and needed, so nothing is tested
    auto step = [&](int e, auto first, auto bulk) {
        constexpr bool FIRST = decltype(first)::value, BULK = decltype(bulk)::value;
        TC ev[N];
        #pragma unroll
        for (int c = 0; c < N; ++c) ev[c] = TC(Storage<TE>::cvt(er[c]));
        if (BULK || e + 2 <= x1) {
            bits2 = put_u(at2);
            if (BULK || e + 3 <= x1) load_u(e + 3, BULK);
            load_e(e + 1, BULK);
        }
        typename Storage<TR>::raw_t rr[N][3], dd[N][3];
        if constexpr (HAS_R && !FIRST) {
            #pragma unroll
            for (int c = 0; c < N; ++c)
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rr[c][k] = Storage<TR>::raw(a.r + 3 * n_out[c] + k);
                    if constexpr (HAS_D) dd[c][k] = Storage<TR>::raw(a.invd + 3 * n_out[c] + k);
                }
        }
        P hown[3];
        {
            const P E = C::make(ev);
            const TC nv[2] = {-ev[0], -ev[N - 1]};
            const P nE = C::make(nv);
            P ya[3][2], yb[3][2];
            y_stage(at1, ya);
            #pragma unroll
            for (int k = 0; k < 3; ++k)
                #pragma unroll
                for (int py = 0; py < 2; ++py) yb[k][py] = next_lane<LZ>(ya[k][py]);
            P fx[3][2][2];                                   // totals of node plane e's faces
            auto cls = [&](auto PYc, auto PZc) {
                constexpr int PY = decltype(PYc)::value, PZ = decltype(PZc)::value;
                constexpr int py[3] = {PY, 1 - PY, PY}, pz[3] = {PZ, PZ, 1 - PZ};
                P s[3], d[3];
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const P c0 = pz[k] ? sub2(ya[k][py[k]], yb[k][py[k]]) : add2(ya[k][py[k]], yb[k][py[k]]);
                    const P p0 = pp[k][py[k]][pz[k]];
                    if constexpr (SUM_FIRST) {
                        s[k] = mul2(E, add2(p0, c0));
                        d[k] = mul2(E, sub2(p0, c0));
                    } else {
                        const P m = mul2(E, p0);
                        s[k] = fma2(E, c0, m);
                        d[k] = fma2(nE, c0, m);
                    }
                    pp[k][py[k]][pz[k]] = c0;
                }
                march_blocks<TC, CUBIC, PY, PZ>(args, s, d);
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    P& gk = gg[k][py[k]][pz[k]];
                    if (py[k] == 0 && pz[k] == 0) {          // translation: only the px = 1 part; gg holds its negative
                        fx[k][0][0] = sub2(d[k], gk);
                        gk = d[k];
                    } else {
                        fx[k][py[k]][pz[k]] = add2(add2(s[k], d[k]), gk);
                        gk = sub2(s[k], d[k]);
                    }
                }
            };
            using I0 = std::integral_constant<int, 0>;
            using I1 = std::integral_constant<int, 1>;
            cls(I0{}, I0{});
            cls(I1{}, I0{});
            cls(I0{}, I1{});
            cls(I1{}, I1{});
            // inverse z: own column + the element column of lane - 1; inverse y: own row, row + 1
            #pragma unroll
            for (int k = 0; k < 3 && !FIRST; ++k) {
                P fz[2];
                #pragma unroll
                for (int py = 0; py < 2; ++py) {
                    const P f0 = fx[k][py][0], f1 = fx[k][py][1];
                    fz[py] = add2(add2(f0, f1), prev_lane<LZ>(sub2(f0, f1)));
                }
                hown[k] = add2(fz[0], fz[1]);
                hs[hat + own_at + LZ * k] = sub2(fz[0], fz[1]);
            }
        }
        __syncthreads();
        if (!FIRST) {
            P yv[3];
            #pragma unroll
            for (int k = 0; k < 3; ++k) {
                P h = hs[hat + dn_at + LZ * k];
                if constexpr (N == 2) { if (row == 0) h = mk2(h.lo(), h.lo()); }     // row ROWS gets row ROWS - 1's
                yv[k] = add2(hown[k], h);
            }
            P xv[3];
            if constexpr (USES_X) {
                #pragma unroll
                for (int k = 0; k < 3; ++k) xv[k] = us[at0 + own_at + LZ * k];
            }
            const bool sums = e >= a.dot_x0 && e < a.dot_x1;
            TC xr[N][3], ax[N][3];
            #pragma unroll
            for (int c = 0; c < N; ++c)
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    ax[c][k] = C::get(yv[k], c);
                    xr[c][k] = USES_X ? C::get(xv[k], c) : TC(0);
                }
            auto fix = [&](int c) {                          // fixed DOFs: the unmasked operand, or a zero residual
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if ((bits0 >> (8 * c + k)) & 1u) continue;
                    if constexpr (EPI == EPI_RESIDUAL) {
                        rr[c][k] = typename Storage<TR>::raw_t(0.0f);
                        ax[c][k] = TC(0);
                    } else {
                        ax[c][k] = xr[c][k] = TC(Storage<TU>::load(a.u + 3 * n_out[c] + k));
                    }
                }
            };
            auto put = [&](int c) {
                TC o[3];
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if constexpr (EPI == EPI_RAW || EPI == EPI_APPLY_DOT) o[k] = ax[c][k];
                    else {
                        const TC r_ = TC(Storage<TR>::cvt(rr[c][k]));
                        if constexpr (EPI == EPI_JACOBI)
                            o[k] = xr[c][k] + a.omega * TC(Storage<TR>::cvt(dd[c][k])) * (r_ - ax[c][k]);
                        else o[k] = r_ - ax[c][k];
                    }
                }
                if (!owner[c]) return;
                #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    Storage<TY>::store(a.y + 3 * n_out[c] + k, o[k]);
                    if constexpr (EPI == EPI_APPLY_DOT || EPI == EPI_TRUE_RES) {
                        if (sums) acc += double(EPI == EPI_TRUE_RES ? o[k] : xr[c][k]) * double(o[k]);
                    }
                }
            };
            if constexpr (!VOTE) {
                #pragma unroll
                for (int c = 0; c < N; ++c) {
                    if (!owner[c]) continue;
                    if (MASK == MASK_NODE && ((bits0 >> (8 * c)) & 7u) != 7u) fix(c);
                    put(c);
                }
            } else {
                if (MASK == MASK_NODE && !__all_sync(0xffffffffu, (bits0 & 0x0707u) == 0x0707u)) {
                    #pragma unroll
                    for (int c = 0; c < N; ++c) fix(c);
                }
                #pragma unroll
                for (int c = 0; c < N; ++c) put(c);
            }
        }
        #pragma unroll
        for (int c = 0; c < N; ++c) n_out[c] += plane_nodes;
        const int t = at0;
        at0 = at1; at1 = at2; at2 = t;
        hat = RING - hat;
        bits0 = bits1; bits1 = bits2;
    };
    step(x0 - 1, std::true_type{}, std::false_type{});
    int e = x0;
    #pragma unroll 1
    for (const int eb = LEAN ? x0 : min(x1, g.nx - 1) - 2; e < eb; ++e) step(e, std::false_type{}, std::true_type{});
    #pragma unroll 1
    for (; e < x1; ++e) step(e, std::false_type{}, std::false_type{});
    if constexpr (EPI == EPI_TRUE_RES || EPI == EPI_APPLY_DOT) {
        const int64_t bid = (int64_t(blockIdx.z) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        block_sum_store<C::NW * 32>(acc, a.partials + bid);
        if (a.counter) {
            static_assert(C::NW * 32 == FT, "the last CTA finishes the reduction with FT threads");
            finalize_last(a.fin, int64_t(gridDim.x) * gridDim.y * gridDim.z, a.partials, a.S, a.counter);
        }
    }
}

// x chunk of parity_march: with w waves of resident CTAs the (y, z) tiles split into at most
// w * slots / tiles chunks; a chunk of cx node planes takes cx + 1 element planes and a prologue of
// about one more.  The cheapest of 1 .. 16 waves is taken, so the last wave is never nearly empty.
inline int march_cx(const Grid& g, int tiles, int slots) {
    const int planes = g.nx + 1;
    int best = planes;
    int64_t cost = INT64_MAX;
    for (int w = 1; w <= 16; ++w) {
        const int chunks = std::min(planes, std::max(1, w * slots / tiles));
        const int cx = (planes + chunks - 1) / chunks;
        const int64_t ctas = int64_t(tiles) * ((planes + cx - 1) / cx);
        const int64_t c = (ctas + slots - 1) / slots * (cx + 2);
        if (c < cost) { cost = c; best = cx; }
        if (cx == 1) break;                                  // more waves split no further
    }
    return best;
}

}  // namespace vx
