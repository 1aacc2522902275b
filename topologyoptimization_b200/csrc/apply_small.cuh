// The structured apply on small grids: the coarse levels of a hierarchy and small problems.
//
// The strip kernel (apply_walsh.cuh) gives a CTA 512 or 1024 element columns of a node plane and
// one barrier per plane.  A grid of 16x8x8 elements has 81 columns: its launch is a chain of
// latencies (5.7 to 6.2 us in a graph whatever the size up to 60x20x20).  Here a CTA owns a small box
// of nodes, 8 x 16 columns of one or two planes: every load of the launch is issued at its start
// (node planes, moduli and the epilogue's operands), each thread runs its element column
// through the box's planes in registers, and two barriers separate load, transform and sum.
// The operations of an element and the order of a node's four contributions are the strip
// kernel's, so K u has the same bits from both (in FP32 packed and scalar arithmetic round
// alike).  A fused dot product is added up by other blocks: launches with one differ in its
// rounding, and a batched solve, which may take the other kernel, can differ from a single one
// there.  The rule that chooses and its table are at small_planes.  What is left is a launch's
// own 2 us and one round of loads, transforms and stores.
#pragma once
#include "apply_walsh.cuh"

namespace tpo {

// A value with unfused operations: what the packed arithmetic of the strip kernel does.
struct F1 {
    float v;
};
__device__ __forceinline__ F1 operator+(F1 a, F1 b) { return {__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 operator-(F1 a, F1 b) { return {__fadd_rn(a.v, -b.v)}; }
__device__ __forceinline__ F1 operator*(F1 a, F1 b) { return {__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vfma(F1 a, F1 b, F1 c) { return {__fmaf_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
template <typename T>
struct SmallV {
    using V = double;
    static __device__ V in(double x) { return x; }
    static __device__ double out(V x) { return x; }
};
template <>
struct SmallV<float> {
    using V = F1;
    static __device__ V in(float x) { return {x}; }
    static __device__ float out(V x) { return x.v; }
};

// Blocks of one element between the x stages.  The blocks couple the coefficients (s, c) in four
// closed groups of three; with a, b, c the members and suffix 0 / 1 for sigma_x:
//   (2,2) (1,1) (3,0)   twist a1, b1, c0; shear a0-b0; (111,x) c1
//   (0,0) (2,1) (1,2)   normal a1, b0, c0; rigid a0; bending b1-c1
//   (0,1) (2,0) (3,2)   shear a1-b0; rigid a0; bending b1-c0; (111,z) c1
//   (0,2) (1,0) (3,1)   the same for z
// P (node plane k's transform) becomes the contributions to node plane k; carry takes those to
// plane k + 1.
template <bool kGeneral, typename T>
__device__ __forceinline__ void small_step(const WalshKe<T> &wk, T Em, typename SmallV<T>::V (&P)[4][3],
                                           const typename SmallV<T>::V (&Q)[4][3],
                                           typename SmallV<T>::V (&carry)[4][3]) {
    using S = SmallV<T>;
    using V = typename S::V;
    const V E = S::in(Em);
    const V ps = E * S::in(wk.p), ds = E * S::in(wk.d), es = E * S::in(wk.e), fs = E * S::in(wk.f);
    auto shear = [&](V &u0, V &u1) {
        if constexpr (kGeneral) {
            const V qs = E * S::in(wk.q), w0 = u0, w1 = u1;
            u0 = vfma(ps, w0, qs * w1);
            u1 = vfma(qs, w0, ps * w1);
        } else {
            const V t = ps * (u0 + u1);
            u0 = t;
            u1 = t;
        }
    };
    auto rigid = [&](V &u) {
        if constexpr (kGeneral) u = (E * S::in(wk.s)) * u;
        else u = S::in(T(0));
    };
    auto bend = [&](V &u, V &w) {
        const V pp = u, qq = w;
        u = vfma(es, pp, fs * qq);
        w = vfma(fs, pp, es * qq);
    };
    auto group = [&](int sa, int ca, int sb, int cb, int sc, int cc, auto blocks) {
        V a0 = P[sa][ca] + Q[sa][ca], a1 = P[sa][ca] - Q[sa][ca];
        V b0 = P[sb][cb] + Q[sb][cb], b1 = P[sb][cb] - Q[sb][cb];
        V c0 = P[sc][cc] + Q[sc][cc], c1 = P[sc][cc] - Q[sc][cc];
        blocks(a0, a1, b0, b1, c0, c1);
        P[sa][ca] = (a0 + a1) + carry[sa][ca];
        carry[sa][ca] = a0 - a1;
        P[sb][cb] = (b0 + b1) + carry[sb][cb];
        carry[sb][cb] = b0 - b1;
        P[sc][cc] = (c0 + c1) + carry[sc][cc];
        carry[sc][cc] = c0 - c1;
    };
    group(2, 2, 1, 1, 3, 0, [&](V &a0, V &a1, V &b0, V &b1, V &c0, V &c1) {
        const V k1 = E * S::in(wk.a1), t = (E * S::in(wk.a2)) * ((a1 + b1) + c0);
        a1 = vfma(k1, a1, t);
        b1 = vfma(k1, b1, t);
        c0 = vfma(k1, c0, t);
        shear(a0, b0);
        c1 = ds * c1;
    });
    group(0, 0, 2, 1, 1, 2, [&](V &a0, V &a1, V &b0, V &b1, V &c0, V &c1) {
        const V k1 = E * S::in(wk.g1), t = (E * S::in(wk.g2)) * ((a1 + b0) + c0);
        a1 = vfma(k1, a1, t);
        b0 = vfma(k1, b0, t);
        c0 = vfma(k1, c0, t);
        rigid(a0);
        bend(b1, c1);
    });
    auto last = [&](V &a0, V &a1, V &b0, V &b1, V &c0, V &c1) {
        shear(a1, b0);
        c1 = ds * c1;
        rigid(a0);
        bend(b1, c0);
    };
    group(0, 1, 2, 0, 3, 2, last);
    group(0, 2, 1, 0, 3, 1, last);
}

// Tile of a CTA: kSR x kSZ element columns; tile t of an axis starts at element t (size - 1) and
// writes the nodes of its rows except the first one's (of tiles after the first), so that
// tiles x (size - 1) >= elements covers every node: powers of two leave nothing over.
constexpr int kSR = 9, kSZ = 17, kSCols = kSR * kSZ;
constexpr int kSThreads = 160;
constexpr int kSPitch = 3 * (kSZ + 1), kSPlane = (kSR + 1) * kSPitch;
template <typename T>
inline size_t small_smem(int tx) {
    return sizeof(T) * ((size_t)(tx + 2) * kSPlane + (size_t)tx * 12 * kSCols);
}
inline dim3 small_grid(const Grid &g, int tx, unsigned nrhs) {
    const int ty = (g.nely + kSR - 2) / (kSR - 1), tz = (g.nelz + kSZ - 2) / (kSZ - 1);
    return dim3((unsigned)(ty * tz), (unsigned)((g.nnx + tx - 1) / tx), nrhs);
}

template <typename T, class Epi, bool kGeneral, int TX>
__global__ void __launch_bounds__(kSThreads)
k_apply_small(const __grid_constant__ WalshKe<T> wk, const Grid g, const T *p, const T *Eact, Epi epi,
              const CGState *st) {
    chain_sync();
    using S = SmallV<T>;
    using V = typename S::V;
    if (blockIdx.z) {  // right-hand side of a batched solve
        const long long zr = blockIdx.z;
        p += zr * g.ndof;
        if (st) st += zr;
        epi.shift(zr, g.ndof);
    }
    if ((st && st->done) || epi.skip()) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *slab = reinterpret_cast<T *>(smem_raw);  // TX + 2 node planes
    T *xch = slab + (TX + 2) * kSPlane;         // TX x [corner 4][component 3][column]
    const int tid = threadIdx.x, nnz = g.nnz;
    const int tz = (g.nelz + kSZ - 2) / (kSZ - 1);
    const int yti = blockIdx.x / tz, zti = blockIdx.x - yti * tz;
    const int yb = yti * (kSR - 1), zb = zti * (kSZ - 1);
    const int x0 = blockIdx.y * TX, nx = min(TX, g.nnx - x0);
    const int row3 = 3 * nnz;
    const long long plane3 = (long long)g.nny * row3;

    // node planes x0 - 1 .. x0 + TX; 0 outside the grid (elements there have E = 0)
    const int srows = min(kSR + 1, g.nny - yb), scols = min(kSPitch, 3 * (nnz - zb));
    const T *src = p + ((x0 - 1) * plane3 + (long long)yb * row3 + 3 * zb);
#pragma unroll
    for (int x = 0; x < TX + 2; x++) {
        const bool in = (unsigned)(x0 - 1 + x) < (unsigned)g.nnx;
#pragma unroll
        for (int i0 = 0; i0 < kSPlane; i0 += kSThreads) {
            const int i = i0 + tid, r = i / kSPitch, c = i - r * kSPitch;
            if (i < kSPlane) slab[x * kSPlane + i] = in && r < srows && c < scols ? src[x * plane3 + r * row3 + c] : T(0);
        }
    }
    // this thread's element column and its moduli, planes x0 - 1 .. x0 + TX - 1
    const int col = min(tid, kSCols - 1), eb = col / kSZ, ez = col - eb * kSZ;
    const bool eok = tid < kSCols && yb + eb < g.nely && zb + ez < g.nelz;
    const T *ep = Eact + ((long long)(x0 - 1) * g.nely + yb + eb) * g.nelz + zb + ez;
    T E[TX + 1];
#pragma unroll
    for (int x = 0; x < TX + 1; x++)
        E[x] = eok && (unsigned)(x0 - 1 + x) < (unsigned)g.nelx ? ep[(long long)x * g.nely * g.nelz] : T(0);
    // the node this thread finishes: column `col` of every plane
    const bool nok = tid < kSCols && yb + eb < g.nny && zb + ez < nnz && (eb > 0 || yti == 0) && (ez > 0 || zti == 0);
    const long long dof = x0 * plane3 + (long long)(yb + eb) * row3 + 3 * (zb + ez);
    typename Epi::Pre opnd[TX];
#pragma unroll
    for (int x = 0; x < TX; x++)
        if (nok && x < nx) epi.pre(dof + x * plane3, opnd[x]);

    __syncthreads();
    if (tid < kSCols) {
        auto transform = [&](int x, V (&h)[4][3]) {
            const T *r0 = slab + (x * kSPlane + eb * kSPitch + 3 * ez), *r1 = r0 + kSPitch;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const V n00 = S::in(r0[c]), n01 = S::in(r0[3 + c]), n10 = S::in(r1[c]), n11 = S::in(r1[3 + c]);
                const V a = n00 + n01, b = n00 - n01, cc = n10 + n11, d = n10 - n11;
                h[0][c] = a + cc;
                h[1][c] = b + d;
                h[2][c] = a - cc;
                h[3][c] = b - d;
            }
        };
        V A[4][3], B[4][3], carry[4][3];
        transform(0, A);
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int c = 0; c < 3; c++) carry[s][c] = S::in(T(0));
#pragma unroll
        for (int x = 0; x < TX + 1; x++) {  // element plane x0 - 1 + x
            V(&P)[4][3] = (x & 1) ? B : A;
            V(&Q)[4][3] = (x & 1) ? A : B;
            transform(x + 1, Q);
            small_step<kGeneral, T>(wk, E[x], P, Q, carry);
            if (x > 0) {  // inverse (y, z) butterfly -> corners (by, bz) of node plane x0 + x - 1
                T *xo = xch + ((x - 1) * 12 * kSCols + tid);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const V a = P[0][c] + P[1][c], b = P[0][c] - P[1][c], d = P[2][c] + P[3][c], e = P[2][c] - P[3][c];
                    xo[(0 * 3 + c) * kSCols] = S::out(a + d);  // (0,0)
                    xo[(1 * 3 + c) * kSCols] = S::out(b + e);  // (0,1)
                    xo[(2 * 3 + c) * kSCols] = S::out(a - d);  // (1,0)
                    xo[(3 * 3 + c) * kSCols] = S::out(b - e);  // (1,1)
                }
            }
        }
    }
    __syncthreads();

    double part[Epi::NV > 0 ? Epi::NV : 1];
#pragma unroll
    for (int k = 0; k < (Epi::NV > 0 ? Epi::NV : 1); k++) part[k] = 0.0;
    if (nok) {
#pragma unroll
        for (int x = 0; x < TX; x++) {
            if (x >= nx) break;
            const T *xn = xch + (x * 12 * kSCols + col), *pn = slab + ((x + 1) * kSPlane + eb * kSPitch + 3 * ez);
            T acc[3], pc[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                // own column, z - 1, y - 1, both (0 at the grid's first column and row)
                acc[c] = xn[c * kSCols];
                if (ez > 0) acc[c] = acc[c] + xn[(3 + c) * kSCols - 1];
                if (eb > 0) acc[c] = acc[c] + xn[(6 + c) * kSCols - kSZ];
                if (ez > 0 && eb > 0) acc[c] = acc[c] + xn[(9 + c) * kSCols - kSZ - 1];
                pc[c] = pn[c];
            }
            const long long i = dof + x * plane3;
            add_spring(g, i, acc, pc);
            epi.emit(i, acc, pc, opnd[x], part);
        }
    }
    if constexpr (Epi::NV > 0) {
        __shared__ double sh[32 * Epi::NV];
        double tot[Epi::NV];
        if (grid_sum<Epi::NV>(part, epi.partials, epi.counter, sh, tot)) {
            if (threadIdx.x == 0) epi.finalize(tot);
        }
    }
}

}  // namespace tpo
