// Kernels whose arithmetic must follow the reference operation by operation.  This file
// is compiled with --fmad=false so that a*b+c stays two rounded operations, as in
// WebAssembly f64 and JavaScript.  Sums run in the reference's order.
#include "cg_coop.cuh"
#include "kernels.cuh"

namespace tpo {

// JavaScript Math.max / Math.min: NaN propagates; +0 wins max, -0 wins min.
__device__ __forceinline__ double js_max(double a, double b) {
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
    if (a == b) return signbit(a) ? b : a;
    return a > b ? a : b;
}
__device__ __forceinline__ double js_min(double a, double b) {
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
    if (a == b) return signbit(a) ? a : b;
    return a < b ? a : b;
}

// lk() (js/optimizer-worker-3d.js:3404-3491): one thread per entry (m, n), same
// sequence of operations as the reference's Gauss loop.
__global__ void k_lk(double nu, double *Ke) {
    const int t = threadIdx.x;
    if (t >= 576) return;
    const int m = t / 24, n = t % 24;
    const double E = 1.0;
    double C[6][6];
    for (int a = 0; a < 6; a++)
        for (int b = 0; b < 6; b++) C[a][b] = 0.0;
    const double fact = E / ((1 + nu) * (1 - 2 * nu));
    C[0][0] = fact * (1 - nu); C[0][1] = fact * nu; C[0][2] = fact * nu;
    C[1][0] = fact * nu; C[1][1] = fact * (1 - nu); C[1][2] = fact * nu;
    C[2][0] = fact * nu; C[2][1] = fact * nu; C[2][2] = fact * (1 - nu);
    C[3][3] = fact * (1 - 2 * nu) / 2;
    C[4][4] = fact * (1 - 2 * nu) / 2;
    C[5][5] = fact * (1 - 2 * nu) / 2;
    const double gp[2] = {-1 / sqrt(3.0), 1 / sqrt(3.0)};
    double acc = 0.0;
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++)
            for (int k = 0; k < 2; k++) {
                const double xi = gp[i], eta = gp[j], zeta = gp[k];
                const double weight = 1.0 * 1.0 * 1.0;
                double dN[8][3] = {
                    {-(1 - eta) * (1 - zeta), -(1 - xi) * (1 - zeta), -(1 - xi) * (1 - eta)},
                    {(1 - eta) * (1 - zeta), -(1 + xi) * (1 - zeta), -(1 + xi) * (1 - eta)},
                    {(1 + eta) * (1 - zeta), (1 + xi) * (1 - zeta), -(1 + xi) * (1 + eta)},
                    {-(1 + eta) * (1 - zeta), (1 - xi) * (1 - zeta), -(1 - xi) * (1 + eta)},
                    {-(1 - eta) * (1 + zeta), -(1 - xi) * (1 + zeta), (1 - xi) * (1 - eta)},
                    {(1 - eta) * (1 + zeta), -(1 + xi) * (1 + zeta), (1 + xi) * (1 - eta)},
                    {(1 + eta) * (1 + zeta), (1 + xi) * (1 + zeta), (1 + xi) * (1 + eta)},
                    {-(1 + eta) * (1 + zeta), (1 - xi) * (1 + zeta), (1 - xi) * (1 + eta)}};
                for (int a = 0; a < 8; a++)
                    for (int q = 0; q < 3; q++) dN[a][q] *= 0.125;
                double B[6][24];
                for (int a = 0; a < 6; a++)
                    for (int b = 0; b < 24; b++) B[a][b] = 0.0;
                for (int a = 0; a < 8; a++) {
                    const int col = a * 3;
                    B[0][col] = dN[a][0];
                    B[1][col + 1] = dN[a][1];
                    B[2][col + 2] = dN[a][2];
                    B[3][col] = dN[a][1];
                    B[3][col + 1] = dN[a][0];
                    B[4][col + 1] = dN[a][2];
                    B[4][col + 2] = dN[a][1];
                    B[5][col] = dN[a][2];
                    B[5][col + 2] = dN[a][0];
                }
                for (int p = 0; p < 6; p++) {
                    double cb = 0.0;
                    for (int q = 0; q < 6; q++) cb += C[p][q] * B[q][n];
                    acc += B[p][m] * cb * 1.0 * weight;
                }
            }
    Ke[t] = acc;
}

// applyAEbe3D / ebePCG general path, step 1: y[a*es + i] = E_e * sum_j Ke[i][j] p[edof_e[j]]
// for element e = elist[a] (explicit list) or e = a (all elements, inactive -> 0).
__global__ void k_elem_products(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                                const double *__restrict__ evals, const int32_t *__restrict__ elist, int count,
                                double thresh, const double *__restrict__ p, double *__restrict__ y,
                                const CGState *st) {
    if (st && st->done) return;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)count * es) return;
    const int a = (int)(t / es), i = (int)(t % es);
    const int e = elist ? elist[a] : a;
    const double E = evals[e];
    if (!elist && !(E > thresh)) {
        y[t] = 0.0;
        return;
    }
    const int32_t *ed = edofs + (long long)e * es;
    double sum = 0.0;
    for (int j = 0; j < es; j++) sum += Ke[i * es + j] * p[ed[j]];
    y[t] = E * sum;
}

// step 2: out[d] = sum of its element products in list order, starting from 0.
__global__ void k_csr_gather(const int64_t *__restrict__ rowptr, const int64_t *__restrict__ cols,
                             const double *__restrict__ y, int ndof, double *__restrict__ out,
                             const uint8_t *__restrict__ fixed, const CGState *st) {
    if (st && st->done) return;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= ndof) return;
    double s = 0.0;
    for (int64_t k = rowptr[d]; k < rowptr[d + 1]; k++) s = s + y[cols[k]];
    out[d] = (fixed && fixed[d]) ? 0.0 : s;
}

// Steps 1 and 2 in one launch for the structured element list (no active list): DOF d
// forms each of its element products (e, i) as k_elem_products does and adds them in CSR
// order as k_csr_gather does, so the result is theirs bit for bit.  Every product belongs
// to exactly one DOF, so none is computed twice.
__global__ void k_csr_apply(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                            const double *__restrict__ evals, double thresh, const double *__restrict__ p,
                            const int64_t *__restrict__ rowptr, const int64_t *__restrict__ cols, int ndof,
                            double *__restrict__ out, const uint8_t *__restrict__ fixed, const CGState *st) {
    if (st && st->done) return;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= ndof) return;
    double s = 0.0;
    for (int64_t k = rowptr[d]; k < rowptr[d + 1]; k++) {
        const long long t = cols[k];
        const int e = (int)(t / es), i = (int)(t % es);
        const double E = evals[e];
        double y = 0.0;
        if (E > thresh) {
            const int32_t *ed = edofs + (long long)e * es;
            double sum = 0.0;
            for (int j = 0; j < es; j++) sum += Ke[i * es + j] * p[ed[j]];
            y = E * sum;
        }
        s = s + y;
    }
    out[d] = (fixed && fixed[d]) ? 0.0 : s;
}

// ebePCG step 1 (:540-550): stiffness per element with Math.pow.
__global__ void k_ebe_evals(const double *__restrict__ dens, int nel, double Emin, double E0, double penal,
                            double *__restrict__ E) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nel) return;
    E[e] = Emin + pow(dens[e], penal) * (E0 - Emin);
}

// ebePCG step 2 (:552-566): diagonal contributions of active elements.
__global__ void k_diag_general(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                               const double *__restrict__ evals, int nel, double thresh,
                               double *__restrict__ ydiag) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nel * es) return;
    const int e = (int)(t / es), i = (int)(t % es);
    const double E = evals[e];
    ydiag[t] = E > thresh ? E * Ke[i * es + i] : 0.0;
}

__global__ void k_invdiag_general(const double *__restrict__ diag, const uint8_t *__restrict__ fixed, int n,
                                  double *__restrict__ invD) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = diag[i];
    invD[i] = (!fixed[i] && d > 1e-30) ? 1.0 / d : 0.0;
}

// denseMatVecRaw (assembly/index.ts:450-464): one thread per row, sequential sum.
__global__ void k_dense_matvec_seq(const double *__restrict__ K, int n, const double *__restrict__ p,
                                   double *__restrict__ Ap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *Kr = K + (long long)i * n;
    double s = 0.0;
    for (int j = 0; j < n; j++) s += Kr[j] * p[j];
    Ap[i] = s;
}

// prepareFilter Hs (:3006-3050): float accumulation in the triplet order
// (neighbour x outer, y, z inner).  One thread per element, reference element order.
__global__ void k_filter_hs(Grid g, double rmin, float *__restrict__ Hs) {
    const long long e1 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e1 >= g.nel) return;
    const int i = (int)(e1 % g.nelx);
    const long long r = e1 / g.nelx;
    const int j = (int)(r % g.nely);
    const int m = (int)(r / g.nely);
    const int R = (int)floor(rmin);
    float acc = 0.0f;
    for (int k = max(i - R, 0); k <= min(i + R, g.nelx - 1); k++)
        for (int l = max(j - R, 0); l <= min(j + R, g.nely - 1); l++)
            for (int n = max(m - R, 0); n <= min(m + R, g.nelz - 1); n++) {
                const double dist = sqrt((double)((i - k) * (i - k) + (j - l) * (j - l) + (m - n) * (m - n)));
                if (dist <= rmin) acc = (float)((double)acc + js_max(0.0, rmin - dist));
            }
    Hs[e1] = acc;
}

// filterSensitivities (:3052-3064): dcn_i = sum_j H_ij x_j dc_j (float accumulation in
// triplet order) / (Hs_i * max(1e-3, x_i)).
__global__ void k_filter_sens(Grid g, double rmin, const float *__restrict__ Hs, const float *__restrict__ x,
                              const float *__restrict__ dc, float *__restrict__ dcn) {
    const long long e1 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e1 >= g.nel) return;
    const int i = (int)(e1 % g.nelx);
    const long long r = e1 / g.nelx;
    const int j = (int)(r % g.nely);
    const int m = (int)(r / g.nely);
    const int R = (int)floor(rmin);
    const long long sy = g.nelx, sz = (long long)g.nelx * g.nely;
    float acc = 0.0f;
    for (int k = max(i - R, 0); k <= min(i + R, g.nelx - 1); k++)
        for (int l = max(j - R, 0); l <= min(j + R, g.nely - 1); l++)
            for (int n = max(m - R, 0); n <= min(m + R, g.nelz - 1); n++) {
                const double dist = sqrt((double)((i - k) * (i - k) + (j - l) * (j - l) + (m - n) * (m - n)));
                if (dist <= rmin) {
                    const long long e2 = k + l * sy + n * sz;
                    const double s = js_max(0.0, rmin - dist);
                    acc = (float)((double)acc + s * (double)__ldg(&x[e2]) * (double)__ldg(&dc[e2]));
                }
            }
    dcn[e1] = (float)((double)acc / ((double)Hs[e1] * js_max(1e-3, (double)x[e1])));
}

// applyDensityFilter (assembly/index.ts:224-273): +-ceil(r) box, dist^2 <= r^2, z outer.
__global__ void k_density_filter(Grid g, double radius, const double *__restrict__ in, double *__restrict__ out) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nel) return;
    const int ex = (int)(e % g.nelx);
    const long long r = e / g.nelx;
    const int ey = (int)(r % g.nely);
    const int ez = (int)(r / g.nely);
    const int R = (int)ceil(radius);
    const double r2 = radius * radius;
    double sum = 0.0, sw = 0.0;
    for (int kz = max(0, ez - R); kz <= min(g.nelz - 1, ez + R); kz++)
        for (int ky = max(0, ey - R); ky <= min(g.nely - 1, ey + R); ky++)
            for (int kx = max(0, ex - R); kx <= min(g.nelx - 1, ex + R); kx++) {
                const double dx = ex - kx, dy = ey - ky, dz = ez - kz;
                const double d2 = dx * dx + dy * dy + dz * dz;
                if (d2 <= r2) {
                    const double w = radius - sqrt(d2);
                    sum += w * __ldg(&in[kx + (long long)ky * g.nelx + (long long)kz * g.nelx * g.nely]);
                    sw += w;
                }
            }
    out[e] = sum / sw;
}

// ---- shared-memory tiled filters ---------------------------------------------------------
// A CTA owns an 8x8x8 block of elements and stages the block with its halo of R elements
// per side into shared memory once; the stencil weights, which depend only on the offset,
// come from a table built once per CTA.  Every element then sums its neighbours from
// shared memory in the same order and with the same roundings as the one-thread-per-element
// kernels above (bit-identical results).  Tiles of FT^3 elements, 512 threads.
constexpr int kFT = 8;

// The stencil as a compact list in the loop order of the per-element kernel: the offsets
// inside the radius (packed 8-bit dx, dy, dz), their shared-memory distance from the centre
// element and their weights.  At most (2R+1)^3 entries.
struct FilterTap {
    int packed;  // (dx + 128) | (dy + 128) << 8 | (dz + 128) << 16
    int soff;    // shared-memory offset from the centre element
};
__device__ __forceinline__ int tap_d(int packed, int k) { return ((packed >> (8 * k)) & 255) - 128; }

// filterSensitivities with the +-floor(rmin) box of prepareFilter; R = floor(rmin) <= 4.
// Neighbour order: x outer, y, z inner.
__global__ void __launch_bounds__(512) k_filter_sens_tiled(Grid g, double rmin, const float *__restrict__ Hs,
                                                           const float *__restrict__ x, const float *__restrict__ dc,
                                                           float *__restrict__ dcn) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = (int)floor(rmin);
    const int W = 2 * R + 1, T = kFT + 2 * R, W3 = W * W * W;
    double *wt = reinterpret_cast<double *>(smem_raw);  // W^3 tap weights
    FilterTap *taps = reinterpret_cast<FilterTap *>(wt + W3);
    float *sx = reinterpret_cast<float *>(taps + W3);
    float *sd = sx + T * T * T;
    __shared__ int ntaps;
    const int ox = blockIdx.x * kFT, oy = blockIdx.y * kFT, oz = blockIdx.z * kFT;
    if (threadIdx.x < 32) {  // taps in the per-element loop order, compacted by warp 0
        int n = 0;
        for (int c0 = 0; c0 < W3; c0 += 32) {
            const int t = c0 + (int)threadIdx.x;
            const int dk = t / (W * W) - R, dl = (t / W) % W - R, dn = t % W - R;
            const double dist = sqrt((double)(dk * dk + dl * dl + dn * dn));
            const bool in = t < W3 && dist <= rmin;
            const unsigned ball = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int q = n + __popc(ball & ((1u << threadIdx.x) - 1u));
                wt[q] = js_max(0.0, rmin - dist);
                taps[q].packed = (dk + 128) | ((dl + 128) << 8) | ((dn + 128) << 16);
                taps[q].soff = (dn * T + dl) * T + dk;
            }
            n += __popc(ball);
        }
        if (threadIdx.x == 0) ntaps = n;
    }
    for (int t = threadIdx.x; t < T * T * T; t += blockDim.x) {
        const int lx = t % T, ly = (t / T) % T, lz = t / (T * T);
        const int gx = ox - R + lx, gy = oy - R + ly, gz = oz - R + lz;
        if (gx >= 0 && gx < g.nelx && gy >= 0 && gy < g.nely && gz >= 0 && gz < g.nelz) {
            const long long e2 = gx + (long long)gy * g.nelx + (long long)gz * g.nelx * g.nely;
            sx[t] = x[e2];
            sd[t] = dc[e2];
        }
    }
    __syncthreads();
    const int tx = threadIdx.x % kFT, ty = (threadIdx.x / kFT) % kFT, tz = threadIdx.x / (kFT * kFT);
    const int i = ox + tx, j = oy + ty, m = oz + tz;
    if (i >= g.nelx || j >= g.nely || m >= g.nelz) return;
    const int c = ((tz + R) * T + (ty + R)) * T + (tx + R);
    const bool inner = i >= R && i + R < g.nelx && j >= R && j + R < g.nely && m >= R && m + R < g.nelz;
    float acc = 0.0f;
    for (int q = 0; q < ntaps; q++) {
        const FilterTap tp = taps[q];
        if (!inner) {
            const int k = i + tap_d(tp.packed, 0), l = j + tap_d(tp.packed, 1), n = m + tap_d(tp.packed, 2);
            if (k < 0 || k >= g.nelx || l < 0 || l >= g.nely || n < 0 || n >= g.nelz) continue;
        }
        acc = (float)((double)acc + wt[q] * (double)sx[c + tp.soff] * (double)sd[c + tp.soff]);
    }
    const long long e1 = i + (long long)j * g.nelx + (long long)m * g.nelx * g.nely;
    dcn[e1] = (float)((double)acc / ((double)Hs[e1] * js_max(1e-3, (double)sx[c])));
}

// applyDensityFilter (assembly/index.ts:224-273) with its +-ceil(r) box and dist^2 <= r^2,
// neighbour order z outer, y, x inner; R = ceil(r) <= 4.  mode 0: out = sum w in / sum w
// (the filter); mode 1: out = in / sum w (the first half of the transpose); mode 2: out =
// sum w in (the second half).
__global__ void __launch_bounds__(512) k_density_tiled(Grid g, double radius, int mode, const double *__restrict__ in,
                                                       double *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = (int)ceil(radius);
    const int W = 2 * R + 1, T = kFT + 2 * R, W3 = W * W * W;
    double *wt = reinterpret_cast<double *>(smem_raw);
    FilterTap *taps = reinterpret_cast<FilterTap *>(wt + W3);
    double *sv = reinterpret_cast<double *>(taps + W3 + (W3 & 1));  // 8-byte aligned after the int pairs
    __shared__ int ntaps;
    const int ox = blockIdx.x * kFT, oy = blockIdx.y * kFT, oz = blockIdx.z * kFT;
    const double r2 = radius * radius;
    if (threadIdx.x < 32) {  // taps in the per-element loop order, compacted by warp 0
        int n = 0;
        for (int c0 = 0; c0 < W3; c0 += 32) {
            const int t = c0 + (int)threadIdx.x;
            const int dz = t / (W * W) - R, dy = (t / W) % W - R, dx = t % W - R;
            // the per-element kernel's d = (ex - kx, ey - ky, ez - kz) = -offset
            const double fx = -dx, fy = -dy, fz = -dz;
            const double d2 = fx * fx + fy * fy + fz * fz;
            const bool in = t < W3 && d2 <= r2;
            const unsigned ball = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int q = n + __popc(ball & ((1u << threadIdx.x) - 1u));
                wt[q] = radius - sqrt(d2);
                taps[q].packed = (dx + 128) | ((dy + 128) << 8) | ((dz + 128) << 16);
                taps[q].soff = (dz * T + dy) * T + dx;
            }
            n += __popc(ball);
        }
        if (threadIdx.x == 0) ntaps = n;
    }
    if (mode != 1) {
        for (int t = threadIdx.x; t < T * T * T; t += blockDim.x) {
            const int lx = t % T, ly = (t / T) % T, lz = t / (T * T);
            const int gx = ox - R + lx, gy = oy - R + ly, gz = oz - R + lz;
            if (gx >= 0 && gx < g.nelx && gy >= 0 && gy < g.nely && gz >= 0 && gz < g.nelz)
                sv[t] = in[gx + (long long)gy * g.nelx + (long long)gz * g.nelx * g.nely];
        }
    }
    __syncthreads();
    const int tx = threadIdx.x % kFT, ty = (threadIdx.x / kFT) % kFT, tz = threadIdx.x / (kFT * kFT);
    const int ex = ox + tx, ey = oy + ty, ez = oz + tz;
    if (ex >= g.nelx || ey >= g.nely || ez >= g.nelz) return;
    const int c = ((tz + R) * T + (ty + R)) * T + (tx + R);
    const bool inner = ex >= R && ex + R < g.nelx && ey >= R && ey + R < g.nely && ez >= R && ez + R < g.nelz;
    double sum = 0.0, sw = 0.0;
    for (int q = 0; q < ntaps; q++) {
        const FilterTap tp = taps[q];
        if (!inner) {
            const int kx = ex + tap_d(tp.packed, 0), ky = ey + tap_d(tp.packed, 1), kz = ez + tap_d(tp.packed, 2);
            if (kx < 0 || kx >= g.nelx || ky < 0 || ky >= g.nely || kz < 0 || kz >= g.nelz) continue;
        }
        const double w = wt[q];
        if (mode != 1) sum += w * sv[c + tp.soff];
        sw += w;
    }
    const long long e = ex + (long long)ey * g.nelx + (long long)ez * g.nelx * g.nely;
    out[e] = mode == 0 ? sum / sw : (mode == 1 ? in[e] / sw : sum);
}

// ---- OC bisection (:3066-3101) --------------------------------------------------------
__device__ __forceinline__ float oc_xnew(float xf, float dcf, const uint8_t *pres, const uint8_t *voidm,
                                         long long i, double lmid, double move) {
    if (pres && pres[i]) return 1.0f;
    if (voidm && voidm[i]) return 0.0f;
    const double x = (double)xf;
    const double Be = -(double)dcf / lmid;
    return (float)js_max(0.0, js_max(x - move, js_min(1.0, js_min(x + move, x * sqrt(Be)))));
}

// ---- exact volume sum of the bisection ------------------------------------------------
// Every float in [0, 1] is an integer multiple of 2^-149, so a sum of up to 2^31 of them
// is an integer below 2^180 in those units: three 64-bit limbs hold it exactly.  Integer
// addition is associative, so the total is the same for every grid shape and block order,
// and it is rounded to double once, to nearest-even, before the reference's comparison
// with volfrac * nel.  A NaN (a positive sensitivity under the square root) makes the sum
// NaN, as in the reference.
struct Exact192 {
    unsigned long long w0, w1, w2;
    unsigned int nan;
};

__device__ __forceinline__ void x192_add(Exact192 &a, const Exact192 &b) {
    const unsigned long long s0 = a.w0 + b.w0;
    const unsigned long long c0 = s0 < a.w0;
    unsigned long long s1 = a.w1 + b.w1;
    unsigned long long c1 = s1 < a.w1;
    s1 += c0;
    c1 += s1 < c0;
    a.w0 = s0;
    a.w1 = s1;
    a.w2 = a.w2 + b.w2 + c1;
    a.nan |= b.nan;
}

// a += v for a float v in [0, 1] (or NaN)
__device__ __forceinline__ void x192_add_float(Exact192 &a, float v) {
    if (v != v) {
        a.nan = 1u;
        return;
    }
    const unsigned bits = __float_as_uint(v) & 0x7fffffffu;  // xnew >= +0; a -0 counts as 0
    const unsigned e = bits >> 23;
    const unsigned long long m = e ? (unsigned long long)((bits & 0x7fffffu) | 0x800000u)
                                   : (unsigned long long)(bits & 0x7fffffu);
    const int sh = e ? (int)e - 1 : 0;  // v = m 2^(sh - 149); sh <= 126 for v <= 1
    const int li = sh >> 6, off = sh & 63;
    Exact192 t{0ULL, 0ULL, 0ULL, 0u};
    const unsigned long long lo = m << off, hi = off > 40 ? m >> (64 - off) : 0ULL;
    if (li == 0) {
        t.w0 = lo;
        t.w1 = hi;
    } else {
        t.w1 = lo;
        t.w2 = hi;
    }
    x192_add(a, t);
}

__device__ __forceinline__ Exact192 x192_shfl_down(const Exact192 &a, int o) {
    Exact192 r;
    r.w0 = __shfl_down_sync(0xffffffffu, a.w0, o);
    r.w1 = __shfl_down_sync(0xffffffffu, a.w1, o);
    r.w2 = __shfl_down_sync(0xffffffffu, a.w2, o);
    r.nan = __shfl_down_sync(0xffffffffu, a.nan, o);
    return r;
}

// 64 bits of W starting at bit s (0 <= s < 192)
__device__ __forceinline__ unsigned long long x192_bits(const Exact192 &a, int s) {
    const unsigned long long w[4] = {a.w0, a.w1, a.w2, 0ULL};
    const int li = s >> 6, off = s & 63;
    return off ? (w[li] >> off) | (w[li + 1] << (64 - off)) : w[li];
}

// W 2^-149 rounded to the nearest double (ties to even)
__device__ double x192_to_double(const Exact192 &a) {
    if (a.nan) return __longlong_as_double(0x7ff8000000000000LL);
    int p = -1;  // highest set bit
    if (a.w2) p = 128 + 63 - __clzll((long long)a.w2);
    else if (a.w1) p = 64 + 63 - __clzll((long long)a.w1);
    else if (a.w0) p = 63 - __clzll((long long)a.w0);
    if (p < 0) return 0.0;
    if (p < 53) return ldexp((double)a.w0, -149);  // exact: W < 2^53
    const int sh = p - 52;
    unsigned long long mant = x192_bits(a, sh) & ((1ULL << 53) - 1ULL);
    const bool round = (x192_bits(a, sh - 1) & 1ULL) != 0;
    bool sticky = false;
    const int below = sh - 1;  // bits [0, below) decide the tie
    {
        const unsigned long long w[3] = {a.w0, a.w1, a.w2};
        for (int li = 0; li < 3 && li * 64 < below; li++) {
            const int nb = below - li * 64;
            const unsigned long long m = nb >= 64 ? ~0ULL : ((1ULL << nb) - 1ULL);
            if (w[li] & m) sticky = true;
        }
    }
    if (round && (sticky || (mant & 1ULL))) mant += 1ULL;  // 2^53 stays exact
    return ldexp((double)mant, sh - 149);
}

// ---- the whole bisection in one cooperative launch ---------------------------------------
// Values a thread adds before its 64-bit sums go to the 192-bit one: 4096 below 2 in units of
// 2^-51 (below 2^-28 in units of 2^-79) stay inside 64 bits.
constexpr int kFastFlush = 4096;

__device__ __forceinline__ void x192_add_u51(Exact192 &a, unsigned long long u) {
    // u 2^-51 = u 2^98 2^-149: limb 1, offset 34
    const Exact192 t{0ULL, u << 34, u >> 30, 0u};
    x192_add(a, t);
}

__device__ __forceinline__ void x192_add_u79(Exact192 &a, unsigned long long u) {
    // u 2^-79 = u 2^70 2^-149: limb 1, offset 6
    const Exact192 t{0ULL, u << 6, u >> 58, 0u};
    x192_add(a, t);
}

// Sum over the block in thread 0.
__device__ __forceinline__ Exact192 x192_block_sum(Exact192 acc, Exact192 *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const Exact192 b = x192_shfl_down(acc, o);
        x192_add(acc, b);
    }
    if (lane == 0) sh[wid] = acc;
    __syncthreads();
    if (wid == 0) {
        acc = lane < nw ? sh[lane] : Exact192{0ULL, 0ULL, 0ULL, 0u};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const Exact192 b = x192_shfl_down(acc, o);
            x192_add(acc, b);
        }
    }
    return acc;
}

// One element of the bisection.  xnew(lmid) rounds max(0, max(lo, min(1, min(hi, s)))) to FP32, with
// lo, hi = x -+ move and s = x sqrt(-dc / lmid).  Rounding is monotone, so it is the same to
// clamp (float)s by (float)lo and (float)hi, and lmid only enters s = t / sqrt(lmid), t = x
// sqrt(-dc): one FP64 product a step instead of a division and a root.
struct __align__(16) OcElem {
    double t;      // NaN: take oc_xnew
    int lo, hi;    // bits of max(0, (float)lo) and min(1, (float)hi); floats >= 0 order as integers
};
static_assert(sizeof(OcElem) == kOcElemBytes, "shared-memory size of an element");
__device__ __forceinline__ OcElem oc_elem(float xf, float dcf, double move) {
    const double x = (double)xf, lo = x - move, hi = x + move;
    OcElem e;
    e.t = lo == lo && hi == hi ? x * sqrt(-(double)dcf) + 0.0 : __longlong_as_double(0x7ff8000000000000LL);
    e.lo = max(0, __float_as_int((float)lo));
    e.hi = min(0x3f800000, __float_as_int((float)hi));
    return e;
}
// The bits of xnew, or -1 where the product does not decide.  s' = t rl, rl = lmid^-1/2, is within
// 8 units of the last place of the reference's FP64 s (each takes at most four roundings), so
// both round to the same float unless s' lies within 16 units of a midpoint of two floats
// (6e-8 of all values).  NaN, negative values and those too small to round here are not
// decided either; from 2^30 on min(1, hi) decides.
__device__ __forceinline__ int oc_bits(const OcElem &e, double rl) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(e.t * rl);
    const unsigned h = (unsigned)(b >> 32), low = (unsigned)b & 0x1fffffffu;
    const bool in = h >= 0x38700000u && h < 0x7ff00000u && low - (0x10000000u - 16u) > 32u;
    int f = (int)((unsigned)((b + 0x10000000ULL) >> 29) - (896u << 23));  // nearest float
    f = h >= 0x41d00000u ? 0x4e800000 : f;
    f = b == 0 ? 0 : f;
    return in || b == 0 ? max(e.lo, min(e.hi, f)) : -1;
}

// OC (js/optimizer-worker-3d.js:3066-3101): bisection on the multiplier, then xnew at the last
// one and change = max |xnew - xold|.  Block b owns elements [b per, (b + 1) per); it keeps the
// first `cap` of them in shared memory for all steps.  Each step every block sums its xnew
// exactly and adds the sum to the step's words (integers: the total does not depend on the
// order), and after a grid barrier every block reads the totals and takes the same steps.
// Preserved and void elements contribute a constant, added once.
//
// A value in [2^-28, 2) is a multiple of 2^-51 and adds to one 64-bit sum, one in [2^-56, 2^-28) a
// multiple of 2^-79 to another; what else there is goes through the 192-bit sum.
//
// One launch per step took 47-54 us a step whatever the size.  In this launch a pass is bound by
// its barrier and two block reductions (3 to 4 us) up to 200,000 elements and by 25 instructions
// an element and step beyond.  With a division and a root for every warp that holds an element
// between its limits, and every block adding up all blocks' words, a call of nine steps took
// 74, 112, 210, 347 us for 24,000, 524,288, 2.05M and 4.2M elements; it takes 67, 80, 118, 234
// (the last keeps only half of its elements in shared memory).  Several steps a pass take the
// design update of 2.05M elements (some 40 steps, all kernels) from 0.82 to 0.75 ms.  The steps
// that are dropped at the end cost as much as the barriers saved near kOcAheadMax: calls of 49
// and 32 steps, one at a time / four, take 945 / 884 and 637 / 625 us with 28,340 elements a block,
// 1216 / 1157 and 815 / 810 with 35,425, 1991 / 1940 and 1327 / 1349 with 55,352, 2612 / 2561 and
// 1745 / 1805 with 70,850.
__global__ void __launch_bounds__(kOcThreads) k_oc_bisect(const float *x, const float *dc,
                                                          const uint8_t *__restrict__ pres,
                                                          const uint8_t *__restrict__ voidm, long long n, long long per,
                                                          int cap, double volfrac, double move, int max_bisections,
                                                          OCState *s, const float *xold, float *xnew, unsigned polls) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    OcElem *sv = reinterpret_cast<OcElem *>(smem_raw);
    __shared__ Exact192 sh[32];
    __shared__ unsigned piece[kOcAhead][4][32];
    __shared__ double s_l[4];
    __shared__ int s_done, s_nb;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    const int ne = (int)max(0LL, b1 - b0);
    const int ns = min(ne, cap);
    auto elem = [&](int i) {
        const long long e = b0 + i;
        if (pres && pres[e]) return OcElem{0.0, 0x3f800000, 0x3f800000};  // 1
        if (voidm && voidm[e]) return OcElem{0.0, 0, 0};
        return oc_elem(x[e], dc[e], move);
    };
    for (int i = threadIdx.x; i < ns; i += blockDim.x) sv[i] = elem(i);
    double l1 = 0.0, l2 = 1e9, lmid = 0.0, rl = 0.0, sum = 0.0;
    auto value = [&](int i) {  // bits of xnew(lmid)
        int r = oc_bits(i < ns ? sv[i] : elem(i), rl);
        // with the masks: without a root (lmid near 0) no element is decided, masked ones neither
        if (r < 0) r = __float_as_int(oc_xnew(x[b0 + i], dc[b0 + i], pres, voidm, b0 + i, lmid, move));
        return r;
    };
    // lmid^-1/2; NaN, which decides no element, for multipliers near the end of the range (where a
    // bracket ends whose volume target no multiplier exceeds)
    auto root = [](double l) { return l > 1e-290 ? rsqrt(l) : __longlong_as_double(0x7ff8000000000000LL); };
    int nb = 0, pass = 0;
    bool done = !((l2 - l1) / (l2 + l1) > 1e-3);
    while (!done && nb < max_bisections) {
        // Steps between two barriers.  From 1e9 the multiplier falls by halves for some thirty steps
        // until a sum exceeds the target: while it does, four at a time, each the one that
        // follows if the sum before it is small; the step that is not drops those after it.
        const int nk = l1 == 0.0 && nb > 0 && per <= kOcAheadMax ? min(kOcAhead, max_bisections - nb) : 1;
        OcWords *words = s->words[pass % 3];
        for (int k = 0; k < nk; k++) {
            lmid = 0.5 * ((k == 0 ? l2 : lmid) + l1);
            rl = root(lmid);
            Exact192 acc{0ULL, 0ULL, 0ULL, 0u};
            unsigned long long fast = 0ULL, tiny = 0ULL;
            bool rare = false;
            int nf = 0;
            for (int i = threadIdx.x; i < ne; i += blockDim.x) {
                const int r = value(i);
                const unsigned e = (unsigned)r >> 23;
                const unsigned long long m = ((unsigned)r & 0x7fffffu) | 0x800000u;
                if (e - 99u < 29u) {
                    fast += m << (e - 99u);
                } else if (e - 71u < 28u) {
                    tiny += m << (e - 71u);
                } else if (r != 0) {
                    x192_add_float(acc, __int_as_float(r));
                    rare = true;
                }
                if (++nf == kFastFlush) {
                    x192_add_u51(acc, fast);
                    x192_add_u79(acc, tiny);
                    fast = tiny = 0ULL;
                    rare = true;
                    nf = 0;
                }
            }
            OcWords *w = words + k;
#pragma unroll
            for (int q = 0; q < 4; q++) {  // 16 bits of every thread's sum at a time
                const unsigned p = __reduce_add_sync(0xffffffffu, (unsigned)(fast >> (16 * q)) & 0xffffu);
                if (lane == 0) piece[k][q][wid] = p;
            }
            if (__syncthreads_or(rare || tiny != 0ULL)) {
                x192_add_u79(acc, tiny);
                acc = x192_block_sum(acc, sh);
                if (threadIdx.x == 0) {
                    const unsigned long long l[3] = {acc.w0, acc.w1, acc.w2};
                    for (int q = 0; q < 3; q++) {
                        if (!l[q]) continue;
                        atomicAdd(&w->limb[2 * q], l[q] & 0xffffffffULL);
                        atomicAdd(&w->limb[2 * q + 1], l[q] >> 32);
                    }
                    if (acc.nan) atomicAdd(&w->nan, 1ULL);
                }
            }
            if (wid < 4) {
                const unsigned p =
                    __reduce_add_sync(0xffffffffu, lane < (int)(blockDim.x >> 5) ? piece[k][wid][lane] : 0u);
                if (lane == 0 && p) atomicAdd(&w->piece[wid], (unsigned long long)p);
            }
        }
        if (!grid_barrier(&s->bar, (unsigned)(pass + 1) * gridDim.x, &s->err, polls)) return;
        // the words of the pass before are read everywhere: clear them for the pass after the next
        if (blockIdx.x == 0 && wid == 1)
            for (int i = lane; i < kOcAhead * kOcWords; i += 32)
                reinterpret_cast<unsigned long long *>(s->words[(pass + 2) % 3])[i] = 0ULL;
        if (wid == 0) {
            double t = 0.0;
            if (lane < nk) {  // lane k adds up step k
                unsigned long long v[kOcWords];
#pragma unroll
                for (int i = 0; i < kOcWords; i++)
                    v[i] = __ldcg(reinterpret_cast<unsigned long long *>(words + lane) + i);
                // 2^-19 = 2^130 2^-149
                Exact192 tot{0ULL, 0ULL, (v[2] + (v[3] << 16)) << 2, (unsigned)(v[10] != 0ULL)};
                x192_add_u51(tot, v[0] + (v[1] << 16));
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    const unsigned long long lo = (q & 1) ? v[4 + q] << 32 : v[4 + q], hi = (q & 1) ? v[4 + q] >> 32 : 0ULL;
                    const Exact192 a{q < 2 ? lo : 0ULL, q < 2 ? hi : (q < 4 ? lo : 0ULL), q < 2 ? 0ULL : (q < 4 ? hi : lo), 0u};
                    if (v[4 + q]) x192_add(tot, a);
                }
                t = x192_to_double(tot);
            }
            double tk[kOcAhead];
#pragma unroll
            for (int k = 0; k < kOcAhead; k++) tk[k] = __shfl_sync(0xffffffffu, t, k);
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < kOcAhead; k++) {
                    if (k >= nk || done) break;
                    lmid = 0.5 * (l2 + l1);
                    sum = tk[k];
                    const bool up = sum > volfrac * (double)n;
                    if (up) l1 = lmid;
                    else l2 = lmid;
                    nb++;
                    done = !((l2 - l1) / (l2 + l1) > 1e-3);
                    if (up) break;
                }
                s_l[0] = l1;
                s_l[1] = l2;
                s_l[2] = sum;
                s_l[3] = lmid;
                s_nb = nb;
                s_done = done;
            }
        }
        __syncthreads();
        l1 = s_l[0];
        l2 = s_l[1];
        sum = s_l[2];
        lmid = s_l[3];
        nb = s_nb;
        done = s_done != 0;
        pass++;
    }
    rl = root(lmid);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->l1 = l1;
        s->l2 = l2;
        s->lmid = s->last_lmid = lmid;
        s->sum = sum;
        s->nb = nb;
        s->done = done;
    }
    if (!done) return;
    // xnew at the last evaluated lmid; change = max |xnew - xold| (exact, order-free max)
    double mx = 0.0;
    for (int i = threadIdx.x; i < ne; i += blockDim.x) {
        const long long e = b0 + i;
        const float v = __int_as_float(value(i));
        if (xold) mx = js_max(mx, fabs((double)v - (double)xold[e]));
        xnew[e] = v;
    }
    if (xold) {
        // non-negative doubles order like their bit patterns
        unsigned long long b = (unsigned long long)__double_as_longlong(mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ob = __shfl_xor_sync(0xffffffffu, b, o);
            b = ob > b ? ob : b;
        }
        if ((threadIdx.x & 31) == 0) atomicMax(&s->change_bits, b);
    }
}

// _assembleGalerkinFromElements (js/optimizer-worker-3d.js:628-662) as a gather: one
// thread per coarse entry (R, C) of the 27-point stencil, no atomics.  The reference scatters,
// for every active fine element in ascending element order, for i, for j >= i, for the
// prolongation pairs (pi, pj): K[cr][cc] += w_i E Ke_ij w_j and, for i != j, K[cc][cr] += the
// same value.  The thread walks the fine elements whose nodes interpolate from both coarse
// nodes in that element order and adds the terms that land on (R, C) in that (i, j, pi,
// pj) order, so the sum is the reference's, bit for bit, and the same on every run.
// The weights are powers of two, so every term is exactly E Ke_ij w w'.
//
// Per element the corners that interpolate from R (and from C) are a bit mask, and only the
// pairs in both masks are visited.  Threads are numbered with the coarse node fastest, so the
// lanes of a warp share neighbour offset and components and walk the same pairs.  (A thread
// for each of the n^2 entries that tested all 300 (i, j) pairs of every element took 2.0 ms
// for 675 coarse DOFs and 3.9 ms for 1728; this takes 0.12 and 0.13 ms, the chain of the
// diagonal entries: 1000 terms added one after the other.)
// Halvings of the weight with which fine index f interpolates from coarse index c (w1d): 0 or
// 1, -1 for no weight.
__device__ __forceinline__ int half_weight(int f, int c, int nC) {
    const int c0 = min(f >> 1, nC - 1), c1 = min(c0 + 1, nC - 1);
    const bool t = c0 != c1 && (f & 1);
    if (c0 == c) return t ? 1 : 0;
    return (t && c1 == c) ? 1 : -1;
}

// One axis' share of the corner masks: bit b of m where corner b's node along the axis
// (element e's node 0: mask m0, node 1: m1) interpolates from coarse index c, and nibble b of
// h its halvings.
struct Corners {
    unsigned m, h;
};
__device__ __forceinline__ Corners corners(int e, int c, int nC, unsigned m0, unsigned m1, unsigned n0, unsigned n1) {
    const int w0 = half_weight(e, c, nC), w1 = half_weight(e + 1, c, nC);
    return {(w0 >= 0 ? m0 : 0u) | (w1 >= 0 ? m1 : 0u), (w0 > 0 ? n0 : 0u) | (w1 > 0 ? n1 : 0u)};
}

__global__ void __launch_bounds__(128) k_galerkin_gather(const __grid_constant__ KeParam<double> ke, Grid gf, Grid gc,
                                                         const double *__restrict__ EactF, double *__restrict__ Kc) {
    __shared__ double sk[576];
    for (int i = threadIdx.x; i < 576; i += blockDim.x) sk[i] = ke.v[i];
    __syncthreads();
    const long long n = gc.ndof, t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int q = (int)(t / gc.nnodes);  // neighbour offset and components
    if (q >= 243) return;
    const int node = (int)(t - (long long)q * gc.nnodes);
    const int nb = q / 9, dR = (q % 9) / 3, dC = q % 3;
    int rx, ry, rz;
    node_xyz(gc, node, rx, ry, rz);
    const int cx = rx + nb / 9 - 1, cy = ry + (nb / 3) % 3 - 1, cz = rz + nb % 3 - 1;
    if (cx < 0 || cx >= gc.nnx || cy < 0 || cy >= gc.nny || cz < 0 || cz >= gc.nnz) return;
    // Elements with a node in both supports: [2 max - 2, 2 min + 1] per axis.  The loops start
    // there at every lane, also outside the grid, so that a warp's lanes stay on the same
    // pairs at the grid's faces.
    const int lx = 2 * max(rx, cx) - 2, ly = 2 * max(ry, cy) - 2, lz = 2 * max(rz, cz) - 2;
    const int hx = 2 * min(rx, cx) + 1, hy = 2 * min(ry, cy) + 1, hz = 2 * min(rz, cz) + 1;
    // Both terms of a pair land on (R, C) when dR == dC and all four weights are positive; the
    // one with the smaller prolongation list positions comes first, and a node's list runs z,
    // y, x from the lower coarse index to the upper.
    const bool dfirst = rz != cz ? rz < cz : (ry != cy ? ry < cy : rx <= cx);
    const bool same = dR == dC;
    const int dmin = min(dR, dC), dmax = max(dR, dC);
    double sum = 0.0;
    for (int ez = lz; ez <= hz; ez++) {
        if (ez < 0 || ez >= gf.nelz) continue;
        const Corners azR = corners(ez, rz, gc.nnz, 0x0fu, 0xf0u, 0x00001111u, 0x11110000u);
        const Corners azC = corners(ez, cz, gc.nnz, 0x0fu, 0xf0u, 0x00001111u, 0x11110000u);
        for (int ey = ly; ey <= hy; ey++) {
            if (ey < 0 || ey >= gf.nely) continue;
            const Corners ayR = corners(ey, ry, gc.nny, 0x33u, 0xccu, 0x00110011u, 0x11001100u);
            const Corners ayC = corners(ey, cy, gc.nny, 0x33u, 0xccu, 0x00110011u, 0x11001100u);
            for (int ex = lx; ex <= hx; ex++) {
                if (ex < 0 || ex >= gf.nelx) continue;
                const Corners axR = corners(ex, rx, gc.nnx, 0x99u, 0x66u, 0x10011001u, 0x01100110u);
                const Corners axC = corners(ex, cx, gc.nnx, 0x99u, 0x66u, 0x10011001u, 0x01100110u);
                const unsigned mR = axR.m & ayR.m & azR.m, mC = axC.m & ayC.m & azC.m;
                if (!mR || !mC) continue;
                const unsigned hR = axR.h + ayR.h + azR.h, hC = axC.h + ayC.h + azC.h;
                const double E = EactF[((long long)ex * gf.nely + ey) * gf.nelz + ez];
                if (E == 0.0) continue;
                // E Ke_ij w w' for i = 3 bi + ci, j = 3 bj + cj
                auto term = [&](int bi, int ci, int bj, int cj, unsigned hi_, unsigned hj) {
                    const int h = (int)((hi_ >> (4 * bi)) & 15u) + (int)((hj >> (4 * bj)) & 15u);
                    return E * sk[(3 * bi + ci) * 24 + 3 * bj + cj] * __hiloint2double((1023 - h) << 20, 0);
                };
                if (same) {
                    for (unsigned mi = mR | mC; mi; mi &= mi - 1) {
                        const int bi = __ffs((int)mi) - 1;
                        const bool iR = (mR >> bi) & 1u, iC = (mC >> bi) & 1u;
                        const unsigned md = iR ? mC & (0xffu << bi) : 0u, mt = iC ? mR & (0xfeu << bi) : 0u;
                        for (unsigned mj = md | mt; mj; mj &= mj - 1) {
                            const int bj = __ffs((int)mj) - 1;
                            const bool dir = (md >> bj) & 1u, tr = (mt >> bj) & 1u;
                            const double vd = dir ? term(bi, dR, bj, dC, hR, hC) : 0.0;
                            const double vt = tr ? term(bi, dR, bj, dC, hC, hR) : 0.0;
                            if (dir && tr) {
                                sum += dfirst ? vd : vt;
                                sum += dfirst ? vt : vd;
                            } else {
                                sum += dir ? vd : vt;
                            }
                        }
                    }
                } else {
                    // i = 3 bi + dmin, j >= i: the direct term if dR < dC, else the transposed
                    // one; then i = 3 bi + dmax, j > i: the other
                    const unsigned mA = dR < dC ? mR : mC, mB = dR < dC ? mC : mR;
                    const unsigned hA = dR < dC ? hR : hC, hB = dR < dC ? hC : hR;
                    for (unsigned mi = mA | mB; mi; mi &= mi - 1) {
                        const int bi = __ffs((int)mi) - 1;
                        if ((mA >> bi) & 1u)
                            for (unsigned mj = mB & (0xffu << bi); mj; mj &= mj - 1) {
                                const int bj = __ffs((int)mj) - 1;
                                sum += term(bi, dmin, bj, dmax, hA, hB);
                            }
                        if ((mB >> bi) & 1u)
                            for (unsigned mj = mA & (0xfeu << bi); mj; mj &= mj - 1) {
                                const int bj = __ffs((int)mj) - 1;
                                sum += term(bi, dmax, bj, dmin, hB, hA);
                            }
                    }
                }
            }
        }
    }
    const long long cn = ((long long)cx * gc.nny + cy) * gc.nnz + cz;
    Kc[(3LL * node + dR) * n + 3 * cn + dC] = sum;
}

// GPUCompute.computeElementEnergies (js/gpu-compute.js:187-303): the reference's WGSL
// kernel, one invocation per element, energy = sum_i sum_j u_i KE_ij u_j in f32 in that
// order, DOF indices < 0 skipped.  Unfused f32 operations (this file is built without
// FMA contraction).
__global__ void k_energy_wgsl(const float *__restrict__ U, const float *__restrict__ KE,
                              const int32_t *__restrict__ edofs, int nel, int es, float *__restrict__ out) {
    const int el = blockIdx.x * blockDim.x + threadIdx.x;
    if (el >= nel) return;
    const long long off = (long long)el * es;
    float energy = 0.0f;
    for (int i = 0; i < es; i++) {
        const int di = edofs[off + i];
        if (di < 0) continue;
        const float ui = U[di];
        for (int j = 0; j < es; j++) {
            const int dj = edofs[off + j];
            if (dj < 0) continue;
            energy = energy + ui * KE[i * es + j] * U[dj];
        }
    }
    out[el] = energy;
}

// ---- the 2D worker's hot path (js/optimizer-worker.js, TopologyOptimizerWorker) ------------
// _precomputeStiffness (:270-285): E = Emin + Math.pow(x, penal) (E0 - Emin) from the float
// (projected) densities, two roundings.
__global__ void k_evals_pow_f32(const float *__restrict__ x, int nel, double Emin, double E0, double penal,
                                double *__restrict__ E) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nel) return;
    E[e] = Emin + pow((double)x[e], penal) * (E0 - Emin);
}

// Jacobi-PCG of the 2D worker as one cooperative launch (cg_coop.cuh): one DOF per thread, its
// four elements' products and their sum as k_csr_apply forms them, the vector updates and the
// dot products as k_cg_alpha, k_cg_update_jacobi and k_cg_p do (their multiply-adds are fused,
// and a block here is two of theirs: 256 DOFs a part), so the iterates are theirs bit for bit.
__global__ void __launch_bounds__(kCoop2Threads) k_cg_coop2(const double *__restrict__ Ke, int nelx, int nely,
                                                            const double *__restrict__ Em, double thresh,
                                                            const double *__restrict__ invD,
                                                            const uint8_t *__restrict__ fixed, double *U, double *r,
                                                            double *z, double *pa, double *pb, CGState *st,
                                                            double *parts, int iters, unsigned polls) {
    constexpr int NT = kCoop2Threads / 2, SEG = (NT + 2) * 2;
    __shared__ double sp[3 * SEG], sK[64], sh[64], sh2[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nny = nely + 1, ndof = 2 * (nelx + 1) * nny, nparts = (ndof + 255) / 256;
    const int n0 = blockIdx.x * NT, d = 2 * n0 + tid, node = n0 + (tid >> 1), c = tid & 1;
    if (tid < 64) sK[tid] = Ke[tid];
    const bool own = d < ndof;
    const int x = node / nny, y = node - x * nny;
    // elements in ascending order; corner (ox, oy) of an element is its local node
    // 0 (0,0), 1 (1,0), 2 (1,1), 3 (0,1)
    double E[4];
    bool have[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int ex = x - 1 + (k >> 1), ey = y - 1 + (k & 1);
        have[k] = own && ex >= 0 && ex < nelx && ey >= 0 && ey < nely;
        E[k] = have[k] ? Em[ey + ex * nely] : 0.0;
    }
    const bool fx = own ? fixed[d] != 0 : true;
    double Ud = own ? U[d] : 0.0, rd = own ? r[d] : 0.0;
    const double dd = own ? invD[d] : 0.0;
    const double eps = st->eps, tolSq = st->tolSq;
    const int maxIter = st->maxIter;
    CoopScalars s{st->rz, st->alpha, st->beta, st->rr, st->it, st->done};
    const int it0 = s.it;
    double *pold = pa, *pnew = pb;
    unsigned epoch = 0;
    bool ok = true;
    // block sums of 256 threads each, as block_sum forms them
    auto part_sums = [&](double a, double b, int nv, double *out) {
        a = warp_sum(a);
        if (nv == 2) b = warp_sum(b);
        if (lane == 0) {
            sh[warp] = a;
            sh[32 + warp] = b;
        }
        __syncthreads();
        if ((warp & 7) == 0) {
            const int vb = 2 * blockIdx.x + (warp >> 3);
            const double ta = warp_sum(lane < 8 ? sh[warp + lane] : 0.0);
            const double tb = nv == 2 ? warp_sum(lane < 8 ? sh[32 + warp + lane] : 0.0) : 0.0;
            if (lane == 0 && vb < nparts) {
                out[vb] = ta;
                if (nv == 2) out[nparts + vb] = tb;
            }
        }
    };
    while (!s.done && s.it - it0 < iters) {
        constexpr int kLoads = (3 * SEG + kCoop2Threads - 1) / kCoop2Threads;
        double zv[kLoads], pv[kLoads];
#pragma unroll
        for (int l = 0; l < kLoads; l++) {
            const int i = l * kCoop2Threads + tid, sg = i / SEG, q = 2 * (n0 - 1 + (sg - 1) * nny) + (i - sg * SEG);
            const bool in = i < 3 * SEG && q >= 0 && q < ndof;
            zv[l] = in ? __ldcg(z + q) : 0.0;
            pv[l] = in ? __ldcg(pold + q) : 0.0;
        }
#pragma unroll
        for (int l = 0; l < kLoads; l++) {
            const int i = l * kCoop2Threads + tid;
            if (i < 3 * SEG) sp[i] = fma(s.beta, pv[l], zv[l]);
        }
        __syncthreads();
        const double pd = sp[SEG + 2 + tid];
        double ap = 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int ax = k >> 1, ay = k & 1;                                  // element (x-1+ax, y-1+ay)
            const int i = 2 * (ay ? (ax ? 0 : 1) : (ax ? 3 : 2)) + c;           // this DOF in it
            const double *col0 = sp + ax * SEG + 2 * ((tid >> 1) + ay), *col1 = col0 + SEG;  // nodes (ex, ey), (ex+1, ey)
            if (have[k]) {
                double yk = 0.0;
                if (E[k] > thresh) {
                    const double *Ki = sK + i * 8;
                    double sum = 0.0;
                    sum += Ki[0] * col0[0];
                    sum += Ki[1] * col0[1];
                    sum += Ki[2] * col1[0];
                    sum += Ki[3] * col1[1];
                    sum += Ki[4] * col1[2];
                    sum += Ki[5] * col1[3];
                    sum += Ki[6] * col0[2];
                    sum += Ki[7] * col0[3];
                    yk = E[k] * sum;
                }
                ap = ap + yk;
            }
        }
        if (fx) ap = 0.0;
        if (own) pnew[d] = pd;
        part_sums(own ? pd * ap : 0.0, 0.0, 1, parts);
        if (!(ok = grid_barrier(&st->wait.bar, ++epoch * gridDim.x, &st->wait.err, polls))) break;
        double t1[1];
        coop_total<1>(parts, nparts, sh2, t1);
        if (!coop_alpha(s, t1[0], eps, st, blockIdx.x == 0 && tid == 0)) break;
        rd = fma(-s.alpha, ap, rd);
        const double zd = dd * rd;
        Ud = fma(s.alpha, pd, Ud);
        if (own) z[d] = zd;
        part_sums(own ? rd * zd : 0.0, own ? rd * rd : 0.0, 2, parts + nparts);
        if (!(ok = grid_barrier(&st->wait.bar, ++epoch * gridDim.x, &st->wait.err, polls))) break;
        double t2[2];
        coop_total<2>(parts + nparts, nparts, sh2, t2);
        coop_beta(s, t2[0], t2[1], eps, tolSq, maxIter, st, blockIdx.x == 0 && tid == 0);
        double *t = pold;
        pold = pnew;
        pnew = t;
    }
    if (own) {
        U[d] = Ud;
        r[d] = rd;
    }
    if (ok && blockIdx.x == 0 && tid == 0) {
        st->rz = s.rz;
        st->beta = s.beta;
        st->rr = s.rr;
        st->it = s.it;
        st->done = s.done;
    }
}

// _computeElementEnergyFlat (:335-345; js/optimizer-worker-3d.js:1561-1571): energy = sum_i
// sum_j u_i KE_ij u_j in FP64 in that order over the element's DOFs, stored as float.
__global__ void k_energy_general(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                                 const double *__restrict__ U, int nel, float *__restrict__ energy) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nel) return;
    const int32_t *ed = edofs + (long long)e * es;
    double en = 0.0;
    for (int i = 0; i < es; i++) {
        const double ui = U[ed[i]];
        for (int j = 0; j < es; j++) en += ui * Ke[i * es + j] * U[ed[j]];
    }
    energy[e] = (float)en;
}

// 2D prepareFilter (:1391-1429): element e = i*nely + j (column-major); neighbours k (x)
// outer, l (y) inner within +-floor(rmin), weight max(0, rmin - dist) where dist <= rmin;
// Hs accumulated into a Float32Array.
__global__ void k_filter_hs2d(int nelx, int nely, double rmin, float *__restrict__ Hs) {
    const int e1 = blockIdx.x * blockDim.x + threadIdx.x;
    if (e1 >= nelx * nely) return;
    const int i = e1 / nely, j = e1 % nely;
    const int R = (int)floor(rmin);
    float acc = 0.0f;
    for (int k = max(i - R, 0); k <= min(i + R, nelx - 1); k++)
        for (int l = max(j - R, 0); l <= min(j + R, nely - 1); l++) {
            const double dist = sqrt((double)((i - k) * (i - k) + (j - l) * (j - l)));
            if (dist <= rmin) acc = (float)((double)acc + js_max(0.0, rmin - dist));
        }
    Hs[e1] = acc;
}

// 2D filterSensitivities (:1431-1443): dcn_e = sum H x dc (float accumulation in the
// triplet order) / (Hs_e max(1e-3, x_e)).
__global__ void k_filter_sens2d(int nelx, int nely, double rmin, const float *__restrict__ Hs,
                                const float *__restrict__ x, const float *__restrict__ dc, float *__restrict__ dcn) {
    const int e1 = blockIdx.x * blockDim.x + threadIdx.x;
    if (e1 >= nelx * nely) return;
    const int i = e1 / nely, j = e1 % nely;
    const int R = (int)floor(rmin);
    float acc = 0.0f;
    for (int k = max(i - R, 0); k <= min(i + R, nelx - 1); k++)
        for (int l = max(j - R, 0); l <= min(j + R, nely - 1); l++) {
            const double dist = sqrt((double)((i - k) * (i - k) + (j - l) * (j - l)));
            if (dist <= rmin) {
                const int e2 = k * nely + l;
                acc = (float)((double)acc + js_max(0.0, rmin - dist) * (double)x[e2] * (double)dc[e2]);
            }
        }
    dcn[e1] = (float)((double)acc / ((double)Hs[e1] * js_max(1e-3, (double)x[e1])));
}

}  // namespace tpo
