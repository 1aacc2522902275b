// Jacobi-PCG on small problems as one cooperative launch (ebePCG assembly/index.ts:504-733, FE
// js/optimizer-worker-3d.js:4189-4371, solveCG js/optimizer-worker.js:1799-1873).
//
// At these sizes an iteration as separate launches (operator, update with its sums, direction)
// is three or four launch latencies and as many last-block reductions: 18 us at 11,253 DOFs in
// 3D, 21 us at 60,802 in 2D, for under 3 MB of traffic.  Here every block keeps its DOFs' U, r
// and 1/D in registers for the whole solve and two grid barriers separate the phases:
//   1  p = z + beta p at the block's nodes and their neighbours (each block forms the
//      neighbours' values itself from z and the old p, so the new p needs no barrier of its
//      own); Ap = K p; the block's part of p.Ap
//      -- barrier, every block adds up all parts: alpha
//   2  U += alpha p, r -= alpha Ap, z = r / D; the block's parts of r.z and r.r
//      -- barrier, every block adds up all parts: beta, the stop test
// All blocks take the same decisions from the same numbers.  p alternates between two arrays, so
// that no block overwrites a value another still reads.
//
// Cooperative launches of several streams run one after the other, where separate launches ran
// side by side.  300 iterations on each of 1, 2, 4, 8 handles with a thread each took, as separate
// launches and as one: 5.7, 6.1, 6.4, 9.0 and 1.9, 2.9, 5.4, 10.9 ms at 30x10x10; 6.0, 6.3, 7.6,
// 13.2 and 3.1, 6.1, 12.2, 24.2 ms at 60x20x20.  Up to two solves at a time gain or lose nothing;
// from four on at 60x20x20 (eight at 30x10x10) they lose.
#pragma once
#include "common.cuh"

namespace tpo {

// Iterations of one launch unless the caller sets another even number; the host launches again if
// need be.  Even: p is back in its first array when a launch ends without being done.
constexpr int kCoopIters = 4096;
static_assert(kCoopIters % 2 == 0, "p alternates between two arrays");

// Scalars of the recurrence, the same in every block.
struct CoopScalars {
    double rz, alpha, beta, rr;
    int it, done;
};

// alpha from p.Ap with EpiCG's breakdown rules; true when the solve goes on.
__device__ __forceinline__ bool coop_alpha(CoopScalars &s, double pAp, double eps, CGState *st, bool first) {
    if (eps > 0.0) s.alpha = s.rz / (pAp + eps);
    else s.alpha = pAp > 0.0 ? s.rz / pAp : 0.0;
    const bool broke = !(eps > 0.0) && !(pAp > 0.0), bad = !isfinite(s.alpha);
    if (first) {
        st->pAp = pAp;
        st->alpha = s.alpha;
        if (broke || bad) {
            st->iters = s.it;
            if (bad) st->nonfinite = 1;
        }
    }
    if (broke || bad) s.done = 1;
    return !s.done;
}
// beta and the decision of cg_decide.
__device__ __forceinline__ void coop_beta(CoopScalars &s, double rz_new, double rr, double eps, double tolSq,
                                          int maxIter, CGState *st, bool first) {
    if (eps > 0.0) s.beta = rz_new / (s.rz + eps);
    else s.beta = s.rz > 0.0 ? rz_new / s.rz : 0.0;
    s.rz = rz_new;
    s.rr = rr;
    s.it += 1;
    const bool bad = !isfinite(rr), conv = !bad && rr < tolSq, cap = !bad && !conv && s.it >= maxIter;
    if (bad || conv || cap) {
        s.done = 1;
        if (first) {
            if (bad) st->nonfinite = 1;
            if (conv) st->converged = 1;
            st->iters = cap ? maxIter : s.it;
        }
    }
}

// Total of NV sums over np parts each (part i of sum k at parts[k np + i]) after the barrier that
// follows their writes: the order of grid_sum's last block (256 threads, strided, then the
// block tree), in every block.  Valid in every thread.  sh: 8 NV doubles.  (Polling the parts
// themselves, in place of a counter and then the parts, took twice the time: 148 x 148 polls.)
template <int NV>
__device__ __forceinline__ void coop_total(const double *parts, int np, double *sh, double (&tot)[NV]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < 256) {
        double acc[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) acc[k] = 0.0;
        for (int i = threadIdx.x; i < np; i += 256) {
#pragma unroll
            for (int k = 0; k < NV; k++) acc[k] += __ldcg(&parts[k * np + i]);
        }
#pragma unroll
        for (int k = 0; k < NV; k++) {
            acc[k] = warp_sum(acc[k]);
            if (lane == 0) sh[k * 8 + wid] = acc[k];
        }
    }
    __syncthreads();
    // every warp adds the eight sums itself, as grid_sum's warp 0 does
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = warp_sum(lane < 8 ? sh[k * 8 + lane] : 0.0);
}

// ---- 3D: the structured hex8 operator ----------------------------------------------------
// A block owns 32 M consecutive nodes.  Warp a forms, for each of them, the product of one of
// the node's eight elements (corner a); Ke's entries are uniform in the warp.  The nodes within
// one step of the block's lie in nine runs of 32 M + 2 nodes, staged as p.
constexpr int kCoop3Threads = 256;
constexpr int kCoop3MaxM = 6;
constexpr size_t coop3_smem(int m) { return sizeof(double) * (9 * (size_t)(32 * m + 2) * 3 + 8 * 3 * (size_t)32 * m + 8 * (size_t)32 * m); }

template <int M>
__global__ void __launch_bounds__(kCoop3Threads) k_cg_coop3(const __grid_constant__ KeParam<double> ke, const Grid g,
                                                            const double *__restrict__ Eact,
                                                            const double *__restrict__ invD,
                                                            const uint8_t *__restrict__ fixed, double *U, double *r,
                                                            double *z, double *pa, double *pb, CGState *st,
                                                            double *parts, int iters, unsigned polls) {
    constexpr int NT = 32 * M, SEG = (NT + 2) * 3, Q = (3 * NT + kCoop3Threads - 1) / kCoop3Threads;
    constexpr int kLoads = (9 * SEG + kCoop3Threads - 1) / kCoop3Threads, kBatch = 6;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sh[32 * 2], sh2[16];
    double *sp = reinterpret_cast<double *>(smem_raw);  // [9][SEG]
    double *sT = sp + 9 * SEG;                          // [corner 8][component 3][NT]
    double *sE = sT + 24 * NT;                          // [corner 8][NT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x;
    const int n0 = blockIdx.x * NT, ncol = g.nny * g.nnz, ndof = (int)g.ndof;
    const int ax = warp & 1, ay = (warp >> 1) & 1, az = warp >> 2;
    const int L = local_node(1 - ax, 1 - ay, 1 - az);
#pragma unroll
    for (int q = lane; q < NT; q += 32) {
        double E = 0.0;
        if (n0 + q < g.nnodes) {
            int x, y, zz;
            node_xyz(g, n0 + q, x, y, zz);
            const int ex = x - 1 + ax, ey = y - 1 + ay, ez = zz - 1 + az;
            if (ex >= 0 && ex < g.nelx && ey >= 0 && ey < g.nely && ez >= 0 && ez < g.nelz)
                E = Eact[((long long)ex * g.nely + ey) * g.nelz + ez];
        }
        sE[warp * NT + q] = E;
    }
    const double eps = st->eps, tolSq = st->tolSq;
    const int maxIter = st->maxIter;
    CoopScalars s{st->rz, st->alpha, st->beta, st->rr, st->it, st->done};
    const int it0 = s.it;
    double Ur[Q], rr_[Q], dr[Q], pr[Q], apr[Q];
    bool own[Q], fx[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int i = q * kCoop3Threads + tid, d = 3 * n0 + i;
        own[q] = i < 3 * NT && d < ndof;
        fx[q] = own[q] ? fixed[d] != 0 : true;
        Ur[q] = own[q] ? U[d] : 0.0;
        rr_[q] = own[q] ? r[d] : 0.0;
        dr[q] = own[q] ? invD[d] : 0.0;
        pr[q] = apr[q] = 0.0;
    }
    double *pold = pa, *pnew = pb;
    unsigned epoch = 0;
    bool ok = true;
    while (!s.done && s.it - it0 < iters) {
        // 1: p at the block's nodes and their neighbours, the loads of several in flight together
#pragma unroll
        for (int l0 = 0; l0 < kLoads; l0 += kBatch) {
            double zv[kBatch], pv[kBatch];
#pragma unroll
            for (int l = 0; l < kBatch; l++) {
                const int i = (l0 + l) * kCoop3Threads + tid, sg = i / SEG;
                const int d = 3 * (n0 - 1 + (sg / 3 - 1) * ncol + (sg % 3 - 1) * g.nnz) + (i - sg * SEG);
                const bool in = l0 + l < kLoads && i < 9 * SEG && d >= 0 && d < ndof;
                zv[l] = in ? __ldcg(z + d) : 0.0;
                pv[l] = in ? __ldcg(pold + d) : 0.0;
            }
#pragma unroll
            for (int l = 0; l < kBatch; l++) {
                const int i = (l0 + l) * kCoop3Threads + tid;
                if (l0 + l < kLoads && i < 9 * SEG) sp[i] = zv[l] + s.beta * pv[l];
            }
        }
        __syncthreads();
#pragma unroll
        for (int q0 = 0; q0 < M; q0++) {
            const int q = 32 * q0 + lane;
            double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const int ox = (b == 1 || b == 2 || b == 5 || b == 6), oy = (b == 2 || b == 3 || b == 6 || b == 7),
                          oz = (b >= 4);
                const double *pv = sp + ((ax + ox) * 3 + ay + oy) * SEG + 3 * (q + az + oz);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double v = pv[c];
#pragma unroll
                    for (int d = 0; d < 3; d++) acc[d] = fma(ke.v[(3 * L + d) * 24 + 3 * b + c], v, acc[d]);
                }
            }
            const double E = sE[warp * NT + q];
#pragma unroll
            for (int d = 0; d < 3; d++) sT[(warp * 3 + d) * NT + q] = E * acc[d];
        }
        __syncthreads();
        double v1[1] = {0.0};
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = q * kCoop3Threads + tid;
            if (!own[q]) continue;
            const int nd = i / 3, d = i - 3 * nd;
            double a = 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++) a += sT[(k * 3 + d) * NT + nd];
            pr[q] = sp[4 * SEG + 3 + i];
            if (3 * n0 + i == g.sdof) a += g.sk * pr[q];
            apr[q] = fx[q] ? 0.0 : a;
            pnew[3 * n0 + i] = pr[q];
            v1[0] += pr[q] * apr[q];
        }
        block_sum<1>(v1, sh);
        if (tid == 0) parts[blockIdx.x] = v1[0];
        if (!(ok = grid_barrier(&st->wait.bar, ++epoch * nb, &st->wait.err, polls))) break;
        double t1[1];
        coop_total<1>(parts, nb, sh2, t1);
        if (!coop_alpha(s, t1[0], eps, st, blockIdx.x == 0 && tid == 0)) break;
        // 2
        double v2[2] = {0.0, 0.0};
#pragma unroll
        for (int q = 0; q < Q; q++) {
            if (!own[q]) continue;
            Ur[q] = Ur[q] + s.alpha * pr[q];
            rr_[q] = rr_[q] - s.alpha * apr[q];
            const double zi = dr[q] * rr_[q];
            z[3 * n0 + q * kCoop3Threads + tid] = zi;
            v2[0] += rr_[q] * zi;
            v2[1] += rr_[q] * rr_[q];
        }
        block_sum<2>(v2, sh);
        if (tid == 0) {
            parts[nb + blockIdx.x] = v2[0];
            parts[2 * nb + blockIdx.x] = v2[1];
        }
        if (!(ok = grid_barrier(&st->wait.bar, ++epoch * nb, &st->wait.err, polls))) break;
        double t2[2];
        coop_total<2>(parts + nb, nb, sh2, t2);
        coop_beta(s, t2[0], t2[1], eps, tolSq, maxIter, st, blockIdx.x == 0 && tid == 0);
        double *t = pold;
        pold = pnew;
        pnew = t;
    }
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (own[q]) {
            U[3 * n0 + q * kCoop3Threads + tid] = Ur[q];
            r[3 * n0 + q * kCoop3Threads + tid] = rr_[q];
        }
    if (ok && blockIdx.x == 0 && tid == 0) {
        st->rz = s.rz;
        st->beta = s.beta;
        st->rr = s.rr;
        st->it = s.it;
        st->done = s.done;
    }
}

}  // namespace tpo
