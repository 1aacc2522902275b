// Declarations of the non-apply kernels of libtpo (definitions in kernels.cu).
#pragma once
#include "common.cuh"

namespace tpo {

// Bracket and result of one OC bisection; zeroed before the launch.
struct OcWords {  // the sum of one bisection step over all blocks
    unsigned long long piece[4];  // units of 2^-51, 2^-35, 2^-19, 2^-3
    unsigned long long limb[6];   // units of 2^-149, 2^-117, ...: values the pieces do not hold
    unsigned long long nan;
};
constexpr int kOcWords = sizeof(OcWords) / 8;
constexpr int kOcAhead = 4;            // bisection steps between two grid barriers at most
constexpr long long kOcAheadMax = 32768;  // elements a block up to which steps are taken ahead
struct OCState {
    double l1, l2, lmid, last_lmid, sum;
    unsigned long long change_bits;  // max |xnew - xold| as the bits of a non-negative double
    int done, nb;
    unsigned int bar;  // arrivals at the launch's grid barrier
    int err;           // the barrier's wait ran out
    OcWords words[3][kOcAhead];  // of the last passes and the next; zero at the start
};
constexpr int kOcThreads = 1024, kOcElemBytes = 16;

// element stiffness
__global__ void k_lk(double nu, double *Ke);

// densities -> element moduli (internal z-fastest order) and thresholded copies
__global__ void k_evals_fine(const float *__restrict__ x_ref, Grid g, double penal, double E0,
                             double Emin, int intpow, double *__restrict__ E, double *__restrict__ Eact,
                             float *__restrict__ Eact32);
__global__ void k_evals_fine_f64(const double *__restrict__ x_ref, Grid g, double penal, double E0,
                                 double Emin, int intpow, double *__restrict__ E, double *__restrict__ Eact,
                                 float *__restrict__ Eact32);
__global__ void k_evals_avg(const double *__restrict__ Ef, Grid gf, Grid gc, double Emin,
                            double *__restrict__ Ec, double *__restrict__ Eact, float *__restrict__ Eact32);
__global__ void k_diag(const __grid_constant__ KeParam<double> ke, Grid g, const double *__restrict__ Eact,
                       const uint8_t *__restrict__ fixed, double *__restrict__ invD, float *__restrict__ invD32);

// dense coarse levels
__global__ void k_zero_d(double *a, long long n);
// one thread per entry of the coarse 27-point stencil (243 per coarse node)
__global__ void __launch_bounds__(128) k_galerkin_gather(const __grid_constant__ KeParam<double> ke, Grid gf, Grid gc,
                                                         const double *__restrict__ EactF, double *__restrict__ Kc);
__global__ void k_galerkin_T(Grid gf, Grid gc, const double *__restrict__ Kf, double *__restrict__ T);
__global__ void k_galerkin_PtT(Grid gf, Grid gc, const double *__restrict__ T, double *__restrict__ Kc);
// womega: 3 doubles (damping, two words of scratch) or null
__global__ void k_dense_rows(const double *__restrict__ K, const Grid g, const uint8_t *__restrict__ fixed, double omega,
                             double *__restrict__ invD, float *__restrict__ invD32, double *__restrict__ womega);
__global__ void k_dense_matvec_seq(const double *__restrict__ K, int n, const double *__restrict__ p,
                                   double *__restrict__ Ap);
// coarsest level: its Jacobi sweeps from zero as a matrix
constexpr int kPolyMaxN = 384;  // largest level that takes this form (choose_coarse_poly of api.cu)
inline size_t coarse_poly_smem(int n) { return (size_t)n * (2 * sizeof(double2) + 81 * sizeof(unsigned short)); }
__global__ void k_coarse_pack(const double *__restrict__ K, const Grid g, double *__restrict__ Ks);
__global__ void __launch_bounds__(1024) k_coarse_poly(const double *__restrict__ Ks, const Grid g,
                                                      const double *__restrict__ invD,
                                                      const uint8_t *__restrict__ fixed, double omega,
                                                      const double *__restrict__ womega, int sweeps,
                                                      double *__restrict__ S);
// coarsest level: explicit inverse
__global__ void k_coarse_prepare(const double *__restrict__ K, int n, const double *__restrict__ invD,
                                 double *__restrict__ A);
constexpr int kGjNb = 32, kGjTile = 64, kGjThreads = 256;  // pivots a launch, tile of a CTA
constexpr int kGjPitch = kGjNb + 1;
constexpr size_t kGjSmem = sizeof(double) * (2 * kGjNb * kGjPitch + kGjTile * kGjPitch + 2 * kGjNb * kGjTile + kGjNb);
__global__ void k_gj_block(const double *__restrict__ A, double *__restrict__ B, int n, int k0,
                           const double *__restrict__ invD);
__global__ void k_coarse_mask_inverse(const double *__restrict__ Ainv, int n, const double *__restrict__ invD,
                                      double *__restrict__ Kinv);

// PCG
__global__ void k_cg_setup(CGState *st, double tol, int maxIter, double eps);
__global__ void k_cg_init_r(const double *__restrict__ F, const double *__restrict__ Ku,
                            const uint8_t *__restrict__ fixed, double *__restrict__ U,
                            double *__restrict__ r, long long n, CGState *st, double *partials);
__global__ void k_cg_pz(const double *__restrict__ r, double *__restrict__ z, const double *__restrict__ invD,
                        const uint8_t *__restrict__ fixed, double *__restrict__ p, long long n, int jacobi,
                        CGState *st, double *partials);
__global__ void k_cg_update_mg(double *__restrict__ U, double *__restrict__ r, const double *__restrict__ p,
                               const double *__restrict__ Ap, long long n, CGState *st, double *partials);
__global__ void k_cg_rz(const double *__restrict__ r, double *__restrict__ z, const uint8_t *__restrict__ fixed,
                        long long n, CGState *st, double *partials);
__global__ void k_cg_update_jacobi(double *__restrict__ U, double *__restrict__ r, double *__restrict__ z,
                                   const double *__restrict__ p, const double *__restrict__ Ap,
                                   const double *__restrict__ invD, long long n, CGState *st, double *partials);
__global__ void k_cg_p(double *__restrict__ p, const double *__restrict__ z, long long n, const CGState *st);
__global__ void k_cg_alpha(const double *__restrict__ p, const double *__restrict__ Ap, long long n, CGState *st,
                           double *partials);
__global__ void k_mask_zero(double *__restrict__ a, const uint8_t *__restrict__ fixed, long long n);
__global__ void k_dot(const double *__restrict__ a, const double *__restrict__ b, long long n,
                      double *out, unsigned *counter, double *partials);

// general-edof apply (WASM ABI): per-element products, then a CSR gather per DOF
__global__ void k_elem_products(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                                const double *__restrict__ evals, const int32_t *__restrict__ elist,
                                int count, double thresh, const double *__restrict__ p,
                                double *__restrict__ y, const CGState *st);
__global__ void k_csr_gather(const int64_t *__restrict__ rowptr, const int64_t *__restrict__ cols,
                             const double *__restrict__ y, int ndof, double *__restrict__ out,
                             const uint8_t *__restrict__ fixed, const CGState *st);
__global__ void k_csr_apply(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                            const double *__restrict__ evals, double thresh, const double *__restrict__ p,
                            const int64_t *__restrict__ rowptr, const int64_t *__restrict__ cols, int ndof,
                            double *__restrict__ out, const uint8_t *__restrict__ fixed, const CGState *st);
__global__ void k_ebe_evals(const double *__restrict__ dens, int nel, double Emin, double E0, double penal,
                            double *__restrict__ E);
__global__ void k_diag_general(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                               const double *__restrict__ evals, int nel, double thresh,
                               double *__restrict__ ydiag);
__global__ void k_invdiag_general(const double *__restrict__ diag, const uint8_t *__restrict__ fixed,
                                  int n, double *__restrict__ invD);

// SIMP
__global__ void k_energy(const __grid_constant__ KeParam<double> ke, Grid g, const double *__restrict__ U,
                         float *__restrict__ energy);
__global__ void k_heaviside(const float *__restrict__ x, long long n, double beta, float *__restrict__ xp);
__global__ void k_sensitivity(const float *__restrict__ x, const float *__restrict__ xp, const float *__restrict__ en,
                              long long n, double penal, double E0, double beta, int useProj, int guard,
                              float *__restrict__ dc, double Emin, float *__restrict__ stress,
                              unsigned long long *__restrict__ max_stress_bits);
__global__ void k_filter_hs(Grid g, double rmin, float *__restrict__ Hs);
__global__ void k_filter_sens(Grid g, double rmin, const float *__restrict__ Hs, const float *__restrict__ x,
                              const float *__restrict__ dc, float *__restrict__ dcn);
__global__ void k_density_filter(Grid g, double radius, const double *__restrict__ in, double *__restrict__ out);
constexpr int kFilterTile = 8;     // elements per side of a tiled filter CTA
constexpr int kFilterMaxHalo = 4;  // largest stencil half-width of the tiled filters
__global__ void k_filter_sens_tiled(Grid g, double rmin, const float *__restrict__ Hs, const float *__restrict__ x,
                                    const float *__restrict__ dc, float *__restrict__ dcn);
__global__ void k_density_tiled(Grid g, double radius, int mode, const double *__restrict__ in,
                                double *__restrict__ out);
// adjoint: dJ/dxPhys (reference order) and the density-filter transpose
__global__ void k_adjoint_sens(const __grid_constant__ KeParam<double> ke, Grid g, const double *__restrict__ xphys,
                               const double *__restrict__ U, const double *__restrict__ Lam, double penal, double E0,
                               double Emin, double *__restrict__ out);
__global__ void k_density_scale(Grid g, double radius, const double *__restrict__ gin, double *__restrict__ t);
__global__ void k_density_stencil(Grid g, double radius, const double *__restrict__ t, double *__restrict__ out);
__global__ void __launch_bounds__(kOcThreads) k_oc_bisect(const float *x, const float *dc,
                                                          const uint8_t *__restrict__ pres,
                                                          const uint8_t *__restrict__ voidm, long long n, long long per,
                                                          int cap, double volfrac, double move, int max_bisections,
                                                          OCState *s, const float *xold, float *xnew, unsigned polls);

__global__ void k_energy_wgsl(const float *__restrict__ U, const float *__restrict__ KE,
                              const int32_t *__restrict__ edofs, int nel, int es, float *__restrict__ out);

// Structured subdomain partition of the reference's KSP "BDDC" preconditioner: block
// boundaries per axis (ns[a] blocks, b[k] .. b[k+1]).
constexpr int kBddcMaxBlocks = 64;
struct BddcPart {
    int ns[3];
    int bx[kBddcMaxBlocks + 1], by[kBddcMaxBlocks + 1], bz[kBddcMaxBlocks + 1];
};
__global__ void k_bddc_setup(const __grid_constant__ KeParam<double> ke, Grid g, const double *__restrict__ E,
                             const uint8_t *__restrict__ fixed, const __grid_constant__ BddcPart part,
                             double *__restrict__ S, uint8_t *__restrict__ W);
__global__ void k_bddc_local(const double *__restrict__ S, const uint8_t *__restrict__ W,
                             const double *__restrict__ r, double *__restrict__ z, long long n,
                             const CGState *__restrict__ st);

// the 2D worker's hot path
__global__ void k_evals_pow_f32(const float *__restrict__ x, int nel, double Emin, double E0, double penal,
                                double *__restrict__ E);
__global__ void k_energy_general(const double *__restrict__ Ke, int es, const int32_t *__restrict__ edofs,
                                 const double *__restrict__ U, int nel, float *__restrict__ energy);
__global__ void k_filter_hs2d(int nelx, int nely, double rmin, float *__restrict__ Hs);
__global__ void k_filter_sens2d(int nelx, int nely, double rmin, const float *__restrict__ Hs,
                                const float *__restrict__ x, const float *__restrict__ dc, float *__restrict__ dcn);

constexpr int kCoop2Threads = 512;
__global__ void __launch_bounds__(kCoop2Threads) k_cg_coop2(const double *__restrict__ Ke, int nelx, int nely,
                                                            const double *__restrict__ Em, double thresh,
                                                            const double *__restrict__ invD,
                                                            const uint8_t *__restrict__ fixed, double *U, double *r,
                                                            double *z, double *pa, double *pb, CGState *st,
                                                            double *parts, int iters, unsigned polls);
__global__ void k_cg_abs_tol(CGState *st, double tol);

}  // namespace tpo
