// Table-driven thermochemistry (any chem.dat / diff.dat of more than two
// species) over one box: TEMPER, primitives and enthalpies; transport; CHRATE.
//
// The tables index species at run time. As one kernel over register arrays
// (MechTables of thermo.cuh) every indexed read or update became a select
// chain over 18 species, at 255 registers and 8 warps per SM: 492 us a launch
// for 48x40x36 points of the 16-species methane mechanism, with the FP64 pipe
// mostly idle. Here each thread's species arrays live in shared memory,
// [species][thread], where an index is an address, the loops run over the
// species and steps that exist, and the three parts are separate launches
// with their own shared memory and registers: 27 + 67 + 61 us. The expressions and
// their order are those of MechTables, so the values are the same.
#include <cuda_runtime.h>

#include "senga_internal.h"
#include "thermo.cuh"

namespace senga {
namespace {

// array number `a` of the block's dynamic shared memory
__device__ __forceinline__ SpArray sp_array(double* sm, int nspec, int a) {
  return SpArray{sm + (int64_t)a * nspec * kTabBlock + threadIdx.x};
}

// TEMPER, p, primitives, species and mixture enthalpies; with constant-Lewis
// transport also lambda, rho D and mu.
__global__ void __launch_bounds__(kTabBlock) k_tab_temper(Geo g, Fields f, const senga_chem* __restrict__ C, int nspec,
                                                         int flmavt) {
  extern __shared__ double sm[];
  const int64_t n = g.n, q = (int64_t)blockIdx.x * kTabBlock + threadIdx.x;
  if (q >= n) return;
  const SpArray ry = sp_array(sm, nspec, 0);
  const double* U = f.uin;
#pragma unroll 4
  for (int s = 0; s < nspec; ++s) ry[s] = U[(5 + s) * n + q];
  const double rho = U[q], ru = U[n + q], rv = U[2 * n + q], rw = U[3 * n + q], re = U[4 * n + q];
  const double ukuk = (ru * ru + rv * rv + rw * rw) / rho;
  double tc[6], td[6];
  tc[0] = 0.5 * ukuk - re;
#pragma unroll
  for (int i = 1; i < 6; ++i) tc[i] = td[i] = 0.0;
  double rmix = 0.0;
  const uint64_t itn0 = itn_load(f, n, q, nspec);
  for (int s = 0; s < nspec; ++s) {
    const int it = tint_of(itn0, s);
    const double y = ry[s];
    const int np = C->ncpoly[s][it];
    tc[0] = tc[0] + y * C->amascp[s][it][C->ncenth[s][it] - 1];
    tc[1] = tc[1] + y * C->amasct[s][it][0];
    td[1] = tc[1];
#pragma unroll
    for (int icp = 2; icp <= 5; ++icp)
      if (icp <= np) {
        tc[icp] = tc[icp] + y * C->amasct[s][it][icp - 1];
        td[icp] = td[icp] + y * C->amascp[s][it][icp - 1];
      }
    rmix = rmix + y * C->rgspec[s];
  }
  const double toltmp = (double)1.0e-10f;  // TOLTMP is a single-precision literal
  double T = f.t[q];
  int iters = 1;
  for (;;) {
    double tf = tc[5], tdp = td[5];
#pragma unroll
    for (int icp = 4; icp >= 1; --icp) {
      tf = tc[icp] + tf * T;
      tdp = td[icp] + tdp * T;
    }
    tf = tc[0] + tf * T;
    const double del = -tf / tdp;
    if (fabs(del) > toltmp) {
      if (iters < 100) {
        T = T + del;
        ++iters;
        continue;
      }
      atomicOr(f.status, 1u);  // reported through senga_get_status
    }
    break;
  }
  uint64_t itn = 0;
  double cpm = 0.0, hm = 0.0;
  for (int s = 0; s < nspec; ++s) {
    int it = 0;
    while (T > C->tinthi[s][it] && it + 1 < C->ntint[s]) ++it;
    itn += (uint64_t)it << (2 * s);
    const int np = C->ncpoly[s][it];
    const double* cp = C->amascp[s][it];
    double c = cp[np - 1];
    for (int icp = np - 1; icp >= 1; --icp) c = c * T + cp[icp - 1];
    const double r = ry[s];
    cpm = cpm + r * c;
    const double y = r / rho;
    f.y[s * n + q] = y;
    const int ih = tint_of(itn, s);
    const double* ch = C->amasch[s][ih];
    const int nh = C->ncpoly[s][ih];
    double v = ch[nh - 1];
    for (int icp = nh - 1; icp >= 1; --icp) v = v * T + ch[icp - 1];
    const double h = ch[C->ncenth[s][ih] - 1] + v * T;
    f.h[s * n + q] = h;
    hm = hm + h * y;
  }
  cpm = cpm / rho;
  f.hmix[q] = hm;
  f.t[q] = T;
  itn_store(f.itn, n, q, nspec, itn);
  f.p[q] = T * rmix;
  if (f.cp) {  // NSCBC face data (cp_mix, rho R_mix of TEMPER)
    f.cp[q] = cpm;
    f.rmix[q] = rmix;
  }
  f.vel[q] = ru / rho;
  f.vel[n + q] = rv / rho;
  f.vel[2 * n + q] = rw / rho;
  if (f.mom) {
    f.mom[q] = ru;
    f.mom[n + q] = rv;
    f.mom[2 * n + q] = rw;
  }
  f.e[q] = re / rho;
  if (flmavt) return;
  const double lcp = C->alamda * exp(kRlamda * log(T));
  f.lam[q] = lcp * cpm;
  f.lcp[q] = lcp;
  f.mu[q] = lcp * kPrantl;
  for (int s = 0; s < nspec; ++s) f.rd[s * n + q] = lcp * C->olewis[s];
}

// Polynomial in lt of n coefficients; N > 0: n == N, known at compile time (a
// loop of run-time length between the exps keeps them from overlapping).
template <int N>
__device__ __forceinline__ double table_poly(const double* __restrict__ c, int n, double lt) {
  const int m = N > 0 ? N : n;
  double fp = c[m - 1];
#pragma unroll
  for (int icp = m - 1; icp >= 1; --icp) fp = fp * lt + c[icp - 1];
  return fp;
}

// Mixture-averaged conductivity, diffusivities and Wilke viscosity.
template <int N>
__device__ __forceinline__ void tab_mixture(const Geo& g, const Fields& f, const senga_chem* __restrict__ C,
                                            const senga_diff* __restrict__ Dt, int nspec, double* sm, int64_t q) {
  const int64_t n = g.n;
  const double T = f.t[q], p = f.p[q], rho = f.uin[q];
  const double lt = log(T / Dt->tdifgb);
  const SpArray x = sp_array(sm, nspec, 0), a = sp_array(sm, nspec, 1), rq = sp_array(sm, nspec, 2);
  double c1 = 0.0, c2 = 0.0, c3 = 0.0, sumy = 0.0;
#pragma unroll 2
  for (int s = 0; s < nspec; ++s) {
    const double lk = exp(table_poly<N>(Dt->condco[s], Dt->ncocon, lt));
    const double fm = f.uin[(5 + s) * n + q] * C->ovwmol[s];
    c1 = c1 + fm * lk;
    c2 = c2 + fm / lk;
    c3 = c3 + fm;
    const double ye = f.y[s * n + q] + kDfctol;
    sumy += ye;
    x[s] = ye * C->ovwmol[s];
    a[s] = 0.0;
  }
  c3 = 1.0 / c3;
  c1 = c1 * c3;
  c2 = c2 * c3;
  f.lam[q] = 0.5 * (c1 + 1.0 / c2);
  const double wmix = rho * c3;
  const double povr = p / Dt->pdifgb;
  for (int s = 0; s < nspec; ++s) {
    const double xs = x[s];
    double den = a[s];
#pragma unroll 4
    for (int t = s + 1; t < nspec; ++t) {
      const double inv = exp(-table_poly<N>(Dt->diffco[s][t], Dt->ncodif, lt)) * povr;  // 1/D_st (DIFFCO is symmetric: one exp per pair)
      den += x[t] * inv;
      a[t] += xs * inv;
    }
    f.rd[s * n + q] = rho * (sumy - (f.y[s * n + q] + kDfctol)) / (den * wmix);
  }
  // Wilke: a holds sqrt(mu_s), rq its reciprocal, x the Y_s / W_s
#pragma unroll 2
  for (int s = 0; s < nspec; ++s) {
    const double sq = sqrt(exp(table_poly<N>(Dt->viscco[s], Dt->ncovis, lt)));
    a[s] = sq;
    rq[s] = 1.0 / sq;
    x[s] = f.y[s * n + q] * C->ovwmol[s];
  }
  double mu = 0.0;
  for (int s = 0; s < nspec; ++s) {
    double cc = 0.0;
    const double sq = a[s];
#pragma unroll 8
    for (int t = 0; t < nspec; ++t) {
      double fw = 1.0 + sq * rq[t] * Dt->wilko2[s][t];
      fw = Dt->wilko1[s][t] * fw * fw;
      cc = cc + x[t] * fw;
    }
    // mu_s itself: squaring the root would round again
    mu = mu + x[s] * (exp(table_poly<N>(Dt->viscco[s], Dt->ncovis, lt)) / cc);
  }
  f.mu[q] = mu;
}
__global__ void __launch_bounds__(kTabBlock) k_tab_mixture(Geo g, Fields f, const senga_chem* __restrict__ C,
                                                          const senga_diff* __restrict__ Dt, int nspec) {
  extern __shared__ double sm[];
  const int64_t q = (int64_t)blockIdx.x * kTabBlock + threadIdx.x;
  if (q >= g.n) return;
  // four coefficients in every table: what the transport tools write
  if (Dt->ncocon == 4 && Dt->ncodif == 4 && Dt->ncovis == 4) tab_mixture<4>(g, f, C, Dt, nspec, sm, q);
  else tab_mixture<0>(g, f, C, Dt, nspec, sm, q);
}

// CHRATE (chrate_point of thermo.cuh) over shared-memory arrays.
__global__ void __launch_bounds__(kTabBlock) k_tab_chrate(Geo g, Fields f, const senga_chem* __restrict__ C, int nspec) {
  extern __shared__ double sm[];
  const int64_t n = g.n, q = (int64_t)blockIdx.x * kTabBlock + threadIdx.x;
  if (q >= n) return;
  const SpArray ry = sp_array(sm, nspec, 0), gib = sp_array(sm, nspec, 1), rate = sp_array(sm, nspec, 2);
#pragma unroll 4
  for (int s = 0; s < nspec; ++s) ry[s] = f.uin[(5 + s) * n + q];
  chrate_point<0>(C, nspec, ry, f.t[q], itn_load(f, n, q, nspec), gib, rate);
#pragma unroll 4
  for (int s = 0; s < nspec; ++s) f.wdot[s * n + q] = rate[s];
}

}  // namespace

cudaError_t load_thermo_tables() { return load_kernels(k_tab_temper, k_tab_mixture, k_tab_chrate); }

int launch_thermo_tables(const Geo& g, const Fields& f, const senga_chem* dchem, const senga_diff* ddiff, int nspec,
                         int flmavt, cudaStream_t s) {
  const unsigned grid = (unsigned)((g.n + kTabBlock - 1) / kTabBlock);
  const size_t arr = (size_t)nspec * kTabBlock * sizeof(double);
  k_tab_temper<<<grid, kTabBlock, arr, s>>>(g, f, dchem, nspec, flmavt);
  if (flmavt) k_tab_mixture<<<grid, kTabBlock, 3 * arr, s>>>(g, f, dchem, ddiff, nspec);
  k_tab_chrate<<<grid, kTabBlock, 3 * arr, s>>>(g, f, dchem, nspec);
  return flmavt ? 3 : 2;
}

}  // namespace senga
