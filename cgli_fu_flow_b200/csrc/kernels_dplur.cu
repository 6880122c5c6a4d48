// DP-LUR inner solver (DPLUSGS.cpp): four Jacobi relaxations of the
// split-Jacobian operator of the LU-SGS sweeps, then the primitive-variable
// update with the pressure increment as the first norm.
//
// A relaxation is a 7-point stencil with no ordering between cells: a thread
// per cell gathers the product of each neighbour's split Jacobian with that
// neighbour's previous iterate.  The split Jacobians come from the coefficient
// record of the LU-SGS sweeps (make_record), formed once per inner iteration
// by the residual kernel, so that a product is ten loads and some 25 FP64
// operations and the kernel needs no exchange between threads.  A cell outside
// the interior contributes nothing, which is the reference's zero NL ghost
// rows (DPLUSGS.cpp:190-318).
#include "cgli_dev.cuh"
#include "cgli_launch.h"

namespace cgli {

struct RelaxPtrs {
  const double *src[5];
  double *dst[5];
  double *rec;                    // [REC_N] fields of coefficient records
  long long n;                    // words of a field
  double rdt;                     // 1 / deltaT
  const double *Jtab, *etdytab;   // per-j J and etdy of a grid uniform in x and z
};

// The product of one direction that cell c's neighbour sees, -A+ n (UP: A* n),
// from the record of cell c and the iterate of cell cn (c, or its periodic
// image); m, q: the face metric of the cell's row and the component of it that
// is not zero on the channel grid (CH)
template <int DIR, bool UP, bool CH>
__device__ __forceinline__ void product(const Dev &d, const RelaxPtrs &a, long long c, long long cn, double m, double o[5]) {
  constexpr int q = DIR + 1;
  double r[REC_N], n[5];
  for (int v : {(int)R_BETA, (int)R_H, (int)R_HR, (int)R_UX + DIR, (int)R_LX + DIR}) r[v] = a.rec[v * a.n + c];
#pragma unroll
  for (int v = 0; v < 5; v++) n[v] = a.src[v][cn];
  if (CH) {
    const double U = 0.5 * r[R_UX + DIR], l = 0.5 * r[R_LX + DIR], bU = r[R_BETA] * U;
    const double a0 = r[R_H] * m * n[q], aq = r[R_HR] * m * n[0];
    const double a4 = rec_g<double>(r) * r[R_UX + DIR] * n[0] + rec_hbt<double>(r) * m * n[q];
    const double p = UP ? U - l : -(U + l);
    o[0] = UP ? (bU - l) * n[0] + a0 : -(bU + l) * n[0] - a0;
#pragma unroll
    for (int v = 1; v <= 3; v++) o[v] = p * n[v];
    o[q] += UP ? aq : -aq;
    o[4] = UP ? p * n[4] + a4 : p * n[4] - a4;
  } else {
    const Split<double> A = split_from_record<double>(r, DIR, d.m[3 * DIR][c], d.m[3 * DIR + 1][c], d.m[3 * DIR + 2][c]);
    if (UP) upper_terms<double>(A, n, o); else lower_terms<double>(A, n, o);
  }
}

// One Jacobi relaxation, DPLUSGS.cpp:488-1141: dst = D^-1 (MR - LL(src) -
// UU(src)) on the interior; src on planes 2 and ie+1 is read at its periodic
// images ie and 3 (the self-copy exchange of :510-531).  The diagonal is that
// of DPLUSGS.cpp:1068-1107 (inviscid).  CH: the metrics are those of a grid
// uniform in x and z, read per row from etdytab.
// Bound by the loads: 26 words a cell from memory (38 us at 128x96x96), the
// neighbours' from L1 (along j and k, blocks of 8 rows) and L2 (along x), four
// blocks a SM to cover their latency (64 registers; general metrics spill 24 B).
// 128x96x96: 53.5 us, where tiles that marched along x, staged the state in
// shared memory and formed each split Jacobian once took 116 (two CTAs a SM, one
// plane's latency after another).
template <bool CH>
__global__ void __launch_bounds__(256, 4) k_dplur_relax(Dev d, RelaxPtrs a) {
  const int k = 2 + blockIdx.x * 32 + (threadIdx.x & 31);
  const int j = 2 + blockIdx.y * 8 + (threadIdx.x >> 5);
  const int i = 3 + blockIdx.z;
  const int ie = d.nx + 2;
  if (k > d.nz + 1 || j > d.ny + 1) return;
  const long long c = ix(d, i, j, k);
  const double idx = d.rdxi, idy = d.rdet, idz = d.rdzt;
  double o[5], LL[5] = {0, 0, 0, 0, 0}, UU[5] = {0, 0, 0, 0, 0}, ux[5] = {0, 0, 0, 0, 0};
  // an open slab's end planes hold zero iterates (DPLUSGS.cpp:191-233)
  if (!(d.x_open && i == 3)) {
    product<0, false, CH>(d, a, c - d.di, i == 3 ? ix(d, ie, j, k) : c - d.di, 1.0, o);
#pragma unroll
    for (int v = 0; v < 5; v++) LL[v] = o[v] * idx;
  }
  if (!(d.x_open && i == ie)) product<0, true, CH>(d, a, c + d.di, i == ie ? ix(d, 3, j, k) : c + d.di, 1.0, ux);
  if (j > 2) {
    product<1, false, CH>(d, a, c - d.dj, c - d.dj, CH ? a.etdytab[j - 1] : 0.0, o);
#pragma unroll
    for (int v = 0; v < 5; v++) LL[v] += o[v] * idy;
  }
  if (j < d.ny + 1) {
    product<1, true, CH>(d, a, c + d.dj, c + d.dj, CH ? a.etdytab[j + 1] : 0.0, o);
#pragma unroll
    for (int v = 0; v < 5; v++) UU[v] = o[v] * idy;
  }
  if (k > 2) {
    product<2, false, CH>(d, a, c - 1, c - 1, 1.0, o);
#pragma unroll
    for (int v = 0; v < 5; v++) LL[v] += o[v] * idz;
  }
  if (k < d.nz + 1) {
    product<2, true, CH>(d, a, c + 1, c + 1, 1.0, o);
#pragma unroll
    for (int v = 0; v < 5; v++) UU[v] += o[v] * idz;
  }
  double r[5], rec[REC_N];
#pragma unroll
  for (int v = 0; v < 5; v++) r[v] = d.MR[v][c] - LL[v] - UU[v] - ux[v] * idx;
  for (int v : {(int)R_BETA, (int)R_HR, (int)R_D11, (int)R_D22}) rec[v] = a.rec[v * a.n + c];
  a.dst[0][c] = rec[R_D11] * r[0];
  a.dst[1][c] = rec[R_D22] * r[1];
  a.dst[2][c] = rec[R_D22] * r[2];
  a.dst[3][c] = rec[R_D22] * r[3];
  a.dst[4][c] = rec_d51<double>(rec, a.rdt) * r[0] + rec[R_D22] * r[4];
}

// Residual of DPLUSGS.cpp:324-478 (the same values as Dual_time_stepping.cpp:
// 737-908 without its zero sponge terms): MR and the first iterate
// NL = D^-1 MR on the interior cells, with each repeated divisor as one
// (Newton-refined) reciprocal, and the coefficient records of planes 2..ie+1.
// CH as for the relaxation.  Bound by its 55 words a cell (80 us at 128x96x96).
// In the channel form the balance comes first, four blocks a SM, so that its 33
// loads are under way together: a step of ten iterations there 5.79 -> 5.46 ms,
// 256x192x192 42.9 -> 40.9; six and eight blocks give 5.55 and 5.62.  With nine
// metric terms more to load (general grids) the same order is slower (7.68 ->
// 7.73 at four blocks, 7.81 at three).
template <bool CH>
__global__ void __launch_bounds__(128, CH ? 4 : 8) k_dplur_residual(Dev d, RelaxPtrs a) {
  int k = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  int j = 2 + blockIdx.y;
  int i = 2 + blockIdx.z;
  if (k > d.nz + 1) return;
  const long long c = ix(d, i, j, k);
  double mm[9], J;
  if (CH) {
    J = a.Jtab[j];
    mm[0] = 1; mm[1] = 0; mm[2] = 0; mm[3] = 0; mm[4] = a.etdytab[j]; mm[5] = 0; mm[6] = 0; mm[7] = 0; mm[8] = 1;
  } else {
    J = d.J[c];
#pragma unroll
    for (int v = 0; v < 9; v++) mm[v] = d.m[v][c];
  }
  const double q1 = d.U_[0][c], q2 = d.U_[1][c], q3 = d.U_[2][c], q4 = d.U_[3][c], q5 = d.U_[4][c];
  const bool halo = i == 2 || i == d.nx + 3;   // the halo planes enter the products only
  double Rk[5];
  const auto balance = [&]() {   // time derivative, flux differences, viscous terms
    const long long fx1 = ix(d, i, j - 1, k - 1), f0 = ix(d, i - 1, j - 1, k - 1);
    const long long fy1 = ix(d, i - 1, j, k - 1), fz1 = ix(d, i - 1, j - 1, k);
    const double i2dt = nr_rcp(2 * d.dt), idx = d.rdxi, idy = d.rdet, idz = d.rdzt;
    const double U_[5] = {q1, q2, q3, q4, q5};
#pragma unroll
    for (int n = 0; n < 5; n++) {
      const double Rp = -(3 * U_[n] - 4 * d.U[n][c] + d.Uq[n][c]) * i2dt;
      const double Rf = -((d.inF[0][n][fx1] - d.inF[0][n][f0]) * idx + (d.inF[1][n][fy1] - d.inF[1][n][f0]) * idy +
                          (d.inF[2][n][fz1] - d.inF[2][n][f0]) * idz);
      Rk[n] = Rp + Rf;
    }
#pragma unroll
    for (int n = 1; n < 5; n++) Rk[n] = Rk[n] + d.vF[n - 1][c];
  };
  if (CH && !halo) balance();
  double rec[REC_N];
  make_record(q1, q2, q3, q4, q5, J, mm, d.e, d.rdxi, d.rdet, d.rdzt, d.dt, rec);
#pragma unroll
  for (int v = 0; v < REC_N; v++) a.rec[v * a.n + c] = rec[v];
  if (halo) return;
  const CPrim<double> q = cprim<double>(q1, q2, q3, q4, q5, J, d.e);
  const double rho = q.rho, u = q.u, v = q.v, w = q.w, VV = q.VV, T = q.Tt, H = q.H, beta = q.beta;
  const double irho = nr_rcp(rho), itemp = irho * (1.0 / KG);
  const double d11 = -(H * (KG - 1) + VV - KG * (T + VV)) * beta;
  const double d12 = -(KG - 1) * u * beta, d13 = -(KG - 1) * v * beta, d14 = -(KG - 1) * w * beta;
  const double d15 = (KG - 1) * beta;
  const double d51 = (KG - 1) * (VV + KG * T * beta + (KG - 1) * VV * beta + H * (-1 + beta - KG * beta)) * itemp;
  const double g5 = -(KG - 1) * (1 + (KG - 1) * beta) * itemp;
  if (!CH) balance();
  const double iJ = nr_rcp(J), f = d.scal[0];
  Rk[1] = Rk[1] + f * iJ;
  Rk[4] = Rk[4] + f * u * iJ;
  double MR[5];
  MR[0] = d11 * Rk[0] + d12 * Rk[1] + d13 * Rk[2] + d14 * Rk[3] + d15 * Rk[4];
  MR[1] = (Rk[1] - u * Rk[0]) * irho;
  MR[2] = (Rk[2] - v * Rk[0]) * irho;
  MR[3] = (Rk[3] - w * Rk[0]) * irho;
  MR[4] = d51 * Rk[0] + g5 * (u * Rk[1] + v * Rk[2] + w * Rk[3] - Rk[4]);
#pragma unroll
  for (int n = 0; n < 5; n++) d.MR[n][c] = MR[n];
  const double g51 = rec_d51<double>(rec, a.rdt);
  a.dst[0][c] = rec[R_D11] * MR[0];
  a.dst[1][c] = rec[R_D22] * MR[1];
  a.dst[2][c] = rec[R_D22] * MR[2];
  a.dst[3][c] = rec[R_D22] * MR[3];
  a.dst[4][c] = g51 * MR[0] + rec[R_D22] * MR[4];
}

// Update of DPLUSGS.cpp:1152-1196 from the last relaxation's result, with
// per-block partial sums of the squared squared increments (:1203-1215);
// one block per (j, i) row of k
__global__ void __launch_bounds__(128, 8) k_dplur_update(Dev d, RelaxPtrs a) {
  int k = 2 + threadIdx.x;
  int j = 2 + blockIdx.x;
  int i = 3 + blockIdx.y;
  const double *const *nr = a.src;
  double acc[5] = {0, 0, 0, 0, 0};
  if (*(volatile int *)d.status) return;   // an iteration before this one failed: keep the state
  for (int kk = k; kk <= d.nz + 1; kk += blockDim.x) {
    long long c = ix(d, i, j, kk);
    // the divisions by q1, rho, T and J as (Newton-refined) reciprocals (1/J
    // from the table)
    const double J = d.J[c], iJ = d.iJ[c];
    double q1 = d.U_[0][c], iq1 = nr_rcp(q1);
    double rhoold = q1 * J;
    double Uold = d.U_[1][c] * iq1, Vold = d.U_[2][c] * iq1, Wold = d.U_[3][c] * iq1;
    double VVold = Uold * Uold + Vold * Vold + Wold * Wold;
    double Pold = (d.U_[4][c] * J - 0.5 * rhoold * VVold) * (KG - 1);
    double Told = Pold * (iq1 * iJ);   // 1 / rho = 1 / (q1 J)
    double P = Pold + nr[0][c] * J;
    double U = Uold + nr[1][c] * J;
    double V = Vold + nr[2][c] * J;
    double W = Wold + nr[3][c] * J;
    double T = Told + nr[4][c] * J;
    double rho = P * nr_rcp(T), rJ = rho * iJ;
    d.U_[0][c] = rJ;
    d.U_[1][c] = rJ * U;
    d.U_[2][c] = rJ * V;
    d.U_[3][c] = rJ * W;
    d.U_[4][c] = (P * (1 / (KG - 1)) + 0.5 * rho * (U * U + V * V + W * W)) * iJ;
    double r[5] = {(P - Pold) * (P - Pold), (U - Uold) * (U - Uold), (V - Vold) * (V - Vold),
                   (W - Wold) * (W - Wold), (T - Told) * (T - Told)};
#pragma unroll
    for (int v = 0; v < 5; v++) acc[v] += r[v] * r[v];
  }
  block_sum5(acc, d.partial + 5 * ((long long)blockIdx.y * gridDim.x + blockIdx.x));
}

namespace {

RelaxPtrs ptrs(const Dev &d, double *const *src, double *const *dst, const SweepArgs &sw) {
  RelaxPtrs a;
  a.rec = sw.drec;
  a.n = (long long)d.X * d.di;
  a.rdt = 1.0 / d.dt;
  for (int v = 0; v < 5; v++) { a.src[v] = src[v]; a.dst[v] = dst[v]; }
  a.Jtab = sw.Jtab;
  a.etdytab = sw.etdytab;
  return a;
}

}  // namespace

// one relaxation NR -> NL (from_nr) or NL -> NR
static void relax(const Dev &d, const SweepArgs &sw, cudaStream_t s, bool from_nr) {
  const RelaxPtrs a = from_nr ? ptrs(d, d.NR, d.NL, sw) : ptrs(d, d.NL, d.NR, sw);
  const dim3 g((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx);
  if (sw.channel_metrics) k_dplur_relax<true><<<g, 256, 0, s>>>(d, a);
  else k_dplur_relax<false><<<g, 256, 0, s>>>(d, a);
}

// residual (MR, NR = D^-1 MR), four relaxations NR->NL->NR->NL->NR, update
void launch_dplur(const Dev &d, const SweepArgs &sw, cudaStream_t s) {
  RelaxPtrs r = ptrs(d, d.NL, d.NR, sw);
  dim3 g((d.nz + 127) / 128, d.ny, d.nx + 2);
  if (sw.channel_metrics) k_dplur_residual<true><<<g, 128, 0, s>>>(d, r);
  else k_dplur_residual<false><<<g, 128, 0, s>>>(d, r);
  for (int sweep = 0; sweep < 4; sweep++) relax(d, sw, s, sweep % 2 == 0);
  RelaxPtrs a = ptrs(d, d.NR, d.NL, sw);
  k_dplur_update<<<dim3(d.ny, d.nx), 128, 0, s>>>(d, a);
}

}  // namespace cgli
