// High-order filter sensor of Filter.cpp:12-1720 (EpX/EpY/EpZ from U_).
//
// Per scale (h: (1,6,1)/8 weights, 2h: (1,2,1)/4) the reference applies six
// iterated filter levels, each an x pass, a y pass on the stretched grid and
// a z pass over full-size scratch arrays, then the high-pass
// fU = 6 L1 - 15 L2 + 20 L3 - 15 L4 + 6 L5 - L6 and E = |u - fu/frho|^2.
//
// Here one kernel launch is one level: a CTA owns an (8 x 32) (j, k) tile
// and marches over a chunk of x planes with a 3-plane ring of the previous
// level in shared memory, so each level reads its input once and writes its
// output once; the x, y and z passes of a plane are done in shared memory.
// The high-pass sum is accumulated in the order the reference writes it as
// the levels are produced, and the last level computes E in its epilogue,
// so no level is kept beyond the next one.  A last kernel forms the face
// ratios and EpX/EpY/EpZ.
//
// Every operation is an explicitly rounded double operation (no fused
// multiply-add) in the reference's evaluation order, so E and the face
// ratios are bit-identical to the reference's and Ep is exact.
#include <cuda_runtime.h>

#include "cgli_filter.h"

namespace cgli {
namespace {

constexpr int FTJ = 8, FTK = 32;                 // output tile (j, k)
constexpr int FRJ = FTJ + 2, FRK = FTK + 2;      // tile with a one-cell halo
constexpr int FTHREADS = (FRJ * FRK + 31) / 32 * 32;   // a thread per cell of the tile with halo

__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

// (a + w*b + c) * s: the x and z passes (Filter.cpp:160, :227; :841, :902)
template <bool TWO_H>
__device__ __forceinline__ double smooth3(double a, double b, double c) {
  return TWO_H ? mul(0.25, add(add(a, mul(2.0, b)), c)) : mul(0.125, add(add(a, mul(6.0, b)), c));
}

struct LevelArgs {
  const double *P[4];   // previous level (U_ for level 0)
  double *L[4];         // this level (not written by the last level)
  double *acc[4];       // running high-pass sum on the interior planes
  const double *U[4];   // U_: wall and z ghost values and E
  const double *J, *Yp;
  double *E;            // written by the last level
  int nx, ny, nz;       // interior cells
  int X, Y, Z;
  int i0, i1;           // x planes of this level
  int level;            // 0..5
  int wrap;             // read P through its periodic image: the 3-plane
                        // exchange of level 3 on a single periodic slab
                        // (Filter.cpp:447-466) without a copy
  int chunk;            // x planes per CTA
};

__device__ __forceinline__ int wrap_plane(int p, int nx) { return p < 3 ? p + nx : (p > nx + 2 ? p - nx : p); }

// The quotients a / b of one divisor, correctly rounded, from its correctly
// rounded reciprocal: q <- q + (a - q b) (1 / b) with fused multiply-adds, the
// second of which starts within half a unit in the last place and so rounds
// correctly (P. Markstein, IBM J. Res. Dev. 34(1), 1990), for operands and
// quotients far from over- and underflow; any other goes through the IEEE
// division (a divisor out of range through its NaN for a reciprocal).
__device__ __forceinline__ double divisor(double b) {
  const double m = fabs(b);
  return m > 1e-200 && m < 1e200 ? __drcp_rn(b) : __longlong_as_double(0x7ff8000000000000LL);
}
__device__ __forceinline__ double quotient(double a, double b, double rb) {
  double q = mul(a, rb);
  q = __fma_rn(__fma_rn(-q, b, a), rb, q);
  q = __fma_rn(__fma_rn(-q, b, a), rb, q);
  const double m = fabs(q), n = fabs(a);
  return m > 1e-200 && m < 1e200 && n > 1e-200 && n < 1e200 ? q : dvd(a, b);
}

// One level.  Bound by the latency of its chain of planes (load, x, y and z
// pass, a barrier each): every plane's loads (the next plane of the previous
// level, the next J and Y, the running sum) are issued a plane ahead, a thread
// per cell of the tile with halo keeps each pass to one round, and the x
// chunk is chosen so that the CTAs fill the chip (launch_filter).  Two CTAs per
// SM hold it at 80 registers (32 B of spill stores, 40 of loads).  At
// 96x72x72 a level takes 51.5 us; with chunks of 16 planes, a division where
// the quotient stands and loads inside the passes it took 137.
template <bool TWO_H>
__global__ void __launch_bounds__(FTHREADS, 2) k_filter_level(LevelArgs a) {
  extern __shared__ double sm[];
  double *ring = sm;                                // [3][4][FRJ*FRK]
  double *gx = ring + 3 * 4 * FRJ * FRK;            // [4][FRJ*FRK]
  double *gy = gx + 4 * FRJ * FRK;                  // [4][FTJ*FRK]
  double *w1 = gy + 4 * FTJ * FRK;                  // [FTJ*FRK]
  double *w3 = w1 + FTJ * FRK;                      // [FTJ*FRK]
  double *jt = w3 + FTJ * FRK;                      // [FRJ*FRK]

  const int tid = threadIdx.x;
  const int k0 = 2 + blockIdx.x * FTK, j0 = 2 + blockIdx.y * FTJ;
  const int ia = a.i0 + blockIdx.z * a.chunk;
  const int ib = min(a.i1, ia + a.chunk - 1);
  const int ny = a.ny + 1, nz = a.nz + 1;           // the reference's ny, nz
  const long long di = (long long)a.Y * a.Z, dj = a.Z;
  const int gend = a.nx + 2;

  // this thread's cell of the tile with halo (x pass), of the tile with the
  // z halo (y pass) and of the tile (z pass)
  const int jh = j0 - 1 + tid / FRK, kh = k0 - 1 + tid % FRK;
  const bool in_h = tid < FRJ * FRK;
  const bool ring_cell = in_h && jh >= 2 && jh <= ny && kh >= 2 && kh <= nz;
  const bool j_cell = in_h && jh >= 1 && jh <= ny + 1 && kh >= 1 && kh <= nz + 1;
  const bool wall_cell = in_h && (jh == 1 || jh == ny + 1) && kh >= 2 && kh <= nz;
  const int jy = j0 + tid / FRK, ky = k0 - 1 + tid % FRK;
  const bool in_y = tid < FTJ * FRK && jy <= ny;
  const bool y_cell = in_y && ky >= 2 && ky <= nz, z_ghost = in_y && (ky == 1 || ky == nz + 1);
  const int rz = tid / FTK, cz = tid % FTK;
  const bool z_cell = tid < FTJ * FTK && j0 + rz <= ny && k0 + cz <= nz;
  const long long oh = jh * dj + kh, oy = jy * dj + ky, oz = (j0 + rz) * dj + k0 + cz;

  double np[4], nj = 0, ym = 0, yc = 0, yp = 0, ac[4], ug[4];
  auto fetch_plane = [&](int p) {
    const long long o = (long long)(a.wrap ? wrap_plane(p, a.nx) : p) * di + oh;
    if (ring_cell)
#pragma unroll
      for (int v = 0; v < 4; v++) np[v] = a.P[v][o];
  };
  auto put_plane = [&](int p) {
    if (ring_cell)
#pragma unroll
      for (int v = 0; v < 4; v++) ring[((p % 3) * 4 + v) * FRJ * FRK + tid] = np[v];
  };
  auto fetch_metric = [&](int i) {   // J on the tile with halo, Y for the weights of the y pass
    if (j_cell) nj = a.J[i * di + oh];
    if (y_cell) { ym = a.Yp[i * di + oy - dj]; yc = a.Yp[i * di + oy]; yp = a.Yp[i * di + oy + dj]; }
  };

  for (int p = ia - 1; p <= ia + 1; p++) {
    fetch_plane(p);
    put_plane(p);
  }
  fetch_metric(ia);
  for (int i = ia; i <= ib; i++) {
    // J of plane i, y-pass weights (Filter.cpp:187-191)
    if (j_cell) jt[tid] = nj;
    if (y_cell) {
      const double A = sub(yp, ym), B = sub(yp, yc), C = sub(yc, ym), rA = divisor(A);
      w1[tid] = quotient(TWO_H ? B : mul(2.0, B), A, rA);
      w3[tid] = quotient(TWO_H ? C : mul(2.0, C), A, rA);
    }
    __syncthreads();
    const bool interior = i >= 3 && i <= gend;
    if (i < ib) {
      fetch_plane(i + 2);
      fetch_metric(i + 1);
    }
    if (z_cell && interior && a.level > 0)
#pragma unroll
      for (int v = 0; v < 4; v++) ac[v] = a.acc[v][i * di + oz];
    if (wall_cell)
#pragma unroll
      for (int v = 0; v < 4; v++) ug[v] = a.U[v][i * di + oh];
    // x pass; the wall rows keep U_ (the scratch arrays start as U_ copies,
    // Filter.cpp:121-138, and the passes only write j = 2..ny)
    const int sm1 = (i - 1) % 3, s0 = i % 3, sp1 = (i + 1) % 3;
    if (ring_cell) {
#pragma unroll
      for (int v = 0; v < 4; v++)
        gx[v * FRJ * FRK + tid] = smooth3<TWO_H>(ring[(sm1 * 4 + v) * FRJ * FRK + tid], ring[(s0 * 4 + v) * FRJ * FRK + tid],
                                                 ring[(sp1 * 4 + v) * FRJ * FRK + tid]);
    } else if (wall_cell) {
#pragma unroll
      for (int v = 0; v < 4; v++) gx[v * FRJ * FRK + tid] = ug[v];
    }
    __syncthreads();
    // y pass (Filter.cpp:193 for h, :875 for 2h); z ghosts keep U_
    if (y_cell) {
      const int tm = tid, tc = tm + FRK, tp = tc + FRK;   // rows jy - 1, jy, jy + 1 of the tile with halo
      const double Jm = jt[tm], Jc = jt[tc], Jp = jt[tp], rJ = divisor(Jc);
      const double wa = w1[tid], wc = w3[tid];
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const double *g = gx + v * FRJ * FRK;
        const double s = add(add(mul(mul(wa, g[tm]), Jm), mul(mul(TWO_H ? 1.0 : 6.0, g[tc]), Jc)), mul(mul(wc, g[tp]), Jp));
        gy[v * FTJ * FRK + tid] = quotient(mul(TWO_H ? 0.5 : 0.125, s), Jc, rJ);
      }
    } else if (z_ghost) {
#pragma unroll
      for (int v = 0; v < 4; v++) gy[v * FTJ * FRK + tid] = a.U[v][i * di + oy];
    }
    __syncthreads();
    // z pass, high-pass accumulation, E on the last level
    if (z_cell) {
      const long long o = i * di + oz;
      double f[4];
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const double *g = gy + v * FTJ * FRK + rz * FRK + cz;
        const double L = smooth3<TWO_H>(g[0], g[1], g[2]);
        if (a.level < 5) a.L[v][o] = L;
        if (interior) {
          // Filter.cpp:769 / :1444, left to right
          switch (a.level) {
            case 0: a.acc[v][o] = mul(6.0, L); break;
            case 1: a.acc[v][o] = sub(ac[v], mul(15.0, L)); break;
            case 2: a.acc[v][o] = add(ac[v], mul(20.0, L)); break;
            case 3: a.acc[v][o] = sub(ac[v], mul(15.0, L)); break;
            case 4: a.acc[v][o] = add(ac[v], mul(6.0, L)); break;
            default: f[v] = sub(ac[v], L); break;
          }
        }
      }
      if (a.level == 5 && interior) {
        // Filter.cpp:796-800 / :1471-1475
        const double u1 = a.U[0][o];
        const double ue = sub(dvd(a.U[1][o], u1), dvd(f[1], f[0]));
        const double ve = sub(dvd(a.U[2][o], u1), dvd(f[2], f[0]));
        const double we = sub(dvd(a.U[3][o], u1), dvd(f[3], f[0]));
        a.E[o] = add(add(mul(ue, ue), mul(ve, ve)), mul(we, we));
      }
    }
    if (i < ib) put_plane(i + 2);   // over plane i - 1, last read by the x pass
  }
}

struct EpArgs {
  const double *Eh, *E2h;
  double *Ep[3];
  double crit, e_high, e_low;
  int nx, ny, nz, X, Y, Z;
};

// E with the ghost rules of Filter.cpp:1521-1552 (nearest interior cell in
// y and z) and the periodic image in x
__device__ __forceinline__ long long e_at(const EpArgs &a, int i, int j, int k) {
  const int ny = a.ny + 1, nz = a.nz + 1, gend = a.nx + 2;
  if (j == 1) j = 2;
  else if (j == ny + 1) j = ny;
  if (k == 1) k = 2;
  else if (k == nz + 1) k = nz;
  if (i == 2) i = gend;
  else if (i == gend + 1) i = 3;
  return (long long)i * a.Y * a.Z + (long long)j * a.Z + k;
}

__device__ __forceinline__ double ep_of(const EpArgs &a, long long p, long long q) {
  const double r = dvd(add(a.Eh[p], a.Eh[q]), add(a.E2h[p], a.E2h[q]));
  return r >= a.crit ? a.e_high : a.e_low;
}

// EpX: i = 2..gend, j = 1..ny-1, k = 1..nz-1 (Filter.cpp:1564-1585);
// EpY: i = 2..gend-1, j = 1..ny, k = 1..nz-1 (:1593-1615);
// EpZ: i = 2..gend-1, j = 1..ny-1, k = 1..nz (:1624-1645)
__global__ void k_filter_ep(EpArgs a) {
  const int k = 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = 1 + blockIdx.y;
  const int i = 2 + blockIdx.z;
  const int ny = a.ny + 1, nz = a.nz + 1, gend = a.nx + 2;
  if (k > nz) return;
  const long long o = (long long)i * a.Y * a.Z + (long long)j * a.Z + k;
  if (j < ny && k < nz) a.Ep[0][o] = ep_of(a, e_at(a, i, j + 1, k + 1), e_at(a, i + 1, j + 1, k + 1));
  if (i < gend) {
    if (k < nz) a.Ep[1][o] = ep_of(a, e_at(a, i + 1, j, k + 1), e_at(a, i + 1, j + 1, k + 1));
    if (j < ny) a.Ep[2][o] = ep_of(a, e_at(a, i + 1, j + 1, k), e_at(a, i + 1, j + 1, k + 1));
  }
}

constexpr size_t level_smem() {
  return sizeof(double) * (3 * 4 * FRJ * FRK + 4 * FRJ * FRK + 4 * FTJ * FRK + 2 * FTJ * FRK + FRJ * FRK);
}

}  // namespace

int filter_smem_bytes() { return (int)level_smem(); }

cudaError_t launch_filter(const Dev &d, const FilterBufs &b, double crit, double e_high, double e_low,
                          cudaStream_t s) {
  cudaError_t err = cudaFuncSetAttribute(k_filter_level<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)level_smem());
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_filter_level<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)level_smem());
  if (err != cudaSuccess) return err;
  const int gend = d.nx + 2;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int slots = 2 * sms;   // CTAs the chip holds (registers and shared memory of two per SM)
  const int range[6][2] = {{1, gend + 2}, {2, gend + 1}, {3, gend}, {1, gend + 2}, {2, gend + 1}, {3, gend}};
  for (int sc = 0; sc < 2; sc++) {
    LevelArgs a{};
    for (int lev = 0; lev < 6; lev++) {
      for (int v = 0; v < 4; v++) {
        a.P[v] = lev == 0 ? d.U_[v] : b.lev[(lev - 1) & 1][v];
        a.L[v] = b.lev[lev & 1][v];
        a.acc[v] = b.acc[v];
        a.U[v] = d.U_[v];
      }
      a.J = d.J;
      a.Yp = b.yp;
      a.E = sc == 0 ? b.eh : b.e2h;
      a.nx = d.nx; a.ny = d.ny; a.nz = d.nz;
      a.X = d.X; a.Y = d.Y; a.Z = d.Z;
      a.i0 = range[lev][0];
      a.i1 = range[lev][1];
      a.level = lev;
      a.wrap = lev == 3;
      // planes per CTA: the fewest plane steps in a row on one of the chip's
      // slots, waves x (chunk + 3, the three planes loaded before the first)
      const int tiles = (d.nz + FTK - 1) / FTK * ((d.ny + FTJ - 1) / FTJ), planes = a.i1 - a.i0 + 1;
      long long least = -1;
      for (int x = 1; x <= planes; x++) {
        const long long ctas = (long long)tiles * ((planes + x - 1) / x), cost = (ctas + slots - 1) / slots * (x + 3);
        if (least < 0 || cost < least) { least = cost; a.chunk = x; }
      }
      dim3 grid((d.nz + FTK - 1) / FTK, (d.ny + FTJ - 1) / FTJ, (planes + a.chunk - 1) / a.chunk);
      if (sc == 0) k_filter_level<false><<<grid, FTHREADS, level_smem(), s>>>(a);
      else k_filter_level<true><<<grid, FTHREADS, level_smem(), s>>>(a);
    }
  }
  EpArgs e{};
  e.Eh = b.eh; e.E2h = b.e2h;
  for (int f = 0; f < 3; f++) e.Ep[f] = b.ep[f];
  e.crit = crit; e.e_high = e_high; e.e_low = e_low;
  e.nx = d.nx; e.ny = d.ny; e.nz = d.nz; e.X = d.X; e.Y = d.Y; e.Z = d.Z;
  // j = 1..ny (Y_out + 1 rows cover every face range), i = 2..gend
  dim3 grid((d.nz + 1 + 127) / 128, d.ny + 1, d.nx + 1);
  k_filter_ep<<<grid, 128, 0, s>>>(e);
  return cudaGetLastError();
}

}  // namespace cgli
