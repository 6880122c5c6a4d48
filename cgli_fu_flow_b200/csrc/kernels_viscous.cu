// Viscous terms (Viscous_terms.cpp:260-904) in one pass over the grid:
// velocity and temperature of the cells, the viscous fluxes of the three face
// sets and their divergence.
//
// A CTA owns a column of ROWS j rows x 32 k columns and marches through a
// chunk of x planes.  Velocity and temperature of four planes (one behind,
// the current, one ahead, one being filled) lie in shared memory with a halo
// of one cell; a warp holds one row, and one more warp (the edge warp) loads
// the two halo columns and forms the z faces of the last column.  Every face
// flux is formed once: its x face waits for the next plane in registers, its
// y face goes to the row below through shared memory, its z face to the lane
// before by shuffle.  The raw state of a plane is loaded two planes ahead, and
// one barrier a plane orders both the planes and the exchanged fluxes.
//
// Bound by latency (the stencil's shared-memory loads and the FP64 chain with
// 16 warps per SM): 418 us at 256x192x192, where the bytes (six arrays in,
// four out) take 115 us and the FP64 operations 170; three kernels, which
// moved 22 arrays more (velocities and face fluxes through memory), took 663.
// 160x128x128: 208 -> 129 us, with general metrics 412 -> 360.
#include "cgli_dev.cuh"
#include "cgli_launch.h"
#include "viscous_face.cuh"

namespace cgli {

namespace {

struct VP { double U, V, W, T; };

template <int ROWS>
struct ViscTile {
  static constexpr int NR = ROWS + 2, NC = 34;      // rows and columns with halo
  static constexpr int THREADS = (NR + 1) * 32;     // a warp per row, the edge warp
  static constexpr int VAR = NR * NC, SLOT = 4 * VAR;
  static constexpr int YX = NR * 4 * 32, ZX = NR * 4;   // exchanged y and z faces of a plane
  static constexpr size_t SMEM = sizeof(double) * (4 * SLOT + 2 * YX + 2 * ZX);
  static_assert(NR <= 16, "the edge warp holds a halo column per half warp");
};

template <int VAR>
__device__ __forceinline__ VP vp(const double *p) {
  VP r; r.U = p[0]; r.V = p[VAR]; r.W = p[2 * VAR]; r.T = p[3 * VAR]; return r;
}

}  // namespace

// planes 3 + chunk blockIdx.z ...; CH: the face metrics have the channel's
// form (d.face_tables), so the per-row tables give eta_y and 1/J and the
// channel forms of the face fluxes apply
template <bool CH, int ROWS, int MINB>
__global__ void __launch_bounds__(ViscTile<ROWS>::THREADS, MINB) k_viscous(Dev d, int chunk) {
  using S = ViscTile<ROWS>;
  constexpr int NC = S::NC, VAR = S::VAR;
  extern __shared__ double sm[];
  double *const yx = sm + 4 * S::SLOT, *const zx = yx + 2 * S::YX;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ie = d.nx + 2, jn = d.ny + 1, kn = d.nz + 1;
  const int ilo = 3 + blockIdx.z * chunk, ihi = min(ie, ilo + chunk - 1);
  const int J0 = 2 + blockIdx.y * ROWS, K0 = 2 + blockIdx.x * 32;
  const bool edge = w == S::NR;
  // this thread's cell of the tile: the edge warp's halves hold the columns
  // K0+32 and K0-1
  const int row = edge ? lane & 15 : w;
  const int col = edge ? (lane < 16 ? 33 : 0) : lane + 1;
  const bool held = row < S::NR;
  const int j = J0 - 1 + row, k = K0 - 1 + col;
  const long long base = ix(d, 0, min(j, jn + 1), min(k, kn + 1));
  const int cell = min(row, S::NR - 1) * NC + col;
  const bool outrow = row >= 1 && row <= ROWS && j <= jn;   // an output row
  const bool do_x = !edge && outrow && k <= kn;
  const bool do_y = !edge && row >= 1 && j <= jn + 1 && k <= kn;
  const bool do_z = outrow && col >= 1 && k <= kn + 1;
  const double rxi = d.rdxi, ret = d.rdet, rzt = d.rdzt;

  double q[5], J = 1;
  auto load = [&](int p) {
    if (!held) return;
    const long long c = base + p * d.di;
#pragma unroll
    for (int v = 0; v < 5; v++) q[v] = d.U_[v][c];
    J = d.J[c];
  };
  // the divisions by rho, rho R and J as Newton-refined reciprocals
  auto store = [&](int p) {
    if (!held) return;
    double *s = sm + (p & 3) * S::SLOT + cell;
    const double irho = nr_rcp(q[0]);
    const double U = q[1] * irho, V = q[2] * irho, W = q[3] * irho;
    const double P = (q[4] - 0.5 * q[0] * (U * U + V * V + W * W)) * (KG - 1) * J;
    s[0] = U; s[VAR] = V; s[2 * VAR] = W;
    s[3 * VAR] = P * (irho * (1.0 / RG)) * nr_rcp(J);
  };
  for (int p = ilo - 1; p <= ilo + 1; p++) { load(p); store(p); }

  double xo[4] = {0, 0, 0, 0}, yo[4] = {0, 0, 0, 0}, dz[4] = {0, 0, 0, 0};   // of plane p-1
  for (int p = ilo; p <= ihi + 1; p++) {
    __syncthreads();   // planes up to p+1 and the exchanged faces of p-1 are in shared memory
    const bool ahead = p + 2 <= ihi + 1, inner = p <= ihi;
    if (ahead) load(p + 2);
    const double *const b = sm + (p & 3) * S::SLOT + cell;
    const double *const bm = sm + ((p - 1) & 3) * S::SLOT + cell;
    const double *const bp = sm + ((p + 1) & 3) * S::SLOT + cell;
    const long long f = ix(d, p - 1, j - 1, k - 1);
    const VP o = vp<VAR>(b);
    double F[4] = {0, 0, 0, 0};
    if (do_x) {
      if (CH) {
        const double *t = d.ftab + (0LL * d.Y + (j - 1)) * 4;
        visc_face_x_channel(rxi, ret, rzt, d.mu, d.rpr, t[0], o, vp<VAR>(bm), vp<VAR>(b + NC), vp<VAR>(bm + NC),
                            vp<VAR>(b - NC), vp<VAR>(bm - NC), vp<VAR>(b + 1), vp<VAR>(bm + 1), vp<VAR>(b - 1),
                            vp<VAR>(bm - 1), t[2], F);
      } else {
        double mm[9], Jf, iJf;
        face_metrics(d, 0, f, j - 1, mm, Jf, iJf);
        visc_face_x(rxi, ret, rzt, d.mu, d.rpr, o, vp<VAR>(bm), vp<VAR>(b + NC), vp<VAR>(bm + NC), vp<VAR>(b - NC),
                    vp<VAR>(bm - NC), vp<VAR>(b + 1), vp<VAR>(bm + 1), vp<VAR>(b - 1), vp<VAR>(bm - 1), mm, iJf, F);
      }
      if (p > ilo) {   // plane p-1 is complete
        const long long c = ix(d, p - 1, j, k);
        const double *const yn = yx + ((p - 1) & 1) * S::YX + (row + 1) * 128 + lane;
        const double *const zn = zx + ((p - 1) & 1) * S::ZX + row * 4;
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const double z = lane == 31 ? zn[v] + dz[v] : dz[v];
          d.vF[v][c] = (F[v] - xo[v]) * rxi + (yn[v * 32] - yo[v]) * ret + z * rzt;
        }
      }
#pragma unroll
      for (int v = 0; v < 4; v++) xo[v] = F[v];
    }
    if (inner && do_y) {
      if (CH) {
        const double *t = d.ftab + (1LL * d.Y + (j - 1)) * 4;
        visc_face_y_channel(rxi, ret, rzt, d.mu, d.rpr, t[0], o, vp<VAR>(b - NC), vp<VAR>(bp), vp<VAR>(bp - NC),
                            vp<VAR>(bm), vp<VAR>(bm - NC), vp<VAR>(b + 1), vp<VAR>(b - NC + 1), vp<VAR>(b - 1),
                            vp<VAR>(b - NC - 1), t[2], yo);
      } else {
        double mm[9], Jf, iJf;
        face_metrics(d, 1, f, j - 1, mm, Jf, iJf);
        visc_face_y(rxi, ret, rzt, d.mu, d.rpr, o, vp<VAR>(b - NC), vp<VAR>(bp), vp<VAR>(bp - NC), vp<VAR>(bm),
                    vp<VAR>(bm - NC), vp<VAR>(b + 1), vp<VAR>(b - NC + 1), vp<VAR>(b - 1), vp<VAR>(b - NC - 1), mm, iJf,
                    yo);
      }
      double *const y = yx + (p & 1) * S::YX + row * 128 + lane;
#pragma unroll
      for (int v = 0; v < 4; v++) y[v * 32] = yo[v];
    }
    if (inner && __any_sync(0xffffffffu, do_z)) {
      double G[4] = {0, 0, 0, 0};
      if (do_z) {
        if (CH) {
          const double *t = d.ftab + (2LL * d.Y + (j - 1)) * 4;
          visc_face_z_channel(rxi, ret, rzt, d.mu, d.rpr, t[0], o, vp<VAR>(b - 1), vp<VAR>(bp), vp<VAR>(bp - 1),
                              vp<VAR>(bm), vp<VAR>(bm - 1), vp<VAR>(b + NC), vp<VAR>(b + NC - 1), vp<VAR>(b - NC),
                              vp<VAR>(b - NC - 1), t[2], G);
        } else {
          double mm[9], Jf, iJf;
          face_metrics(d, 2, f, j - 1, mm, Jf, iJf);
          visc_face_z(rxi, ret, rzt, d.mu, d.rpr, o, vp<VAR>(b - 1), vp<VAR>(bp), vp<VAR>(bp - 1), vp<VAR>(bm),
                      vp<VAR>(bm - 1), vp<VAR>(b + NC), vp<VAR>(b + NC - 1), vp<VAR>(b - NC), vp<VAR>(b - NC - 1),
                      vp<VAR>(bm + NC), mm, iJf, G);
        }
        if (edge) {
          double *const z = zx + (p & 1) * S::ZX + row * 4;
#pragma unroll
          for (int v = 0; v < 4; v++) z[v] = G[v];
        }
      }
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const double up = __shfl_down_sync(0xffffffffu, G[v], 1);
        dz[v] = lane == 31 ? -G[v] : up - G[v];
      }
    }
    if (ahead) store(p + 2);
  }
}

namespace {

template <bool CH, int ROWS, int MINB>
void viscous(const Dev &d, cudaStream_t s) {
  using S = ViscTile<ROWS>;
  const auto kern = k_viscous<CH, ROWS, MINB>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  dim3 g((d.nz + 31) / 32, (d.ny + ROWS - 1) / ROWS, 1);
  const int chunk = march_chunk(d.nx, (int)(g.x * g.y), MINB, 3);
  g.z = (d.nx + chunk - 1) / chunk;
  kern<<<g, S::THREADS, S::SMEM, s>>>(d, chunk);
}

}  // namespace

// Planes per CTA of a kernel that marches `cols` columns of nx planes, with
// `resident` CTAs per SM and the time of `start` planes for a CTA's start: the
// fewest planes in a row on one SM.
int march_chunk(int nx, int cols, int resident, int start) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int best = nx;
  long long least = -1;
  for (int x = 1; x <= nx; x++) {
    const long long ctas = (long long)cols * ((nx + x - 1) / x), slots = (long long)sms * resident;
    const long long cost = (ctas + slots - 1) / slots * (x + start);
    if (least < 0 || cost < least) { least = cost; best = x; }
  }
  return best;
}

// 13 rows a CTA: 16 warps of up to 128 registers, one CTA per SM.  The channel
// form needs 114 registers; at 256x192x192 7 rows with three CTAs per SM (64
// registers) take 522 us, 9 rows with two (80) 505, 5 rows with three (80) 495,
// 13 rows 418.  General metrics at 160x128x128: 6 rows with two 457, 5 rows
// with two 410, 9 rows with one 442, 13 rows 360 (128 registers, 344 B of spill
// stores and 240 of loads).
void launch_viscous(const Dev &d, cudaStream_t s) {
  if (d.face_tables) viscous<true, 13, 1>(d, s);
  else viscous<false, 13, 1>(d, s);
}

}  // namespace cgli
