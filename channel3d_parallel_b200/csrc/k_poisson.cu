// Pseudo-pressure Poisson solve and projection.
//
// solve_poisson_equation (src/poisson.f90:33-101) restated for one GPU:
//   per y-plane 2-D DFT over (x, z)   -> k_xfft_fwd (k_xfft.cu): x
//                                        real-to-complex FFT of each (j, k)
//                                        line, divergence fused in;
//   per (kx, kz) tridiagonal in y     -> k_slab_fwd, k_slab_inv (k_slab.cu):
//   (Zgtsv, :50-75)                      z FFT, partitioned elimination over
//                                        blocks of rows, inverse z FFT;
//   inverse DFT / (nxp*nzp), real     -> k_xfft_inv (k_xfft.cu):
//   part, periodic copies (:78-88)       complex-to-real x FFT of the Hermitian
//                                        half spectrum.
// gradient (src/differential_operators.f90:16-52) and the projection update
// (src/projection.f90:22-46) are k_grad_sub; in the time step k_grad_sub2,
// which also writes every ghost entry of u, v, w (the boundary conditions)
// and, in the last stage, adds the constant-x-mass-flow shift whose bulk
// flux the forward x FFT reduced (k_xfft_fwd<FROM_DIV_FLUX>).
//
// Two precisions share the kernels (template T): FP64, and FP32 for the
// mixed-precision solve, where the kx = kz = 0 wall-normal mode is computed
// in FP64 (line sums of the right-hand side and an FP64 Thomas solve of the
// pinned mean mode) and the FP32 result is refined by re-projecting with the
// FP64 residual div(u).
//
// Spectrum layout in HBM: spec[(m*Ny + (j-2))*pz + (k-2)], m = 0..Nx/2: a kx
// slab is Ny contiguous rows of pz >= Nz complex values.
#include <algorithm>
#include <cmath>
#include <vector>

#include "c3d_internal.cuh"
#include "fft.cuh"
#include "ghost_images.cuh"

namespace c3d {

// ---------------------------------------------------------------------------
// host set-up
// ---------------------------------------------------------------------------
constexpr int kBandMaxR = 16;       // largest FFT radix of the band solve (128 registers)

static bool make_passes(int n, FftPasses& P) { return make_fft_passes(n, P, 8); }

constexpr int kMaxNx = 512;         // longest x row

static FftPasses get_passes(int n, int maxr) {
  FftPasses P{};
  make_fft_passes(n, P, maxr);
  return P;
}

template <typename C>
static int make_twiddles(Handle* h, int n, C** out) {
  std::vector<C> t(n);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int m = 0; m < n; ++m) {
    long double a = -2.0L * pi * (long double)m / (long double)n;
    t[m].x = (decltype(t[m].x))cosl(a);
    t[m].y = (decltype(t[m].y))sinl(a);
  }
  if (*out == nullptr) {
    int rc = dev_alloc(h, out, n);
    if (rc) return rc;
  }
  C3D_CUDA_TRY(h, cudaMemcpyAsync(*out, t.data(), sizeof(C) * n, cudaMemcpyHostToDevice, h->stream));
  return 0;
}

// Thomas factorisation of every mode, the no-pivot path of the reference's
// LAPACK zgtsv call (src/poisson.f90:72): MULT = DL(k)/D(k), D(k+1) -= MULT*DU(k),
// one thread per mode.  Stored: 1/d'_j, layout [(m*Ny + j)*nkzs + kz'], FP64
// and (if given) FP32, and the multipliers of mode (0, 0).  Rounded operation
// by operation as written.
__global__ void k_tri_table(Dims d, const double* __restrict__ dd, const double* __restrict__ dl,
                            const double* __restrict__ du, const double* __restrict__ kxx,
                            const double* __restrict__ kzz, double* __restrict__ rdp, float* __restrict__ rdp32,
                            double* __restrict__ mult00) {
  const int kz = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
  if (kz >= d.nkzs) return;
  const double kx2 = kxx[m], kz2 = kzz[kz];
  double up = 0.0;                          // MULT(j-1)*DU(j-1)
  for (int j = 0; j < d.Ny; ++j) {
    double D = (dd[j] + kx2) + kz2;
    if (m == 0 && kz == 0 && j == 0) D = 3.0 / 2.0 * D;       // src/poisson.f90:69
    if (j > 0) D = __dsub_rn(D, up);
    const int64_t o = ((int64_t)m * d.Ny + j) * d.nkzs + kz;
    const double r = __ddiv_rn(1.0, D);
    rdp[o] = r;
    if (rdp32) rdp32[o] = (float)r;
    if (j + 1 < d.Ny) {
      const double mu = __ddiv_rn(dl[j], D);
      up = __dmul_rn(mu, du[j]);
      if (m == 0 && kz == 0) mult00[j] = mu;
    }
  }
}

// the tables of the current grid (FP32 copies once the mixed path is set up)
static int build_tri_table(Handle* h) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  const int Ny = d.Ny, nkx = d.nkx, nkzs = d.nkzs;
  const int64_t nt = (int64_t)Ny * nkzs * nkx;
  int rc;
  if (S.rdp == nullptr) {
    if ((rc = dev_alloc(h, &S.rdp, nt))) return rc;
    if ((rc = dev_alloc(h, &S.mult00, Ny))) return rc;
    if ((rc = dev_alloc(h, &S.dl, Ny))) return rc;
    if ((rc = dev_alloc(h, &S.du, Ny))) return rc;
    if ((rc = dev_alloc(h, &S.dl32, Ny))) return rc;
    if ((rc = dev_alloc(h, &S.du32, Ny))) return rc;
    if ((rc = dev_alloc(h, &S.tri, Ny + nkx + nkzs))) return rc;
  }
  if (S.spec32 != nullptr && S.rdp32 == nullptr && (rc = dev_alloc(h, &S.rdp32, nt))) return rc;
  std::vector<double> dl(Ny, 0.0), du(Ny, 0.0), tri(Ny + nkx + nkzs);
  std::vector<float> dl32(Ny, 0.0f), du32(Ny, 0.0f);
  for (int jj = 0; jj + 1 < Ny; ++jj) {
    dl[jj] = h->Dl[jj + 3];   // Dyy(j+1, j), j = jj+2
    du[jj] = h->Du[jj + 2];   // Dyy(j, j+1)
    dl32[jj] = (float)dl[jj];
    du32[jj] = (float)du[jj];
  }
  for (int jj = 0; jj < Ny; ++jj) tri[jj] = h->Dd[jj + 2];
  for (int m = 0; m < nkx; ++m) tri[Ny + m] = h->kxx[m];
  for (int k = 0; k < nkzs; ++k) tri[Ny + nkx + k] = h->kzz[k];
  cudaStream_t s = h->stream;
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.dl, dl.data(), Ny * 8, cudaMemcpyHostToDevice, s));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.du, du.data(), Ny * 8, cudaMemcpyHostToDevice, s));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.dl32, dl32.data(), Ny * 4, cudaMemcpyHostToDevice, s));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.du32, du32.data(), Ny * 4, cudaMemcpyHostToDevice, s));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.tri, tri.data(), tri.size() * 8, cudaMemcpyHostToDevice, s));
  k_tri_table<<<dim3((nkzs + 63) / 64, nkx), 64, 0, s>>>(d, S.tri, S.dl, S.du, S.tri + Ny, S.tri + Ny + nkx, S.rdp,
                                                         S.rdp32, S.mult00);
  C3D_LAUNCH_CHECK(h);
  S.tail_current = false;
  C3D_CUDA_TRY(h, cudaStreamSynchronize(s));   // the host copies end here
  return 0;
}

// ---------------------------------------------------------------------------
// Band-restricted z transform and y solve (FP64), for the Poisson solve of
// the Schur complement: the right-hand side is zero outside the rows
// [rlo, rhi] and only those rows of the solution are read.  Thomas on the
// band alone: the forward sweep starts at rlo from zero, and the back
// substitution starts from x(rhi+1) = S(rhi+1) y(rhi+1), y(rhi+1) =
// -MULT(rhi) y(rhi), where S(j) = x(j)/y(j) of the homogeneous tail is
// tabulated once per grid (build_tail_table).  One CTA per kx slab, the band rows in
// shared memory; the band's own z transform, there and back.
// ---------------------------------------------------------------------------
struct BandYzArgs {
  Dims d;
  double2* __restrict__ spec;
  const double2* __restrict__ tw;
  const double* __restrict__ rdp;
  const double* __restrict__ tail;
  const double* __restrict__ dl;
  const double* __restrict__ du;
  FftPasses P;
  int rs, pz;
  int rlo, rhi;
};

__global__ void __launch_bounds__(256) k_spectral_band(BandYzArgs a) {
  extern __shared__ __align__(16) unsigned char sb_smem[];
  const int m = blockIdx.x;
  const int Ny = a.d.Ny, Nz = a.d.Nz, nkzs = a.d.nkzs, RS = a.rs;
  const int nr = a.rhi - a.rlo + 1;
  double2* data = reinterpret_cast<double2*>(sb_smem);   // [nr][RS]
  double2* tw = data + (size_t)nr * RS;                   // [Nz]
  const int tid = threadIdx.x, nt = blockDim.x;
  double2* g = a.spec + ((int64_t)m * Ny + a.rlo) * a.pz;
  for (int t = tid; t < Nz; t += nt) tw[t] = a.tw[t];
  // eight loads in flight per thread before any store
  for (int t0 = tid; t0 < nr * Nz; t0 += 8 * nt) {
    double2 tv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + u * nt, r = t / Nz, c = t - r * Nz;
      tv[u] = t < nr * Nz ? g[(int64_t)r * a.pz + c] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + u * nt, r = t / Nz, c = t - r * Nz;
      if (t < nr * Nz) data[r * RS + c] = tv[u];
    }
  }
  __syncthreads();
  fft_rows_dif<double, kBandMaxR>(data, nr, RS, tw, a.P);
  const double* rdp_m = a.rdp + (int64_t)m * Ny * nkzs;
  const double* tail_m = a.tail + (int64_t)m * Ny * nkzs;
  for (int col = tid; col < Nz; col += nt) {
    const int kz = dif_position_to_k(col, a.P);
    const int kzs = kz <= Nz - kz ? kz : Nz - kz;
    // forward: y(j) = b(j) - DL(j-1)/D'(j-1) y(j-1), y(rlo-1) = 0
    double2 prev = make_double2(0.0, 0.0);
    for (int r = 0; r < nr; ++r) {
      const int j = a.rlo + r;
      double2 b = data[r * RS + col];
      if (r > 0) {
        const double mu = a.dl[j - 1] * rdp_m[(int64_t)(j - 1) * nkzs + kzs];
        b.x -= mu * prev.x;
        b.y -= mu * prev.y;
      }
      data[r * RS + col] = b;
      prev = b;
    }
    // the rows above the band, through the tail ratio
    double2 xn = make_double2(0.0, 0.0);
    if (a.rhi + 1 < Ny) {
      const double mu = a.dl[a.rhi] * rdp_m[(int64_t)a.rhi * nkzs + kzs];
      const double sx = -mu * tail_m[(int64_t)(a.rhi + 1) * nkzs + kzs];
      xn.x = sx * prev.x;
      xn.y = sx * prev.y;
    }
    // back substitution x(j) = (y(j) - DU(j) x(j+1)) / D'(j)
    for (int r = nr - 1; r >= 0; --r) {
      const int j = a.rlo + r;
      const double rp = rdp_m[(int64_t)j * nkzs + kzs];
      const double u = a.du[j];
      double2 b = data[r * RS + col];
      b.x = (b.x - u * xn.x) * rp;
      b.y = (b.y - u * xn.y) * rp;
      data[r * RS + col] = b;
      xn = b;
    }
  }
  __syncthreads();
  fft_rows_dit_inv<double, kBandMaxR>(data, nr, RS, tw, a.P);
  for (int t = tid; t < nr * Nz; t += nt) {
    const int r = t / Nz, c = t - r * Nz;
    g[(int64_t)r * a.pz + c] = data[r * RS + c];
  }
}

// S(j) = x(j)/y(j) when the right-hand side vanishes from row j on:
// S(Ny-1) = 1/D'(Ny-1), S(j) = (1 + DU(j) MULT(j) S(j+1)) / D'(j), with
// MULT(j) = DL(j)/D'(j) formed as the solves form it
static int build_tail_table(Handle* h) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  const int Ny = d.Ny, nkx = d.nkx, nkzs = d.nkzs;
  const int64_t nt = (int64_t)Ny * nkzs * nkx;
  std::vector<double> rdp(nt), tail(nt), dl(Ny), du(Ny);
  C3D_CUDA_TRY(h, cudaMemcpyAsync(rdp.data(), S.rdp, 8 * nt, cudaMemcpyDeviceToHost, h->stream));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(dl.data(), S.dl, 8 * Ny, cudaMemcpyDeviceToHost, h->stream));
  C3D_CUDA_TRY(h, cudaMemcpyAsync(du.data(), S.du, 8 * Ny, cudaMemcpyDeviceToHost, h->stream));
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  for (int m = 0; m < nkx; ++m)
    for (int kzs = 0; kzs < nkzs; ++kzs) {
      auto o = [&](int j) { return ((int64_t)m * Ny + j) * nkzs + kzs; };
      double sj = rdp[o(Ny - 1)];
      tail[o(Ny - 1)] = sj;
      for (int j = Ny - 2; j >= 0; --j) {
        const double mu = dl[j] * rdp[o(j)];
        sj = (1.0 + du[j] * mu * sj) * rdp[o(j)];
        tail[o(j)] = sj;
      }
    }
  int rc;
  if (!S.tail && (rc = dev_alloc(h, &S.tail, nt))) return rc;
  C3D_CUDA_TRY(h, cudaMemcpyAsync(S.tail, tail.data(), 8 * nt, cudaMemcpyHostToDevice, h->stream));
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  S.tail_current = true;
  return 0;
}

static size_t band_yz_smem(const Dims& d, int rs, int nr) {
  return sizeof(double2) * ((size_t)nr * rs + d.Nz);
}
static const size_t kBandYzSmemMax = 200 * 1024;

// the band solve of rows [blo, bhi] when it fits in shared memory; false
// (nothing launched) otherwise
static int launch_band_yz(Handle* h, int blo, int bhi, bool* done) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  *done = false;
  const int nr = bhi - blo + 1;
  int rs = d.Nz;
  while (rs % 8 != 1) ++rs;
  const size_t smem = band_yz_smem(d, rs, nr);
  if (nr <= 0 || smem > kBandYzSmemMax) return 0;
  int rc;
  if (!S.tail_current) {   // first use on this grid (outside any graph capture: the table build synchronises)
    if ((rc = build_tail_table(h))) return rc;
    C3D_CUDA_TRY(h, cudaFuncSetAttribute(k_spectral_band, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kBandYzSmemMax));
  }
  BandYzArgs a{};
  a.d = d; a.spec = S.spec; a.tw = S.twz; a.rdp = S.rdp; a.tail = S.tail; a.dl = S.dl; a.du = S.du;
  a.P = get_passes(d.Nz, kBandMaxR); a.rs = rs; a.pz = S.pz64; a.rlo = blo; a.rhi = bhi;
  k_spectral_band<<<(unsigned)d.nkx, 256, smem, h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  *done = true;
  return 0;
}

// ---------------------------------------------------------------------------
// FP64 kx = kz = 0 mode of the mixed path: plane sums and the pinned solve
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_mode00(Dims d, const double* __restrict__ linesum,
                                                 const double* __restrict__ mult00, const double* __restrict__ rdp,
                                                 const double* __restrict__ du, double* __restrict__ phi00) {
  extern __shared__ double m00[];
  const int Ny = d.Ny, Nz = d.Nz, nkzs = d.nkzs;
  double* b00 = m00;                 // plane sums, then the solution
  double* sm_ = m00 + Ny;            // the (0, 0) rows of the factor tables
  double* sr = m00 + 2 * Ny;
  double* su = m00 + 3 * Ny;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // plane sums: one warp per row j, a fixed shuffle tree over its z lines
  for (int j = warp; j < Ny; j += nw) {
    double s = 0.0;
    for (int k = lane; k < Nz; k += 32) s += linesum[(int64_t)j * Nz + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) b00[j] = s;
  }
  for (int j = threadIdx.x; j < Ny; j += blockDim.x) {
    sm_[j] = j > 0 ? mult00[j - 1] : 0.0;
    sr[j] = rdp[(int64_t)j * nkzs];
    su[j] = du[j];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // mode (0, 0): table entries (m = 0, kz' = 0), elimination in shared memory
    for (int j = 1; j < Ny; ++j) b00[j] = b00[j] - sm_[j] * b00[j - 1];
    double xn = b00[Ny - 1] * sr[Ny - 1];
    b00[Ny - 1] = xn;
    for (int j = Ny - 2; j >= 0; --j) {
      xn = (b00[j] - su[j] * xn) * sr[j];
      b00[j] = xn;
    }
  }
  __syncthreads();
  const double sd = (double)d.Nx * (double)d.Nz;
  for (int j = threadIdx.x; j < Ny; j += blockDim.x) phi00[j] = b00[j] / sd;
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
// Which form of the z transforms and y solves: the cluster that keeps a slab on
// chip moves the spectrum once in place of twice and has no chain through
// memory, but past 256 columns a thread of it has several, and slabs of many
// rows or columns need 16 CTAs.  Few such slabs, resident at once, are still
// better off there (at most two of their CTAs an SM, three with up to 64 columns;
// where the CTAs are more than three quarters full, two waves of up to four an
// SM): in thin channels the chain over the blocks is what the other form waits
// for.
// Measured, cluster against blocks (us, B200, FP64), clusters of up to 8 CTAs:
// 192x128x192 45 / 67, 256x128x256 93 / 114, 64x256x64 19 / 33; more than 256
// columns: 48x8x384 30 / 18, 12x64x288 34 / 21, 128x64x384 89 / 65, 384x256x384
// 1237 / 417; 16 CTAs: 12x300x12 15 / 25, 36x160x64 17 / 21, 24x160x128 21 / 25,
// 36x160x128 27 / 25, 64x160x128 42 / 32, 24x500x64 21 / 39, 48x500x64 38 / 45, 64x500x64 51 / 50,
// 24x300x36 17 / 25, 36x300x36 30 / 27, 96x300x64 61 / 41, 192x256x192 156 / 134.
// FP32 (mixed steps, six solves): 24x300x64 390 / 429, 36x500x64 723 / 823,
// 96x300x36 670 / 537, 48x8x288 378 / 211.
static bool slab_by_blocks(const Dims& d, const SlabCluster& c) {
  if (d.Nz > 256) return true;
  if (c.cs <= 8) return false;
  const bool filled = 4 * c.jc > 3 * c.jmax;
  const int most = filled ? std::min(2 * c.active, 4 * 148 / c.cs) : std::min(c.active, (d.Nz > 64 ? 2 : 3) * 148 / c.cs);
  return d.nkx > most;
}

// parts: bit0 x FFT, bit1 y-z solve, bit2 inverse x FFT.  rhs_in: the
// right-hand side, or with from_div the potential whose residual
// div((U, V, W) - grad rhs_in) is solved for (FP32).
template <typename T>
static int run_spectral_t(Handle* h, bool from_div, const double* U, const double* V, const double* W,
                          const double* rhs_in, double* out, double* phi1, int accumulate, int parts,
                          int blo = 0, int bhi = -1, double flux_dt = 0.0) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  constexpr bool f32 = sizeof(T) == 4;
  int rc;
  if (bhi < 0) bhi = d.Ny - 1;                 // band of j rows (0-based j-2); full by default
  if (parts & 1) {
    const bool whole = blo == 0 && bhi == d.Ny - 1;
    if ((rc = launch_xfft_fwd<T>(h, from_div, U, V, W, rhs_in, f32 ? S.linesum : nullptr, blo, bhi,
                                 from_div && whole ? flux_dt : 0.0)))
      return rc;
    if (f32) {
      k_mode00<<<1, 1024, 4 * sizeof(double) * d.Ny, h->stream>>>(d, S.linesum, S.mult00, S.rdp, S.du, S.phi00);
      C3D_LAUNCH_CHECK(h);
    }
  }
  if (parts & 2) {
    bool band_done = false;
    if (!f32 && (blo > 0 || bhi < d.Ny - 1)) {   // a band of rows: the band-restricted solve
      if ((rc = launch_band_yz(h, blo, bhi, &band_done))) return rc;
    }
    if (!band_done) {
      typename SlabTables<T>::C* spec;
      if constexpr (f32) spec = S.spec32; else spec = S.spec;
      const SlabCluster& c = f32 ? S.cluster32 : S.cluster;
      rc = slab_by_blocks(d, c) ? launch_slab<T>(h, spec, f32 ? 1 : 0, blo, bhi)
                                : launch_cluster<T>(h, spec, f32 ? 1 : 0, blo, bhi);
      if (rc) return rc;
    }
  }
  if (parts & 4) {
    if ((rc = launch_xfft_inv<T>(h, out, phi1, f32 ? S.phi00 : nullptr, accumulate, blo, bhi))) return rc;
  }
  if (parts == 7) h->stats.poisson_solves++;
  return 0;
}

int profile_spectral(Handle* h, int part) {
  return run_spectral_t<double>(h, true, h->Us, h->Vs, h->Ws, nullptr, h->rhs_p, nullptr, 0, 1 << part);
}

// divergence only (fine entry and diagnostics): rhs_p = div(U,V,W) incl. the
// reference's duplicated planes i = nxg-1 and k = nzg-1, and zero plane nzg
__global__ void k_divergence(Dims d, Metric m, const double* __restrict__ U,
                             const double* __restrict__ V, const double* __restrict__ W,
                             double* __restrict__ rhs) {
  const int64_t n1 = d.nxg - 2, n2 = d.nyg - 2, n3 = d.nzg - 1;
  const int64_t tot = n1 * n2 * n3;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = 2 + (int)(t % n1);
    const int j = 2 + (int)((t / n1) % n2);
    const int k = 2 + (int)(t / (n1 * n2));
    double v = 0.0;
    if (k <= d.nzg - 1) {
      v = (U[idxU(d, i, j, k)] - U[idxU(d, i - 1, j, k)]) * m.rdx[i]
        + (V[idxV(d, i, j, k)] - V[idxV(d, i, j - 1, k)]) * m.rdy[j]
        + (W[idxW(d, i, j, k)] - W[idxW(d, i, j, k - 1)]) * m.rdz[k];
    }
    rhs[t] = v;
  }
}

int launch_divergence(Handle* h, const double* U, const double* V, const double* W, double* rhs) {
  k_divergence<<<148 * 8, 256, 0, h->stream>>>(h->d, h->m, U, V, W, rhs);
  C3D_LAUNCH_CHECK(h);
  return 0;
}

// in place on an rhs_p-shaped array; always FP64 (fine entry, IB operators)
int launch_poisson_solve(Handle* h, double* rhs, int rk_step, double dt) {
  int rc = run_spectral_t<double>(h, false, nullptr, nullptr, nullptr, rhs, rhs,
                                  rk_step == 1 ? h->phi1 : nullptr, 0, 7);
  if (rc) return rc;
  if (rk_step == 1) { h->P_pending = true; h->P_pending_dt = dt; }
  return 0;
}

// solve for the divergence of (U, V, W) into out (rhs_p layout), the
// divergence computed inside the forward x FFT (divergence followed by
// solve_poisson_equation, src/differential_operators.f90:54-74 and
// src/poisson.f90:33-101); P side effect at rk_step 1
int launch_poisson_of_div(Handle* h, const double* U, const double* V, const double* W, double* out,
                          int rk_step, double dt) {
  int rc = run_spectral_t<double>(h, true, U, V, W, nullptr, out, rk_step == 1 ? h->phi1 : nullptr, 0, 7);
  if (rc) return rc;
  if (rk_step == 1) { h->P_pending = true; h->P_pending_dt = dt; }
  return 0;
}

// the same restricted to a band of j rows (Fortran j = jlo..jhi): the
// divergence of (U, V, W) is zero outside the band and the caller reads the
// solution only inside it (the Schur complement's spread field and its
// gathers); rows of `out` outside the band are left as they were
int launch_poisson_of_div_band(Handle* h, const double* U, const double* V, const double* W, double* out,
                               int jlo, int jhi) {
  const int blo = std::max(jlo - 2, 0), bhi = std::min(jhi - 2, h->d.Ny - 1);
  if (bhi < blo) return 0;
  return run_spectral_t<double>(h, true, U, V, W, nullptr, out, nullptr, 0, 7, blo, bhi);
}

// ---------------------------------------------------------------------------
// projection: U = Ui - G phi at interior points (src/projection.f90:40-44),
// optional P_interim = phi/dt; ghosts are filled by the caller
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 6) k_grad_sub(Dims d, Metric m, const double* __restrict__ Ui,
                                                  const double* __restrict__ Vi,
                                                  const double* __restrict__ Wi,
                                                  const double* __restrict__ phi,
                                                  double* __restrict__ Uo, double* __restrict__ Vo,
                                                  double* __restrict__ Wo,
                                                  double* __restrict__ Pint, double rdt, int dup) {
  const int i = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = 2 + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = 2 + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > d.Nx + 1 || j > d.Ny + 1 || k > d.Nz + 1) return;
  const double p0 = __ldg(phi + idxR(d, i, j, k));
  const double px = __ldg(phi + idxR(d, i + 1, j, k));
  const double pz = __ldg(phi + idxR(d, i, j, k + 1));
  const int64_t iu = idxU(d, i, j, k), iw = idxW(d, i, j, k);
  const double un = __ldg(Ui + iu) - (px - p0) * m.rdxg[i];
  const double wn = __ldg(Wi + iw) - (pz - p0) * m.rdzg[k];
  double py = 0.0, vn = 0.0;
  if (j <= d.Ny) {
    py = __ldg(phi + idxR(d, i, j + 1, k));
    vn = __ldg(Vi + idxV(d, i, j, k)) - (py - p0) * m.rdyg[j];
  }
  Uo[iu] = un;
  Wo[iw] = wn;
  if (j <= d.Ny) Vo[idxV(d, i, j, k)] = vn;
  if (dup && k == 2) {
    // the reference's gradient also covers plane nzg-1 (the duplicate of
    // plane 2) for the x and y components (src/differential_operators.f90:38-52);
    // the input's duplicate plane is read as the periodic image of plane 2.
    // Skipped (dup = 0) where the boundary conditions are applied next.
    const int kd = d.Nz + 2;
    Uo[idxU(d, i, j, kd)] = __ldg(Ui + iu) - (px - p0) * m.rdxg[i];
    if (j <= d.Ny) Vo[idxV(d, i, j, kd)] = __ldg(Vi + idxV(d, i, j, k)) - (py - p0) * m.rdyg[j];
  }
  if (Pint) {
    Pint[idxR(d, i, j, k)] = p0 * rdt;
    if (i == 2) Pint[idxR(d, d.Nx + 2, j, k)] = p0 * rdt;
    if (k == 2) {
      Pint[idxR(d, i, j, d.Nz + 2)] = p0 * rdt;
      if (i == 2) Pint[idxR(d, d.Nx + 2, j, d.Nz + 2)] = p0 * rdt;
    }
  }
}

// The same update for two cells (k, k+1) per thread, without the duplicate
// plane and P_interim (the time step's case): both cells' loads are issued
// before any store, and phi(k+1) serves both.  With ghosts = 1 every ghost
// entry of the results is written as well (the boundary conditions of the
// projected field): the x images by the threads of the boundary columns,
// the z and y images (whole blocks and warps) out of line.
__global__ void __launch_bounds__(256, 4) k_grad_sub2(Dims d, Metric m, const double* __restrict__ Ui,
                                                   const double* __restrict__ Vi,
                                                   const double* __restrict__ Wi,
                                                   const double* __restrict__ phi,
                                                   double* __restrict__ Uo, double* __restrict__ Vo,
                                                   double* __restrict__ Wo, int ghosts,
                                                   const double* __restrict__ ushift) {
  const int i = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = 2 + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = 2 + 2 * (int)blockIdx.z;
  if (i > d.Nx + 1 || j > d.Ny + 1) return;
  const bool two = k + 1 <= d.Nz + 1;
  const bool hv = j <= d.Ny;
  const int64_t pr = idxR(d, i, j, k), plr = (int64_t)(d.nxg - 2) * (d.nyg - 2);
  const int64_t iu = idxU(d, i, j, k), iv = idxV(d, i, j, k), iw = idxW(d, i, j, k);
  const int64_t plu = (int64_t)d.nx * d.nyg, plv = (int64_t)d.nxg * d.ny, plw = (int64_t)d.nxg * d.nyg;
  const double p0 = __ldg(phi + pr), px = __ldg(phi + pr + 1), p1 = __ldg(phi + pr + plr);
  const double u0 = __ldg(Ui + iu), w0 = __ldg(Wi + iw);
  double py = 0.0, v0 = 0.0, p1x = 0.0, p2 = 0.0, u1 = 0.0, w1 = 0.0, p1y = 0.0, v1 = 0.0;
  if (hv) {
    py = __ldg(phi + pr + (d.nxg - 2));
    v0 = __ldg(Vi + iv);
  }
  if (two) {
    p1x = __ldg(phi + pr + plr + 1);
    p2 = __ldg(phi + pr + 2 * plr);
    u1 = __ldg(Ui + iu + plu);
    w1 = __ldg(Wi + iw + plw);
    if (hv) {
      p1y = __ldg(phi + pr + plr + (d.nxg - 2));
      v1 = __ldg(Vi + iv + plv);
    }
  }
  const double rx = m.rdxg[i], ry = m.rdyg[j];
  double un0 = u0 - (px - p0) * rx;
  const double wn0 = w0 - (p1 - p0) * m.rdzg[k], vn0 = v0 - (py - p0) * ry;
  double un1 = u1 - (p1x - p1) * rx;
  const double wn1 = w1 - (p2 - p1) * m.rdzg[k + 1], vn1 = v1 - (p1y - p1) * ry;
  if (ushift) {
    // constant-mass-flow correction of u after the projection
    // (src/time_integration.f90:187-193), ghosts included
    const double sh = *ushift;
    un0 += sh;
    un1 += sh;
  }
  if (!ghosts) {
    Uo[iu] = un0;
    Wo[iw] = wn0;
    if (hv) Vo[iv] = vn0;
    if (two) {
      Uo[iu + plu] = un1;
      Wo[iw + plw] = wn1;
      if (hv) Vo[iv + plv] = vn1;
    }
    return;
  }
  // cells k (c = 0) and k+1 (c = 1)
  const bool yu = j == 2 || j == d.nyg - 1;                 // u, w: odd y reflections
  const bool yv = j == 2 || j == d.Ny;                      // v: next to a zero wall
  const XImages xu = x_images(i, d.Nx, d.nx), xw = x_images(i, d.Nx, d.nxg);
  for (int c = 0; c <= (two ? 1 : 0); ++c) {
    const int kc = k + c;
    const double un = c ? un1 : un0, wn = c ? wn1 : wn0, vn = c ? vn1 : vn0;
    const int64_t ou = iu + c * plu, ow = iw + c * plw, ov = iv + c * plv;
    if (yu || kc == d.Nz + 1 || kc + d.Nz <= d.nzg) put_images_all(Uo, d.nx, d.nyg, d.nzg, d.Nx, d.Nz, false, i, j, kc, un);
    else put_row(Uo + ou - (i - 1), i, xu, un);
    if (yu || kc == d.Nz + 1 || kc + d.Nz <= d.nz) put_images_all(Wo, d.nxg, d.nyg, d.nz, d.Nx, d.Nz, false, i, j, kc, wn);
    else put_row(Wo + ow - (i - 1), i, xw, wn);
    if (hv) {
      if (yv || kc == d.Nz + 1 || kc + d.Nz <= d.nzg) {
        put_images_all(Vo, d.nxg, d.ny, d.nzg, d.Nx, d.Nz, true, i, j, kc, vn);
        if (j == 2) put_images_all(Vo, d.nxg, d.ny, d.nzg, d.Nx, d.Nz, true, i, 1, kc, 0.0);
        if (j == d.Ny) put_images_all(Vo, d.nxg, d.ny, d.nzg, d.Nx, d.Nz, true, i, d.ny, kc, 0.0);
      } else {
        put_row(Vo + ov - (i - 1), i, xw, vn);
      }
    }
  }
}

int launch_gradient_subtract(Handle* h, const double* Ui, const double* Vi, const double* Wi,
                             const double* phi, double dt, double* Uo, double* Vo, double* Wo,
                             bool dup_plane, bool with_ghosts, const double* ushift) {
  const Dims& d = h->d;
  dim3 b(32, 4, 2);
  dim3 g((d.Nx + 31) / 32, (d.Ny + 3) / 4, (d.Nz + 1) / 2);
  double* Pint = (h->ib != nullptr || h->write_pinterim) ? h->P_interim : nullptr;
  if (!dup_plane && !Pint) {
    const dim3 b2(32, 8, 1), g2((d.Nx + 31) / 32, (d.Ny + 7) / 8, (d.Nz + 1) / 2);
    k_grad_sub2<<<g2, b2, 0, h->stream>>>(d, h->m, Ui, Vi, Wi, phi, Uo, Vo, Wo, with_ghosts ? 1 : 0, ushift);
    C3D_LAUNCH_CHECK(h);
    return 0;
  }
  if (ushift) {
    h->last_error = "mass-flow correction inside the projection needs the time step's update kernel";
    return C3D_ERR_UNSUPPORTED;
  }
  k_grad_sub<<<g, b, 0, h->stream>>>(d, h->m, Ui, Vi, Wi, phi, Uo, Vo, Wo, Pint, 1.0 / dt, dup_plane ? 1 : 0);
  C3D_LAUNCH_CHECK(h);
  return with_ghosts ? launch_fill_ghosts3(h, Uo, Vo, Wo) : 0;
}

// The potential of div(star) for one stage (rk_step 1..3), star an interior
// field whose ghosts are taken as the boundary conditions define them; *phi is
// where it lies.  The stage-1 potential, kept for the pressure
// (src/poisson.f90:91-99), goes into its own array.  Mixed: an FP32 solve, then
// refinement sweeps that solve for the FP64 residual div(star - grad phi) and
// add to phi.  flux: the first forward x FFT also yields the constant-x-mass-
// flow shift (the bulk flux of d(phi)/dx over the periodic uniform x grid is
// zero, so the flux of the projected u is that of star).
int launch_stage_solve(Handle* h, double* const star[3], int rk_step, double dt, bool flux, double** phi) {
  const bool stage1 = rk_step == 1 && h->ib == nullptr;
  double* p = stage1 ? h->phi1 : h->rhs_p;
  int rc;
  if (h->poisson_mode == C3D_POISSON_MIXED) {
    rc = run_spectral_t<float>(h, true, star[0], star[1], star[2], nullptr, p, nullptr, 0, 7, 0, -1, flux ? dt : 0.0);
    for (int sw = 1; sw <= h->refine_sweeps && !rc; ++sw)
      rc = run_spectral_t<float>(h, true, star[0], star[1], star[2], p, p, nullptr, 1, 7);
    h->stats.refinement_sweeps = h->refine_sweeps;
  } else {
    rc = run_spectral_t<double>(h, true, star[0], star[1], star[2], nullptr, p, nullptr, 0, 7, 0, -1, flux ? dt : 0.0);
  }
  if (rc) return rc;
  if (stage1) { h->P_pending = true; h->P_pending_dt = dt; }
  *phi = p;
  return 0;
}

// compute_non_IB_projection with U* in (Us,Vs,Ws) and the result in (U,V,W),
// all ghost entries included
int launch_projection_step(Handle* h, int rk_step, double dt) {
  double* const star[3] = {h->Us, h->Vs, h->Ws};
  double* phi = nullptr;
  const int rc = launch_stage_solve(h, star, rk_step, dt, false, &phi);
  if (rc) return rc;
  return launch_gradient_subtract(h, h->Us, h->Vs, h->Ws, phi, dt, h->U, h->V, h->W, false, true);
}

// P = phi1/(dt*rk_coef(1,1)) with the copies of src/poisson.f90:92-98
__global__ void k_build_P(Dims d, const double* __restrict__ phi, double* __restrict__ P, double den) {
  const int64_t tot = (int64_t)d.nxg * d.nyg * d.nzg;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    int i = 1 + (int)(t % d.nxg);
    int j = 1 + (int)((t / d.nxg) % d.nyg);
    int k = 1 + (int)(t / ((int64_t)d.nxg * d.nyg));
    // P(1,:,:)=P(2,:,:), P(nxg,:,:)=P(nxg-1,:,:), same in y and z
    if (i == 1) i = 2;
    if (i == d.nxg) i = d.nxg - 1;
    if (j == 1) j = 2;
    if (j == d.nyg) j = d.nyg - 1;
    if (k == 1) k = 2;
    if (k == d.nzg) k = d.nzg - 1;
    P[t] = phi[idxR(d, i, j, k)] / den;
  }
}

int rebuild_pressure(Handle* h) {
  if (!h->P_pending) return 0;
  const double den = h->P_pending_dt * (8.0 / 15.0);
  k_build_P<<<148 * 8, 256, 0, h->stream>>>(h->d, h->phi1, h->P, den);
  C3D_LAUNCH_CHECK(h);
  h->P_pending = false;
  return 0;
}

int poisson_setup(Handle* h) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  FftPasses P;
  if (!make_passes(d.Nx, P) || !make_passes(d.Nz, P)) {
    h->last_error = "nxp and nzp must be products of 2 and 3 (nx_global-2, nz_global-2)";
    return C3D_ERR_PARAM;
  }
  if (d.Nx % 2) {
    h->last_error = "nx_global must be even";
    return C3D_ERR_PARAM;
  }
  if (d.Nx > kMaxNx) {
    h->last_error = "nx_global too large for the x FFT kernels (nx_global - 2 <= 512)";
    return C3D_ERR_UNSUPPORTED;
  }
  int rc;
  if (S.spec == nullptr) {
    S.pz64 = d.Nz;
    if ((rc = cluster_setup<double>(h))) return rc;
    if ((rc = make_twiddles(h, d.Nx, &S.twx))) return rc;
    if ((rc = make_twiddles(h, d.Nz, &S.twz))) return rc;
    if ((rc = xfft_setup<double>(h))) return rc;
    const int64_t ns = (int64_t)d.Ny * S.pz64 * d.nkx;
    if ((rc = dev_alloc(h, &S.spec, ns))) return rc;
    const int64_t nbx = xfft_blocks(d);
    if ((rc = dev_alloc(h, &h->flux_part, nbx))) return rc;
    h->flux_part_len = nbx;
  }
  if ((rc = build_tri_table(h))) return rc;
  if (S.mixed_ready && slab_by_blocks(d, S.cluster32) && (rc = slab_setup(h, true))) return rc;
  return slab_by_blocks(d, S.cluster) ? slab_setup(h, false) : 0;
}

int mixed_setup(Handle* h) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  if (S.mixed_ready) return 0;
  S.pz32 = d.Nz + (d.Nz & 1);
  int rc;
  if ((rc = cluster_setup<float>(h))) return rc;
  if ((rc = make_twiddles(h, d.Nx, &S.twx32))) return rc;
  if ((rc = make_twiddles(h, d.Nz, &S.twz32))) return rc;
  const int64_t ns = (int64_t)d.Ny * S.pz32 * d.nkx;
  if ((rc = dev_alloc(h, &S.spec32, ns))) return rc;
  if ((rc = dev_alloc(h, &S.linesum, (int64_t)d.Ny * d.Nz))) return rc;
  if ((rc = dev_alloc(h, &S.phi00, d.Ny))) return rc;
  if ((rc = xfft_setup<float>(h))) return rc;
  if ((rc = build_tri_table(h))) return rc;       // with the FP32 pivots
  if (slab_by_blocks(d, S.cluster32) && (rc = slab_setup(h, true))) return rc;
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  S.mixed_ready = true;
  return 0;
}

}  // namespace c3d
