// The x transforms of the Poisson solve (src/poisson.f90:43-47, 78-88) with
// what stands before and after them: the divergence of the stage field (and
// of the refinement's residual field, and the x bulk flux), and the periodic
// copies of the potential.
//
// Two real x lines form one complex line; a CTA
// takes kLines complex lines.  The last stage of the forward transform keeps
// the two butterflies that hold wavenumbers m and Nx - m in one thread, which
// splits them into the two real lines' coefficients and writes these; the
// inverse starts the same way and its last stage writes the potential: neither
// the split nor the result goes through shared memory again.
#include <vector>

#include "c3d_internal.cuh"
#include "fft.cuh"
#include "fft_tables.h"

namespace c3d {

namespace {

constexpr int kLines = 8;        // complex lines per CTA
// threads per CTA: the forward kernel waits on memory and takes its fields
// through L1, which many CTAs' rows leave little of (four CTAs of 192 threads
// at 384 x 256 x 384: 400 us, two of 384: 289; 43 either way at 192 x 128 x
// 192); the inverse is bound by its stages (288 columns: 86 us with 192
// threads, 97 with 384) as long as several CTAs share an SM: with one or none
// its rounds follow one another, and up to 384 threads take fewer of them
// (512x16x16 12.4 -> 10.4 us, 486x20x24 14.5 -> 10.4, 384x64x24 10.4 -> 8.3)
constexpr int kFwdThreads = 384;
constexpr int kInvThreads = 192;
constexpr int kInvFewThreads = 384;
constexpr int kMaxR = 8;         // largest radix (register budget)
constexpr unsigned kRecLines = (unsigned)((1ull << 32) / kLines);   // reciprocal of kLines for div_by

// shared-memory row stride: FP64 1 mod 8, FP32 odd (conflict-free across rows)
template <typename T>
constexpr int x_stride(int Nx) {
  return sizeof(T) == 8 ? (Nx + 6) / 8 * 8 + 1 : Nx | 1;
}

// what the first stage reads
enum { FROM_RHS = 0, FROM_DIV = 1, FROM_DIV_FLUX = 2, FROM_RESIDUAL = 3 };

template <typename T>
struct XfwdArgs {
  Dims d;
  Metric m;
  const double* __restrict__ U;
  const double* __restrict__ V;
  const double* __restrict__ W;
  const double* __restrict__ rhs;             // right-hand side (FROM_RHS), potential (FROM_RESIDUAL)
  typename cplx<T>::t* __restrict__ spec;
  const typename cplx<T>::t* __restrict__ tw;
  double* __restrict__ linesum;               // FP64 line sums (mixed path) or null
  const int* __restrict__ pos;                // digit-reversed position of coefficient m
  FftPasses P;
  int pz;                                     // spectrum row pitch
  int rs;                                     // shared-memory row stride
  int rbase, nlines;                          // lines rbase .. rbase+nlines-1 (a band of j rows)
  unsigned recN;                              // ceil(2^32 / Nx)
  // FROM_DIV_FLUX: per-block partials, the last block writes the
  // constant-mass-flow correction to scw
  double* flux_part;
  DevScalars* scw;
  double q0, norm, dt;
};

// per real line of the CTA: element offsets of its x = 2 cell (-1: no line;
// for v: the zero wall value) and factors
struct LineInfo {
  int u, v, vm, w, wm;     // u(j,k) or the right-hand side, v(j,k), v(j-1,k), w(j,k), w(j,k-1)
  int off;                 // place in a spectrum slab
  int p, pym, pzm;         // phi(j,k), phi(j-1,k), phi(j,k-1)
  double ry, rz, cq;       // 1/dy, 1/dz, bulk-flux weight
  double gy, gym, gz, gzm; // 1/dyg, 1/dzg of the gradient at v(j), v(j-1), w(k), w(k-1); 0 on the walls
};

// real x-line r = (k-2) + Nz*(j-2); its spectrum goes to slab offset (j-2)*pz + (k-2)
template <int SRC>
__device__ __forceinline__ void line_info(const Dims& d, const Metric& m, int pz, int r, int rend, LineInfo& L) {
  L.u = -1;
  L.cq = 0.0;
  if (r >= rend) return;
  const int jj = r / d.Nz, kk = r - jj * d.Nz, j = 2 + jj, k = 2 + kk;
  L.off = jj * pz + kk;
  if (SRC == FROM_RHS) {
    L.u = (int)idxR(d, 2, j, k);
    return;
  }
  // the ghost values are read as the boundary conditions define them (periodic
  // images in x and z, zero V walls), so the fields need no ghost fill
  const int km = k == 2 ? d.Nz + 1 : k - 1;
  L.u = (int)idxU(d, 2, j, k);
  L.v = j == d.ny ? -1 : (int)idxV(d, 2, j, k);
  L.vm = j == 2 ? -1 : (int)idxV(d, 2, j - 1, k);
  L.w = (int)idxW(d, 2, j, k);
  L.wm = (int)idxW(d, 2, j, km);
  L.ry = m.rdy[j];
  L.rz = m.rdz[k];
  if (SRC == FROM_DIV_FLUX) L.cq = m.cqu[j] * (k == 2 ? 2.0 : 1.0);
  if (SRC == FROM_RESIDUAL) {
    L.p = (int)idxR(d, 2, j, k);
    L.pym = j == 2 ? L.p : (int)idxR(d, 2, j - 1, k);
    L.pzm = (int)idxR(d, 2, j, km);
    L.gy = j == d.ny ? 0.0 : m.rdyg[j];
    L.gym = j == 2 ? 0.0 : m.rdyg[j - 1];
    L.gz = m.rdzg[k];
    L.gzm = m.rdzg[km];
  }
}

// the loads behind the value that enters the transform at x index i (0-based)
// of a line, and that value
template <int SRC>
struct LineLoads {
  double x1, x0, y1, y0, z1, z0;
};
template <int SRC, typename T>
__device__ __forceinline__ LineLoads<SRC> line_load(const XfwdArgs<T>& a, const LineInfo& L, int N, int i) {
  LineLoads<SRC> v;
  v.x1 = v.x0 = v.y1 = v.y0 = v.z1 = v.z0 = 0.0;
  if (L.u < 0) return v;
  if (SRC == FROM_RHS) {
    v.x1 = a.rhs[L.u + i];
    return v;
  }
  const int xo = (i == 0 ? N : i) - 1;    // u(i-1) of i = 2 is u(N+1)
  v.x1 = a.U[L.u + i];
  v.x0 = a.U[L.u + xo];
  if (L.v >= 0) v.y1 = a.V[L.v + i];
  if (L.vm >= 0) v.y0 = a.V[L.vm + i];
  v.z1 = a.W[L.w + i];
  v.z0 = a.W[L.wm + i];
  if (SRC == FROM_RESIDUAL) {
    const double* ph = a.rhs + L.p;
    const double* pm = a.rhs + L.pzm;
    const int ny1 = L.gy == 0.0 ? 0 : N + 1, nz1 = (N + 1) * a.d.Ny;    // rows of phi are Nx+1 long
    const double p0 = ph[i];
    v.x1 -= (ph[i + 1] - p0) * a.m.rdxg[2 + i];
    v.x0 -= (ph[xo + 1] - ph[xo]) * a.m.rdxg[2 + xo];
    v.y1 -= (ph[ny1 + i] - p0) * L.gy;
    v.y0 -= (p0 - a.rhs[L.pym + i]) * L.gym;
    v.z1 -= (ph[nz1 + i] - p0) * L.gz;
    v.z0 -= (pm[nz1 + i] - pm[i]) * L.gzm;
  }
  return v;
}
template <int SRC>
__device__ __forceinline__ double line_value(const LineInfo& L, const LineLoads<SRC>& v, double rdx, double& flux) {
  if (SRC == FROM_RHS) return v.x1;
  if (L.u < 0) return 0.0;
  if (SRC == FROM_DIV_FLUX) flux += L.cq * v.x1;
  return (v.x1 - v.x0) * rdx + (v.y1 - v.y0) * L.ry + (v.z1 - v.z0) * L.rz;
}

// The transform's inputs into shared memory (rows [kLines][rs] of two real
// lines each).  A thread takes one x of kBatch lines at a time and issues all
// their loads before it uses any: with the first butterfly formed straight
// from the loads (8 points a thread, 96 loads in batches of 24) the kernel
// waited for memory, 49 us against 46 at 192 x 128 x 192.
// FP32: the FP64 values also to val [2*kLines][Nx], for the line sums.
template <int SRC, int NX, typename T>
__device__ __forceinline__ void xfwd_values(const XfwdArgs<T>& a, const LineInfo* L, typename cplx<T>::t* buf, int RS,
                                            double* val, double& flux) {
  constexpr int kBatch = SRC == FROM_RESIDUAL ? 2 : 4;
  const int N = NX > 0 ? NX : a.d.Nx;
  T* out = reinterpret_cast<T*>(buf);
  for (int t = threadIdx.x; t < N * (2 * kLines / kBatch); t += blockDim.x) {
    const int g = NX > 0 ? t / N : div_by(t, a.recN), i = t - g * N;
    const LineInfo* l = L + g * kBatch;
    LineLoads<SRC> v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) v[u] = line_load<SRC>(a, l[u], N, i);
    const double rdx = SRC == FROM_RHS ? 0.0 : a.m.rdx[2 + i];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const double x = line_value<SRC>(l[u], v[u], rdx, flux);
      const int rl = g * kBatch + u;
      out[2 * ((rl >> 1) * RS + i) + (rl & 1)] = (T)x;
      if (sizeof(T) == 4) val[rl * N + i] = x;
    }
  }
}

// last stage and split: the butterflies of wavenumbers k0 + s K and of their
// mirror images N - k0 - s K = (K - k0) + (R-1-s) K, K = N/R
template <int R, typename T>
__device__ __forceinline__ void xfwd_last(const XfwdArgs<T>& a, const LineInfo* L, const typename cplx<T>::t* buf,
                                          int N, int RS) {
  using C = typename cplx<T>::t;
  const int K = N / R, slab = a.d.Ny * a.pz;
  for (int t = threadIdx.x; t < kLines * (K / 2 + 1); t += blockDim.x) {
    const int l = t % kLines, k0 = t / kLines, kp = k0 == 0 ? 0 : K - k0;
    const LineInfo &La = L[2 * l], &Lb = L[2 * l + 1];
    if (La.u < 0) continue;
    const bool self = kp == k0;
    C v[R], w[R];
    const C* pv = buf + l * RS + a.pos[k0];
    const C* pw = buf + l * RS + a.pos[kp];
#pragma unroll
    for (int s = 0; s < R; ++s) { v[s] = pv[s]; w[s] = pw[s]; }
    Dft<T, false, R>::run(v);
    Dft<T, false, R>::run(w);
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int m = k0 + s * K;
      const bool up = 2 * m > N;                  // coefficient N - m is the one kept
      if (self && up) continue;
      const C Z = v[s], Zr = k0 == 0 ? v[(R - s) % R] : w[R - 1 - s];
      // A = (Z_m + conj Z_{N-m})/2, B = (Z_m - conj Z_{N-m})/(2i); conjugates at N - m
      C A, B;
      A.x = (T)0.5 * (Z.x + Zr.x);
      A.y = (T)0.5 * (Z.y - Zr.y);
      B.x = (T)0.5 * (Z.y + Zr.y);
      B.y = (T)-0.5 * (Z.x - Zr.x);
      if (up) { A.y = -A.y; B.y = -B.y; }
      C* out = a.spec + (up ? N - m : m) * slab;
      out[La.off] = A;
      if (Lb.u >= 0) out[Lb.off] = B;
    }
  }
}

// (hi, lo) += (b, c), the rounding of hi + b kept in lo
__device__ __forceinline__ void two_sum(double& hi, double& lo, double b, double c) {
  const double s = hi + b, t = s - hi;
  lo = ((hi - (s - t)) + (b - t)) + (lo + c);
  hi = s;
}

// FROM_DIV_FLUX: the bulk flux of u (src/mass_flow.f90:24-53, 144-175) is
// reduced from the u values this kernel reads (compute_time_step_RK3's
// correction, src/time_integration.f90:187-193, then needs no pass of its
// own): weights wq(j) + wq(j+1) per row and plane 2 twice (plane nzg-1 is its
// copy).
// FROM_RESIDUAL (refinement of the FP32 solve): the divergence of
// U - grad(phi), formed as the projection update forms it, so that field is
// neither written nor read back (32 bytes a cell read in place of 56 for the
// update and 24 for its divergence).
template <int SRC, typename T, int NX>
__global__ void __launch_bounds__(kFwdThreads, 2) k_xfft_fwd(XfwdArgs<T> a) {
  using C = typename cplx<T>::t;
  extern __shared__ __align__(16) unsigned char xf_smem[];
  __shared__ LineInfo L[2 * kLines];
  C* buf = reinterpret_cast<C*>(xf_smem);
  const int Nx = NX > 0 ? NX : a.d.Nx, RS = NX > 0 ? x_stride<T>(NX) : a.rs;
  C* tw = buf + (size_t)kLines * RS;
  double* val = reinterpret_cast<double*>(tw + Nx);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int r0 = a.rbase + (int)blockIdx.x * 2 * kLines, rend = a.rbase + a.nlines;
  if (tid < 2 * kLines) line_info<SRC>(a.d, a.m, a.pz, r0 + tid, rend, L[tid]);
  for (int t = tid; t < Nx; t += nt) tw[t] = a.tw[t];
  __syncthreads();
  double flux = 0.0;
  xfwd_values<SRC, NX>(a, L, buf, RS, val, flux);
  __syncthreads();
  if (sizeof(T) == 4 && a.linesum) {   // FP64 line sums: one warp per line, a fixed shuffle tree
    const int warp = tid >> 5, lane = tid & 31;
    for (int rl = warp; rl < 2 * kLines; rl += nt >> 5) {
      double sum = 0.0;
      for (int q = lane; q < Nx; q += 32) sum += val[rl * Nx + q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0 && L[rl].u >= 0) a.linesum[r0 + rl] = sum;
    }
  }
  if constexpr (NX > 0) {
    constexpr int RL = plan_last_radix(NX, kMaxR);
    fft_fixed_dif<T, NX, kMaxR, NX, RL>(buf, kLines, kRecLines, RS, tw);
    xfwd_last<RL>(a, L, buf, NX, RS);
  } else {
    fft_rows_dif<T, kMaxR, kLines>(buf, kLines, RS, tw, a.P, 0, a.P.npass - 1);
    switch (a.P.radix[a.P.npass - 1]) {
      case 8: xfwd_last<8>(a, L, buf, Nx, RS); break;
      case 6: xfwd_last<6>(a, L, buf, Nx, RS); break;
      case 4: xfwd_last<4>(a, L, buf, Nx, RS); break;
      case 3: xfwd_last<3>(a, L, buf, Nx, RS); break;
      default: xfwd_last<2>(a, L, buf, Nx, RS); break;
    }
  }
  if (SRC == FROM_DIV_FLUX) {
    // block partial by a fixed tree (any thread count up to kFwdThreads); the
    // last block adds the partials the same way as unevaluated sums hi + lo,
    // then shift = Qflow_x_0 - flux/norm, formed before it is rounded (the two
    // are nearly equal), and dPdx = (dPdx + shift/dt)/2
    __shared__ double red[kFwdThreads], rel[kFwdThreads];
    __shared__ bool last;
    auto tree = [&](double v, double e, double& lo) {
      red[tid] = v;
      rel[tid] = e;
      __syncthreads();
      for (int st = 256; st > 0; st >>= 1) {
        if (tid < st && tid + st < nt) two_sum(red[tid], rel[tid], red[tid + st], rel[tid + st]);
        __syncthreads();
      }
      const double r = red[0];
      lo = rel[0];
      __syncthreads();
      return r;
    };
    double lo;
    const double bsum = tree(flux, 0.0, lo);
    if (tid == 0) {
      a.flux_part[blockIdx.x] = bsum + lo;
      __threadfence();
      last = atomicAdd(&a.scw->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      double t = 0.0, e = 0.0;
      for (unsigned b = tid; b < gridDim.x; b += nt) two_sum(t, e, __ldcg(a.flux_part + b), 0.0);
      const double hi = tree(t, e, lo);
      if (tid == 0) {
        const double shift = (__fma_rn(a.q0, a.norm, -hi) - lo) / a.norm;
        DevScalars* sc = a.scw;
        sc->qflow = (hi + lo) / a.norm;
        sc->shift = shift;
        sc->dpdx_prev = sc->dPdx;
        sc->dPdx = 0.5 * (sc->dPdx + shift / a.dt);
        sc->ticket = 0u;
      }
    }
  }
}

template <typename T>
struct XinvArgs {
  Dims d;
  const typename cplx<T>::t* __restrict__ spec;
  const typename cplx<T>::t* __restrict__ tw;
  const typename cplx<T>::t* __restrict__ tw1;
  double* __restrict__ rhs;      // output phi (rhs_p layout)
  double* __restrict__ phi1;     // optional second copy (P side effect)
  const double* __restrict__ phi00;   // FP64 mean mode added to the output (mixed path)
  int accumulate;                // 1: rhs += result (refinement)
  const int* __restrict__ pos;
  FftPasses P;
  int pz, rs;
  int rbase, nlines;             // lines rbase .. rbase+nlines-1 (a band of j rows)
  double inv_scale;              // 1/(nxp*nzp)
};

// per real line: place in a spectrum slab, offset of the x = 2 value of
// phi(j,k) (-1: no line), and of phi(j,nzp+2) for the plane k = 2 that the
// reference duplicates (else -1)
struct OutLine {
  int off, o, o2;
  double p00;
};

template <int R, typename T>
__device__ __forceinline__ void xinv_first(const XinvArgs<T>& a, const OutLine* L, typename cplx<T>::t* buf, int N,
                                           int RS) {
  using C = typename cplx<T>::t;
  const int K = N / R, slab = a.d.Ny * a.pz;
  for (int t = threadIdx.x; t < kLines * (K / 2 + 1); t += blockDim.x) {
    const int l = t % kLines, k0 = t / kLines, kp = k0 == 0 ? 0 : K - k0;
    const OutLine &La = L[2 * l], &Lb = L[2 * l + 1];
    C A[R], B[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int m = k0 + s * K;
      const C* in = a.spec + (2 * m > N ? N - m : m) * slab;
      A[s] = B[s] = C{(T)0, (T)0};
      if (La.o >= 0) A[s] = in[La.off];
      if (Lb.o >= 0) B[s] = in[Lb.off];
    }
    // Z = A + iB on the full circle from the two half spectra
    C v[R], w[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int m = k0 + s * K;
      C As = A[s], Bs = B[s];
      if (m == 0 || 2 * m == N) { As.y = (T)0; Bs.y = (T)0; }   // Hermitian projection
      if (2 * m > N) { As.y = -As.y; Bs.y = -Bs.y; }
      v[s] = C{As.x - Bs.y, As.y + Bs.x};
      w[R - 1 - s] = C{As.x + Bs.y, Bs.x - As.y};
    }
    C* pv = buf + l * RS + a.pos[k0];
    Dft<T, true, R>::run(v);
#pragma unroll
    for (int s = 0; s < R; ++s) pv[s] = v[s];
    if (kp != k0) {
      C* pw = buf + l * RS + a.pos[kp];
      Dft<T, true, R>::run(w);
#pragma unroll
      for (int s = 0; s < R; ++s) pw[s] = w[s];
    }
  }
}

// phi at x index i of a line, with the copies of apply_periodic_xz_centers
// (src/poisson.f90:106-125): x plane nxg-1 and z plane nzp+2 duplicate plane 2
template <typename T>
__device__ __forceinline__ void put_phi(const XinvArgs<T>& a, const OutLine& L, int N, int i, double v) {
  if (L.o < 0) return;
  if (a.phi00) v += L.p00;
  if (a.accumulate) v += a.rhs[L.o + i];
  auto put = [&](double* f) {
    f[L.o + i] = v;
    if (i == 0) f[L.o + N] = v;
    if (L.o2 >= 0) {
      f[L.o2 + i] = v;
      if (i == 0) f[L.o2 + N] = v;
    }
  };
  put(a.rhs);
  if (a.phi1) put(a.phi1);
}

template <typename T, int NX>
__global__ void __launch_bounds__(kInvFewThreads, 2) k_xfft_inv(XinvArgs<T> a) {
  using C = typename cplx<T>::t;
  extern __shared__ __align__(16) unsigned char xi_smem[];
  __shared__ OutLine L[2 * kLines];
  C* buf = reinterpret_cast<C*>(xi_smem);
  const int Nx = NX > 0 ? NX : a.d.Nx, RS = NX > 0 ? x_stride<T>(NX) : a.rs;
  C* tw = buf + (size_t)kLines * RS;
  const Dims& d = a.d;
  const int tid = threadIdx.x;
  if (tid < 2 * kLines) {
    const int r = a.rbase + (int)blockIdx.x * 2 * kLines + tid;
    OutLine o{0, -1, -1, 0.0};
    if (r < a.rbase + a.nlines) {
      const int jj = r / d.Nz, kk = r - jj * d.Nz;
      o.off = jj * a.pz + kk;
      o.o = (int)idxR(d, 2, 2 + jj, 2 + kk);
      if (kk == 0) o.o2 = (int)idxR(d, 2, 2 + jj, d.Nz + 2);
      if (a.phi00) o.p00 = a.phi00[jj];
    }
    L[tid] = o;
  }
  for (int t = tid; t < Nx; t += blockDim.x) tw[t] = a.tw[t];
  __syncthreads();
  const double rsd = a.inv_scale;
  auto in = [&](int l, int e) { return buf[l * RS + e]; };
  auto out = [&](int l, int e, C v) {
    put_phi(a, L[2 * l], Nx, e, (double)v.x * rsd);
    put_phi(a, L[2 * l + 1], Nx, e, (double)v.y * rsd);
  };
  if constexpr (NX > 0) {
    constexpr int R0 = plan_radix(NX, kMaxR), RL = plan_last_radix(NX, kMaxR);
    xinv_first<RL>(a, L, buf, NX, RS);
    __syncthreads();
    fft_fixed_dit_inv<T, NX, kMaxR, NX / R0, RL>(buf, kLines, kRecLines, RS, tw);
    ct_edge<T, true, R0>(kLines, NX, a.tw1, a.P.rec[0], in, out);
  } else {
    switch (a.P.radix[a.P.npass - 1]) {
      case 8: xinv_first<8>(a, L, buf, Nx, RS); break;
      case 6: xinv_first<6>(a, L, buf, Nx, RS); break;
      case 4: xinv_first<4>(a, L, buf, Nx, RS); break;
      case 3: xinv_first<3>(a, L, buf, Nx, RS); break;
      default: xinv_first<2>(a, L, buf, Nx, RS); break;
    }
    __syncthreads();
    fft_rows_dit_inv<T, kMaxR, kLines>(buf, kLines, RS, tw, a.P, 1, a.P.npass - 1);
    ct_edge_any<T, true>(kLines, a.tw1, a.P, in, out);
  }
}

// at least two stages (a first and a last)
FftPasses x_plan(int Nx) {
  FftPasses P{};
  if (Nx <= kMaxR) {
    P.n = Nx;
    P.npass = 2;
    P.radix[0] = Nx / 2;
    P.radix[1] = 2;
    set_strides(P);
  } else {
    make_fft_passes(Nx, P, kMaxR);
  }
  return P;
}

// a butterfly of the whole span per thread, in equal rounds of at most most threads
int x_threads(const FftPasses& P, int most) {
  const int items = kLines * P.n / P.radix[0], rounds = (items + most - 1) / most;
  const int nt = ((items + rounds - 1) / rounds + 31) / 32 * 32;
  return nt < 64 ? 64 : nt;
}

template <typename T>
size_t x_smem(const FftPasses& P, bool fwd) {
  return sizeof(typename cplx<T>::t) * ((size_t)kLines * x_stride<T>(P.n) + P.n) +
         (fwd && sizeof(T) == 4 ? sizeof(double) * 2 * kLines * P.n : 0);
}

// The kernels for lines of Nx points: lines of 32 to 512 points, but 36 and 54,
// have the length compiled in (FP64: inverse at 384 x 256 x 384 188 -> 170 us, forward 288 ->
// 281; time step 4969 -> 4874 us there, 661 -> 653 at 192 x 128 x 192, 368 ->
// 358 at 162 x 113 x 108, 83 -> 82 at 32 x 64 x 32; FP32 mixed steps 1117 -> 1064
// us at 192 x 128 x 192, 7771 -> 7535 at 384 x 256 x 384).  Right-hand
// sides from memory (the Poisson solve called by itself) take the run-time
// stages.
template <typename T>
struct XKernels {
  void (*div)(XfwdArgs<T>);
  void (*flux)(XfwdArgs<T>);
  void (*residual)(XfwdArgs<T>);     // FP32
  void (*inv)(XinvArgs<T>);
};
template <typename T, int NX>
XKernels<T> x_set() {
  XKernels<T> k{k_xfft_fwd<FROM_DIV, T, NX>, k_xfft_fwd<FROM_DIV_FLUX, T, NX>, nullptr, k_xfft_inv<T, NX>};
  if constexpr (sizeof(T) == 4) k.residual = k_xfft_fwd<FROM_RESIDUAL, T, NX>;
  return k;
}
template <typename T, int... NX>
XKernels<T> x_pick(int Nx) {
  XKernels<T> k = x_set<T, 0>();
  ((Nx == NX ? (void)(k = x_set<T, NX>()) : (void)0), ...);
  return k;
}
template <typename T>
XKernels<T> x_kernels(int Nx) {
  return x_pick<T, 32, 48, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512>(Nx);
}

template <typename T>
struct XTables {
  const typename cplx<T>::t *tw, *tw1;
  typename cplx<T>::t* spec;
  int pz;
};
template <typename T>
XTables<T> x_tables(const SpectralState& S) {
  if constexpr (sizeof(T) == 8) return {S.twx, S.tw1x, S.spec, S.pz64};
  else return {S.twx32, S.tw1x32, S.spec32, S.pz32};
}

}  // namespace

int64_t xfft_blocks(const Dims& d) { return ((int64_t)d.Ny * d.Nz + 2 * kLines - 1) / (2 * kLines); }

// forward transform of rows blo..bhi (0-based j-2) of the divergence of (U, V,
// W) (from_div), of div((U, V, W) - grad rhs) (from_div with rhs) or of rhs;
// flux_dt > 0: with the constant-x-mass-flow correction
template <typename T>
int launch_xfft_fwd(Handle* h, bool from_div, const double* U, const double* V, const double* W, const double* rhs,
                    double* linesum, int blo, int bhi, double flux_dt) {
  const Dims& d = h->d;
  const XTables<T> t = x_tables<T>(h->sp);
  XfwdArgs<T> a{};
  a.d = d; a.m = h->m; a.U = U; a.V = V; a.W = W; a.rhs = rhs;
  a.spec = t.spec; a.tw = t.tw; a.linesum = linesum; a.pos = h->sp.posx;
  a.P = x_plan(d.Nx); a.pz = t.pz; a.rs = x_stride<T>(d.Nx);
  a.recN = (unsigned)(((1ull << 32) + d.Nx - 1) / d.Nx);
  a.rbase = blo * d.Nz; a.nlines = (bhi - blo + 1) * d.Nz;
  const unsigned nb = (unsigned)((a.nlines + 2 * kLines - 1) / (2 * kLines));
  const int nt = x_threads(a.P, kFwdThreads);
  const size_t smem = x_smem<T>(a.P, true);
  if (flux_dt > 0.0) {
    if (h->flux_part_len < (int64_t)nb) {
      h->last_error = "x bulk-flux partials not allocated";
      return C3D_ERR_CUDA;
    }
    a.flux_part = h->flux_part; a.scw = h->sc;
    a.q0 = h->Qflow_x_0; a.norm = h->norm_u; a.dt = flux_dt;
    x_kernels<T>(d.Nx).flux<<<nb, nt, smem, h->stream>>>(a);
  } else if (from_div && rhs) {
    if constexpr (sizeof(T) == 4) x_kernels<T>(d.Nx).residual<<<nb, nt, smem, h->stream>>>(a);
  } else if (from_div) {
    x_kernels<T>(d.Nx).div<<<nb, nt, smem, h->stream>>>(a);
  } else {
    k_xfft_fwd<FROM_RHS, T, 0><<<nb, nt, smem, h->stream>>>(a);
  }
  C3D_LAUNCH_CHECK(h);
  return 0;
}
template int launch_xfft_fwd<double>(Handle*, bool, const double*, const double*, const double*, const double*,
                                     double*, int, int, double);
template int launch_xfft_fwd<float>(Handle*, bool, const double*, const double*, const double*, const double*,
                                    double*, int, int, double);

// inverse transform of rows blo..bhi into out (rhs_p layout) and phi1 if given
template <typename T>
int launch_xfft_inv(Handle* h, double* out, double* phi1, const double* phi00, int accumulate, int blo, int bhi) {
  const Dims& d = h->d;
  const XTables<T> t = x_tables<T>(h->sp);
  XinvArgs<T> a{};
  a.d = d; a.spec = t.spec; a.tw = t.tw; a.tw1 = t.tw1; a.rhs = out; a.phi1 = phi1; a.phi00 = phi00;
  a.accumulate = accumulate; a.pos = h->sp.posx;
  a.P = x_plan(d.Nx); a.pz = t.pz; a.rs = x_stride<T>(d.Nx);
  a.rbase = blo * d.Nz; a.nlines = (bhi - blo + 1) * d.Nz;
  a.inv_scale = 1.0 / ((double)d.Nx * (double)d.Nz);
  const unsigned nb = (unsigned)((a.nlines + 2 * kLines - 1) / (2 * kLines));
  x_kernels<T>(d.Nx).inv<<<nb, x_threads(a.P, nb <= 148 ? kInvFewThreads : kInvThreads), x_smem<T>(a.P, false), h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  return 0;
}
template int launch_xfft_inv<double>(Handle*, double*, double*, const double*, int, int, int);
template int launch_xfft_inv<float>(Handle*, double*, double*, const double*, int, int, int);

// first-stage twiddles and (FP64 set-up, done first) the digit-reversed
// positions; the kernels' dynamic shared-memory limits are process-wide, so
// they are set to what the longest rows need
template <typename T>
int xfft_setup(Handle* h) {
  using C = typename cplx<T>::t;
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  const FftPasses P = x_plan(d.Nx);
  int rc;
  const std::vector<C> tw1 = edge_twiddles<C>(d.Nx, P.radix[0]);
  C* dst = nullptr;
  if ((rc = dev_alloc(h, &dst, d.Nx))) return rc;
  C3D_CUDA_TRY(h, cudaMemcpyAsync(dst, tw1.data(), sizeof(C) * d.Nx, cudaMemcpyHostToDevice, h->stream));
  std::vector<int> pos(d.Nx);
  if constexpr (sizeof(T) == 8) {
    S.tw1x = dst;
    for (int m = 0; m < d.Nx; ++m) pos[m] = dif_k_to_position(m, P);
    if ((rc = dev_alloc(h, &S.posx, d.Nx))) return rc;
    C3D_CUDA_TRY(h, cudaMemcpyAsync(S.posx, pos.data(), sizeof(int) * d.Nx, cudaMemcpyHostToDevice, h->stream));
  } else {
    S.tw1x32 = dst;
  }
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));     // the host copies end here
  FftPasses longest = x_plan(512);
  const int smem = (int)x_smem<T>(longest, true);
  auto limit = [&](auto* k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); };
  C3D_CUDA_TRY(h, limit(k_xfft_fwd<FROM_RHS, T, 0>));
  const XKernels<T> k = x_kernels<T>(d.Nx);
  C3D_CUDA_TRY(h, limit(k.div));
  C3D_CUDA_TRY(h, limit(k.flux));
  if constexpr (sizeof(T) == 4) C3D_CUDA_TRY(h, limit(k.residual));
  C3D_CUDA_TRY(h, limit(k.inv));
  return 0;
}
template int xfft_setup<double>(Handle*);
template int xfft_setup<float>(Handle*);

}  // namespace c3d
