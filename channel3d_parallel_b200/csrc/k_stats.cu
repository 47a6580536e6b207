// On-device diagnostics: compute_statistics (src/statistics.f90:22-148) and
// the reductions of output_monitor (src/monitor.f90:21-110), one domain.
//
// Statistics: with term_1 = interpolate_x(U) = (U(i-1)+U(i))/2 and term_2 =
// interpolate_y(V) = (V(j-1)+V(j))/2 (rows 1 and nyg the negatives of rows 2
// and nyg-1), per y row jj = 1..nyg the sums over i = 2..nxg-2 and
// k = 2..nzg-2 (W: k = 2..nz-1) of term_1, term_2, W, their squares and
// term_1*term_2, divided by (nxg-3)(nzg-3) (W: (nxg-3)(nz-2)); the wall
// derivatives of the mean profiles give utau, wtau and Retau.  Row sums are
// per (row, z chunk) block partials added in chunk order (deterministic).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "c3d_internal.cuh"

namespace c3d {

namespace {
constexpr int kStatQ = 7;        // Umean, Vmean, Wmean, U2mean, V2mean, W2mean, UVmean
constexpr int kStatChunks = 12;  // z chunks per y row
constexpr int kStatThreads = 256;
constexpr int kBoxBlocks = 148 * 4;
}  // namespace

__global__ void __launch_bounds__(kStatThreads) k_stat_rows(Dims d, const double* __restrict__ U,
                                                           const double* __restrict__ V,
                                                           const double* __restrict__ W,
                                                           double* __restrict__ part) {
  const int j = 1 + blockIdx.x;
  const int c = blockIdx.y;
  const int ni = d.nxg - 3, nk = d.nzg - 3;
  const int k0 = 2 + (int)((int64_t)c * nk / gridDim.y), k1 = 2 + (int)((int64_t)(c + 1) * nk / gridDim.y);
  double s[kStatQ] = {0, 0, 0, 0, 0, 0, 0};
  // one warp per x row of the chunk; rows of V either side of the row (the
  // walls' own for the ghost rows, with the opposite sign)
  const int ja = j == 1 ? 1 : (j == d.nyg ? d.nyg - 2 : j - 1);
  const double sg = j == 1 || j == d.nyg ? -0.5 : 0.5;
  for (int k = k0 + (int)(threadIdx.x >> 5); k < k1; k += kStatThreads / 32) {
    const double* u = U + idxU(d, 2, j, k);
    const double* va = V + idxV(d, 2, ja, k);
    const double* wr = W + idxW(d, 2, j, k);
#pragma unroll 2
    for (int i = threadIdx.x & 31; i < ni; i += 32) {
      const double t1 = 0.5 * (u[i - 1] + u[i]), t2 = sg * (va[i] + va[i + d.nxg]), w = wr[i];
      s[0] += t1; s[1] += t2; s[2] += w;
      s[3] += t1 * t1; s[4] += t2 * t2; s[5] += w * w;
      s[6] += t1 * t2;
    }
  }
  __shared__ double red[kStatQ][kStatThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kStatQ; ++q) {
    double v = s[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[q][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < kStatQ) {
    double v = 0.0;
    for (int w_ = 0; w_ < kStatThreads / 32; ++w_) v += red[threadIdx.x][w_];
    part[((int64_t)(j - 1) * gridDim.y + c) * kStatQ + threadIdx.x] = v;
  }
}

// out[q*nyg + jj-1] = (sum over chunks in order) / count
__global__ void k_stat_final(int nyg, int nch, double cnt_uv, double cnt_w, const double* __restrict__ part,
                             double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nyg * kStatQ) return;
  const int q = t / nyg, j = t - q * nyg;
  double v = 0.0;
  for (int c = 0; c < nch; ++c) v += part[((int64_t)j * nch + c) * kStatQ + q];
  out[t] = v / ((q == 2 || q == 5) ? cnt_w : cnt_uv);
}

// Sums and maxima of U, V, W over the interior boxes of output_monitor
// (blockIdx.y: component), one warp per x row; per block (sum, max)
__global__ void __launch_bounds__(256) k_box_sum_max(Dims d, const double* __restrict__ U,
                                                    const double* __restrict__ V, const double* __restrict__ W,
                                                    double2* __restrict__ part) {
  const int c = blockIdx.y, lane = threadIdx.x & 31;
  const double* F = c == 0 ? U : (c == 1 ? V : W);
  const int n1 = c == 0 ? d.nx : d.nxg, n2 = c == 1 ? d.ny : d.nyg, n3 = c == 2 ? d.nz : d.nzg;
  const int nrows = (n2 - 2) * (n3 - 2);
  double s = 0.0, mx = -INFINITY;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < nrows; row += gridDim.x * 8) {
    const int k = row / (n2 - 2), j = row - k * (n2 - 2);
    const double* f = F + 1 + (int64_t)n1 * (j + 1 + (int64_t)n2 * (k + 1));
#pragma unroll 4
    for (int i = lane; i < n1 - 2; i += 32) {
      const double v = f[i];
      s += v;
      mx = fmax(mx, v);
    }
  }
  __shared__ double ss[8], sm[8];
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  const int wid = threadIdx.x >> 5;
  if (lane == 0) { ss[wid] = s; sm[wid] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = -INFINITY;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { a += ss[w]; b = fmax(b, sm[w]); }
    part[blockIdx.y * gridDim.x + blockIdx.x] = make_double2(a, b);
  }
}


// compute_statistics: profiles[7*nyg] (Umean, Vmean, Wmean, U2mean, V2mean,
// W2mean, UVmean at yg(1:nyg)); scalars[8] = utau, wtau, Retau_u, Retau_w,
// Qflow_x, Qflow_y, Qflow_z, and 1 if U, V or W holds a NaN or infinity
// (the reference stops there, src/statistics.f90:142-144)
int compute_statistics(Handle* h, double* profiles, double* scalars) {
  const Dims& d = h->d;
  const int nyg = d.nyg;
  // device results: the profiles, then the three flows and the finiteness
  // flag; one copy and one synchronisation bring them all
  int rc;
  const int64_t nout = (int64_t)nyg * kStatQ + 4;
  const int64_t need = (int64_t)nyg * kStatChunks * kStatQ + nout;
  if (h->stat_cap < need) {
    if ((rc = dev_alloc(h, &h->stat_buf, need))) return rc;
    h->stat_cap = need;
  }
  double* part = h->stat_buf;
  double* out = h->stat_buf + (int64_t)nyg * kStatChunks * kStatQ;
  k_stat_rows<<<dim3((unsigned)nyg, kStatChunks), kStatThreads, 0, h->stream>>>(d, h->U, h->V, h->W, part);
  C3D_LAUNCH_CHECK(h);
  const double cnt = (double)(d.nxg - 3) * (double)(d.nzg - 3), cntw = (double)(d.nxg - 3) * (double)(d.nz - 2);
  k_stat_final<<<(nyg * kStatQ + 127) / 128, 128, 0, h->stream>>>(nyg, kStatChunks, cnt, cntw, part, out);
  C3D_LAUNCH_CHECK(h);
  double* flows = out + (int64_t)nyg * kStatQ;
  if ((rc = launch_statistics_flows(h, flows))) return rc;
  if ((rc = launch_finite(h, (int*)(flows + 3)))) return rc;
  std::vector<double> res(nout);
  C3D_CUDA_TRY(h, cudaMemcpyAsync(res.data(), out, sizeof(double) * nout, cudaMemcpyDeviceToHost, h->stream));
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  std::memcpy(profiles, res.data(), sizeof(double) * nyg * kStatQ);
  const double* Um = profiles;
  const double* Wm = profiles + 2 * nyg;
  const std::vector<double>& yg = h->yg;
  const std::vector<double>& y = h->y;
  const double nu = h->p.nu;
  // src/statistics.f90:109-127 (the wall Reynolds stresses are zero)
  const double dUb = (Um[1] - Um[0]) / (yg[2] - yg[1]);
  const double dUt = (Um[nyg - 1] - Um[nyg - 2]) / (yg[nyg] - yg[nyg - 1]);
  const double dWb = (Wm[1] - Wm[0]) / (yg[2] - yg[1]);
  const double dWt = (Wm[nyg - 1] - Wm[nyg - 2]) / (yg[nyg] - yg[nyg - 1]);
  const double utau = std::pow((0.0 - 0.0 - nu * dUt + nu * dUb) / h->Ly, 0.5);
  const double wtau = std::pow((0.0 - 0.0 - nu * dWt + nu * dWb) / h->Ly, 0.5);
  scalars[0] = utau;
  scalars[1] = wtau;
  scalars[2] = utau * (y[d.ny] - y[1]) / 2.0 / nu;
  scalars[3] = wtau * (y[d.ny] - y[1]) / 2.0 / nu;
  int bad = 0;
  std::memcpy(&bad, &res[(size_t)nyg * kStatQ + 3], sizeof(bad));
  for (int c = 0; c < 3; ++c) scalars[4 + c] = res[(size_t)nyg * kStatQ + c];
  scalars[7] = bad ? 1.0 : 0.0;
  return 0;
}

// output_monitor (src/monitor.f90:21-50): out[0..2] mean U, V, W over the
// interior divided by nxm*nym*nzm (as printed, :78-80), out[3..5] their
// maxima, out[6] the maximum |div u| (check_divergence, :210-221)
int monitor_values(Handle* h, double* out) {
  const Dims& d = h->d;
  int rc;
  const double vol = (double)(d.nx - 1) * (double)(d.ny - 1) * (double)(d.nz - 1);
  // partials of the three components, then those of the divergence, in one copy
  constexpr int64_t nbox = 3 * 2 * (int64_t)kBoxBlocks, nres = nbox + kBoxBlocks;
  if (h->mon_buf == nullptr && (rc = dev_alloc(h, &h->mon_buf, nres))) return rc;
  k_box_sum_max<<<dim3(kBoxBlocks, 3), 256, 0, h->stream>>>(d, h->U, h->V, h->W, (double2*)h->mon_buf);
  C3D_LAUNCH_CHECK(h);
  if ((rc = launch_maxdiv(h, h->mon_buf + nbox))) return rc;
  std::vector<double> p(nres);
  C3D_CUDA_TRY(h, cudaMemcpyAsync(p.data(), h->mon_buf, sizeof(double) * nres, cudaMemcpyDeviceToHost, h->stream));
  C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  for (int c = 0; c < 3; ++c) {
    double s = 0.0, m = -INFINITY;
    for (int b = 0; b < kBoxBlocks; ++b) {
      s += p[2 * ((size_t)c * kBoxBlocks + b)];
      m = std::max(m, p[2 * ((size_t)c * kBoxBlocks + b) + 1]);
    }
    out[c] = s / vol;
    out[3 + c] = m;
  }
  double mx = 0.0;
  for (int b = 0; b < kBoxBlocks; ++b) mx = p[nbox + b] > mx ? p[nbox + b] : mx;
  out[6] = mx;
  return 0;
}

}  // namespace c3d
