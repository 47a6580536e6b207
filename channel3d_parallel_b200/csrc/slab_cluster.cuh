// The z transforms and wall-normal solves of the Poisson equation
// (src/poisson.f90:45-80), one thread-block cluster per kx slab: the slab stays
// in the cluster's shared memory from its first read to its last write (the
// two-kernel form in k_slab.cu is for slabs that this holds badly).  Compiled for
// FP64 in k_slab_cluster.cu and for FP32 in k_slab_cluster32.cu: each holds a
// kernel per row length.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>

#include "bulk.cuh"
#include "c3d_internal.cuh"
#include "fft.cuh"

namespace cg = cooperative_groups;

namespace c3d {

__host__ __device__ inline unsigned reciprocal(int n) {
  return n > 1 ? (unsigned)(((1ull << 32) + n - 1) / n) : 0u;
}

constexpr int kYzMaxRWide = 16;     // largest FFT radix (register budget)
constexpr int kYzMaxRNarrow = 8;

// ---------------------------------------------------------------------------
// kernel 2: z FFT, Thomas in y, inverse z FFT of one kx slab per cluster
// ---------------------------------------------------------------------------
// Two launch shapes: wide CTAs (at most 256 threads, two per SM) and narrow
// CTAs (at most 192 threads, three per SM, half the rows).  The whole FP64
// spectrum does not fit the aggregate shared memory at once, so the grid runs
// in two waves either way; narrow CTAs keep more warps per SM in flight and
// shorten each CTA's sequential sweeps.  yz_jmax: rows of j per CTA (the
// pivots of one column are held in registers).
template <typename T, bool NARROW>
__host__ __device__ constexpr int yz_jmax() { return (sizeof(T) == 8 ? 32 : 64) / (NARROW ? 2 : 1); }
template <bool NARROW>
__host__ __device__ constexpr int yz_threads() { return NARROW ? 192 : 256; }
template <bool NARROW>
__host__ __device__ constexpr int yz_min_blocks() { return NARROW ? 3 : 2; }

template <typename T>
struct YzArgs {
  Dims d;
  typename cplx<T>::t* __restrict__ spec;
  const typename cplx<T>::t* __restrict__ tw;
  const T* __restrict__ rdp;     // 1/D'(j) per (m, j, kz')
  const T* __restrict__ dl;      // Dyy(j+1, j)
  const T* __restrict__ du;      // Dyy(j, j+1)
  unsigned long long* err;       // sticky error bits
  FftPasses P;
  unsigned rec_jc;   // ceil(2^32 / jc)
  int cs;        // CTAs per cluster
  int jc;        // j rows per CTA
  int rs;        // shared-memory row stride (complex values)
  int pz;        // HBM row pitch (complex values)
  int zero00;    // 1: leave the kx = kz = 0 column to the FP64 mean-mode solve
  int rlo, rhi;  // rows (j-2) with a nonzero right-hand side and rows of the
                 // solution needed: the band [rlo, rhi]; other rows start at
                 // zero and are not transformed back or stored
};

// CTA c of the cluster owns rows j0 = c*jc .. j0+jn-1 of the slab.  Shared
// memory: rows [jc][rs] (the z FFT runs along a row), twiddles, DL and DU.
// The Thomas sweeps walk a column (one kz per thread) down the rows, CTA by
// CTA: forward elimination from CTA 0 to cs-1, back substitution from cs-1 to
// 0, each CTA starting from the neighbour row read through distributed
// shared memory.  After the forward transform column `col` holds wavenumber
// kz = dif_position_to_k(col); the inverse transform takes that order back.
template <typename T, bool NARROW, int NZ = 0>
__global__ void __launch_bounds__(yz_threads<NARROW>(), yz_min_blocks<NARROW>()) k_spectral_yz(YzArgs<T> a) {
  using C = typename cplx<T>::t;
  constexpr int JM = yz_jmax<T, NARROW>();
  extern __shared__ __align__(128) unsigned char yz_smem[];
  __shared__ __align__(8) uint64_t bar;
  cg::cluster_group cl = cg::this_cluster();
  const Dims& d = a.d;
  const int cs = a.cs;
  const int crank = (int)cl.block_rank();
  const int m = blockIdx.x / cs;
  const int Ny = d.Ny, Nz = NZ ? NZ : d.Nz, nkzs = d.nkzs;
  const int RS = a.rs, Jc = a.jc;
  const int j0 = crank * Jc;
  const int jn = min(Jc, Ny - j0);             // rows owned by this CTA (>= 1)
  C* data = reinterpret_cast<C*>(yz_smem);
  C* tw = data + (size_t)Jc * RS;
  C* ylast = tw + Nz;                          // local forward value of the last row
  C* xfirst = ylast + Nz;                      // local back-substituted first row
  C* yin = xfirst + Nz;                        // carry Y_in of this CTA
  T* sdl = reinterpret_cast<T*>(yin + Nz);
  T* sdu = sdl + Ny;
  const int tid = threadIdx.x, nt = blockDim.x;
  C* g = a.spec + ((int64_t)m * Ny + j0) * a.pz;
  const unsigned rowbytes = (unsigned)(a.pz * sizeof(C));

  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  // this CTA's rows of the band: [blo, bhi)
  const int blo = min(max(a.rlo - j0, 0), jn), bhi = max(min(a.rhi + 1 - j0, jn), blo);
  if (tid < 32) {
    if (tid == 0) mbar_arrive_expect_tx(&bar, rowbytes * (unsigned)(bhi - blo));
    __syncwarp();
    for (int r = blo + tid; r < bhi; r += 32)
      bulk_load(data + (size_t)r * RS, g + (int64_t)r * a.pz, rowbytes, &bar);
  }
  for (int t = tid; t < (jn - (bhi - blo)) * Nz; t += nt) {   // rows outside the band start at zero
    const int rr = t / Nz, col = t - rr * Nz;
    const int r = rr < blo ? rr : rr + (bhi - blo);
    data[(size_t)r * RS + col] = C{(T)0, (T)0};
  }
  for (int t = tid; t < Nz; t += nt) tw[t] = a.tw[t];
  for (int t = tid; t < Ny; t += nt) { sdl[t] = a.dl[t]; sdu[t] = a.du[t]; }

  const bool loaded = mbar_wait(&bar, 0, kWaitCycles);
  if (!loaded) atomicOr(a.err, 1ull);
  __syncthreads();

  constexpr int MAXR = NARROW ? kYzMaxRNarrow : kYzMaxRWide;
  const unsigned nrec = bhi - blo == Jc ? a.rec_jc : reciprocal(bhi - blo);
  if constexpr (NZ > 0) fft_fixed_dif<T, NZ, MAXR>(data + (size_t)blo * RS, bhi - blo, nrec, RS, tw);
  else fft_rows_dif<T, MAXR>(data + (size_t)blo * RS, bhi - blo, RS, tw, a.P);

  // pivots of this thread's column for rows j0-1 .. j0+jn-1 (one column per
  // thread when Nz <= blockDim; otherwise reloaded per column below)
  const T* rdp_m = a.rdp + (int64_t)m * Ny * nkzs;
  const bool one_col = Nz <= nt;
  T rdv[JM];
  T rdm1 = (T)0;                               // pivot of row j0-1 (previous CTA)
  auto load_pivots = [&](int col) {
    const int kz = dif_position_to_k(col, a.P);
    const int kzs = kz <= Nz - kz ? kz : Nz - kz;
#pragma unroll
    for (int jl = 0; jl < JM; ++jl)
      rdv[jl] = jl < jn ? __ldg(rdp_m + (int64_t)(j0 + jl) * nkzs + kzs) : (T)0;
    rdm1 = j0 > 0 ? __ldg(rdp_m + (int64_t)(j0 - 1) * nkzs + kzs) : (T)0;
  };
  if (one_col && tid < Nz) load_pivots(tid);

  // Partitioned elimination: every CTA sweeps its own rows at once, then
  // corrects them with carries from its neighbours (no tables):
  //   forward: y(j) = yl(j) + h(j) Y_in,  h(j0-1) = 1, h(j) = -MULT(j-1) h(j-1),
  //            Y_in(c+1) = yl_c(j1) + h_c(j1) Y_in(c);
  //   backward (on the corrected y): x(j) = xl(j) + g(j) X_in,  g(j1+1) = 1,
  //            g(j) = -DU(j)/D'(j) g(j+1),  X_in(c-1) = xl_c(j0) + g_c(j0) X_in(c).
  // The sweeps take rows in chunks of kCh: loads of a chunk are issued
  // together, the recurrence runs in registers, then the chunk is stored.
  constexpr int kCh = 4;
  // ylast / xfirst: published end values; hg[col] = (h(j1), g(j0))
  C* hg = yin;
  for (int col = tid; col < Nz; col += nt) {
    if (!one_col) load_pivots(col);
    // local forward elimination B(j) -= DL(j-1)/D'(j-1) * B(j-1) from y(j0-1) = 0
    C prev = C{(T)0, (T)0};
    T hcur = (T)1;
#pragma unroll
    for (int c0 = 0; c0 < JM; c0 += kCh) {
      if (c0 < jn) {
        C bv[kCh];
        T dlv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          bv[u] = C{(T)0, (T)0};
          dlv[u] = (T)0;
          if (jl < jn) {
            bv[u] = data[jl * RS + col];
            if (j0 + jl > 0) dlv[u] = sdl[j0 + jl - 1];
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          if (jl < jn) {
            const T mu = dlv[u] * (jl == 0 ? rdm1 : rdv[jl > 0 ? jl - 1 : 0]);
            if (jl > 0) {
              bv[u].x = bv[u].x - mu * prev.x;
              bv[u].y = bv[u].y - mu * prev.y;
            }
            hcur = -mu * hcur;
            prev = bv[u];
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u)
          if (c0 + u < jn) data[(c0 + u) * RS + col] = bv[u];
      }
    }
    ylast[col] = prev;
    hg[col].x = hcur;
  }
  cl.sync();
  for (int col = tid; col < Nz; col += nt) {
    if (!one_col) load_pivots(col);
    // Y_in = y(j0-1) from the predecessors' end values
    C Y = C{(T)0, (T)0};
    for (int c = 0; c < crank; ++c) {
      const C yl = cl.map_shared_rank(ylast, c)[col];
      const T he = cl.map_shared_rank(hg, c)[col].x;
      const T yx = yl.x + he * Y.x, yy = yl.y + he * Y.y;
      Y.x = yx;
      Y.y = yy;
    }
    // forward correction y += h Y_in (h recomputed), then the local back
    // substitution x(j) = (y(j) - DU(j) x(j+1)) / D'(j) from x(j1+1) = 0
    T hcur = (T)1;
#pragma unroll
    for (int c0 = 0; c0 < JM; c0 += kCh) {
      if (c0 < jn && crank > 0) {
        C bv[kCh];
        T dlv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          bv[u] = C{(T)0, (T)0};
          dlv[u] = (T)0;
          if (jl < jn) {
            bv[u] = data[jl * RS + col];
            dlv[u] = sdl[j0 + jl - 1];
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          if (jl < jn) {
            const T mu = dlv[u] * (jl == 0 ? rdm1 : rdv[jl > 0 ? jl - 1 : 0]);
            hcur = -mu * hcur;
            bv[u].x += hcur * Y.x;
            bv[u].y += hcur * Y.y;
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u)
          if (c0 + u < jn) data[(c0 + u) * RS + col] = bv[u];
      }
    }
    C xn = C{(T)0, (T)0};
    T gcur = (T)1;
#pragma unroll
    for (int c0 = JM - kCh; c0 >= 0; c0 -= kCh) {
      if (c0 < jn) {
        C bv[kCh];
        T duv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          bv[u] = C{(T)0, (T)0};
          duv[u] = (T)0;
          if (jl < jn) {
            bv[u] = data[jl * RS + col];
            duv[u] = sdu[j0 + jl];
          }
        }
#pragma unroll
        for (int u = kCh - 1; u >= 0; --u) {
          const int jl = c0 + u;
          if (jl < jn) {
            bv[u].x = (bv[u].x - duv[u] * xn.x) * rdv[jl];
            bv[u].y = (bv[u].y - duv[u] * xn.y) * rdv[jl];
            gcur = -duv[u] * rdv[jl] * gcur;
            xn = bv[u];
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u)
          if (c0 + u < jn) data[(c0 + u) * RS + col] = bv[u];
      }
    }
    xfirst[col] = xn;
    hg[col].y = gcur;
  }
  cl.sync();
  for (int col = tid; col < Nz; col += nt) {
    if (!one_col) load_pivots(col);
    // X_in = x(j1+1) from the successors' first values
    C X = C{(T)0, (T)0};
    for (int c = cs - 1; c > crank; --c) {
      const C xf = cl.map_shared_rank(xfirst, c)[col];
      const T ge = cl.map_shared_rank(hg, c)[col].y;
      const T xx = xf.x + ge * X.x, xy = xf.y + ge * X.y;
      X.x = xx;
      X.y = xy;
    }
    // backward correction x += g X_in (g recomputed from the last row up)
    T gcur = (T)1;
#pragma unroll
    for (int c0 = JM - kCh; c0 >= 0; c0 -= kCh) {
      if (c0 < jn && crank < cs - 1) {
        C bv[kCh];
        T duv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; ++u) {
          const int jl = c0 + u;
          bv[u] = C{(T)0, (T)0};
          duv[u] = (T)0;
          if (jl < jn) {
            bv[u] = data[jl * RS + col];
            duv[u] = sdu[j0 + jl];
          }
        }
#pragma unroll
        for (int u = kCh - 1; u >= 0; --u) {
          const int jl = c0 + u;
          if (jl < jn) {
            gcur = -duv[u] * rdv[jl] * gcur;
            bv[u].x += gcur * X.x;
            bv[u].y += gcur * X.y;
          }
        }
#pragma unroll
        for (int u = 0; u < kCh; ++u)
          if (c0 + u < jn) data[(c0 + u) * RS + col] = bv[u];
      }
    }
    if (a.zero00 && m == 0 && col == 0)
      for (int jl = 0; jl < jn; ++jl) data[jl * RS] = C{(T)0, (T)0};
  }
  __syncthreads();

  if constexpr (NZ > 0) fft_fixed_dit_inv<T, NZ, MAXR>(data + (size_t)blo * RS, bhi - blo, nrec, RS, tw);
  else fft_rows_dit_inv<T, MAXR>(data + (size_t)blo * RS, bhi - blo, RS, tw, a.P);
  // no CTA leaves while another may still read its ylast / xfirst
  cl.sync();

  fence_async_shared();
  __syncthreads();
  if (tid < 32) {
    if (loaded) {
      for (int r = blo + tid; r < bhi; r += 32) bulk_store(g + (int64_t)r * a.pz, data + (size_t)r * RS, rowbytes);
      bulk_commit();
      bulk_wait_read_all();
    } else {
      // the rows never arrived: let the copies in flight finish before exit
      mbar_wait(&bar, 0, kWaitCycles);
    }
  }
}

// cluster decomposition of a kx slab: the narrow shape when it fits (Nz <=
// 192, a CTA within 72 KB so three share an SM), else the wide shape (two
// CTAs per SM within 112 KB; 16-CTA clusters may use up to one SM each); in
// each the smallest power-of-two cluster whose CTAs own at most yz_jmax rows.
// Row stride: FP64 rows of 16-byte values padded to rs = 1 (mod 8) make
// row-to-row steps conflict-free; FP32 rows stay 16-byte aligned for the
// bulk copies (rs even) with rs = 2 (mod 4).
template <typename T, bool NARROW>
static bool choose_shape(const Dims& d, int rs, int& cs, int& jc, int& nt, int& smem) {
  const size_t esz = sizeof(typename cplx<T>::t);
  const int ntmax = yz_threads<NARROW>();
  // a multiple of Nz (one column per thread, fixed FFT butterflies) when
  // Nz <= ntmax
  nt = ntmax;
  if (d.Nz <= ntmax) {
    nt = d.Nz * (ntmax / d.Nz);
    if (nt > 128 && d.Nz >= 128) nt = d.Nz;
  } else if (NARROW) {
    return false;
  }
  const size_t limit = NARROW ? 72 * 1024 : 112 * 1024;
  for (cs = 1; cs <= 16; cs *= 2) {
    jc = (d.Ny + cs - 1) / cs;
    if ((cs - 1) * jc >= d.Ny) continue;      // every CTA must own a row
    if (jc > yz_jmax<T, NARROW>()) continue;
    const size_t bytes = esz * ((size_t)jc * rs + 4 * (size_t)d.Nz) + 2 * sizeof(T) * d.Ny;
    if (bytes <= limit || (!NARROW && cs == 16 && bytes <= 224 * 1024)) {
      smem = (int)bytes;
      return true;
    }
  }
  return false;
}

// Function attributes are process-wide and handles of different sizes share
// them, so a kernel's dynamic shared-memory limit only ever grows (per
// device; handles are created from one host thread at a time).
template <auto KERN>
static cudaError_t raise_smem_limit(int bytes) {
  static int cur[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (bytes <= cur[dev]) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) cur[dev] = bytes;
  return e;
}

template <typename T, bool NARROW>
static int active_clusters(int cs, int nt, int smem) {
  if (raise_smem_limit<k_spectral_yz<T, NARROW>>(smem) != cudaSuccess) return 0;
  if (cs > 8 &&
      cudaFuncSetAttribute(k_spectral_yz<T, NARROW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)cs, 1, 1);
  cfg.blockDim = dim3((unsigned)nt, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_spectral_yz<T, NARROW>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// Picks the shape whose kx slabs (one cluster each) run in fewer waves of
// co-resident clusters, as the device reports them; the narrow shape on a tie.
template <typename T>
static bool choose_cluster(const Dims& d, int pz, SlabCluster& c) {
  int rs = pz;
  if (sizeof(T) == 8) { while (rs % 8 != 1) ++rs; }
  else { while (rs % 4 != 2) ++rs; }
  int ncs, njc, nnt, nsm, wcs, wjc, wnt, wsm;
  const bool okn = choose_shape<T, true>(d, rs, ncs, njc, nnt, nsm);
  const bool okw = choose_shape<T, false>(d, rs, wcs, wjc, wnt, wsm);
  auto waves = [&](int active) { return active > 0 ? (d.nkx + active - 1) / active : 1 << 30; };
  const int an = okn ? active_clusters<T, true>(ncs, nnt, nsm) : 0;
  const int aw = okw ? active_clusters<T, false>(wcs, wnt, wsm) : 0;
  if (okn && (!okw || waves(an) <= waves(aw))) {
    c = SlabCluster{ncs, njc, rs, nnt, nsm, 1, yz_jmax<T, true>(), an};
    return true;
  }
  if (!okw) return false;
  c = SlabCluster{wcs, wjc, rs, wnt, wsm, 0, yz_jmax<T, false>(), aw};
  return true;
}

// The kernel for rows of Nz columns.  Rows of 64 to 256 columns have the
// length compiled in: the kernel passes through its code about once, so its
// size costs instruction fetches (49 -> 45 us at 192 x 128 x 192 on its own, 710
// -> 673 us a time step, where other kernels run in between; FP32 mixed steps
// 1063 -> 1035 us there, 264 -> 250 at 64 x 64 x 64).  Shorter rows take the form
// with run-time stages.
template <typename T>
using YzKernel = void (*)(YzArgs<T>);
template <typename T, bool NARROW, int... NZ>
static YzKernel<T> yz_pick(int Nz) {
  YzKernel<T> k = k_spectral_yz<T, NARROW>;
  ((Nz == NZ ? (void)(k = k_spectral_yz<T, NARROW, NZ>) : (void)0), ...);
  return k;
}
template <typename T>
static YzKernel<T> yz_kernel(int Nz, int narrow) {
  return narrow ? yz_pick<T, true, 64, 72, 96, 108, 128, 144, 162, 192>(Nz)
                : yz_pick<T, false, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256>(Nz);
}

// z transforms and y solves of the whole spectrum in place, one launch
template <typename T>
int launch_cluster(Handle* h, typename SlabTables<T>::C* spec, int zero00, int rlo, int rhi) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  constexpr bool f32 = sizeof(T) == 4;
  const SlabCluster& c = f32 ? S.cluster32 : S.cluster;
  YzArgs<T> a{};
  a.d = d;
  a.spec = spec;
  if constexpr (f32) {
    a.tw = S.twz32; a.rdp = S.rdp32; a.dl = S.dl32; a.du = S.du32; a.pz = S.pz32;
  } else {
    a.tw = S.twz; a.rdp = S.rdp; a.dl = S.dl; a.du = S.du; a.pz = S.pz64;
  }
  a.err = &h->sc->err;
  make_fft_passes(d.Nz, a.P, c.narrow ? kYzMaxRNarrow : kYzMaxRWide);
  a.cs = c.cs; a.jc = c.jc; a.rs = c.rs; a.zero00 = zero00;
  a.rlo = rlo; a.rhi = rhi;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(c.cs * d.nkx), 1, 1);
  cfg.blockDim = dim3((unsigned)c.nt, 1, 1);
  cfg.dynamicSmemBytes = (size_t)c.smem;
  cfg.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = c.cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  a.rec_jc = reciprocal(c.jc);
  C3D_CUDA_TRY(h, cudaLaunchKernelEx(&cfg, yz_kernel<T>(d.Nz, c.narrow), a));
  C3D_LAUNCH_CHECK(h);
  return 0;
}

// the cluster shape of the handle's slabs; C3D_ERR_UNSUPPORTED when there is none
template <typename T>
int cluster_setup(Handle* h) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  constexpr bool f32 = sizeof(T) == 4;
  SlabCluster& c = f32 ? S.cluster32 : S.cluster;
  if (!choose_cluster<T>(d, f32 ? S.pz32 : S.pz64, c)) {
    h->last_error = f32 ? "ny_global too large for the FP32 cluster decomposition"
                        : "ny_global too large for one 16-CTA cluster per kx slab";
    return C3D_ERR_UNSUPPORTED;
  }
  // process-wide, and handles of one Nz may differ in Ny: the most any needs
  const YzKernel<T> k = yz_kernel<T>(d.Nz, c.narrow);
  C3D_CUDA_TRY(h, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
  if (c.cs > 8) C3D_CUDA_TRY(h, cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return 0;
}

}  // namespace c3d
