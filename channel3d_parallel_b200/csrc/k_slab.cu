// The z transforms and wall-normal solves of the Poisson equation
// (src/poisson.f90:45-80): z DFT of every row of a kx slab, one tridiagonal
// system in y per (kx, kz), inverse z DFT.
//
// Two kernels over blocks of kRows rows of j, a CTA a block, so that a slab of
// any size spreads over the chip:
//   k_slab_fwd: z FFT of the block's rows (the first stage reads them from
//     memory, the last leaves them in shared memory), then one thread per
//     column sweeps the block's rows forward and back in registers with zero
//     values outside the block, and stores them;
//   k_slab_inv: adds the two neighbours' contributions, and transforms back
//     (the last stage writes to memory).
// The elimination is that of the whole column (L U = T, factors from the
// whole matrix), partitioned: with Y the forward value before the block and X
// the solution after it,
//   y(j) = yl(j) + h(j) Y,          h(j) = -MULT(j-1) h(j-1),    h = 1 before the block,
//   x(j) = xl(j) + p(j) Y + g(j) X, g(j) = -DU(j)/D'(j) g(j+1),  g = 1 after the block,
//                                   p(j) = (h(j) - DU(j) p(j+1))/D'(j), p = 0 after it,
// where yl, xl are the block's own sweeps.  The chain over the blocks needs a
// block's last yl and first xl only; the last CTA of a slab to finish (a
// ticket per slab) runs it for every column and leaves Y and X per block.
//
// Why two passes over the spectrum and not one that keeps a slab on chip: a
// slab of 128 x 192 values takes 2 SMs' shared memory and one of 256 x 384
// takes 7, so a cluster that holds it runs 8 to 12 warps per SM, in whole
// waves of clusters, with the sweeps of 16 to 32 rows one after another.
// 384 x 256 x 384: 1237 us in clusters, 417 here (1.4 GB moved: 210 us at the
// copy rate); what is left is latency at 24 warps per SM and about 100
// instructions a value.  Few slabs in a thin channel are the other way round:
// the chain over the blocks is what they wait for (slab_by_blocks,
// k_poisson.cu).  Four rounds of 64 registers or 16 rows a block were
// slower at 384 x 256 x 384 (553 and 603 us with 256 threads, against 539).
#include <algorithm>
#include <cmath>
#include <vector>

#include "c3d_internal.cuh"
#include "fft.cuh"
#include "fft_tables.h"

namespace c3d {

namespace {

constexpr int kRows = 8;            // rows of j per block, held in registers per column
constexpr int kMaxR = 8;            // largest FFT radix
constexpr unsigned kRecRows = (unsigned)((1ull << 32) / kRows);   // reciprocal of kRows for div_by
// one column per thread up to 384: the row's columns in two rounds of 192
// threads took 539 us at 384 x 256 x 384 against 467
constexpr int kSlabThreads = 384;

// row stride in shared memory: FP64 1 mod 8, FP32 odd
template <typename T>
constexpr int slab_stride(int Nz) {
  return sizeof(T) == 8 ? (Nz + 6) / 8 * 8 + 1 : Nz | 1;
}

template <typename T>
struct SlabArgs {
  Dims d;
  typename cplx<T>::t* __restrict__ spec;
  const typename cplx<T>::t* __restrict__ tw;    // w_N^m
  const typename cplx<T>::t* __restrict__ tw1;   // first-stage twiddles, [r][q]
  const T* __restrict__ rdp;      // 1/D'(j) per (m, j, kz')
  const T* __restrict__ dl;       // Dyy(j+1, j)
  const T* __restrict__ du;       // Dyy(j, j+1)
  const T* __restrict__ link;     // h(last), p(first), g(first) per (m, block): [m][block][3][kz']
  const int* __restrict__ kzs;    // kz' of the column at each transformed position
  typename cplx<T>::t* __restrict__ ends;   // [m][block][2][Nz]: yl(last), xl(first), then Y, X
  unsigned* __restrict__ ticket;  // per slab
  FftPasses P;
  int jr, nblk;                   // rows per block, blocks of a slab
  int rs, pz;                     // row stride in shared memory, in memory
  int zero00;                     // 1: leave the kx = kz = 0 column to the FP64 mean-mode solve
  int rlo, rhi;                   // rows with a right-hand side and rows of the solution wanted
  int b0;                         // first block launched
};

// shared memory: rows [jr][rs], twiddles [Nz], pivots [jr+1][nkzs] of rows
// j0-1 .. j0+jr-1, DL and DU of the same rows
template <typename T>
struct SlabSmem {
  typename cplx<T>::t *data, *tw;
  T *rdp, *dl, *du;
};
template <typename T>
__device__ __forceinline__ SlabSmem<T> slab_carve(unsigned char* base, const SlabArgs<T>& a) {
  SlabSmem<T> s;
  s.data = reinterpret_cast<typename cplx<T>::t*>(base);
  s.tw = s.data + (size_t)a.jr * a.rs;
  s.rdp = reinterpret_cast<T*>(s.tw + a.d.Nz);
  s.dl = s.rdp + (size_t)(a.jr + 1) * a.d.nkzs;
  s.du = s.dl + a.jr + 1;
  return s;
}
template <typename T>
size_t slab_smem(int Nz, int nkzs, int jr, int rs) {
  return sizeof(typename cplx<T>::t) * ((size_t)jr * rs + Nz) + sizeof(T) * (size_t)(jr + 1) * (nkzs + 2);
}

template <typename T>
__device__ __forceinline__ void cp_async_t(T* s, const T* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
               "n"(sizeof(T)));
}

// the block's tables, asynchronously
template <typename T>
__device__ __forceinline__ void slab_tables(const SlabArgs<T>& a, const SlabSmem<T>& s, int m, int j0, int jn) {
  using C = typename cplx<T>::t;
  const int nk = a.d.nkzs, Ny = a.d.Ny;
  const int first = j0 > 0 ? 0 : nk;       // row j0-1 exists
  const T* src = a.rdp + ((int64_t)m * Ny + j0 - 1) * nk;
  for (int t = first + (int)threadIdx.x; t < (jn + 1) * nk; t += blockDim.x) cp_async_t(s.rdp + t, src + t);
  for (int t = threadIdx.x; t <= jn; t += blockDim.x) {
    const int j = j0 - 1 + t;
    s.dl[t] = j >= 0 ? a.dl[j] : (T)0;
    s.du[t] = j >= 0 ? a.du[j] : (T)0;
  }
  for (int t = threadIdx.x; t < a.d.Nz; t += blockDim.x) {
    const C w = a.tw[t];
    s.tw[t] = w;
  }
  asm volatile("cp.async.commit_group;\n" ::);
}

// the chain over a slab's blocks, one thread per column
template <typename T>
__device__ __forceinline__ void slab_chain(const SlabArgs<T>& a, int m) {
  using C = typename cplx<T>::t;
  const int Nz = a.d.Nz, nk = a.d.nkzs, nb = a.nblk;
  const int b0 = a.b0, b1 = a.b0 + (int)gridDim.x - 1;
  for (int col = threadIdx.x; col < Nz; col += blockDim.x) {
    const T* lk = a.link + (int64_t)m * nb * 3 * nk + a.kzs[col];
    C* e = a.ends + (int64_t)m * nb * 2 * Nz + col;
    C Y = C{(T)0, (T)0}, X = C{(T)0, (T)0};
    // blocks before b0 have no right-hand side: Y = 0 there.  The loads of a
    // batch of blocks are issued together.
    constexpr int kB = 8;
    for (int c = b0; c < nb; c += kB) {
      C yl[kB];
      T h[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        yl[u] = C{(T)0, (T)0};
        if (c + u <= b1) yl[u] = __ldcg(e + (int64_t)(c + u) * 2 * Nz);
        h[u] = c + u < nb ? lk[(int64_t)(c + u) * 3 * nk] : (T)0;
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        if (c + u < nb) e[(int64_t)(c + u) * 2 * Nz] = Y;
        Y = C{yl[u].x + h[u] * Y.x, yl[u].y + h[u] * Y.y};
      }
    }
    constexpr int kC = 4;
    for (int c = nb - 1; c >= b0; c -= kC) {
      C xl[kC], Yb[kC];
      T p[kC], g[kC];
#pragma unroll
      for (int u = 0; u < kC; ++u) {
        const int b = c - u;
        xl[u] = Yb[u] = C{(T)0, (T)0};
        p[u] = g[u] = (T)0;
        if (b >= b0) {
          if (b <= b1) xl[u] = __ldcg(e + ((int64_t)b * 2 + 1) * Nz);
          Yb[u] = e[(int64_t)b * 2 * Nz];
          p[u] = lk[((int64_t)b * 3 + 1) * nk];
          g[u] = lk[((int64_t)b * 3 + 2) * nk];
        }
      }
#pragma unroll
      for (int u = 0; u < kC; ++u) {
        const int b = c - u;
        if (b >= b0 && b <= b1) e[((int64_t)b * 2 + 1) * Nz] = X;
        X = C{xl[u].x + p[u] * Yb[u].x + g[u] * X.x, xl[u].y + p[u] * Yb[u].y + g[u] * X.y};
      }
    }
  }
}

// one column of a block: the sweeps with zero values outside the block.
// FULL: kRows rows, all in the band
template <bool FULL, typename T>
__device__ __forceinline__ void slab_sweeps(const SlabArgs<T>& a, const SlabSmem<T>& s, int col, int blo, int bhi,
                                            int jn, typename cplx<T>::t* g, typename cplx<T>::t* e) {
  using C = typename cplx<T>::t;
  const int nk = a.d.nkzs, RS = a.rs, Nz = a.d.Nz;
  const T* rd = s.rdp + nk + a.kzs[col];     // row j0
  C v[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    v[r] = C{(T)0, (T)0};
    if (FULL || (r >= blo && r < bhi)) v[r] = s.data[r * RS + col];
  }
  T rp[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) rp[r] = FULL || r < jn ? rd[r * nk] : (T)0;
  C yl = v[0];
#pragma unroll
  for (int r = 1; r < kRows; ++r) {
    if (FULL || r < jn) {
      const T mu = s.dl[r] * rp[r - 1];              // DL of row j0+r-1
      v[r].x -= mu * v[r - 1].x;
      v[r].y -= mu * v[r - 1].y;
      yl = v[r];
    }
  }
  e[col] = yl;
  C xn = C{(T)0, (T)0};
  C* o = g + col;
#pragma unroll
  for (int r = kRows - 1; r >= 0; --r) {
    if (FULL || r < jn) {
      const T u = s.du[r + 1];
      v[r].x = (v[r].x - u * xn.x) * rp[r];
      v[r].y = (v[r].y - u * xn.y) * rp[r];
      xn = v[r];
      if (FULL || (r >= blo && r < bhi)) o[r * a.pz] = v[r];
    }
  }
  e[Nz + col] = xn;
}

// the neighbours' contributions to one column, v: its own values
template <bool FULL, typename T>
__device__ __forceinline__ void slab_correct(const SlabArgs<T>& a, const SlabSmem<T>& s, int col, int blo, int bhi,
                                             int j0, int jn, bool zero, typename cplx<T>::t (&v)[kRows],
                                             typename cplx<T>::t Y, typename cplx<T>::t X) {
  using C = typename cplx<T>::t;
  const int nk = a.d.nkzs, RS = a.rs;
  const T* rd = s.rdp + a.kzs[col];            // row j0-1
  T h[kRows], rp = j0 > 0 ? rd[0] : (T)0, hc = (T)1;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    h[r] = (T)0;
    if (FULL || r < jn) {
      hc = -(s.dl[r] * rp) * hc;
      h[r] = hc;
      rp = rd[(r + 1) * nk];
    }
  }
  T p = (T)0, gc = (T)1;
#pragma unroll
  for (int r = kRows - 1; r >= 0; --r) {
    if (FULL || r < jn) {
      const T u = s.du[r + 1], q = rd[(r + 1) * nk];
      p = (h[r] - u * p) * q;
      gc = -(u * q) * gc;
      v[r].x += p * Y.x + gc * X.x;
      v[r].y += p * Y.y + gc * X.y;
      if (zero) v[r] = C{(T)0, (T)0};
      if (FULL || (r >= blo && r < bhi)) s.data[r * RS + col] = v[r];
    }
  }
}

template <typename T, int NZ>
__global__ void __launch_bounds__(kSlabThreads, 2) k_slab_fwd(SlabArgs<T> a) {
  using C = typename cplx<T>::t;
  extern __shared__ __align__(16) unsigned char slab_smem_raw[];
  __shared__ bool s_last;
  const int m = blockIdx.y, b = a.b0 + blockIdx.x;
  constexpr int R0 = plan_radix(NZ > 0 ? NZ : 2, kMaxR);
  const int Ny = a.d.Ny, Nz = NZ > 0 ? NZ : a.d.Nz, RS = NZ > 0 ? slab_stride<T>(NZ) : a.rs;
  const int j0 = b * a.jr, jn = min(a.jr, Ny - j0);
  const int blo = max(a.rlo - j0, 0), bhi = min(a.rhi + 1 - j0, jn);   // rows [blo, bhi) of the band
  const bool full = bhi - blo == kRows;
  const SlabSmem<T> s = slab_carve<T>(slab_smem_raw, a);
  C* const g = a.spec + ((int64_t)m * Ny + j0) * a.pz;
  slab_tables(a, s, m, j0, jn);
  auto first_in = [&](int l, int e) { return g[(blo + l) * a.pz + e]; };
  auto first_out = [&](int l, int e, C v) { s.data[(blo + l) * RS + e] = v; };
  if constexpr (NZ > 0) ct_edge<T, false, R0>(bhi - blo, NZ, a.tw1, a.P.rec[0], first_in, first_out);
  else ct_edge_any<T, false>(bhi - blo, a.tw1, a.P, first_in, first_out);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  if constexpr (NZ > 0) {
    if (full) fft_fixed_dif<T, NZ, kMaxR, NZ / R0>(s.data, kRows, kRecRows, RS, s.tw);
  } else if (full) {
    fft_rows_dif<T, kMaxR, kRows>(s.data, kRows, RS, s.tw, a.P, 1);
  }
  if (!full) fft_rows_dif<T, kMaxR>(s.data + blo * RS, bhi - blo, RS, s.tw, a.P, 1);
  C* const e = a.ends + ((int64_t)m * a.nblk + b) * 2 * Nz;
  for (int col = threadIdx.x; col < Nz; col += blockDim.x) {
    if (full) slab_sweeps<true>(a, s, col, blo, bhi, jn, g, e);
    else slab_sweeps<false>(a, s, col, blo, bhi, jn, g, e);
  }
  // the slab's last block runs the chain
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();             // the block's stores, ordered before the ticket by the barrier
    s_last = atomicAdd(a.ticket + m, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    slab_chain(a, m);
    if (threadIdx.x == 0) a.ticket[m] = 0u;
  }
}

template <typename T, int NZ>
__global__ void __launch_bounds__(kSlabThreads, 2) k_slab_inv(SlabArgs<T> a) {
  using C = typename cplx<T>::t;
  extern __shared__ __align__(16) unsigned char slab_smem_raw[];
  // the slabs that k_slab_fwd left last, and L2 still holds, come first (473 ->
  // 448 us at 384 x 256 x 384)
  const int m = (int)gridDim.y - 1 - (int)blockIdx.y, b = a.b0 + blockIdx.x;
  constexpr int R0 = plan_radix(NZ > 0 ? NZ : 2, kMaxR);
  const int Ny = a.d.Ny, Nz = NZ > 0 ? NZ : a.d.Nz, RS = NZ > 0 ? slab_stride<T>(NZ) : a.rs;
  const int j0 = b * a.jr, jn = min(a.jr, Ny - j0);
  const int blo = max(a.rlo - j0, 0), bhi = min(a.rhi + 1 - j0, jn);
  const bool full = bhi - blo == kRows;
  const SlabSmem<T> s = slab_carve<T>(slab_smem_raw, a);
  C* const g = a.spec + ((int64_t)m * Ny + j0) * a.pz;
  slab_tables(a, s, m, j0, jn);
  const C* const e = a.ends + ((int64_t)m * a.nblk + b) * 2 * Nz;
  C v[kRows], Y, X;
  auto load = [&](int col) {
    const C* o = g + col;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      v[r] = C{(T)0, (T)0};
      if (full || (r >= blo && r < bhi)) v[r] = o[r * a.pz];
    }
    Y = e[col];
    X = e[Nz + col];
  };
  if ((int)threadIdx.x < Nz) load(threadIdx.x);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  for (int col = threadIdx.x; col < Nz; col += blockDim.x) {
    if (col >= (int)blockDim.x) load(col);
    const bool zero = a.zero00 && m == 0 && col == 0;
    if (full) slab_correct<true>(a, s, col, blo, bhi, j0, jn, zero, v, Y, X);
    else slab_correct<false>(a, s, col, blo, bhi, j0, jn, zero, v, Y, X);
  }
  __syncthreads();
  if constexpr (NZ > 0) {
    if (full) fft_fixed_dit_inv<T, NZ, kMaxR, NZ / R0>(s.data, kRows, kRecRows, RS, s.tw);
  } else if (full) {
    fft_rows_dit_inv<T, kMaxR, kRows>(s.data, kRows, RS, s.tw, a.P, 1);
  }
  if (!full) fft_rows_dit_inv<T, kMaxR>(s.data + blo * RS, bhi - blo, RS, s.tw, a.P, 1);
  auto last_in = [&](int l, int q) { return s.data[(blo + l) * RS + q]; };
  auto last_out = [&](int l, int q, C v) { g[(blo + l) * a.pz + q] = v; };
  if constexpr (NZ > 0) ct_edge<T, true, R0>(bhi - blo, NZ, a.tw1, a.P.rec[0], last_in, last_out);
  else ct_edge_any<T, true>(bhi - blo, a.tw1, a.P, last_in, last_out);
}

// factors across a block, per mode: h(last), p(first), g(first)
template <typename T>
__global__ void k_slab_link(Dims d, int jr, int nblk, const double* __restrict__ rdp, const double* __restrict__ dl,
                            const double* __restrict__ du, T* __restrict__ link) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
  if (t >= d.nkzs) return;
  for (int b = 0; b < nblk; ++b) {
    const int j0 = b * jr, jn = min(jr, d.Ny - j0);
    auto rd = [&](int j) { return rdp[((int64_t)m * d.Ny + j) * d.nkzs + t]; };
    double h[kRows], hc = 1.0;
    for (int r = 0; r < jn; ++r) {
      const int j = j0 + r;
      hc = j > 0 ? -(dl[j - 1] * rd(j - 1)) * hc : 0.0;
      h[r] = hc;
    }
    double p = 0.0, g = 1.0;
    for (int r = jn - 1; r >= 0; --r) {
      const double u = du[j0 + r], rp = rd(j0 + r);
      p = (h[r] - u * p) * rp;
      g = -(u * rp) * g;
    }
    T* o = link + (((int64_t)m * nblk + b) * 3) * d.nkzs + t;
    o[0] = (T)hc;
    o[d.nkzs] = (T)p;
    o[2 * d.nkzs] = (T)g;
  }
}

constexpr int kSlabSmemMax = 220 * 1024;

// The kernels for rows of Nz columns.  Rows of 192 to 512 columns have the
// length compiled in (384 x 256 x 384: 448 -> 417 us, FP32 mixed steps
// 7480 -> 7370);
// shorter rows reach these kernels only with very many of them.
template <typename T>
struct SlabKernels {
  void (*fwd)(SlabArgs<T>);
  void (*inv)(SlabArgs<T>);
};
template <typename T, int... NZ>
SlabKernels<T> slab_pick(int Nz) {
  SlabKernels<T> k{k_slab_fwd<T, 0>, k_slab_inv<T, 0>};
  ((Nz == NZ ? (void)(k = {k_slab_fwd<T, NZ>, k_slab_inv<T, NZ>}) : (void)0), ...);
  return k;
}
template <typename T>
SlabKernels<T> slab_kernels(int Nz) {
  return slab_pick<T, 192, 216, 256, 288, 324, 384, 432, 486, 512>(Nz);
}

}  // namespace

// tables of the slab kernels; after every change of the grid (f32: the FP32
// copies too)
template <typename T>
static int slab_setup_t(Handle* h, SlabTables<T>& t) {
  using C = typename cplx<T>::t;
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  int rc;
  if (t.ticket == nullptr) {      // the last of its buffers
    t.jr = kRows;
    while (t.jr > 1 && slab_smem<T>(d.Nz, d.nkzs, t.jr, slab_stride<T>(d.Nz)) > (size_t)kSlabSmemMax) t.jr /= 2;
    t.nblk = (d.Ny + t.jr - 1) / t.jr;
    FftPasses P;
    make_fft_passes(d.Nz, P, kMaxR);
    const std::vector<C> tw1 = edge_twiddles<C>(d.Nz, P.radix[0]);
    std::vector<int> kzs(d.Nz);
    for (int c = 0; c < d.Nz; ++c) {
      const int k = dif_position_to_k(c, P);
      kzs[c] = k <= d.Nz - k ? k : d.Nz - k;
    }
    if ((rc = dev_alloc(h, &t.tw1, d.Nz))) return rc;
    if ((rc = dev_alloc(h, &t.kzs, d.Nz))) return rc;
    if ((rc = dev_alloc(h, &t.link, (int64_t)d.nkx * t.nblk * 3 * d.nkzs))) return rc;
    if ((rc = dev_alloc(h, &t.ends, (int64_t)d.nkx * t.nblk * 2 * d.Nz))) return rc;
    if ((rc = dev_alloc(h, &t.ticket, d.nkx))) return rc;
    C3D_CUDA_TRY(h, cudaMemcpyAsync(t.tw1, tw1.data(), sizeof(C) * d.Nz, cudaMemcpyHostToDevice, h->stream));
    C3D_CUDA_TRY(h, cudaMemcpyAsync(t.kzs, kzs.data(), sizeof(int) * d.Nz, cudaMemcpyHostToDevice, h->stream));
    const SlabKernels<T> k = slab_kernels<T>(d.Nz);
    C3D_CUDA_TRY(h, cudaFuncSetAttribute(k.fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmemMax));
    C3D_CUDA_TRY(h, cudaFuncSetAttribute(k.inv, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmemMax));
    C3D_CUDA_TRY(h, cudaStreamSynchronize(h->stream));   // the host copies end here
  }
  k_slab_link<T><<<dim3((d.nkzs + 63) / 64, d.nkx), 64, 0, h->stream>>>(d, t.jr, t.nblk, S.rdp, S.dl, S.du, t.link);
  C3D_LAUNCH_CHECK(h);
  return 0;
}

int slab_setup(Handle* h, bool f32) {
  return f32 ? slab_setup_t<float>(h, h->sp.slab32) : slab_setup_t<double>(h, h->sp.slab);
}

// z transforms and y solves of the whole spectrum, in place; rows (0-based
// j-2) outside [rlo, rhi] have no right-hand side and keep what they hold
template <typename T>
int launch_slab(Handle* h, typename SlabTables<T>::C* spec, int zero00, int rlo, int rhi) {
  const Dims& d = h->d;
  SpectralState& S = h->sp;
  constexpr bool f32 = sizeof(T) == 4;
  SlabArgs<T> a{};
  a.d = d;
  a.spec = spec;
  if constexpr (f32) {
    a.tw = S.twz32; a.rdp = S.rdp32; a.dl = S.dl32; a.du = S.du32; a.pz = S.pz32;
  } else {
    a.tw = S.twz; a.rdp = S.rdp; a.dl = S.dl; a.du = S.du; a.pz = S.pz64;
  }
  const SlabTables<T>* t;
  if constexpr (f32) t = &S.slab32; else t = &S.slab;
  a.tw1 = t->tw1; a.link = t->link; a.kzs = t->kzs; a.ends = t->ends; a.ticket = t->ticket;
  make_fft_passes(d.Nz, a.P, kMaxR);
  a.jr = t->jr; a.nblk = t->nblk;
  a.rs = slab_stride<T>(d.Nz);
  a.zero00 = zero00; a.rlo = rlo; a.rhi = rhi;
  a.b0 = rlo / a.jr;
  const dim3 grid(rhi / a.jr - a.b0 + 1, d.nkx);
  // a column per thread and a butterfly of the 8-row, radix-8 stages; longer
  // rows in equal rounds of at most kSlabThreads
  const int rounds = (d.Nz + kSlabThreads - 1) / kSlabThreads;
  const int nt = std::max(64, ((d.Nz + rounds - 1) / rounds + 31) / 32 * 32);
  const size_t smem = slab_smem<T>(d.Nz, d.nkzs, a.jr, a.rs);
  const SlabKernels<T> k = slab_kernels<T>(d.Nz);
  k.fwd<<<grid, nt, smem, h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  k.inv<<<grid, nt, smem, h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  return 0;
}
template int launch_slab<double>(Handle*, double2*, int, int, int);
template int launch_slab<float>(Handle*, float2*, int, int, int);

}  // namespace c3d
