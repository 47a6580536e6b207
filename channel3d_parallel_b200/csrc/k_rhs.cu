// Right-hand sides and RK3 stage update.
//
// compute_rhs_u/v/w (src/equations.f90:24-423) evaluated point-wise for all
// three components in one kernel, fused with the stage update of
// compute_time_step_RK3 (src/time_integration.f90:105-107, 134-136, 163-168).
//
// Interpolations are the reference's midpoint averages (src/interpolation.f90);
// every metric division is a precomputed reciprocal factor (Metric).  The
// RK3 tableau a21 = a31 = 1/4 is exploited by keeping one accumulator
// G = Uo + dt/4 F1 instead of Uo and F1:
//   stage 1:  U* = U + dt*8/15*F1,   G = U + dt/4*F1
//   stage 2:  U* = G + dt*5/12*F2
//   stage 3:  U* = G + dt*3/4 *F3     (a32 = 0)
// which is the reference's update up to FP64 rounding order.
#include "c3d_internal.cuh"

namespace c3d {

struct RhsArgs {
  Dims d;
  Metric m;
  const double* __restrict__ U;
  const double* __restrict__ V;
  const double* __restrict__ W;
  const double* __restrict__ Gu;   // accumulators in (stages 2,3)
  const double* __restrict__ Gv;
  const double* __restrict__ Gw;
  double* __restrict__ Us;         // stage outputs (interior)
  double* __restrict__ Vs;
  double* __restrict__ Ws;
  double* __restrict__ Gu_out;     // accumulators out (stage 1)
  double* __restrict__ Gv_out;
  double* __restrict__ Gw_out;
  const double* __restrict__ Hu;   // exterior pressure-gradient masks (IB) or null
  const double* __restrict__ Hv;
  const double* __restrict__ Hw;
  const DevScalars* sc;
  double cs;   // coefficient of F for U*
  double cg;   // coefficient of F for G (stage 1)
  int comp_mask;  // rhs-only mode: which components to write (bit0 u, bit1 v, bit2 w)
  const double* __restrict__ phi;   // potential of the projection formed on the way in
  const double* ushift;             // constant-mass-flow shift of u, or null
  int kc;                           // z planes per CTA
};

// F into the rhs_u/v/w arrays (fine entries), incl. the duplicated periodic
// planes the reference also computes
__global__ void __launch_bounds__(256) k_rhs(RhsArgs a) {
  const Dims& d = a.d;
  const int i = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = 2 + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = 2 + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > d.Nx + 1 || j > d.Ny + 1 || k > d.Nz + 1) return;
  const Metric& m = a.m;
  const double* __restrict__ U = a.U;
  const double* __restrict__ V = a.V;
  const double* __restrict__ W = a.W;
#define LU(ii, jj, kk) __ldg(U + idxU(d, ii, jj, kk))
#define LV(ii, jj, kk) __ldg(V + idxV(d, ii, jj, kk))
#define LW(ii, jj, kk) __ldg(W + idxW(d, ii, jj, kk))
  const double dPdx = a.sc->dPdx, dPdy = a.sc->dPdy, dPdz = a.sc->dPdz;

  // ---- shared loads
  const double u0 = LU(i, j, k), uxm = LU(i - 1, j, k), uxp = LU(i + 1, j, k);
  const double uym = LU(i, j - 1, k), uyp = LU(i, j + 1, k);
  const double uzm = LU(i, j, k - 1), uzp = LU(i, j, k + 1);
  const double v0 = LV(i, j, k), vxp = LV(i + 1, j, k), vym = LV(i, j - 1, k);
  const double w0 = LW(i, j, k), wxp = LW(i + 1, j, k), wzm = LW(i, j, k - 1);

  // ---------------- Fu (src/equations.f90:40-151)
  double Fu;
  {
    const double v1m = LV(i + 1, j - 1, k);
    const double w1m = LW(i + 1, j, k - 1);
    const double ap = u0 + uxp, am = uxm + u0;
    double r = (am * am - ap * ap) * (0.25 * m.rdxg[i]);
    r += ((uym + u0) * (vym + v1m) - (u0 + uyp) * (v0 + vxp)) * (0.25 * m.rdy[j]);
    r += ((uzm + u0) * (wzm + w1m) - (u0 + uzp) * (w0 + wxp)) * (0.25 * m.rdz[k]);
    const double visc = m.cxpF[i] * (uxp - u0) - m.cxmF[i] * (u0 - uxm)
                      + m.cypC[j] * (uyp - u0) - m.cymC[j] * (u0 - uym)
                      + m.czpC[k] * (uzp - u0) - m.czmC[k] * (u0 - uzm);
    r += visc;
    r += a.Hu ? dPdx * __ldg(a.Hu + idxU(d, i, j, k)) : dPdx;
    Fu = r;
  }
  // ---------------- Fw (src/equations.f90:309-421)
  double Fw;
  {
    const double wxm = LW(i - 1, j, k), wym = LW(i, j - 1, k), wyp = LW(i, j + 1, k);
    const double wzp = LW(i, j, k + 1);
    const double umzp = LU(i - 1, j, k + 1);
    const double vzp = LV(i, j, k + 1), vymzp = LV(i, j - 1, k + 1);
    const double am = wzm + w0, ap = w0 + wzp;
    double r = (am * am - ap * ap) * (0.25 * m.rdzg[k]);
    r += ((uxm + umzp) * (wxm + w0) - (u0 + uzp) * (w0 + wxp)) * (0.25 * m.rdx[i]);
    r += ((vym + vymzp) * (wym + w0) - (v0 + vzp) * (w0 + wyp)) * (0.25 * m.rdy[j]);
    const double visc = m.cxpC[i] * (wxp - w0) - m.cxmC[i] * (w0 - wxm)
                      + m.cypC[j] * (wyp - w0) - m.cymC[j] * (w0 - wym)
                      + m.czpF[k] * (wzp - w0) - m.czmF[k] * (w0 - wzm);
    r += visc;
    r += a.Hw ? dPdz * __ldg(a.Hw + idxW(d, i, j, k)) : dPdz;
    Fw = r;
  }
  // ---------------- Fv (src/equations.f90:174-286), faces j = 2..ny-1
  const bool hasv = (j <= d.Ny);
  double Fv = 0.0;
  if (hasv) {
    const double vxm = LV(i - 1, j, k), vyp = LV(i, j + 1, k);
    const double vzm = LV(i, j, k - 1), vzp = LV(i, j, k + 1);
    const double um1 = LU(i - 1, j + 1, k);
    const double wyp = LW(i, j + 1, k), wypzm = LW(i, j + 1, k - 1);
    const double am = vym + v0, ap = v0 + vyp;
    double r = (am * am - ap * ap) * (0.25 * m.rdyg[j]);
    r += ((uxm + um1) * (vxm + v0) - (u0 + uyp) * (v0 + vxp)) * (0.25 * m.rdx[i]);
    r += ((vzm + v0) * (wzm + wypzm) - (v0 + vzp) * (w0 + wyp)) * (0.25 * m.rdz[k]);
    const double visc = m.cxpC[i] * (vxp - v0) - m.cxmC[i] * (v0 - vxm)
                      + m.cypF[j] * (vyp - v0) - m.cymF[j] * (v0 - vym)
                      + m.czpC[k] * (vzp - v0) - m.czmC[k] * (v0 - vzm);
    r += visc;
    r += a.Hv ? dPdy * __ldg(a.Hv + idxV(d, i, j, k)) : dPdy;
    Fv = r;
  }
#undef LU
#undef LV
#undef LW

  // rhs_u(2:nx-1, 2:nyg-1, 2:nzg-1): x 2..Nx+1, z 2..Nz+2 (plane Nz+2 duplicates 2)
  const int nu1 = d.nx - 2, nu2 = d.nyg - 2;
  if (a.comp_mask & 1) {
    double* R = a.Us;
    R[(i - 2) + (int64_t)nu1 * ((j - 2) + (int64_t)nu2 * (k - 2))] = Fu;
    if (k == 2) R[(i - 2) + (int64_t)nu1 * ((j - 2) + (int64_t)nu2 * (d.Nz))] = Fu;
  }
  // rhs_v(2:nxg-1, 2:ny-1, 2:nzg-1): x 2..Nx+2
  if ((a.comp_mask & 2) && hasv) {
    double* R = a.Vs;
    const int n1 = d.nxg - 2, n2 = d.ny - 2;
    const int64_t o = (int64_t)n1 * n2;
    R[(i - 2) + (int64_t)n1 * (j - 2) + o * (k - 2)] = Fv;
    if (i == 2) R[(d.Nx) + (int64_t)n1 * (j - 2) + o * (k - 2)] = Fv;
    if (k == 2) {
      R[(i - 2) + (int64_t)n1 * (j - 2) + o * d.Nz] = Fv;
      if (i == 2) R[(d.Nx) + (int64_t)n1 * (j - 2) + o * d.Nz] = Fv;
    }
  }
  // rhs_w(2:nxg-1, 2:nyg-1, 2:nz-1): x 2..Nx+2
  if (a.comp_mask & 4) {
    double* R = a.Ws;
    const int n1 = d.nxg - 2, n2 = d.nyg - 2;
    const int64_t o = (int64_t)n1 * n2;
    R[(i - 2) + (int64_t)n1 * (j - 2) + o * (k - 2)] = Fw;
    if (i == 2) R[(d.Nx) + (int64_t)n1 * (j - 2) + o * (k - 2)] = Fw;
  }
}

// ---------------------------------------------------------------------------
// Stage kernel of the time step.  A CTA owns a TX x TY tile of (i, j) columns
// and marches over a chunk of z planes, one cell per thread and plane.
//
// PROJ: the input is the previous stage's U*, V*, W* with its potential phi,
// and the velocities are formed on the way in, u = u* - d(phi)/dx (+ the
// mass-flow shift) with the boundary conditions as index folds and signs
// (projection, src/projection.f90:40-44; boundary_conditions.f90:20-252), so
// between two stages the projected fields are neither written nor read:
// 80 bytes a cell (u*, phi, G in; u* out) in place of the 56 of a separate
// projection plus 72.  Without PROJ the input is U, V, W with their ghosts.
//
// The planes (tile plus halo) come by cp.async into a ring of NSLOT slots,
// three planes ahead of the one whose velocities are formed, which in turn is
// two ahead of the one that is computed, so one barrier a plane orders
// everything; each thread forms the velocities of its own cell and most
// threads one component of a halo cell, in place (the three components of a
// cell in one thread: 105 us in place of 103 at 192 x 128 x 192, one warp in
// three held the others at the barrier).  Loads one plane ahead into
// registers took 166-197 us a stage at 192 x 128 x 192 (two to three
// microseconds a plane: the memory's latency under load).
//
// Measured (B200, us a stage 2 or 3): 192 x 128 x 192 101, where the separate
// projection took 53 and the update 92; 384 x 256 x 384 740 (369 and 692);
// 32 x 64 x 32 8 (6 and 31: that update marched 64 planes whatever the grid).
// Two or three planes a turn of the loop took 133 and 147 us: the code of one
// plane is as much as the instruction cache feeds.  Bound by instruction issue (0.55 a cycle at 16 warps,
// 400 a cell) and by the shared-memory pipe (0.7 busy: an 8-byte access of a
// warp is two wavefronts); memory runs at 3.5 TB/s.
//
// The momentum fluxes live on cell edges and centres,
//   Exy = (u + u(j+1)) (v + v(i+1)),  Exz = (u + u(k+1)) (w + w(i+1)),
//   Eyz = (v + v(k+1)) (w + w(j+1)),  and the squares of the face sums,
// each shared by two components; those on a z face, and the viscous z
// differences, are carried in registers from one plane to the next, so plane
// k-1 is not read again.
// ---------------------------------------------------------------------------
constexpr int TX = 32, TY = 8;
constexpr int PX = TX + 2, PY = TY + 2, PN = PX * PY;
constexpr int FX = PX + 1, FY = PY + 1, FN = FX * FY;     // phi: one more column and row
constexpr int RHS_THREADS = TX * TY;
constexpr int NHALO = PN - TX * TY;       // halo cells of a tile, at most one a thread
constexpr int RHS_CTAS = 2;               // resident CTAs per SM
constexpr int NSLOT = 6;                  // planes k .. k+5
static_assert(3 * NHALO <= RHS_THREADS && FN - TX * TY <= RHS_THREADS, "one halo value per thread");

__device__ __forceinline__ void cp_async8(unsigned sdst, const double* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sdst), "l"(gsrc));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Products and sums rounded as written here, so that both forms of the kernel
// (and the separate projection followed by the plain one) give the same bits.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double sqdiff(double a, double b) { return __fma_rn(a, a, -__dmul_rn(b, b)); }
__device__ __forceinline__ double wdiff(double p, double a, double q, double b) {
  return __fma_rn(p, a, -__dmul_rn(q, b));
}

// shared memory: NSLOT planes of U, V, W (PN each) and phi (FN, PROJ), the z
// factors (rdz/4, rdzg/4) of planes k0-1..k1+1 and (czpC, czmC), (czpF, czmF)
// of planes k0..k1
template <bool PROJ>
struct RhsSmem {
  static constexpr int SLOT = 3 * PN + (PROJ ? FN : 0);
  static constexpr int Z0 = NSLOT * SLOT + ((NSLOT * SLOT) & 1);
  static size_t bytes(int kc) { return sizeof(double) * (size_t)(Z0 + 2 * (kc + 2) + 4 * kc); }
};

template <int MODE, bool PROJ>
__global__ void __launch_bounds__(RHS_THREADS, RHS_CTAS) k_rhs_march(RhsArgs a) {
  using L = RhsSmem<PROJ>;
  extern __shared__ __align__(16) double rhs_smem[];
  // 1/dxg per tile column, 1/dyg per tile row (gradient of phi); y factors per
  // row: (rdy/4, rdyg/4), (cypC, cymC), (cypF, cymF)
  __shared__ double sGx[PX], sGy[PY];
  __shared__ double2 sY[3][TY];
  double2* sZ = reinterpret_cast<double2*>(rhs_smem + L::Z0);
  double2* sZ1 = sZ + a.kc + 2;
  const Dims& d = a.d;
  const Metric& m = a.m;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i0 = 2 + blockIdx.x * TX, j0 = 2 + blockIdx.y * TY;
  const int k0 = 2 + blockIdx.z * a.kc, k1 = min(k0 + a.kc - 1, d.Nz + 1);
  const int i = i0 + tx, j = j0 + ty;
  const int plU = d.nx * d.nyg, plV = d.nxg * d.ny, plW = d.nxg * d.nyg, plR = (d.nxg - 2) * (d.nyg - 2);
  auto at = [](int z, int pl) { return (int64_t)z * pl; };     // 32 x 32 -> 64 bits
  auto xfold = [&](int gi) { return gi == 1 ? d.Nx + 1 : 2 + (gi - 2) % d.Nx; };
  auto zfold = [&](int k) { return PROJ ? (k == 1 ? d.Nz + 1 : (k >= d.Nz + 2 ? k - d.Nz : k)) : k; };

  // places in the fields, inside a plane (always legal; what is read at a
  // position that is not needed is not used).  Columns past the grid fold back
  // into it like the periodic images: with one clamped address for all of them
  // a part-filled tile took twice as long as a full one, and copies left out by
  // a condition slowed every tile (105 -> 141 us at 192 x 128 x 192).
  struct Pos {
    int u, v, w;
    bool neg, wall;          // u, w: wall reflection; v: zero
  };
  auto place = [&](int x, int y) {
    Pos p;
    int gi = i0 - 1 + x, gj = min(j0 - 1 + y, d.Ny + 2), gv = min(gj, d.Ny + 1);
    p.neg = p.wall = false;
    if (PROJ) {
      p.neg = gj == 1 || gj == d.Ny + 2;
      p.wall = gj < 2 || gj > d.Ny;
      gi = xfold(gi);
      gj = gj == 1 ? 2 : (gj == d.Ny + 2 ? d.Ny + 1 : gj);
      gv = min(gj, d.Ny);
    }
    if (gi > d.Nx + 2) gi = xfold(gi);
    p.u = (int)idxU(d, gi, gj, 1);
    p.v = (int)idxV(d, gi, gv, 1);
    p.w = (int)idxW(d, gi, gj, 1);
    return p;
  };
  auto phi_place = [&](int x, int y) {      // rows 1 and ny+1: the gradient there is not used as it stands
    const int gi = xfold(i0 - 1 + x), gj = min(max(j0 - 1 + y, 2), d.Ny + 1);
    return (int)idxR(d, gi, gj, 2);
  };
  // halo value of this thread: component hf at a tile position of rows 0 and
  // PY-1 or the side columns (the threads past 3 * NHALO copy the last one too and form nothing);
  // of phi: row 0, the last two rows, the side columns
  const int hv = min(tid, 3 * NHALO - 1), hf = hv / NHALO, hp = hv - hf * NHALO;
  int hx, hy, fx = 1, fy = 1;
  const bool fhalo = PROJ && tid < FN - TX * TY;
  if (hp < 2 * PX) { hy = hp < PX ? 0 : PY - 1; hx = hp < PX ? hp : hp - PX; }
  else { const int t = hp - 2 * PX; hx = t < TY ? 0 : PX - 1; hy = 1 + (t < TY ? t : t - TY); }
  if (tid < 3 * FX) { const int r = tid / FX; fy = r == 0 ? 0 : PY - 2 + r; fx = tid - r * FX; }
  else if (fhalo) { const int t = tid - 3 * FX, q = t / TY; fx = q == 0 ? 0 : PX - 2 + q; fy = 1 + (t - q * TY); }
  const int c = (ty + 1) * PX + (tx + 1);
  const int cf = (ty + 1) * FX + (tx + 1), chf = hy * FX + hx;      // the same places in phi's tile
  const int hs = hf * PN + hy * PX + hx;                            // the halo value's place in a slot
  const int hq = 3 * PN + chf + (hf == 0 ? 1 : (hf == 1 ? FX : 0)); // the other end of its gradient
  const Pos P0 = place(tx + 1, ty + 1), P1 = place(hx, hy);
  const double* const hsrc = hf == 0 ? a.U + P1.u : (hf == 1 ? a.V + P1.v : a.W + P1.w);
  const int hpl = hf == 0 ? plU : (hf == 1 ? plV : plW);
  const bool hneg = hf != 1 && P1.neg, hzero = hf == 1 && P1.wall;
  const int f0 = PROJ ? phi_place(tx + 1, ty + 1) : 0, f1 = PROJ ? phi_place(fx, fy) : 0;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(rhs_smem);

  // plane k of the inputs into ring slot `slot`
  auto issue = [&](int k, int slot) {
    const int z = zfold(k) - 1;
    const unsigned s = sbase + 8u * (unsigned)(slot * L::SLOT);
    const double *Uz = a.U + at(z, plU), *Vz = a.V + at(z, plV), *Wz = a.W + at(z, plW);
    cp_async8(s + 8 * c, Uz + P0.u);
    cp_async8(s + 8 * (PN + c), Vz + P0.v);
    cp_async8(s + 8 * (2 * PN + c), Wz + P0.w);
    cp_async8(s + 8 * hs, hsrc + at(z, hpl));
    if (PROJ) {
      const double* Fz = a.phi + at(z - 1, plR);
      cp_async8(s + 8 * (3 * PN + cf), Fz + f0);
      if (fhalo) cp_async8(s + 8 * (3 * PN + fy * FX + fx), Fz + f1);
    }
  };
  // the last plane whose velocities are needed is k1+1; its w needs phi of k1+2
  const int kend = PROJ ? k1 + 2 : k1 + 1;
  for (int q = 0; q < NSLOT; ++q) {
    if (k0 - 1 + q <= kend) issue(k0 - 1 + q, q);
    cp_async_commit();
  }

  // tables
  if (tid < PX) sGx[tid] = i0 - 1 + tid <= d.Nx + 2 ? m.rdxg[xfold(i0 - 1 + tid)] : 0.0;
  if (tid < PY) sGy[tid] = j0 - 1 + tid >= 2 && j0 - 1 + tid <= d.Ny ? m.rdyg[j0 - 1 + tid] : 0.0;
  if (tid < TY) {
    const int gj = j0 + tid <= d.Ny + 1 ? j0 + tid : 2;
    sY[0][tid] = make_double2(0.25 * m.rdy[gj], 0.25 * m.rdyg[gj]);
    sY[1][tid] = make_double2(m.cypC[gj], m.cymC[gj]);
    sY[2][tid] = make_double2(m.cypF[gj], m.cymF[gj]);
  }
  for (int t = tid; t < a.kc; t += RHS_THREADS) {
    const int kk = min(k0 + t, k1);
    sZ1[t] = make_double2(m.czpC[kk], m.czmC[kk]);
    sZ1[a.kc + t] = make_double2(m.czpF[kk], m.czmF[kk]);
  }
  for (int t = tid; t < a.kc + 2; t += RHS_THREADS) {
    const int kk = zfold(min(k0 - 1 + t, k1 + 1));
    sZ[t] = make_double2(0.25 * m.rdz[kk], 0.25 * m.rdzg[kk]);
  }
  const bool edge = j0 + TY > d.Ny + 1;     // the tile holds wall rows of v or rows past them
  const int ic = min(i, d.Nx + 1);
  const double2 x0 = make_double2(0.25 * m.rdxg[ic], 0.25 * m.rdx[ic]);
  const double2 x1 = make_double2(m.cxpF[ic], m.cxmF[ic]), x2 = make_double2(m.cxpC[ic], m.cxmC[ic]);
  const double shift = MODE == 1 && PROJ && a.ushift ? *a.ushift : 0.0;
  const double dPdx = a.sc->dPdx, dPdy = a.sc->dPdy, dPdz = a.sc->dPdz;

  const double hshift = hf == 0 ? shift : 0.0;
  // velocities of plane k0-1+kz in place: slot s, phi of the next plane in slot
  // sn; p0: phi of the own cell (carried from plane to plane); the own cell's
  // velocities to u, v, w.  The halo goes one component a thread, so that every
  // warp has the same work before the barrier.
  double p0 = 0.0;
  auto form_plane = [&](int kz, int s, int sn, double& u, double& v, double& w) {
    double* S = rhs_smem + s * L::SLOT;
    if (!PROJ) {
      u = S[c];
      v = S[PN + c];
      w = S[2 * PN + c];
      return;
    }
    const double* Sn = rhs_smem + sn * L::SLOT;
    const double gz = 4.0 * sZ[kz].y;
    const double pz = Sn[3 * PN + cf];
    u = __fma_rn(p0 - S[3 * PN + cf + 1], sGx[tx + 1], S[c]);
    v = __fma_rn(p0 - S[3 * PN + cf + FX], sGy[ty + 1], S[PN + c]);
    w = __fma_rn(p0 - pz, gz, S[2 * PN + c]);
    p0 = pz;
    if (MODE == 1) u += shift;
    if (edge) {
      if (P0.neg) { u = -u; w = -w; }
      if (P0.wall) v = 0.0;
    }
    S[c] = u;
    S[PN + c] = v;
    S[2 * PN + c] = w;
    const double g = hf == 0 ? sGx[hx] : (hf == 1 ? sGy[hy] : gz);
    double h = __fma_rn(S[3 * PN + chf] - (hf == 2 ? Sn : S)[hq], g, S[hs]);
    if (MODE == 1) h += hshift;
    if (tid < 3 * NHALO) S[hs] = hzero ? 0.0 : (hneg ? -h : h);
  };

  // planes k0-1, k0, k0+1 formed (k0+2 has landed), slots 0, 1, 2
  cp_async_wait<NSLOT - 4>();
  __syncthreads();
  if (PROJ) {
    p0 = rhs_smem[3 * PN + cf];
  }
  double ua, va, wa, u0, v0, w0, u1, v1, w1;
  form_plane(0, 0, 1, ua, va, wa);
  form_plane(1, 1, 2, u0, v0, w0);
  form_plane(2, 2, 3, u1, v1, w1);
  __syncthreads();
  // fluxes and differences on the cell's lower z face
  double Exz = mul(ua + u0, wa + rhs_smem[2 * PN + c + 1]);
  double Eyz = mul(va + v0, wa + rhs_smem[2 * PN + c + PX]);
  double Cz = mul(wa + w0, wa + w0);
  double du = u0 - ua, dv = v0 - va, dw = w0 - wa;
  double gu = 0.0, gv = 0.0, gw = 0.0;        // accumulators, one plane ahead
  auto load_G = [&](int k) {                  // legal at every position
    const int z = k - 1;
    gu = __ldg(a.Gu + at(z, plU) + P0.u);
    gv = __ldg(a.Gv + at(z, plV) + P0.v);
    gw = __ldg(a.Gw + at(z, plW) + P0.w);
  };
  if (MODE == 2) load_G(k0);
  const bool active = i <= d.Nx + 1 && j <= d.Ny + 1, hasv = active && j <= d.Ny;
  auto next = [](int s) { return s == NSLOT - 1 ? 0 : s + 1; };
  int s0 = 1;                // slot of plane k
  for (int k = k0; k <= k1; ++k) {
    const int t = k - k0;
    const int s1 = next(s0), s2 = next(s1), s3 = next(s2);
    // planes up to k+3 have landed and those up to k+1 are formed; every
    // thread is done with plane k-1, whose slot takes plane k+NSLOT-1
    cp_async_wait<NSLOT - 5>();
    __syncthreads();
    if (k + NSLOT - 1 <= kend) issue(k + NSLOT - 1, s0 == 0 ? NSLOT - 1 : s0 - 1);
    cp_async_commit();
    double u2 = 0.0, v2 = 0.0, w2 = 0.0;
    if (k < k1) form_plane(t + 3, s2, s3, u2, v2, w2);
    const double *U0 = rhs_smem + s0 * L::SLOT + c, *V0 = U0 + PN, *W0 = U0 + 2 * PN;
    const double *U1 = rhs_smem + s1 * L::SLOT + c, *V1 = U1 + PN;
    const double2 z0 = sZ[t + 1], z1 = sZ1[t];
    const double2 y0 = sY[0][ty], y1 = sY[1][ty];
    const double uxm = U0[-1], uxp = U0[1], uym = U0[-PX], uyp = U0[PX];
    const double vxm = V0[-1], vxp = V0[1], vym = V0[-PX], vyp = V0[PX];
    const double wxp = W0[1], wym = W0[-PX], wyp = W0[PX];
    const double exy = mul(u0 + uyp, v0 + vxp), exz = mul(u0 + u1, w0 + wxp), eyz = mul(v0 + v1, w0 + wyp);
    const double eu = u1 - u0, ev = v1 - v0, ew = w1 - w0;
    const int64_t zu = at(k - 1, plU), zv = at(k - 1, plV), zw = at(k - 1, plW);
    auto store = [&](double* S, const double* Hm, double dP, double* Go, double conv, double visc, double f, double g,
                     int64_t z, int o) {
      // the mask of an immersed body: only without PROJ
      const double F = !PROJ && Hm ? __fma_rn(dP, __ldg(Hm + z + o), conv + visc) : (conv + visc) + dP;
      if (MODE == 1) {
        (S + z)[o] = __fma_rn(a.cs, F, f);
        (Go + z)[o] = __fma_rn(a.cg, F, f);
      } else {
        (S + z)[o] = __fma_rn(a.cs, F, g);
      }
    };
    if (active) {
      {
        const double exym = mul(uym + u0, vym + V0[1 - PX]);
        const double conv = __fma_rn(sqdiff(uxm + u0, u0 + uxp), x0.x,
                                     __fma_rn(exym - exy, y0.x, mul(Exz - exz, z0.x)));
        const double visc = (wdiff(x1.x, uxp - u0, x1.y, u0 - uxm) + wdiff(y1.x, uyp - u0, y1.y, u0 - uym)) +
                            wdiff(z1.x, eu, z1.y, du);
        store(a.Us, a.Hu, dPdx, a.Gu_out, conv, visc, u0, gu, zu, P0.u);
      }
      {
        const double2 z2 = sZ1[a.kc + t];
        const double wxm = W0[-1];
        const double exzm = mul(uxm + U1[-1], wxm + w0), eyzm = mul(vym + V1[-PX], wym + w0);
        const double cz = mul(w0 + w1, w0 + w1);
        const double conv = __fma_rn(Cz - cz, z0.y, __fma_rn(exzm - exz, x0.y, mul(eyzm - eyz, y0.x)));
        const double visc = (wdiff(x2.x, wxp - w0, x2.y, w0 - wxm) + wdiff(y1.x, wyp - w0, y1.y, w0 - wym)) +
                            wdiff(z2.x, ew, z2.y, dw);
        store(a.Ws, a.Hw, dPdz, a.Gw_out, conv, visc, w0, gw, zw, P0.w);
        Cz = cz;
      }
      if (hasv) {
        const double2 y2 = sY[2][ty];
        const double exym = mul(uxm + U0[PX - 1], vxm + v0);
        const double conv = __fma_rn(sqdiff(vym + v0, v0 + vyp), y0.y,
                                     __fma_rn(exym - exy, x0.y, mul(Eyz - eyz, z0.x)));
        const double visc = (wdiff(x2.x, vxp - v0, x2.y, v0 - vxm) + wdiff(y2.x, vyp - v0, y2.y, v0 - vym)) +
                            wdiff(z1.x, ev, z1.y, dv);
        store(a.Vs, a.Hv, dPdy, a.Gv_out, conv, visc, v0, gv, zv, P0.v);
      }
    }
    if (MODE == 2 && k < k1) load_G(k + 1);
    Exz = exz; Eyz = eyz;
    du = eu; dv = ev; dw = ew;
    u0 = u1; v0 = v1; w0 = w1;
    u1 = u2; v1 = v2; w1 = w2;
    s0 = s1;
  }
  cp_async_wait<0>();
}

static RhsArgs base_args(Handle* h) {
  RhsArgs a{};
  a.d = h->d;
  a.m = h->m;
  a.U = h->U; a.V = h->V; a.W = h->W;
  a.sc = h->sc;
  if (h->p.exterior_pressure_gradient && h->ib != nullptr) {
    a.Hu = ib_hu(h); a.Hv = ib_hv(h); a.Hw = ib_hw(h);
  }
  return a;
}

static dim3 rhs_block() { return dim3(32, 4, 2); }
static dim3 rhs_grid(const Dims& d) {
  dim3 b = rhs_block();
  return dim3((d.Nx + b.x - 1) / b.x, (d.Ny + b.y - 1) / b.y, (d.Nz + b.z - 1) / b.z);
}

constexpr int kMaxChunk = 128;   // the chunk's z factors stay in shared memory

// z planes per CTA: the chunk count whose waves of resident CTAs march the
// fewest planes; a chunk also forms the planes on its two sides and fills its
// pipeline, worth about four planes
static int rhs_chunk(const Dims& d, int tiles) {
  const int slots = RHS_CTAS * 148;
  int best = 1, cost = 1 << 30;
  for (int n = 1; n <= d.Nz; ++n) {
    const int kc = (d.Nz + n - 1) / n;
    if (kc > kMaxChunk) continue;
    const int ctas = tiles * ((d.Nz + kc - 1) / kc);
    const int t = ((ctas + slots - 1) / slots) * (kc + 4);
    if (t < cost) { cost = t; best = kc; }
  }
  return best;
}

template <int MODE, bool PROJ>
static int launch_march(Handle* h, RhsArgs& a) {
  const Dims& d = h->d;
  const int gx = (d.Nx + TX - 1) / TX, gy = (d.Ny + TY - 1) / TY;
  a.kc = rhs_chunk(d, gx * gy);
  const dim3 grid(gx, gy, (d.Nz + a.kc - 1) / a.kc);
  const size_t smem = RhsSmem<PROJ>::bytes(a.kc);
  k_rhs_march<MODE, PROJ><<<grid, dim3(TX, TY), smem, h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  return 0;
}

int rhs_setup(Handle* h) {
  auto limit = [&](auto* k, size_t b) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  };
  C3D_CUDA_TRY(h, limit(k_rhs_march<1, false>, RhsSmem<false>::bytes(kMaxChunk)));
  C3D_CUDA_TRY(h, limit(k_rhs_march<2, false>, RhsSmem<false>::bytes(kMaxChunk)));
  C3D_CUDA_TRY(h, limit(k_rhs_march<1, true>, RhsSmem<true>::bytes(kMaxChunk)));
  C3D_CUDA_TRY(h, limit(k_rhs_march<2, true>, RhsSmem<true>::bytes(kMaxChunk)));
  return 0;
}

// stage = 1, 2, 3; U,V,W (with valid ghosts) -> Us,Vs,Ws interior (+ G at stage 1)
int launch_rhs_stage(Handle* h, int stage, double dt) {
  RhsArgs a = base_args(h);
  a.Us = h->Us; a.Vs = h->Vs; a.Ws = h->Ws;
  if (stage == 1) {
    a.Gu_out = h->Gu; a.Gv_out = h->Gv; a.Gw_out = h->Gw;
    a.cs = dt * (8.0 / 15.0);
    a.cg = dt * (1.0 / 4.0);
    return launch_march<1, false>(h, a);
  }
  a.Gu = h->Gu; a.Gv = h->Gv; a.Gw = h->Gw;
  a.cs = (stage == 2) ? dt * (5.0 / 12.0) : dt * (3.0 / 4.0);
  return launch_march<2, false>(h, a);
}

// the same from the previous stage's U* (in, interior only) and potential:
// the velocities are the projected ones, plus *ushift for u when given, with
// the boundary conditions applied; out must not be in
int launch_rhs_stage_projected(Handle* h, int stage, double dt, double* const in[3], const double* phi,
                               const double* ushift, double* const out[3]) {
  RhsArgs a = base_args(h);
  a.U = in[0]; a.V = in[1]; a.W = in[2];
  a.phi = phi;
  a.ushift = ushift;
  a.Us = out[0]; a.Vs = out[1]; a.Ws = out[2];
  if (stage == 1) {
    a.Gu_out = h->Gu; a.Gv_out = h->Gv; a.Gw_out = h->Gw;
    a.cs = dt * (8.0 / 15.0);
    a.cg = dt * (1.0 / 4.0);
    return launch_march<1, true>(h, a);
  }
  a.Gu = h->Gu; a.Gv = h->Gv; a.Gw = h->Gw;
  a.cs = (stage == 2) ? dt * (5.0 / 12.0) : dt * (3.0 / 4.0);
  return launch_march<2, true>(h, a);
}

// compute_time_step_Euler (src/time_integration.f90:34-52): U* = U + dt*F
// for the three components (the stage-1 kernel with its accumulator output
// sent to the G work fields, which Euler does not read)
int launch_rhs_euler(Handle* h, double dt) {
  RhsArgs a = base_args(h);
  a.Us = h->Us; a.Vs = h->Vs; a.Ws = h->Ws;
  a.Gu_out = h->Gu; a.Gv_out = h->Gv; a.Gw_out = h->Gw;
  a.cs = dt;
  a.cg = dt;
  return launch_march<1, false>(h, a);
}

// fine entries: component 1/2/3 -> rhsU/rhsV/rhsW
int launch_rhs_only(Handle* h, int component) {
  RhsArgs a = base_args(h);
  a.Us = h->rhsU; a.Vs = h->rhsV; a.Ws = h->rhsW;
  a.comp_mask = 1 << (component - 1);
  k_rhs<<<rhs_grid(h->d), rhs_block(), 0, h->stream>>>(a);
  C3D_LAUNCH_CHECK(h);
  return 0;
}

}  // namespace c3d
