// Cartesian 2-D shallow-water finite-volume step for sm_100a.
//
// One stage = one explicit stage of zoomy_jax's flux operator fused with the
// Shu-Osher update (zoomy_jax/fvm/solver_jax.py:722-895 and 990-1074;
// zoomy_jax/fvm/solver2/blocks.py:129-287, march.py:126-157):
//
//   halo load -> W = (b, eta, u, v) or (b, h, qx, qy) -> LSQ gradient (3x3
//   least-squares stencil, boundary ghosts) -> neighbour bounds -> limiter ->
//   tied / demoted slopes -> face traces with the Audusse clip -> Rusanov or
//   hydrostatic-reconstruction HLL face flux, each face once per tile ->
//   divergence + cell-edge bed source -> Q_out = a Q0 + (1 - a)(Qk + b dt L).
//
// Data layout: SoA planes (the reference's (n_state, n_cells) layout), cell
// (i, j) at i*ny + j.  Order 2: the strip kernel (swe2d_strip_kernel), one
// launch per stage -- a warp marches a 32-column strip down its rows in
// registers; interior items run the bare stencil, boundary items the same body
// with the boundary folded in.  Order 1: the tile kernel (swe2d_stage_kernel),
// a CTA per TX x 32 tile with its halo in shared memory.  Every face of an
// item is evaluated once.  The final stage also folds in Manning friction, the
// troubled-cell flag and the float64 maximum wave speed that sets the next dt,
// so a step queues with no host synchronisation.
#include <cstdio>
#include <cstring>
#include <cmath>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "launch_rules.h"

namespace zb {

constexpr int TY = 32;        // tile cells along y (contiguous)
constexpr int NT = 256;       // threads per CTA

template <typename T>
struct LsqTable {
  // [class 0..8][direction][slot]; slot 0..7 = the 3x3 neighbours (a, b) in
  // row-major order without (0, 0), 8 = x-boundary ghost, 9 = y-boundary ghost
  T w[9][2][10];
};

template <typename T>
struct SweParams {
  int nx, ny;
  T half_dx, half_dy;       // |face centre - cell centre|
  T kx, ky;                 // |face| / |cell| for x- and y-faces
  T g, eps_kp, eps_wet, manning_n;
  T vk_eps2;                // Venkatakrishnan eps^2
  int bc[4];                // left, right, bottom, top
  int limiter;
  int implicit_source;
  double cfl2r;             // cfl * 2 * r_in
  double den_fac;           // d * (2k + 1)
  double dt_max, t_end;
  double alpha, beta;       // Shu-Osher coefficients (generic stage)
  double dt_stage;          // generic stage: dt (< 0: read ctrl->dt)
  T inv6dx, inv6dy;         // interior least-squares gradient factors
  T inv4dx, inv4dy;         // 1 / (4 dx), 1 / (4 dy): side-class closed forms
  T inv5dx, inv5dy;         // 1 / (5 dx), 1 / (5 dy): corner closed forms
  int sx, sxc;              // output rows of an interior and of a boundary-strip item
  int single;               // 1: one launch, every item in the general body
  // the bed's interior gradient and limiter value (planes gx, gy, phi of
  // zb_swe2d_bed_prepare), read by the eta / HLL-HR interior strip body;
  // nullptr: evaluated from b like every other variable
  const T* bed;
};

enum { MODE_STEP1 = 0, MODE_STEP2 = 1, MODE_EULER = 2, MODE_STAGE = 3 };

template <typename T, int TX>
struct Smem {
  static constexpr int RX = TX + 2, RY = TY + 2, N = RX * RY;   // tile + 1-cell halo
  static constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
  T b[N], h[N], qx[N], qy[N], hinv[N];
  T fxh[NFX], fxt[NFX], fxl[NFX], fxr[NFX];
  T fyh[NFY], fyt[NFY], fyl[NFY], fyr[NFY];
};

// ── dt from the phase slot (solver2/blocks.py:64-95) ────────────────────────
__device__ __forceinline__ double dt_from_amax(double amax, double t,
                                               double cfl2r, double den_fac,
                                               double dt_max, double t_end) {
  double dt = cfl2r / (den_fac * amax);   // amax = 0 -> +inf, drops out
  dt = nmin(dt, dt_max);
  dt = nmin(dt, t_end - t);
  return dt;
}

// ── limiter candidates (reconstruction_jax.py:603-691) ──────────────────────
// Minmod / Barth-Jespersen on a Cartesian cell.  The four faces carry the
// increments +a, -a (x) and +c, -c (y).  With dpos = umax - u >= 0 and
// dneg = umin - u <= 0 a face with increment d > eps gives clip(dpos / d) and
// one with d < -eps gives clip(dneg / d) = clip(-dneg / |d|).  IEEE division
// is monotone in both operands, so the minimum over the four faces is exactly
// clip(min(dpos, -dneg) / max(|a|, |c|)) whenever max(|a|, |c|) > eps (a pair
// with |d| <= eps contributes 1 and never the minimum), and 1 otherwise: one
// division per variable instead of four, bit-identical to the per-face form in
// float64 (float32 divides with adiv, within its 2 ulp of that form).
template <typename T>
__device__ __forceinline__ T phi_clipmin(T a, T c, T dpos, T dneg) {
  const T m = fmx(fabs(a), fabs(c));
  const T dm = fmn(dpos, -dneg);
  const T r = clip01(adiv(dm, m));
  return m > T(1e-30) ? r : T(1);
}

template <typename T>
__device__ __forceinline__ T vk_cand(T delta, T dpos, T dneg, T ev2) {
  const T eps = T(1e-30);
  // selects, as phi_clipmin (two branches: 1000 x 1100, four steps, float32 529 us, now
  // 393, float64 1676, now 1327)
  const bool pos = delta > eps, neg = delta < -eps;
  const T d = pos ? dpos : dneg;
  const T num = d * d + ev2 + T(2) * delta * d;
  const T den = d * d + T(2) * delta * delta + delta * d + ev2;
  const T r = clip01(adiv(pos ? num : -num, pos ? zmax(den, eps) : zmin(den, -eps)));
  return pos || neg ? r : T(1);
}

template <typename T>
__device__ __forceinline__ T limiter_phi(int lim, T gx, T gy, T hdx, T hdy,
                                         T dpos, T dneg, T ev2) {
  if (lim == ZB_LIM_NONE) return T(1);
  T a = gx * hdx, c = gy * hdy;
  if (lim == ZB_LIM_VENKATAKRISHNAN) {
    T p = vk_cand(a, dpos, dneg, ev2);
    p = zmin(p, vk_cand(-a, dpos, dneg, ev2));
    p = zmin(p, vk_cand(c, dpos, dneg, ev2));
    p = zmin(p, vk_cand(-c, dpos, dneg, ev2));
    return clip01(p);
  }
  return phi_clipmin(a, c, dpos, dneg);
}

// ── face state and Riemann solvers ──────────────────────────────────────────
template <typename T>
struct Side {
  T b, h, qx, qy, ux, uy;
};

// Numerical flux across a face with unit normal n = sg * e_AXIS (sg = +-1).
// Outputs Fh, Fqx, Fqy and the scalar fluctuations Dm (owner / L side) and Dp
// (neighbour / R side) that multiply n.  Restates numerical_flux of the oracle:
// Rusanov (zoomy_jax/fvm/flux.py:72-82) and hydrostatic-reconstruction
// Rusanov / HLL (Audusse et al. 2004; Harten-Lax-van Leer 1983, Davis speeds).
// With an axis normal u.n = sg * u_AXIS and p n = sg * p e_AXIS exactly, so the
// terms the general form multiplies by a zero normal component are dropped.
template <typename T, int RIEMANN, int AXIS>
__device__ __forceinline__ void riemann(const Side<T>& L, const Side<T>& R, T sg, T g,
                                        T& Fh, T& Fqx, T& Fqy, T& Dm, T& Dp) {
  const T half = T(0.5);
  const T unL = sg * (AXIS == 0 ? L.ux : L.uy);
  const T unR = sg * (AXIS == 0 ? R.ux : R.uy);
  if (RIEMANN == ZB_RIEMANN_RUSANOV) {
    const T cL = asqrt(g * L.h), cR = asqrt(g * R.h);
    const T s = fmx(fabs(unL) + cL, fabs(unR) + cR);
    const T qnL = sg * (AXIS == 0 ? L.qx : L.qy);
    const T qnR = sg * (AXIS == 0 ? R.qx : R.qy);
    const T pL = sg * (half * g * (L.h * L.h)), pR = sg * (half * g * (R.h * R.h));
    T FLx = L.qx * unL, FLy = L.qy * unL, FRx = R.qx * unR, FRy = R.qy * unR;
    if (AXIS == 0) { FLx += pL; FRx += pR; } else { FLy += pL; FRy += pR; }
    const T hs = half * s;
    Fh = half * (qnL + qnR) - hs * (R.h - L.h);
    Fqx = half * (FLx + FRx) - hs * (R.qx - L.qx);
    Fqy = half * (FLy + FRy) - hs * (R.qy - L.qy);
    Dm = T(0);
    Dp = T(0);
    return;
  }
  const T bs = fmx(L.b, R.b);
  const T hLs = fmx(T(0), L.h + L.b - bs);
  const T hRs = fmx(T(0), R.h + R.b - bs);
  const T cL = asqrt(g * hLs), cR = asqrt(g * hRs);
  const T qLx = hLs * L.ux, qLy = hLs * L.uy;
  const T qRx = hRs * R.ux, qRy = hRs * R.uy;
  const T FLh = hLs * unL, FRh = hRs * unR;
  const T pL = sg * (half * g * (hLs * hLs)), pR = sg * (half * g * (hRs * hRs));
  T FLx = qLx * unL, FLy = qLy * unL, FRx = qRx * unR, FRy = qRy * unR;
  if (AXIS == 0) { FLx += pL; FRx += pR; } else { FLy += pL; FRy += pR; }
  if (RIEMANN == ZB_RIEMANN_RUSANOV_HR) {
    const T s = fmx(fabs(unL) + cL, fabs(unR) + cR);
    const T hs = half * s;
    Fh = half * (FLh + FRh) - hs * (hRs - hLs);
    Fqx = half * (FLx + FRx) - hs * (qRx - qLx);
    Fqy = half * (FLy + FRy) - hs * (qRy - qLy);
  } else {
    // Davis speeds clipped at zero: s_L = min(uL - cL, uR - cR, 0), s_R likewise
    const T sl = fmn3(unL - cL, unR - cR, T(0));
    const T sr = fmx3(unL + cL, unR + cR, T(0));
    const T den = sr - sl;
    const T quo = adiv(T(1), den);   // a select, not a branch
    const T inv = den > T(0) ? quo : T(0);
    const T slsr = sl * sr;
    Fh = (sr * FLh - sl * FRh + slsr * (hRs - hLs)) * inv;
    Fqx = (sr * FLx - sl * FRx + slsr * (qRx - qLx)) * inv;
    Fqy = (sr * FLy - sl * FRy + slsr * (qRy - qLy)) * inv;
  }
  Dm = half * g * (L.h * L.h - hLs * hLs);
  Dp = -(half * g * (R.h * R.h - hRs * hRs));
}

// ── the first-order stage kernel (one tile per CTA) ─────────────────────────
// Euler / generic stage without reconstruction for the TX x 32 tile of a CTA:
// the face traces are the cell states.
template <typename T, int TX, int RIEMANN, int MODE>
__global__ void __launch_bounds__(NT)
swe2d_stage_kernel(const T* __restrict__ bP, const T* __restrict__ hP,
                   const T* __restrict__ qxP, const T* __restrict__ qyP,
                   const T* h0P, const T* qx0P, const T* qy0P,
                   T* hO, T* qxO, T* qyO, zb_ctrl* ctrl, int phase,
                   const T* __restrict__ hinv_src,
                   unsigned char* __restrict__ trouble_out,
                   const SweParams<T> p) {
  using S = Smem<T, TX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  __shared__ double red[NT / 32];
  const int tid = threadIdx.x;
  const int i0 = blockIdx.y * TX, j0 = blockIdx.x * TY;
  const int nx = p.nx, ny = p.ny;
  const bool lead_block = blockIdx.x == 0 && blockIdx.y == 0;

  // dt of this step
  double dtd;
  if (MODE == MODE_STAGE) {
    dtd = p.dt_stage >= 0.0 ? p.dt_stage : ctrl->dt;
  } else {
    const int nph = (phase + 1) % 3, nnph = (phase + 2) % 3;
    const double t = ctrl->t[phase];
    dtd = dt_from_amax(ctrl->amax[phase], t, p.cfl2r, p.den_fac, p.dt_max, p.t_end);
    const bool ok = isfinite(dtd) && dtd > 0.0;
    if (lead_block && tid == 0) {
      if (!ok && t < p.t_end) atomicOr(&ctrl->status, (unsigned)ZB_ST_DT_INVALID);
      ctrl->dt = ok ? dtd : 0.0;
      ctrl->t[nph] = ok ? t + dtd : t;
      ctrl->amax[nnph] = 0.0;
      ctrl->troubled = 0u;
      // no-op step (t_end reached or dt invalid): the state is unchanged, so
      // the next slot carries this slot's wave-speed maximum forward
      if (!ok) ctrl->amax[nph] = ctrl->amax[phase];
    }
    if (!ok) {
      // the Euler path writes the workspace that is copied back: keep it equal
      for (int e = tid; e < TX * TY; e += NT) {
        const int gi = i0 + e / TY, gj = j0 + e % TY;
        if (gi < nx && gj < ny) {
          const size_t k = (size_t)gi * ny + gj;
          hO[k] = hP[k]; qxO[k] = qxP[k]; qyO[k] = qyP[k];
        }
      }
      return;
    }
  }
  const bool per_x = p.bc[0] == ZB_BC_PERIODIC;
  const bool per_y = p.bc[2] == ZB_BC_PERIODIC;
  const T dt = T(dtd);
  const T g = p.g, half = T(0.5);

  // ── halo load ──
  for (int e = tid; e < S::N; e += NT) {
    const int r = e / S::RY, c = e - r * S::RY;
    int gi = i0 - 1 + r, gj = j0 - 1 + c;
    bool ix = gi >= 0 && gi < nx, iy = gj >= 0 && gj < ny;
    if (!ix && per_x && iy) { gi = (gi + nx) % nx; ix = true; }
    if (!iy && per_y && ix) { gj = (gj + ny) % ny; iy = true; }
    T vb = T(0), vh = T(0), vqx = T(0), vqy = T(0);
    if (ix && iy) {
      const size_t k = (size_t)gi * ny + gj;
      vb = bP[k]; vh = hP[k]; vqx = qxP[k]; vqy = qyP[k];
    }
    s.b[e] = vb;
    s.h[e] = vh;
    s.qx[e] = vqx;
    s.qy[e] = vqy;
    s.hinv[e] = kp_hinv(vh, p.eps_kp);
  }
  __syncthreads();

  // ── faces ──
  // a cell's state with its velocities from the given hinv (a seam partner
  // takes the OWNER's: the flux pass hands the inner cell's aux to both sides
  // of a boundary face, solver_jax.py:827-866)
  auto side = [&](int e, T hinv, Side<T>& sd) {
    sd.b = s.b[e];
    sd.h = s.h[e];
    sd.qx = s.qx[e];
    sd.qy = s.qy[e];
    sd.ux = sd.qx * hinv;
    sd.uy = sd.qy * hinv;
  };
  auto face = [&](auto axis_tag, int eL, int eR, bool lo, bool hi, int kind, T& Fh, T& Ft, T& l,
                  T& r) {
    constexpr int AX = decltype(axis_tag)::value;
    Side<T> A, B;
    T Fx, Fy, Dm, Dp;
    if (lo || hi) {
      const int eo = lo ? eR : eL;
      const T sg = lo ? T(-1) : T(1);
      side(eo, s.hinv[eo], A);
      if (kind == ZB_BC_PERIODIC) {
        side(lo ? eL : eR, s.hinv[eo], B);
      } else {
        B = A;
        if (kind == ZB_BC_WALL) {   // q - 2 (q.n) n
          if (AX == 0) { B.qx = -A.qx; B.ux = -A.ux; }
          else { B.qy = -A.qy; B.uy = -A.uy; }
        }
      }
      riemann<T, RIEMANN, AX>(A, B, sg, g, Fh, Fx, Fy, Dm, Dp);
      const T Fn = AX == 0 ? Fx : Fy, Ftr = AX == 0 ? Fy : Fx;
      const T own_n = Fn + Dm * sg;
      Fh = lo ? -Fh : Fh;
      Ft = lo ? -Ftr : Ftr;
      r = lo ? own_n : T(0);
      l = lo ? T(0) : own_n;
    } else {
      side(eL, s.hinv[eL], A);
      side(eR, s.hinv[eR], B);
      riemann<T, RIEMANN, AX>(A, B, T(1), g, Fh, Fx, Fy, Dm, Dp);
      const T Fn = AX == 0 ? Fx : Fy;
      Ft = AX == 0 ? Fy : Fx;
      l = Fn + Dm;
      r = -Fn + Dp;
    }
  };
  for (int e = tid; e < S::NFX; e += NT) {
    const int fi = e / TY, fj = e - fi * TY;
    const int gi = i0 + fi, gj = j0 + fj;
    if (gj >= ny || gi > nx) continue;
    const int eL = fi * S::RY + (fj + 1);
    face(std::integral_constant<int, 0>(), eL, eL + S::RY, gi == 0, gi == nx,
         p.bc[gi == 0 ? 0 : 1], s.fxh[e], s.fxt[e], s.fxl[e], s.fxr[e]);
  }
  for (int e = tid; e < S::NFY; e += NT) {
    const int fi = e / (TY + 1), fj = e - fi * (TY + 1);
    const int gi = i0 + fi, gj = j0 + fj;
    if (gi >= nx || gj > ny) continue;
    const int eL = (fi + 1) * S::RY + fj;
    face(std::integral_constant<int, 1>(), eL, eL + 1, gj == 0, gj == ny, p.bc[gj == 0 ? 2 : 3],
         s.fyh[e], s.fyt[e], s.fyl[e], s.fyr[e]);
  }
  __syncthreads();

  // ── divergence, stage update, epilogue ──
  double amax_loc = 0.0;
  bool bad = false;
  for (int e = tid; e < TX * TY; e += NT) {
    const int ti = e / TY, tj = e - ti * TY;
    const int gi = i0 + ti, gj = j0 + tj;
    if (gi >= nx || gj >= ny) continue;
    const int fl = ti * TY + tj, fr = fl + TY;
    const int fb = ti * (TY + 1) + tj, ft = fb + 1;
    const T kx = p.kx, ky = p.ky;
    const T dh = -(kx * (s.fxh[fr] - s.fxh[fl]) + ky * (s.fyh[ft] - s.fyh[fb]));
    const T dqx = -(kx * (s.fxl[fr] + s.fxr[fl]) + ky * (s.fyt[ft] - s.fyt[fb]));
    const T dqy = -(kx * (s.fxt[fr] - s.fxt[fl]) + ky * (s.fyl[ft] + s.fyr[fb]));
    const int e1 = (ti + 1) * S::RY + (tj + 1);
    const T hk = s.h[e1], qxk = s.qx[e1], qyk = s.qy[e1];
    T hn, qxn, qyn;
    const size_t k = (size_t)gi * ny + gj;
    if (MODE == MODE_EULER) {
      hn = hk + dt * dh;
      qxn = qxk + dt * dqx;
      qyn = qyk + dt * dqy;
      if (p.manning_n != T(0)) {
        // source as RK1 after the hyperbolic step with the step's input aux
        // (zoomy_jax/fvm/solver_jax.py:1129; ode.py:14-18)
        const T hi0 = kp_hinv(hk, p.eps_kp);
        const T qn = asqrt(qxn * qxn + qyn * qyn);
        const T kf = (-p.g) * (p.manning_n * p.manning_n) * qn * (hi0 * hi0) * cbrt(hi0);
        if (p.implicit_source) {
          const T den = T(1) + dt * (-kf);
          qxn = qxn / den;
          qyn = qyn / den;
        } else {
          qxn = qxn + dt * (qxn * kf);
          qyn = qyn + dt * (qyn * kf);
        }
      }
    } else {
      const T a = T(p.alpha), bt = T(p.beta);
      T sqx = dqx, sqy = dqy;
      if (hinv_src != nullptr && p.manning_n != T(0)) {
        // solver2 adds the source to the stage residual at Qk with the step's
        // aux (solver2/blocks.py:241-287, march.py:120-124)
        const T hi = hinv_src[k];
        const T qn = asqrt(qxk * qxk + qyk * qyk);
        const T kf = (-p.g) * (p.manning_n * p.manning_n) * qn * (hi * hi) * cbrt(hi);
        sqx = dqx + qxk * kf;
        sqy = dqy + qyk * kf;
      }
      const T h2 = hk + bt * dt * dh, qx2 = qxk + bt * dt * sqx, qy2 = qyk + bt * dt * sqy;
      if (p.alpha != 0.0) {
        const T h0 = h0P[k], qx0 = qx0P[k], qy0 = qy0P[k];
        hn = a * h0 + (T(1) - a) * h2;
        qxn = a * qx0 + (T(1) - a) * qx2;
        qyn = a * qy0 + (T(1) - a) * qy2;
      } else {
        hn = h2; qxn = qx2; qyn = qy2;
      }
    }
    hO[k] = hn;
    qxO[k] = qxn;
    qyO[k] = qyn;
    const bool tr = (hn < T(0)) || !isfinite(hn) || !isfinite(qxn) || !isfinite(qyn) ||
                    !isfinite(s.b[e1]);
    bad = bad || tr;
    if (trouble_out != nullptr) trouble_out[k] = tr ? 1 : 0;
    if (MODE == MODE_EULER) {
      const T hi = kp_hinv(hn, p.eps_kp);
      const T c = asqrt(g * fmx(hn, T(0)));
      const T lx = fabs(qxn * hi) + c, ly = fabs(qyn * hi) + c;
      amax_loc = nmax(amax_loc, (double)nmax(lx, ly));
    }
  }
  const unsigned anybad = __syncthreads_or(bad ? 1 : 0);
  if (anybad && tid == 0) atomicOr(&ctrl->status, (unsigned)ZB_ST_TROUBLED);
  if (MODE == MODE_EULER) {
    const double m = block_max_double(amax_loc, red);
    if (tid == 0) {
      atomic_max_pos_double(&ctrl->amax[(phase + 1) % 3], m);
      if (lead_block) atomicAdd(&ctrl->steps, 1u);
    }
  }
}

// ── the strip kernel ───────────────────────────────────────────────────────
// The order-2 stage organised for registers: one warp owns a strip of 32
// contiguous columns (28 outputs plus two halo columns on each side) and
// marches down its rows.  Each lane keeps a sliding window of three rows of W,
// the limited slopes of two rows and the last x-face's fluxes in registers; the
// column neighbours come from warp shuffles.  Every face is evaluated once.
constexpr int SX = 64;          // output rows per work item at most
constexpr int STRIP_NT = 128;   // four independent warps per CTA
constexpr int SXC_MAX = 32;     // output rows of the ensemble's longest boundary-strip item

template <typename T>
struct RowW {
  T b, w1, w2, w3, h, hinv;
  __device__ T w(int v) const { return v == 0 ? b : (v == 1 ? w1 : (v == 2 ? w2 : w3)); }
};

template <typename T, int RECON>
__device__ __forceinline__ void strip_trace(const RowW<T>& c, const T* sl, T o, Side<T>& sd) {
  const T vb = c.b + sl[0] * o, w1 = c.w1 + sl[1] * o;
  const T w2 = c.w2 + sl[2] * o, w3 = c.w3 + sl[3] * o;
  sd.b = vb;
  if (RECON == ZB_RECON_ETA) {
    const T eta = fmx(w1, vb);
    const T hf = eta - vb;
    sd.h = hf;
    sd.ux = w2;
    sd.uy = w3;
    sd.qx = w2 * hf;
    sd.qy = w3 * hf;
  } else {
    sd.h = w1;
    sd.qx = w2;
    sd.qy = w3;
    sd.ux = w2 * c.hinv;
    sd.uy = w3 * c.hinv;
  }
}

template <typename T>
__device__ __forceinline__ T shd(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <typename T>
__device__ __forceinline__ T shu(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }

// float2 arithmetic on the sm_100 paired-FP32 instructions (one issue slot for
// two lanes of the same operation)
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {   // a - b, one rounding
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// The x-face (rows r-2 | r-1) and the y-face (row r-2, this lane | next lane)
// of an interior strip row evaluated together as the two lanes of float2
// arithmetic: eta traces, the Audusse hydrostatic reconstruction, HLL with
// Davis speeds, the fluctuations and the cell-edge bed terms of riemann() and
// strip_trace() for ZB_RECON_ETA / ZB_RIEMANN_HLL_HR in float32.  Lane x is
// the x-face (normal velocity u, transverse v), lane y the y-face (normal v,
// transverse u).  Square roots, divisions and min / max stay per lane.
// Outputs as the scalar path names them: x-face Fh, Fy, fxl_n, fxr_n; y-face
// Gh, Gx, fyl_t, fyr_own.
// The next lane's row r-2 (the y-face's upper side): W, h and the y-slopes.
struct NextRow {
  float b, w1, w2, w3, h, s4, s5, s6, s7;
};
__device__ __forceinline__ NextRow next_row(const RowW<float>& R0, const float* slA) {
  NextRow n;
  n.b = shd(R0.b); n.w1 = shd(R0.w1); n.w2 = shd(R0.w2); n.w3 = shd(R0.w3); n.h = shd(R0.h);
  n.s4 = shd(slA[4]); n.s5 = shd(slA[5]); n.s6 = shd(slA[6]); n.s7 = shd(slA[7]);
  return n;
}

// The faces of a strip row that lie on the boundary: the x-face (rows r-2 | r-1) where xlo / xhi, the
// y-face where ylo (this lane is the ghost below column 0) / yhi (column
// ny - 1).  A boundary face takes the owner's trace on both sides, its normal
// velocity times sx / sy (-1: a wall mirrors it; +1: extrapolation) on the
// ghost's; a periodic side passes no flag (its ghost lanes and rows hold the
// partner cell with zero slopes).
struct EdgeFaces {
  bool xlo, xhi, ylo, yhi;
  float sx, sy;
};

template <bool EDGE, typename P>
__device__ __forceinline__ void faces_pair(const RowW<float>& R0, const RowW<float>& R1,
                                           const float* slA, const float* slB,
                                           const NextRow& nx_, const P& p,
                                           const EdgeFaces& ef, float& Fh, float& Fy, float& fxl_n, float& fxr_n,
                                           float& Gh, float& Gx, float& fyl_t, float& fyr_own) {
  const float g = p.g, hg = 0.5f * g;
  const float nb_b = nx_.b, nb_w1 = nx_.w1, nb_w2 = nx_.w2, nb_w3 = nx_.w3, nb_h = nx_.h;
  const float sn4 = nx_.s4, sn5 = nx_.s5, sn6 = nx_.s6, sn7 = nx_.s7;
  const float2 o1 = f2(p.half_dx, p.half_dy), o2 = f2(-o1.x, -o1.y);
  // side 1: row r-2 towards +x (x-face) and towards +y (y-face)
  float2 b1 = fma2(f2(slA[0], slA[4]), o1, f2(R0.b, R0.b));
  const float2 e1 = fma2(f2(slA[1], slA[5]), o1, f2(R0.w1, R0.w1));
  float2 un1 = fma2(f2(slA[2], slA[7]), o1, f2(R0.w2, R0.w3));
  float2 ut1 = fma2(f2(slA[3], slA[6]), o1, f2(R0.w3, R0.w2));
  float2 h1 = sub2(f2(fmaxf(e1.x, b1.x), fmaxf(e1.y, b1.y)), b1);   // Audusse clip
  // side 2: row r-1 towards -x and the next lane's row r-2 towards -y
  float2 b2 = fma2(f2(slB[0], sn4), o2, f2(R1.b, nb_b));
  const float2 e2 = fma2(f2(slB[1], sn5), o2, f2(R1.w1, nb_w1));
  float2 un2 = fma2(f2(slB[2], sn7), o2, f2(R1.w2, nb_w3));
  float2 ut2 = fma2(f2(slB[3], sn6), o2, f2(R1.w3, nb_w2));
  float2 h2 = sub2(f2(fmaxf(e2.x, b2.x), fmaxf(e2.y, b2.y)), b2);
  if (EDGE) {
    // x: uniform over the warp
    if (ef.xlo) { b1.x = b2.x; h1.x = h2.x; un1.x = ef.sx * un2.x; ut1.x = ut2.x; }
    if (ef.xhi) { b2.x = b1.x; h2.x = h1.x; un2.x = ef.sx * un1.x; ut2.x = ut1.x; }
    // y: the lane below column 0 and the lane of column ny - 1
    b1.y = ef.ylo ? b2.y : b1.y; h1.y = ef.ylo ? h2.y : h1.y;
    un1.y = ef.ylo ? ef.sy * un2.y : un1.y; ut1.y = ef.ylo ? ut2.y : ut1.y;
    b2.y = ef.yhi ? b1.y : b2.y; h2.y = ef.yhi ? h1.y : h2.y;
    un2.y = ef.yhi ? ef.sy * un1.y : un2.y; ut2.y = ef.yhi ? ut1.y : ut2.y;
  }
  // hydrostatic reconstruction
  const float2 bs = f2(fmaxf(b1.x, b2.x), fmaxf(b1.y, b2.y));
  const float2 t1 = sub2(add2(h1, b1), bs), t2 = sub2(add2(h2, b2), bs);
  const float2 hL = f2(fmaxf(0.f, t1.x), fmaxf(0.f, t1.y));
  const float2 hR = f2(fmaxf(0.f, t2.x), fmaxf(0.f, t2.y));
  const float2 gg = f2(g, g), hg2 = f2(hg, hg), m1 = f2(-1.f, -1.f);
  const float2 ghL = mul2(gg, hL), ghR = mul2(gg, hR);
  const float2 cL = f2(sqrtf(ghL.x), sqrtf(ghL.y)), cR = f2(sqrtf(ghR.x), sqrtf(ghR.y));
  const float2 FLh = mul2(hL, un1), FRh = mul2(hR, un2);      // normal discharges
  const float2 qLt = mul2(hL, ut1), qRt = mul2(hR, ut2);      // transverse discharges
  const float2 FLn = fma2(FLh, un1, mul2(hg2, mul2(hL, hL)));
  const float2 FRn = fma2(FRh, un2, mul2(hg2, mul2(hR, hR)));
  const float2 FLt = mul2(qLt, un1), FRt = mul2(qRt, un2);
  // Davis speeds clipped at zero and the HLL combination
  const float2 sL1 = sub2(un1, cL), sL2 = sub2(un2, cR), sR1 = add2(un1, cL), sR2 = add2(un2, cR);
  const float2 sl = f2(fmn3(sL1.x, sL2.x, 0.f), fmn3(sL1.y, sL2.y, 0.f));
  const float2 sr = f2(fmx3(sR1.x, sR2.x, 0.f), fmx3(sR1.y, sR2.y, 0.f));
  const float2 den = sub2(sr, sl);
  const float2 inv = f2(den.x > 0.f ? __fdividef(1.f, den.x) : 0.f,
                        den.y > 0.f ? __fdividef(1.f, den.y) : 0.f);
  const float2 slsr = mul2(sl, sr), nsl = mul2(sl, m1);
  auto hll = [&](float2 FL, float2 FR, float2 d) {
    return mul2(fma2(slsr, d, fma2(nsl, FR, mul2(sr, FL))), inv);
  };
  const float2 Fh2 = hll(FLh, FRh, sub2(hR, hL));
  const float2 Fn2 = hll(FLn, FRn, sub2(FRh, FLh));
  const float2 Ft2 = hll(FLt, FRt, sub2(qRt, qLt));
  // fluctuations of the reconstruction and the cell-edge bed terms
  const float2 Dm2 = mul2(hg2, fma2(mul2(hL, m1), hL, mul2(h1, h1)));
  const float2 Dp2 = mul2(f2(-hg, -hg), fma2(mul2(hR, m1), hR, mul2(h2, h2)));
  const float2 ces1 = mul2(mul2(hg2, add2(f2(R0.h, R0.h), h1)), sub2(b1, f2(R0.b, R0.b)));
  const float2 ces2 = mul2(mul2(f2(-hg, -hg), add2(f2(R1.h, nb_h), h2)), sub2(b2, f2(R1.b, nb_b)));
  const float2 fl = add2(add2(Fn2, Dm2), ces1);
  const float2 fr = add2(sub2(Dp2, Fn2), ces2);
  Fh = Fh2.x; Fy = Ft2.x; fxl_n = fl.x; fxr_n = fr.x;
  Gh = Fh2.y; Gx = Ft2.y; fyl_t = fl.y; fyr_own = fr.y;
}

// One warp's work item: strip `strip` (28 output columns from column 28 strip)
// over the output rows [r0, r1).  EDGE false, the interior body: every lane's
// cell two cells or more from every boundary.  EDGE true, the general body:
// any rows and columns of the grid.  It is the interior body with the boundary
// folded into per-lane and per-row selects, so that no lane runs a branch of
// its own:
//   * rows and columns outside the grid load zeros (wall, extrapolation) or
//     the periodic image;
//   * least-squares gradient: the 3x3 row and column sums leave out what lies
//     outside, the cell's own ghost enters as -/+ (ghost + 2 u) along its axis
//     and the normal matrix is diag(4 dx^2, 4 dy^2) in place of diag(6, 6)
//     (x of a side column sees five neighbours: 4 dx^2); the four corner cells,
//     whose matrix is not diagonal, take
//     g = s (2 d_n + d_diag - 2 d_ghost - d_t) / 5 along each axis, d the
//     differences to the inner neighbour along the axis, the diagonal one, the
//     ghost and the inner neighbour across it, s = +1 on the low side;
//   * bounds: the neighbour beyond a side is 2 ghost - u;
//   * faces: EdgeFaces.
// The branchy boundary bodies this replaces cost a column-boundary row 1.7 us
// of latency (one lane's slopes and face serially, a launch of its own beside
// the interior): 512^2 float32 27 us per step at best row heights, 64^2 25.
// `lead` (one item of the grid) keeps the control block.  MODE_STAGE: the
// generic Shu-Osher stage with a given dt, optional per-cell first-order mask,
// troubled-mask output and friction inside the stage (hinv_src).
// P: SweParams<T> in kernel-parameter space, or volatile in shared memory (the
// ensemble: fields read where they are used instead of held in registers).
template <typename T, int RECON, int RIEMANN, int MODE, bool EDGE, bool BEDT, typename P>
__device__ __forceinline__ void strip_item(const T* __restrict__ bP, const T* __restrict__ hP,
                                           const T* __restrict__ qxP, const T* __restrict__ qyP,
                                           const T* __restrict__ h0P,
                                           const T* __restrict__ qx0P,
                                           const T* __restrict__ qy0P, T* __restrict__ hO,
                                           T* __restrict__ qxO, T* __restrict__ qyO,
                                           zb_ctrl* ctrl, int phase, const P& p,
                                           const int strip, const int r0, const int r1,
                                           const bool lead, const T* __restrict__ hinv_src = nullptr,
                                           const unsigned char* __restrict__ force_o1 = nullptr,
                                           unsigned char* __restrict__ trouble_out = nullptr) {
  const int lane = threadIdx.x & 31;
  const int nx = p.nx, ny = p.ny;
  const int cj = strip * SW - 2 + lane;
  const bool cin = !EDGE || (cj >= 0 && cj < ny);
  double dtd;
  if (MODE == MODE_STAGE) {
    dtd = p.dt_stage >= 0.0 ? p.dt_stage : ctrl->dt;
  } else {
    const double t = ctrl->t[phase];
    dtd = dt_from_amax(ctrl->amax[phase], t, p.cfl2r, p.den_fac, p.dt_max, p.t_end);
    const bool ok = isfinite(dtd) && dtd > 0.0;
    if (lead && lane == 0) {
      // the duties of swe2d_stage_kernel's lead block
      const int nph = (phase + 1) % 3, nnph = (phase + 2) % 3;
      if (MODE == MODE_STEP1) {
        if (!ok && t < p.t_end) atomicOr(&ctrl->status, (unsigned)ZB_ST_DT_INVALID);
        ctrl->dt = ok ? dtd : 0.0;
        ctrl->t[nph] = ok ? t + dtd : t;
        ctrl->amax[nnph] = 0.0;
        ctrl->troubled = 0u;
      } else if (!ok) {
        ctrl->amax[nph] = ctrl->amax[phase];
      } else {
        atomicAdd(&ctrl->steps, 1u);
      }
    }
    if (!ok) return;                    // no-op step (t_end reached or dt invalid)
  }
  const T dt = T(dtd);
  const T g = p.g, half = T(0.5);
  const bool out_lane = lane >= 2 && lane < 2 + SW && cin;
  // float32 rows of the eta / HLL-HR scheme evaluate their two faces as paired
  // float32 arithmetic (faces_pair)
  constexpr bool PAIR = std::is_same<T, float>::value && RECON == ZB_RECON_ETA &&
                        RIEMANN == ZB_RIEMANN_HLL_HR;
  // BEDT: interior items of the eta / HLL-HR scheme read b's gradient and
  // limiter value from the planes swe2d_bed_kernel prepared (b never
  // changes) instead of evaluating them; the planes are laid out like the
  // state's
  constexpr bool BED = BEDT && !EDGE && RECON == ZB_RECON_ETA && RIEMANN == ZB_RIEMANN_HLL_HR;
  const T* __restrict__ bedP = p.bed;
  const size_t bed_plane = (size_t)nx * ny;
  // EDGE: the lane's column (its periodic image where the sides are periodic)
  // and what the boundary makes of it
  const bool per_x = EDGE && p.bc[0] == ZB_BC_PERIODIC, per_y = EDGE && p.bc[2] == ZB_BC_PERIODIC;
  const bool byl = EDGE && cj == 0, byh = EDGE && cj == ny - 1, by = byl || byh;
  const bool wall_y = by && p.bc[byl ? 2 : 3] == ZB_BC_WALL;
  int lc = cj;
  bool cld = cin;
  if (EDGE && per_y && !cin) {
    lc = cj % ny;
    if (lc < 0) lc += ny;
    cld = true;
  }
  // the row the lane loads for row index r (the periodic image), -1: none
  auto load_row = [&](int r) -> int {
    if (!EDGE || (r >= 0 && r < nx)) return r;
    if (!per_x) return -1;
    const int w = r % nx;
    return w < 0 ? w + nx : w;
  };

  RowW<T> R0, R1, R2;                 // rows r-2, r-1, r
  T Sx0[4], Sx1[4], Sx2[4];           // (W(j-1) + W(j)) + W(j+1) of those rows
  T Wm1[4], Wp1[4], Wm2[4], Wp2[4];   // W(j-1), W(j+1) of rows r-1 and r
  T slA[8], slB[8];                   // [sx0..3, sy0..3] of rows r-2 and r-1
  T fxh_p = T(0), fxt_p = T(0), fxr_p = T(0);
  T amax_loc = T(0);   // reduced in T; float -> double is exact and monotone
  bool bad = false;
  const int nsteps = (r1 - r0) + 4;
  const int limiter = p.limiter;
  const bool clipmin = limiter != ZB_LIM_NONE && limiter != ZB_LIM_VENKATAKRISHNAN;
  // row r + 1 is fetched while row r is processed
  T nbv = T(0), nhv = T(0), nqxv = T(0), nqyv = T(0);
  T nbgx = T(0), nbgy = T(0), nbphi = T(0);   // BED: the next slope row's bed values
  {
    const int lr = load_row(r0 - 2);
    if (!EDGE || (cld && lr >= 0)) {
      const size_t k = (size_t)lr * ny + lc;
      nbv = bP[k]; nhv = hP[k]; nqxv = qxP[k]; nqyv = qyP[k];
    }
  }
  for (int s = 0; s < nsteps; ++s) {
    const int r = r0 - 2 + s;
    // the update of row r - 2 at the end of this iteration reads these: issue
    // the loads now so their latency overlaps the slope and face work
    const int ro = r - 2;
    const bool upd = s >= 4 && out_lane && ro >= r0 && ro < r1;
    T qxk = T(0), qyk = T(0), h0 = T(0), qx0 = T(0), qy0 = T(0), hsrc = T(0);
    if (upd) {
      const size_t k = (size_t)ro * ny + cj;
      if (RECON == ZB_RECON_ETA) { qxk = qxP[k]; qyk = qyP[k]; }
      if (MODE == MODE_STEP2 || (MODE == MODE_STAGE && p.alpha != 0.0)) {
        h0 = h0P[k]; qx0 = qx0P[k]; qy0 = qy0P[k];
      }
      if (MODE == MODE_STAGE && hinv_src != nullptr) hsrc = hinv_src[k];
    }
    // the bed slopes of row r - 1 (the slope block below), fetched in the
    // previous iteration; fetch row r's for the next one
    const T bgx = nbgx, bgy = nbgy, bphi = nbphi;
    if (BED && s >= 1 && r <= r1) {
      const size_t k = (size_t)r * ny + cj;   // BED: interior items, no guards
      nbgx = __ldg(bedP + k);
      nbgy = __ldg(bedP + bed_plane + k);
      nbphi = __ldg(bedP + 2 * bed_plane + k);
    }
    bool o1 = false;   // MODE_STAGE: the cell of row r - 1 is demoted to first order
    if (MODE == MODE_STAGE && force_o1 != nullptr && s >= 2 && cin && r - 1 >= 0 && r - 1 < nx)
      o1 = force_o1[(size_t)(r - 1) * ny + cj] != 0;
    // shift the windows and take row r
    R0 = R1; R1 = R2;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      Sx0[v] = Sx1[v]; Sx1[v] = Sx2[v];
      Wm1[v] = Wm2[v]; Wp1[v] = Wp2[v];
    }
    {
      const T vb = nbv, vh = nhv, vqx = nqxv, vqy = nqyv;
      if (s + 1 < nsteps) {
        const int lr = load_row(r + 1);
        if (!EDGE || (cld && lr >= 0)) {
          const size_t k = (size_t)lr * ny + lc;
          nbv = bP[k]; nhv = hP[k]; nqxv = qxP[k]; nqyv = qyP[k];
        } else {
          nbv = T(0); nhv = T(0); nqxv = T(0); nqyv = T(0);
        }
      }
      const T hinv = kp_hinv(vh, p.eps_kp);
      R2.b = vb;
      R2.h = vh;
      R2.hinv = hinv;
      if (RECON == ZB_RECON_ETA) {
        R2.w1 = vb + vh;
        R2.w2 = vqx * hinv;
        R2.w3 = vqy * hinv;
      } else {
        R2.w1 = vh;
        R2.w2 = vqx;
        R2.w3 = vqy;
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (v == 0 && BED) continue;   // b's windows feed only its slope
        const T w = R2.w(v);
        const T wl = shu(w), wr = shd(w);
        Wm2[v] = wl;
        Wp2[v] = wr;
        Sx2[v] = EDGE ? ((byl ? T(0) : wl) + w) + (byh ? T(0) : wr) : (wl + w) + wr;
      }
    }
    if (s < 2) continue;
    // limited slopes of row r-1
    {
      const int m = r - 1;
      const bool bxl = EDGE && m == 0, bxh = EDGE && m == nx - 1, bx = bxl || bxh;   // uniform
      T phi[4], gxa[4], gya[4], dposa[4], dnega[4];
      // x and y scale of the differences
      const T ix = (EDGE && (by || bx)) ? p.inv4dx : p.inv6dx;
      const T iy = (EDGE && (by || bx)) ? p.inv4dy : p.inv6dy;
      // gradient and bounds of variable v; BX: a boundary row.  The choice of the row is
      // made once for the four variables, so that they run side by side (64^2 solve, all
      // items in this body, 701 -> 679 us; 517 x 389 float32 236 -> 226)
      auto slope = [&](auto BXT, int v) {
        constexpr bool BX = decltype(BXT)::value;
        const T u = R1.w(v);
        T wp0 = R2.w(v), wm0 = R0.w(v), w0p = Wp1[v], w0m = Wm1[v];
        T xhi = Sx2[v], xlo = Sx0[v];       // gx = (xhi - xlo) / ..
        const T tc = BX ? (bxl ? u + wp0 : wm0 + u) : (wm0 + u) + wp0;
        T tl = shu(tc), tr = shd(tc);       // gy = (tr - tl) / ..
        T cgx = T(0), cgy = T(0);           // corner cells: the gradient itself
        if (EDGE) {
          // y: the side's ghost
          const T gyv = per_y ? (byl ? w0m : w0p) : ((v == 3 && wall_y) ? -u : u);
          const T cy = gyv + T(2) * u, gg = T(2) * gyv - u;
          if constexpr (BX) {
            // x: the side's ghost row; the corner cells
            const T gxv = per_x ? (bxl ? wm0 : wp0)
                                : ((v == 2 && p.bc[bxl ? 0 : 1] == ZB_BC_WALL) ? -u : u);
            const T wn = bxl ? wp0 : wm0;                       // inner neighbour along x
            const T ra = shu(wn), rb = shd(wn);
            const T wt = byl ? w0p : w0m, wd = byl ? rb : ra;   // across, diagonal
            const T dn = wn - u, dt_ = wt - u, dd = wd - u;
            cgx = (T(2) * dn + dd - T(2) * (gxv - u) - dt_) * p.inv5dx;
            cgy = (T(2) * dt_ + dd - T(2) * (gyv - u) - dn) * p.inv5dy;
            cgx = bxl ? cgx : -cgx;
            cgy = byl ? cgy : -cgy;
            const T cx = gxv + T(2) * u, ggx = T(2) * gxv - u;
            if (bxl) { xlo = cx; wm0 = ggx; }
            else { xhi = cx; wp0 = ggx; }
          }
          tl = byl ? cy : tl;
          tr = byh ? cy : tr;
          w0m = byl ? gg : w0m;
          w0p = byh ? gg : w0p;
        }
        const T umax = fmx3(u, wp0, fmx3(wm0, w0p, w0m));
        const T umin = fmn3(u, wp0, fmn3(wm0, w0p, w0m));
        T gx, gy, dpos, dneg;
        if constexpr (PAIR) {
          // the x and y components as the two lanes of paired float32
          // arithmetic
          const float2 gv = mul2(sub2(f2(xhi, tr), f2(xlo, tl)), f2(ix, iy));
          const float2 dd = sub2(f2(umax, umin), f2(u, u));
          gx = gv.x; gy = gv.y; dpos = dd.x; dneg = dd.y;
        } else {
          gx = (xhi - xlo) * ix;
          gy = (tr - tl) * iy;
          dpos = umax - u;
          dneg = umin - u;
        }
        if constexpr (BX) {
          gx = by ? cgx : gx;
          gy = by ? cgy : gy;
        }
        gxa[v] = gx;
        gya[v] = gy;
        dposa[v] = dpos;
        dnega[v] = dneg;
      };
      if (BED) {
        gxa[0] = bgx;
        gya[0] = bgy;
        phi[0] = bphi;
      }
      bool plain = true;
      if constexpr (EDGE) {
        if (bx) {
          plain = false;
#pragma unroll
          for (int v = 0; v < 4; ++v) slope(std::true_type(), v);
        }
      }
      if (plain) {
#pragma unroll
        for (int v = BED ? 1 : 0; v < 4; ++v) slope(std::false_type(), v);
      }
      // One choice of the limiter for the four variables, so that their quotients run
      // side by side: a warp waits for dependent instructions most of its time (float64:
      // issue 55 %), and a branch per variable kept the four chains apart.  2048^2
      // float64, three steps, 1723 -> 1585 us, float32, six, 1085 -> 1060; 64 instances
      // 1396 -> 1301.
      if (clipmin) {
#pragma unroll
        for (int v = BED ? 1 : 0; v < 4; ++v) {
          if constexpr (PAIR) {
            const float2 ac = mul2(f2(gxa[v], gya[v]), f2(p.half_dx, p.half_dy));
            phi[v] = phi_clipmin(ac.x, ac.y, dposa[v], dnega[v]);
          } else {
            phi[v] = phi_clipmin(gxa[v] * p.half_dx, gya[v] * p.half_dy, dposa[v], dnega[v]);
          }
        }
      } else {
#pragma unroll
        for (int v = BED ? 1 : 0; v < 4; ++v)
          phi[v] = limiter_phi<T>(limiter, gxa[v], gya[v], p.half_dx, p.half_dy, dposa[v],
                                  dnega[v], p.vk_eps2);
      }
      if (RECON == ZB_RECON_ETA) {
        if (p.eps_wet >= T(0) && R1.h < p.eps_wet) {
          phi[0] = phi[1] = phi[2] = phi[3] = T(0);
        }
        phi[0] = zmin(phi[0], phi[1]);
        phi[2] = zmin(phi[2], phi[1]);
        phi[3] = zmin(phi[3], phi[1]);
      }
      // ghosts (a periodic partner enters the seam's faces unreconstructed)
      // and demoted cells have no slopes
      if ((EDGE && (!cin || m < 0 || m >= nx)) || (MODE == MODE_STAGE && o1)) {
#pragma unroll
        for (int v = 0; v < 4; ++v) { phi[v] = T(0); gxa[v] = T(0); gya[v] = T(0); }
      }
#pragma unroll
      for (int v = 0; v < 8; ++v) slA[v] = slB[v];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if constexpr (PAIR) {
          const float2 sv = mul2(f2(phi[v], phi[v]), f2(gxa[v], gya[v]));
          slB[v] = sv.x;
          slB[4 + v] = sv.y;
        } else {
          slB[v] = phi[v] * gxa[v];
          slB[4 + v] = phi[v] * gya[v];
        }
      }
    }
    if (s < 3) continue;
    // the x-face between rows r-2 (A, lower) and r-1 (B, upper) and the y-face
    // of row r-2 above this lane (the lower lane's is the one below)
    T Fh, Fy, fxl_n, fxr_n, Gh, Gx, fyl_t, fyr_own;
    {
      EdgeFaces ef = {false, false, false, false, 1.0f, 1.0f};
      if (EDGE) {
        ef.xlo = !per_x && r - 1 == 0;
        ef.xhi = !per_x && r - 2 == nx - 1;
        ef.ylo = !per_y && cj == -1;
        ef.yhi = !per_y && cj == ny - 1;
        ef.sx = p.bc[ef.xlo ? 0 : 1] == ZB_BC_WALL ? -1.0f : 1.0f;
        ef.sy = p.bc[ef.ylo ? 2 : 3] == ZB_BC_WALL ? -1.0f : 1.0f;
      }
      if constexpr (PAIR) {
        const NextRow nv = next_row(R0, slA);
        faces_pair<EDGE, P>(R0, R1, slA, slB, nv, p, ef, Fh, Fy, fxl_n, fxr_n, Gh, Gx, fyl_t, fyr_own);
        if (s == 3) {          // face r0 - 1/2: only the next row needs it
          fxh_p = Fh; fxt_p = Fy; fxr_p = fxr_n;
          continue;
        }
      } else {
        T Fx, Dm, Dp;
        RowW<T> LA = R0, LB = R1;
        if (EDGE && per_x && RECON != ZB_RECON_ETA) {
          // a seam partner's velocity is its momentum times the owner's hinv
          if (r - 1 == 0) LA.hinv = R1.hinv;
          if (r - 2 == nx - 1) LB.hinv = R0.hinv;
        }
        Side<T> A, B;
        strip_trace<T, RECON>(LA, slA, p.half_dx, A);
        strip_trace<T, RECON>(LB, slB, -p.half_dx, B);
        if (EDGE && (ef.xlo || ef.xhi)) {   // uniform
          Side<T> O = ef.xlo ? B : A;
          O.qx *= T(ef.sx);
          O.ux *= T(ef.sx);
          if (ef.xlo) A = O;
          else B = O;
        }
        riemann<T, RIEMANN, 0>(A, B, T(1), g, Fh, Fx, Fy, Dm, Dp);
        const T cesA = half * g * (R0.h + A.h) * (A.b - R0.b);
        const T cesB = -(half * g * (R1.h + B.h) * (B.b - R1.b));
        fxl_n = Fx + Dm + cesA;
        fxr_n = -Fx + Dp + cesB;
        if (s == 3) {            // face r0 - 1/2: only the next row needs it
          fxh_p = Fh; fxt_p = Fy; fxr_p = fxr_n;
          continue;
        }
        // y-face of row r-2: this lane | the next lane
        Side<T> C, D;
        T Gy, Em, Ep;
        RowW<T> nb, own = R0;
        nb.b = shd(R0.b); nb.w1 = shd(R0.w1); nb.w2 = shd(R0.w2); nb.w3 = shd(R0.w3);
        nb.h = shd(R0.h); nb.hinv = shd(R0.hinv);
        if (EDGE && per_y && RECON != ZB_RECON_ETA) {
          if (cj == -1) own.hinv = nb.hinv;
          if (cj == ny - 1) nb.hinv = own.hinv;
        }
        T sln[8];
#pragma unroll
        for (int v = 0; v < 4; ++v) sln[4 + v] = shd(slA[4 + v]);
        strip_trace<T, RECON>(own, slA + 4, p.half_dy, C);
        strip_trace<T, RECON>(nb, sln + 4, -p.half_dy, D);
        if (EDGE) {
          const T sy = T(ef.sy);
          const Side<T> O = ef.ylo ? D : C;
          C.b = ef.ylo ? O.b : C.b;
          C.h = ef.ylo ? O.h : C.h;
          C.qx = ef.ylo ? O.qx : C.qx;
          C.ux = ef.ylo ? O.ux : C.ux;
          C.qy = ef.ylo ? sy * O.qy : C.qy;
          C.uy = ef.ylo ? sy * O.uy : C.uy;
          D.b = ef.yhi ? O.b : D.b;
          D.h = ef.yhi ? O.h : D.h;
          D.qx = ef.yhi ? O.qx : D.qx;
          D.ux = ef.yhi ? O.ux : D.ux;
          D.qy = ef.yhi ? sy * O.qy : D.qy;
          D.uy = ef.yhi ? sy * O.uy : D.uy;
        }
        riemann<T, RIEMANN, 1>(C, D, T(1), g, Gh, Gx, Gy, Em, Ep);
        const T cesC = half * g * (R0.h + C.h) * (C.b - R0.b);
        const T cesD = -(half * g * (nb.h + D.h) * (D.b - nb.b));
        fyl_t = Gy + Em + cesC;
        fyr_own = -Gy + Ep + cesD;
      }
      const T fyh_b = shu(Gh), fyt_b = shu(Gx), fyr_b = shu(fyr_own);
      // update of row r-2
      const T kx = p.kx, ky = p.ky;
      const T dh = -(kx * (Fh - fxh_p) + ky * (Gh - fyh_b));
      const T dqx = -(kx * (fxl_n + fxr_p) + ky * (Gx - fyt_b));
      const T dqy = -(kx * (Fy - fxt_p) + ky * (fyl_t + fyr_b));
      fxh_p = Fh; fxt_p = Fy; fxr_p = fxr_n;
      if (!upd) continue;
      const size_t k = (size_t)ro * ny + cj;
      const T hk = R0.h;
      if (RECON != ZB_RECON_ETA) {
        qxk = R0.w2;
        qyk = R0.w3;
      }
      T hn, qxn, qyn;
      if (MODE == MODE_STEP1) {
        hn = hk + dt * dh;
        qxn = qxk + dt * dqx;
        qyn = qyk + dt * dqy;
      } else if (MODE == MODE_STAGE) {
        const T al = T(p.alpha), bt = T(p.beta);
        T sqx = dqx, sqy = dqy;
        if (hinv_src != nullptr && p.manning_n != T(0)) {
          // solver2 adds the source to the stage residual at Qk with the
          // step's aux (solver2/blocks.py:241-287, march.py:120-124)
          const T qn = asqrt(qxk * qxk + qyk * qyk);
          const T kf = (-p.g) * (p.manning_n * p.manning_n) * qn * (hsrc * hsrc) * cbrt(hsrc);
          sqx = dqx + qxk * kf;
          sqy = dqy + qyk * kf;
        }
        const T h2 = hk + bt * dt * dh, qx2 = qxk + bt * dt * sqx, qy2 = qyk + bt * dt * sqy;
        if (p.alpha != 0.0) {
          hn = al * h0 + (T(1) - al) * h2;
          qxn = al * qx0 + (T(1) - al) * qx2;
          qyn = al * qy0 + (T(1) - al) * qy2;
        } else {
          hn = h2; qxn = qx2; qyn = qy2;
        }
      } else {
        const T h2 = hk + dt * dh, qx2 = qxk + dt * dqx, qy2 = qyk + dt * dqy;
        hn = half * (h0 + h2);
        qxn = half * (qx0 + qx2);
        qyn = half * (qy0 + qy2);
        if (p.manning_n != T(0)) {
          // source as RK1 after the hyperbolic step with the step's input aux
          // (zoomy_jax/fvm/solver_jax.py:1129; ode.py:14-18)
          const T hi0 = kp_hinv(h0, p.eps_kp);
          const T qn = asqrt(qxn * qxn + qyn * qyn);
          const T kf = (-p.g) * (p.manning_n * p.manning_n) * qn * (hi0 * hi0) * cbrt(hi0);
          if (p.implicit_source) {
            const T den = T(1) + dt * (-kf);
            qxn = qxn / den;
            qyn = qyn / den;
          } else {
            qxn = qxn + dt * (qxn * kf);
            qyn = qyn + dt * (qyn * kf);
          }
        }
      }
      hO[k] = hn;
      qxO[k] = qxn;
      qyO[k] = qyn;
      if (MODE == MODE_STAGE) {
        const bool tr = (hn < T(0)) || !isfinite(hn) || !isfinite(qxn) || !isfinite(qyn) ||
                        !isfinite(R0.b);
        bad = bad || tr;
        if (trouble_out != nullptr) trouble_out[k] = tr ? 1 : 0;
      } else {
        // troubled: h < 0 or a non-finite value (one non-finite term makes
        // the sum's difference with itself NaN; finite states that overflow
        // the sum, |q| ~ 1e38, would flag too)
        const T chk = (hn + qxn) + (qyn + R0.b);
        bad = bad || !(hn >= T(0)) || !(chk - chk == T(0));
      }
      if (MODE == MODE_STEP2) {
        const T hi = kp_hinv(hn, p.eps_kp);
        const T c = asqrt(g * fmx(hn, T(0)));
        const T lx = fabs(qxn * hi) + c, ly = fabs(qyn * hi) + c;
        amax_loc = nmax(amax_loc, nmax(lx, ly));
      }
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&ctrl->status, (unsigned)ZB_ST_TROUBLED);
  if (MODE == MODE_STEP2) {
    for (int o = 16; o > 0; o >>= 1)
      amax_loc = nmax(amax_loc, __shfl_xor_sync(0xffffffffu, amax_loc, o));
    if (lane == 0) atomic_max_pos_double(&ctrl->amax[(phase + 1) % 3], (double)amax_loc);
  }
}

// Work items of a grid with nx, ny >= 3 (strips of SW columns from column 0).
// The strips whose lanes reach outside the grid (the first, and the last one
// or two) go in chunks of sxc rows; every other strip has two items for the
// rows [0, 2) and [nx - 2, nx) -- these are the boundary items, for the general
// body -- and sx-row chunks of the rows between for the interior body.  Order:
// interior items, boundary strips, boundary rows.  Item 0 keeps the control
// block.  Returns the item count (item = -1), the count of boundary items
// (item = -2), or with item >= 0 fills its strip, rows and kind (1 boundary, 0
// interior).
constexpr int SXC_ENS = 32;
__host__ __device__ inline int full_items(int nx, int ny, int item, int* strip, int* r0,
                                          int* r1, int* kind, int sxc, int sx) {
  const int ns = (ny + SW - 1) / SW;
  const int nmid = full_mid_strips(ny);   // middle strips: 1 <= s <= nmid
  const int nedge = ns - nmid;
  const int nint = nx > 4 ? nmid * ((nx - 4 + sx - 1) / sx) : 0;
  const int ncc = (nx + sxc - 1) / sxc;
  const int nside = nedge * ncc + 2 * nmid;
  if (item == -2) return nside;
  if (item < 0) return nint + nside;
  int st, a, b, k = 1;
  if (item < nint) {
    st = 1 + item % nmid;
    a = 2 + (item / nmid) * sx;
    b = a + sx < nx - 2 ? a + sx : nx - 2;
    k = 0;
  } else if ((item -= nint) < nedge * ncc) {
    const int e = item / ncc;                // boundary strips: 0, nmid + 1, ..., ns - 1
    st = e == 0 ? 0 : nmid + e;
    a = (item % ncc) * sxc;
    b = a + sxc < nx ? a + sxc : nx;
  } else {
    item -= nedge * ncc;
    st = 1 + (item >> 1);
    a = (item & 1) ? (nx - 2 > 2 ? nx - 2 : 2) : 0;
    b = (item & 1) ? nx : 2;
  }
  *strip = st;
  *r0 = a;
  *r1 = b;
  *kind = k;
  return nint + nside;
}

// One stage of a grid: a warp per item, the interior or the general body by
// the item's kind (p.single: the general body for all), both bodies in one
// launch.  BED: the interior items read the prepared bed planes (p.bed).
// float32: 4 CTAs of 4 warps per SM (128 registers; the bodies spill at 96).
template <typename T, int RECON, int RIEMANN, int MODE, bool BED>
__global__ void __launch_bounds__(STRIP_NT, sizeof(T) == 4 ? 4 : 2)
swe2d_strip_kernel(const T* __restrict__ bP, const T* __restrict__ hP,
                   const T* __restrict__ qxP, const T* __restrict__ qyP,
                   const T* __restrict__ h0P, const T* __restrict__ qx0P,
                   const T* __restrict__ qy0P, T* __restrict__ hO, T* __restrict__ qxO,
                   T* __restrict__ qyO, zb_ctrl* ctrl, int phase,
                   const T* __restrict__ hinv_src, const unsigned char* __restrict__ force_o1,
                   unsigned char* __restrict__ trouble_out, const SweParams<T> p) {
  const int item = blockIdx.x * (STRIP_NT / 32) + (threadIdx.x >> 5);
  const bool lead = item == 0;
  int strip, r0, r1, kind = 1;
  if (p.single) {
    const int ns = (p.ny + SW - 1) / SW;
    strip = item % ns;
    r0 = (item / ns) * p.sx;
    r1 = min(r0 + p.sx, p.nx);
    if (r0 >= p.nx) return;   // warp-uniform
  } else {
    if (item >= full_items(p.nx, p.ny, -1, nullptr, nullptr, nullptr, nullptr, p.sxc, p.sx))
      return;
    full_items(p.nx, p.ny, item, &strip, &r0, &r1, &kind, p.sxc, p.sx);
  }
  pdl_enter();
  if (kind)
    strip_item<T, RECON, RIEMANN, MODE, true, false>(
        bP, hP, qxP, qyP, h0P, qx0P, qy0P, hO, qxO, qyO, ctrl, phase, p, strip, r0, r1, lead,
        hinv_src, force_o1, trouble_out);
  else
    strip_item<T, RECON, RIEMANN, MODE, false, BED>(
        bP, hP, qxP, qyP, h0P, qx0P, qy0P, hO, qxO, qyO, ctrl, phase, p, strip, r0, r1, lead,
        hinv_src, force_o1, trouble_out);
}

// ── batched ensemble: one launch per stage over all instances ───────────────
// Each instance is an independent Cartesian grid with its own size, spacing,
// Manning coefficient, dt and control block; the work list holds the strip
// items of every instance, so the whole ensemble advances one stage per launch.
template <typename T>
struct EnsDesc {
  SweParams<T> p;
  long long q_off;   // element offset of the instance's (4, C) state
  long long ws_off;  // element offset of its (3, C) stage buffer
};

// One strip item of an instance: stage 1 reads Q and writes the stage buffer,
// stage 2 reads the stage buffer and Q0 = Q and writes Q.
template <typename T, int MODE, bool EDGE>
__device__ __forceinline__ void ens_item(const volatile SweParams<T>& p, T* q, T* ws,
                                         zb_ctrl* ctrl, int phase, int strip, int r0, int r1,
                                         bool lead) {
  const size_t C = (size_t)p.nx * p.ny;
  if (MODE == MODE_STEP1)
    strip_item<T, ZB_RECON_ETA, ZB_RIEMANN_HLL_HR, MODE_STEP1, EDGE, false>(
        q, q + C, q + 2 * C, q + 3 * C, nullptr, nullptr, nullptr, ws, ws + C, ws + 2 * C,
        ctrl, phase, p, strip, r0, r1, lead);
  else
    strip_item<T, ZB_RECON_ETA, ZB_RIEMANN_HLL_HR, MODE_STEP2, EDGE, false>(
        q, ws, ws + C, ws + 2 * C, q + C, q + 2 * C, q + 3 * C, q + C, q + 2 * C, q + 3 * C,
        ctrl, phase, p, strip, r0, r1, lead);
}

// All instances' strip items, a warp per item: the interior items, then the
// boundary items, each list longest item first (the block scheduler fills the
// tail of the long ones with the short ones).  The work list's header items[0] =
// {interior items, boundary items}; the lists follow it.  A warp's instance
// parameters sit in shared memory: read from global memory they were held in
// registers and spilled (408 bytes a thread with both bodies in one kernel,
// 222 us a stage of 64 instances; now 8 in float32, none in float64).  The work
// list and the parameters are read before the wait for the launch before this one:
// zb_ens_prepare writes them with a copy that has landed when it returns, never a
// launch.
template <typename T, int MODE>
__global__ void __launch_bounds__(STRIP_NT, sizeof(T) == 4 ? 4 : 2)
ens_strip_kernel(const EnsDesc<T>* __restrict__ desc, const int4* __restrict__ items, T* Q,
                 T* W, zb_ctrl* ctrls, int phase) {
  __shared__ SweParams<T> par[STRIP_NT / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int4 hd = items[0];
  const int it = blockIdx.x * (STRIP_NT / 32) + warp;
  if (it >= hd.x + hd.y) return;
  // w = {instance, strip, r0, flags | r1 << 1}; flag bit 0 = the item keeps the
  // instance's control block
  const int4 w = items[1 + it];
  const EnsDesc<T>* d = desc + w.x;
  static_assert(sizeof(SweParams<T>) % 4 == 0, "copied by words");
  for (int k = lane; k < (int)(sizeof(SweParams<T>) / 4); k += 32)
    ((int*)&par[warp])[k] = ((const int*)&d->p)[k];
  __syncwarp();
  pdl_enter();
  const volatile SweParams<T>& p = par[warp];
  T* q = Q + d->q_off;
  T* ws = W + d->ws_off;
  if (it < hd.x)
    ens_item<T, MODE, false>(p, q, ws, ctrls + w.x, phase, w.y, w.z, w.w >> 1, (w.w & 1) != 0);
  else
    ens_item<T, MODE, true>(p, q, ws, ctrls + w.x, phase, w.y, w.z, w.w >> 1, (w.w & 1) != 0);
}

// A march's start: the control blocks, then the wave-speed maximum of every
// instance by AMAX_PARTS CTAs (one CTA per instance left the largest ones to a
// single SM: 64 instances of 64^2 .. 512^2 475 us, now 16).
constexpr int AMAX_PARTS = 16;

__global__ void ens_ctrl_init_kernel(zb_ctrl* ctrls, int n_inst, int phase, double t0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_inst) return;
  zb_ctrl* ctrl = ctrls + i;
  for (int j = 0; j < 3; ++j) { ctrl->amax[j] = 0.0; ctrl->t[j] = 0.0; }
  ctrl->t[phase] = t0;
  ctrl->dt = 0.0;
  ctrl->status = 0u;
  ctrl->steps = 0u;
  ctrl->troubled = 0u;
}

template <typename T>
__global__ void __launch_bounds__(NT)
ens_amax_kernel(const EnsDesc<T>* __restrict__ desc, const T* __restrict__ Q, zb_ctrl* ctrls,
                int n_inst, int phase, T g, T eps) {
  __shared__ double red[NT / 32];
  const int i = blockIdx.x / AMAX_PARTS, part = blockIdx.x % AMAX_PARTS;
  if (i >= n_inst) return;
  const EnsDesc<T>* d = desc + i;
  const size_t C = (size_t)d->p.nx * d->p.ny;
  const T* q = Q + d->q_off;
  double m = 0.0;
  for (size_t k = (size_t)part * NT + threadIdx.x; k < C; k += (size_t)AMAX_PARTS * NT) {
    const T h = q[C + k];
    const T hi = kp_hinv(h, eps);
    const T c = asqrt(g * nmax(h, T(0)));
    m = nmax(m, (double)nmax(fabs(q[2 * C + k] * hi) + c, fabs(q[3 * C + k] * hi) + c));
  }
  m = block_max_double(m, red);
  if (threadIdx.x == 0) atomic_max_pos_double(&ctrls[i].amax[phase], m);
}

// ── wave-speed max / aux / mass kernels ─────────────────────────────────────
template <typename T>
__global__ void __launch_bounds__(NT)
swe2d_amax_kernel(const T* __restrict__ hP, const T* __restrict__ qxP,
                  const T* __restrict__ qyP, size_t C, T g, T eps_kp,
                  double* out) {
  __shared__ double red[NT / 32];
  double m = 0.0;
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < C;
       k += (size_t)gridDim.x * NT) {
    const T h = hP[k];
    const T hi = kp_hinv(h, eps_kp);
    const T c = asqrt(g * nmax(h, T(0)));
    const T lx = fabs(qxP[k] * hi) + c, ly = fabs(qyP[k] * hi) + c;
    m = nmax(m, (double)nmax(lx, ly));
  }
  m = block_max_double(m, red);
  if (threadIdx.x == 0) atomic_max_pos_double(out, m);
}

// The bed's interior least-squares gradient and limiter value, one thread per
// cell: the slope block of strip_item for variable 0 (b) -- the float32
// paired block, the float64 scalar one -- in the same operations and order
// ((left + centre) + right sums, difference and scaling, three-input bounds,
// the limiter), so the strip body that reads these planes produces the same
// bits as the one that evaluates them.  Cells on the domain boundary get zeros
// (the interior body never reads them; boundary cells take the boundary
// classes).
template <typename T>
__global__ void __launch_bounds__(NT)
swe2d_bed_kernel(const T* __restrict__ b, T* __restrict__ bed, const SweParams<T> p) {
  const int nx = p.nx, ny = p.ny;
  const size_t n = (size_t)nx * ny;
  const bool clipmin = p.limiter != ZB_LIM_NONE && p.limiter != ZB_LIM_VENKATAKRISHNAN;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(k / (size_t)ny), j = (int)(k % (size_t)ny);
    T gx = T(0), gy = T(0), phi = T(0);
    if (i >= 1 && i < nx - 1 && j >= 1 && j < ny - 1) {
      const T* rm = b + (k - ny);   // row i - 1
      const T* rc = b + k;          // row i
      const T* rp = b + (k + ny);   // row i + 1
      const T u = rc[0];
      const T sx0 = (rm[-1] + rm[0]) + rm[1];   // row sums of rows i -/+ 1
      const T sx2 = (rp[-1] + rp[0]) + rp[1];
      const T tl = (rm[-1] + rc[-1]) + rp[-1];  // column sums of columns j -/+ 1
      const T tr = (rm[1] + rc[1]) + rp[1];
      const T umax = fmx3(u, rp[0], fmx3(rm[0], rc[1], rc[-1]));
      const T umin = fmn3(u, rp[0], fmn3(rm[0], rc[1], rc[-1]));
      if constexpr (std::is_same<T, float>::value) {
        const float2 gv = mul2(sub2(f2(sx2, tr), f2(sx0, tl)), f2(p.inv6dx, p.inv6dy));
        const float2 dd = sub2(f2(umax, umin), f2(u, u));
        gx = gv.x;
        gy = gv.y;
        if (clipmin) {
          const float2 ac = mul2(gv, f2(p.half_dx, p.half_dy));
          phi = phi_clipmin(ac.x, ac.y, dd.x, dd.y);
        } else {
          phi = limiter_phi(p.limiter, gv.x, gv.y, p.half_dx, p.half_dy, dd.x, dd.y, p.vk_eps2);
        }
      } else {
        gx = (sx2 - sx0) * p.inv6dx;
        gy = (tr - tl) * p.inv6dy;
        phi = limiter_phi(p.limiter, gx, gy, p.half_dx, p.half_dy, umax - u, umin - u, p.vk_eps2);
      }
    }
    bed[k] = gx;
    bed[n + k] = gy;
    bed[2 * n + k] = phi;
  }
}

__global__ void swe2d_ctrl_init_kernel(zb_ctrl* ctrl, int phase, double t0) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) { ctrl->amax[i] = 0.0; ctrl->t[i] = 0.0; }
    ctrl->t[phase] = t0;
    ctrl->dt = 0.0;
    ctrl->status = 0u;
    ctrl->steps = 0u;
    ctrl->troubled = 0u;
  }
}

__global__ void swe2d_dt_finalize_kernel(zb_ctrl* ctrl, double t, double cfl2r,
                                         double den_fac, double dt_max,
                                         double t_end) {
  if (threadIdx.x == 0) {
    const double dt = dt_from_amax(ctrl->reserved[0], t, cfl2r, den_fac, dt_max, t_end);
    ctrl->dt = dt;
    if (!(isfinite(dt) && dt > 0.0) && t < t_end)
      atomicOr(&ctrl->status, (unsigned)ZB_ST_DT_INVALID);
  }
}

__global__ void zero_double_kernel(double* p) { *p = 0.0; }

// LSQ derivative aux rows with extrapolation ghosts (delta 0)
template <typename T>
__global__ void __launch_bounds__(NT)
swe2d_aux_kernel(const T* __restrict__ Q, T* __restrict__ A, int nx, int ny,
                 T eps_kp, const LsqTable<T> lsq) {
  const size_t C = (size_t)nx * ny;
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < C;
       k += (size_t)gridDim.x * NT) {
    const int gi = (int)(k / ny), gj = (int)(k - (size_t)gi * ny);
    const bool bxl = gi == 0, bxh = gi == nx - 1, byl = gj == 0, byh = gj == ny - 1;
    const int cls = (bxl ? 0 : (bxh ? 2 : 1)) * 3 + (byl ? 0 : (byh ? 2 : 1));
    const T* wx = lsq.w[cls][0];
    const T* wy = lsq.w[cls][1];
    T g[4][2];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const T* U = Q + (size_t)v * C;
      const T u = U[k];
      T gx = T(0), gy = T(0);
      int s = 0;
      for (int a = -1; a <= 1; ++a)
        for (int bb = -1; bb <= 1; ++bb) {
          if (a == 0 && bb == 0) continue;
          const bool ok = gi + a >= 0 && gi + a < nx && gj + bb >= 0 && gj + bb < ny;
          const T d = ok ? U[k + (long long)a * ny + bb] - u : T(0);
          gx += wx[s] * d;
          gy += wy[s] * d;
          ++s;
        }
      g[v][0] = gx;
      g[v][1] = gy;
    }
    A[0 * C + k] = g[2][0];
    A[1 * C + k] = g[1][0];
    A[2 * C + k] = g[3][1];
    A[3 * C + k] = g[1][1];
    A[4 * C + k] = g[0][0];
    A[5 * C + k] = g[0][1];
    A[6 * C + k] = kp_hinv(Q[C + k], eps_kp);
  }
}

template <typename T>
__global__ void __launch_bounds__(NT)
mass_partial_kernel(const T* __restrict__ h, size_t C, double vol, double* partial) {
  __shared__ double red[NT];
  double acc = 0.0;
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < C;
       k += (size_t)gridDim.x * NT)
    acc += (double)h[k] * vol;
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void mass_final_kernel(const double* partial, int n, zb_ctrl* ctrl) {
  __shared__ double red[NT];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += NT) acc += partial[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) ctrl->mass = red[0];
}

// Manning friction as RK1 with a given aux hinv0 (ode.py:14-18,
// solver_jax.py:373-397, 1129); implicit = point-implicit closed form
template <typename T>
__global__ void __launch_bounds__(NT)
swe2d_source_kernel(T* __restrict__ qx, T* __restrict__ qy, const T* __restrict__ hinv0,
                    size_t C, T g, T n, T dt, int implicit) {
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < C;
       k += (size_t)gridDim.x * NT) {
    const T hi0 = hinv0[k];
    T a = qx[k], b = qy[k];
    const T qn = asqrt(a * a + b * b);
    const T kf = (-g) * (n * n) * qn * (hi0 * hi0) * cbrt(hi0);
    if (implicit) {
      const T den = T(1) + dt * (-kf);
      a = a / den;
      b = b / den;
    } else {
      a = a + dt * (a * kf);
      b = b + dt * (b * kf);
    }
    qx[k] = a;
    qy[k] = b;
  }
}

// the float64 quotient, square root and reciprocal square root of the
// kernels above, for their accuracy test (zb_newton_check_f64)
__global__ void __launch_bounds__(NT)
newton_check_kernel(const double* __restrict__ a, const double* __restrict__ b,
                    double* __restrict__ out, long long n) {
  for (long long k = blockIdx.x * (long long)NT + threadIdx.x; k < n;
       k += (long long)gridDim.x * NT) {
    out[k] = ndiv(a[k], b[k]);
    out[n + k] = nsqrt(b[k]);
    out[2 * n + k] = nrsqrt(b[k]);
  }
}

// ── host side ───────────────────────────────────────────────────────────────
constexpr int MASS_BLOCKS = 1184;   // 148 SMs x 8

static bool valid_cfg(const zb_swe2d_cfg* c) {
  if (!c) return false;
  if (c->nx < 3 || c->ny < 3) return false;
  if ((long long)c->nx * c->ny > (1LL << 31)) return false;
  if (!(c->dx > 0 && c->dy > 0)) return false;
  if (c->order != 1 && c->order != 2) return false;
  if (c->recon < 0 || c->recon > 2 || c->riemann < 0 || c->riemann > 2) return false;
  if (c->limiter < 0 || c->limiter > 3) return false;
  for (int i = 0; i < 4; ++i)
    if (c->bc[i] < 0 || c->bc[i] > 2) return false;
  if ((c->bc[0] == ZB_BC_PERIODIC) != (c->bc[1] == ZB_BC_PERIODIC)) return false;
  if ((c->bc[2] == ZB_BC_PERIODIC) != (c->bc[3] == ZB_BC_PERIODIC)) return false;
  if (c->dtype != ZB_F32 && c->dtype != ZB_F64) return false;
  if (c->order == 1 && c->recon != ZB_RECON_CONSTANT) return false;
  if (c->order == 2 && c->recon == ZB_RECON_CONSTANT) return false;
  if (c->dim_factor < 1 || c->degree < 0) return false;
  return true;
}

// Least-squares weights of the 9 Cartesian cell classes: pseudo-inverse of the
// offsets of the in-domain 3x3 neighbours plus, per derivative direction, the
// ghost of the boundary face normal to that direction (oracle/mesh.py,
// _lsq_weights; pinned against the reference's derivative aux rows).
template <typename T>
static LsqTable<T> make_lsq(double dx, double dy) {
  LsqTable<T> tab;
  std::memset(&tab, 0, sizeof(tab));
  for (int ci = 0; ci < 3; ++ci)
    for (int cj = 0; cj < 3; ++cj) {
      const int cls = ci * 3 + cj;
      for (int d = 0; d < 2; ++d) {
        double px[10], py[10];
        int slot[10], n = 0, k = 0;
        for (int a = -1; a <= 1; ++a)
          for (int b = -1; b <= 1; ++b) {
            if (a == 0 && b == 0) continue;
            const bool okx = !(ci == 0 && a < 0) && !(ci == 2 && a > 0);
            const bool oky = !(cj == 0 && b < 0) && !(cj == 2 && b > 0);
            if (okx && oky) { px[n] = a * dx; py[n] = b * dy; slot[n] = k; ++n; }
            ++k;
          }
        if (d == 0 && ci != 1) { px[n] = (ci == 0 ? -1.0 : 1.0) * dx; py[n] = 0.0; slot[n] = 8; ++n; }
        if (d == 1 && cj != 1) { px[n] = 0.0; py[n] = (cj == 0 ? -1.0 : 1.0) * dy; slot[n] = 9; ++n; }
        double sxx = 0, sxy = 0, syy = 0;
        for (int m = 0; m < n; ++m) { sxx += px[m] * px[m]; sxy += px[m] * py[m]; syy += py[m] * py[m]; }
        const double det = sxx * syy - sxy * sxy;
        const double i00 = syy / det, i01 = -sxy / det, i11 = sxx / det;
        for (int m = 0; m < n; ++m) {
          const double wxm = i00 * px[m] + i01 * py[m];
          const double wym = i01 * px[m] + i11 * py[m];
          tab.w[cls][d][slot[m]] = (T)(d == 0 ? wxm : wym);
        }
      }
    }
  return tab;
}

// the scheme whose interior body reads prepared bed slopes: order 2, eta
// reconstruction, HLL with hydrostatic reconstruction (float32 or float64)
static bool bed_scheme(const zb_swe2d_cfg* c) {
  return c->order == 2 && c->recon == ZB_RECON_ETA && c->riemann == ZB_RIEMANN_HLL_HR;
}

template <typename T>
static SweParams<T> make_params(const zb_swe2d_cfg* c, double alpha, double beta,
                                double dt_stage = -1.0) {
  SweParams<T> p;
  std::memset(&p, 0, sizeof(p));
  p.nx = c->nx;
  p.ny = c->ny;
  p.half_dx = (T)(0.5 * c->dx);
  p.half_dy = (T)(0.5 * c->dy);
  const double vol = c->dx * c->dy;
  p.kx = (T)(c->dy / vol);
  p.ky = (T)(c->dx / vol);
  p.g = (T)c->g;
  p.eps_kp = (T)c->wet_dry_eps;
  p.eps_wet = (T)(c->eps_wet < 0 ? -1.0 : c->eps_wet);
  p.manning_n = (T)c->manning_n;
  const double hv = std::pow(vol, 0.5);
  p.vk_eps2 = (T)(hv * hv);
  for (int i = 0; i < 4; ++i) p.bc[i] = c->bc[i];
  p.limiter = c->limiter;
  p.implicit_source = c->implicit_source;
  const double r_in = c->dx * c->dy / (c->dx + c->dy);
  p.cfl2r = c->cfl * 2.0 * r_in;
  p.den_fac = (double)c->dim_factor * (double)(2 * c->degree + 1);
  p.dt_max = c->dt_max;
  p.t_end = c->t_end;
  p.alpha = alpha;
  p.beta = beta;
  p.dt_stage = dt_stage;
  p.inv6dx = (T)(1.0 / (6.0 * c->dx));
  p.inv6dy = (T)(1.0 / (6.0 * c->dy));
  p.inv4dx = (T)(1.0 / (4.0 * c->dx));
  p.inv4dy = (T)(1.0 / (4.0 * c->dy));
  p.inv5dx = (T)(1.0 / (5.0 * c->dx));
  p.inv5dy = (T)(1.0 / (5.0 * c->dy));
  p.sx = p.sxc = SX;
  p.single = 0;
  p.bed = (bed_scheme(c) && (c->dtype == ZB_F64) == std::is_same<T, double>::value)
              ? (const T*)c->bed : nullptr;
  return p;
}

template <typename T>
constexpr int tile_x() { return sizeof(T) == 4 ? 16 : 8; }

template <typename T, int RIEMANN, int MODE, int TX = tile_x<T>()>
static int launch_stage(const zb_swe2d_cfg* c, const T* b, const T* h, const T* qx,
                        const T* qy, const T* h0, const T* qx0, const T* qy0,
                        T* ho, T* qxo, T* qyo, zb_ctrl* ctrl, int phase,
                        const SweParams<T>& p, cudaStream_t st, const T* hinv_src = nullptr,
                        unsigned char* trouble_out = nullptr) {
  auto kern = swe2d_stage_kernel<T, TX, RIEMANN, MODE>;
  const size_t sm = sizeof(Smem<T, TX>);
  static std::atomic<unsigned> attr_mask{0u};   // per instantiation, one bit per device
  int dev = 0;
  ZB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 32) return ZB_E_UNSUPPORTED;
  if (!(attr_mask.load() & (1u << dev))) {
    ZB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr_mask.fetch_or(1u << dev);
  }
  const dim3 grid((c->ny + TY - 1) / TY, (c->nx + TX - 1) / TX);
  kern<<<grid, NT, sm, st>>>(b, h, qx, qy, h0, qx0, qy0, ho, qxo, qyo, ctrl, phase,
                             hinv_src, trouble_out, p);
  return zb_launch_check();
}

// One order-2 stage of a single grid: one launch of the strip kernel.
template <typename T, int RECON, int RIEMANN, int MODE>
static int launch_strips(const zb_swe2d_cfg* c, const T* b, const T* h, const T* qx, const T* qy,
                         const T* h0, const T* qx0, const T* qy0, T* ho, T* qxo, T* qyo,
                         zb_ctrl* ctrl, int phase, SweParams<T> p, cudaStream_t st,
                         const T* hinv_src = nullptr, const unsigned char* force_o1 = nullptr,
                         unsigned char* trouble_out = nullptr) {
  const StripRows rows = strip_rows(c->nx, c->ny, sizeof(T) == 4);
  p.sx = rows.sx;
  p.sxc = rows.sxc;
  p.single = rows.single ? 1 : 0;
  const int n = p.single ? ((c->ny + SW - 1) / SW) * ((c->nx + p.sx - 1) / p.sx)
                         : full_items(c->nx, c->ny, -1, nullptr, nullptr, nullptr, nullptr, p.sxc,
                                      p.sx);
  const int wpb = STRIP_NT / 32;
  auto go = [&](auto bed) -> int {
    ZB_CUDA_TRY(pdl_launch(swe2d_strip_kernel<T, RECON, RIEMANN, MODE, decltype(bed)::value>,
                           dim3((n + wpb - 1) / wpb), dim3(STRIP_NT), 0, st, b, h, qx, qy, h0, qx0,
                           qy0, ho, qxo, qyo, ctrl, phase, hinv_src, force_o1, trouble_out, p));
    return zb_launch_check();
  };
  if constexpr (RECON == ZB_RECON_ETA && RIEMANN == ZB_RIEMANN_HLL_HR && MODE != MODE_STAGE)
    if (p.bed && !p.single) return go(std::true_type());
  return go(std::false_type());
}

// part: -1 = the whole step, 0 = first launch only, 1 = second launch only
template <typename T, int ORDER, int RECON, int RIEMANN>
static int run_step(const zb_swe2d_cfg* c, T* Q, T* ws, zb_ctrl* ctrl, int phase,
                    int part, cudaStream_t st) {
  const size_t C = (size_t)c->nx * c->ny;
  T *b = Q, *h = Q + C, *qx = Q + 2 * C, *qy = Q + 3 * C;
  const SweParams<T> p = make_params<T>(c, 0.0, 1.0);
  T *h1 = ws, *qx1 = ws + C, *qy1 = ws + 2 * C;
  if constexpr (ORDER == 1) {
    // Euler reads the stencil of Q and cannot write Q in place: write the
    // workspace (launch 0), then copy the three evolving planes back (part 1)
    if (part != 1) {
      int rc = launch_stage<T, RIEMANN, MODE_EULER>(
          c, b, h, qx, qy, nullptr, nullptr, nullptr, h1, qx1, qy1, ctrl, phase, p, st);
      if (rc) return rc;
    }
    if (part != 0)
      ZB_CUDA_TRY(cudaMemcpyAsync(h, h1, 3 * C * sizeof(T), cudaMemcpyDeviceToDevice, st));
    return ZB_OK;
  }
  if constexpr (ORDER == 2) {
    if (part != 1) {
      const int rc = launch_strips<T, RECON, RIEMANN, MODE_STEP1>(
          c, b, h, qx, qy, nullptr, nullptr, nullptr, h1, qx1, qy1, ctrl, phase, p, st);
      if (rc) return rc;
    }
    if (part == 0) return ZB_OK;
    return launch_strips<T, RECON, RIEMANN, MODE_STEP2>(c, b, h1, qx1, qy1, h, qx, qy, h, qx, qy,
                                                        ctrl, phase, p, st);
  }
  return ZB_OK;
}

template <typename T, int ORDER, int RECON, int RIEMANN>
static int run_generic_stage(const zb_swe2d_cfg* c, const T* Qk, const T* Q0, T* Qo,
                             double alpha, double beta, double dt, zb_ctrl* ctrl,
                             const T* hinv_src, const unsigned char* force_o1,
                             unsigned char* trouble_out, cudaStream_t st) {
  const size_t C = (size_t)c->nx * c->ny;
  const SweParams<T> p = make_params<T>(c, alpha, beta, dt);
  const T* b0 = Q0 ? Q0 : Qk;
  if constexpr (ORDER == 2)
    return launch_strips<T, RECON, RIEMANN, MODE_STAGE>(
        c, b0, Qk + C, Qk + 2 * C, Qk + 3 * C, Q0 ? Q0 + C : nullptr, Q0 ? Q0 + 2 * C : nullptr,
        Q0 ? Q0 + 3 * C : nullptr, Qo + C, Qo + 2 * C, Qo + 3 * C, ctrl, 0, p, st, hinv_src,
        force_o1, trouble_out);
  else   // first order already: force_o1 changes nothing
    return launch_stage<T, RIEMANN, MODE_STAGE>(
        c, b0, Qk + C, Qk + 2 * C, Qk + 3 * C, Q0 ? Q0 + C : nullptr, Q0 ? Q0 + 2 * C : nullptr,
        Q0 ? Q0 + 3 * C : nullptr, Qo + C, Qo + 2 * C, Qo + 3 * C, ctrl, 0, p, st, hinv_src,
        trouble_out);
}

// dispatch over (order, recon, riemann)
template <typename T, typename F>
static int dispatch(const zb_swe2d_cfg* c, F&& f) {
#define ZB_CASE(O, R, M)                                                       \
  if (c->order == O && c->recon == R && c->riemann == M)                       \
    return f(std::integral_constant<int, O>(), std::integral_constant<int, R>(), \
             std::integral_constant<int, M>());
  ZB_CASE(1, ZB_RECON_CONSTANT, ZB_RIEMANN_RUSANOV)
  ZB_CASE(1, ZB_RECON_CONSTANT, ZB_RIEMANN_RUSANOV_HR)
  ZB_CASE(1, ZB_RECON_CONSTANT, ZB_RIEMANN_HLL_HR)
  ZB_CASE(2, ZB_RECON_CONSERVATIVE, ZB_RIEMANN_RUSANOV)
  ZB_CASE(2, ZB_RECON_CONSERVATIVE, ZB_RIEMANN_RUSANOV_HR)
  ZB_CASE(2, ZB_RECON_CONSERVATIVE, ZB_RIEMANN_HLL_HR)
  ZB_CASE(2, ZB_RECON_ETA, ZB_RIEMANN_RUSANOV_HR)
  ZB_CASE(2, ZB_RECON_ETA, ZB_RIEMANN_HLL_HR)
#undef ZB_CASE
  return ZB_E_UNSUPPORTED;
}

template <typename T>
static int amax_into(const zb_swe2d_cfg* c, const T* Q, double* dst, cudaStream_t st) {
  const size_t C = (size_t)c->nx * c->ny;
  zero_double_kernel<<<1, 1, 0, st>>>(dst);
  const int blocks = (int)std::min<size_t>((C + NT - 1) / NT, 148 * 16);
  swe2d_amax_kernel<T><<<blocks, NT, 0, st>>>(Q + C, Q + 2 * C, Q + 3 * C, C, (T)c->g,
                                              (T)c->wet_dry_eps, dst);
  return zb_launch_check();
}


// ── ensemble host side ──────────────────────────────────────────────────────
template <typename T>
static size_t ens_desc_bytes(int n_inst) {
  return ((size_t)n_inst * sizeof(EnsDesc<T>) + 255) / 256 * 256;
}

// the chunk heights of an instance's size class (zb_ens_tuning)
static void ens_class_rows(const zb_ens_tuning& t, const zb_ens_instance& in, int* sxc,
                           int* sx) {
  const int side = std::max(in.nx, in.ny);
  int c = 0;
  while (c < t.n_classes - 1 && side > t.class_max_side[c]) ++c;
  *sxc = t.edge_rows[c];
  *sx = t.interior_rows[c];
}

// strip items of an instance (the single grid's list): {strip, r0, r1, kind,
// first item}
template <typename F>
static void ens_strip_items(const zb_ens_instance& in, const zb_ens_tuning& t, F&& visit) {
  int sxc, sx;
  ens_class_rows(t, in, &sxc, &sx);
  const int n = full_items(in.nx, in.ny, -1, nullptr, nullptr, nullptr, nullptr, sxc, sx);
  for (int it = 0; it < n; ++it) {
    int st, r0, r1, kind;
    full_items(in.nx, in.ny, it, &st, &r0, &r1, &kind, sxc, sx);
    visit(st, r0, r1, kind, it == 0);
  }
}

static size_t ens_count(const zb_ens_instance* inst, int n, const zb_ens_tuning& t) {
  size_t strips = 0;
  for (int i = 0; i < n; ++i) {
    int sxc, sx;
    ens_class_rows(t, inst[i], &sxc, &sx);
    strips += (size_t)full_items(inst[i].nx, inst[i].ny, -1, nullptr, nullptr, nullptr, nullptr,
                                 sxc, sx);
  }
  return strips;
}

// the launch shape of the untuned entry points: one size class, 32-row
// boundary-strip chunks, 64-row interior chunks (the CTAs per SM are a field that
// no launch reads)
static zb_ens_tuning ens_default_tuning(const zb_swe2d_cfg* c, int tile_x) {
  zb_ens_tuning t;
  std::memset(&t, 0, sizeof(t));
  t.tile_x = tile_x;
  t.ctas_per_sm = c && c->dtype == ZB_F64 ? 2 : 4;
  t.n_classes = 1;
  t.class_max_side[0] = 1 << 30;
  t.edge_rows[0] = SXC_ENS;
  t.interior_rows[0] = SX;
  return t;
}

static bool ens_tuning_valid(const zb_swe2d_cfg* c, const zb_ens_tuning* t) {
  if (!c || !t || (t->tile_x != 8 && t->tile_x != 16)) return false;
  if (t->ctas_per_sm < 1 || t->ctas_per_sm > (c->dtype == ZB_F64 ? 2 : 4)) return false;
  if (t->n_classes < 1 || t->n_classes > 4) return false;
  for (int k = 0; k < t->n_classes; ++k) {
    if (t->edge_rows[k] < 4 || t->edge_rows[k] > SXC_MAX) return false;
    if (t->interior_rows[k] < 8 || t->interior_rows[k] > 1024) return false;
    if (k > 0 && t->class_max_side[k] <= t->class_max_side[k - 1]) return false;
  }
  return true;
}

static bool ens_valid(const zb_swe2d_cfg* c, const zb_ens_instance* inst, int n, int tile_x) {
  if (!c || !inst || n < 1 || (tile_x != 8 && tile_x != 16)) return false;
  if (c->order != 2 || c->recon != ZB_RECON_ETA || c->riemann != ZB_RIEMANN_HLL_HR) return false;
  if (c->dtype != ZB_F32 && c->dtype != ZB_F64) return false;
  for (int i = 0; i < 4; ++i)
    if (c->bc[i] != ZB_BC_WALL && c->bc[i] != ZB_BC_EXTRAPOLATION) return false;
  for (int i = 0; i < n; ++i)
    if (inst[i].nx < 3 || inst[i].ny < 3 || !(inst[i].dx > 0) || !(inst[i].dy > 0) ||
        inst[i].q_offset < 0 || inst[i].ws_offset < 0)
      return false;
  return true;
}

template <typename T>
static int ens_launch(int part, const void* table, int n_inst, int n_items, void* Q, void* W,
                      zb_ctrl* ctrls, int phase, cudaStream_t st) {
  const EnsDesc<T>* desc = (const EnsDesc<T>*)table;
  const int4* items = (const int4*)((const char*)table + ens_desc_bytes<T>(n_inst));
  const int sgrid = (n_items + STRIP_NT / 32 - 1) / (STRIP_NT / 32);
  if (part == 0)
    ZB_CUDA_TRY(pdl_launch(ens_strip_kernel<T, MODE_STEP1>, dim3(sgrid), dim3(STRIP_NT), 0, st, desc,
                           items, (T*)Q, (T*)W, ctrls, phase));
  else
    ZB_CUDA_TRY(pdl_launch(ens_strip_kernel<T, MODE_STEP2>, dim3(sgrid), dim3(STRIP_NT), 0, st, desc,
                           items, (T*)Q, (T*)W, ctrls, phase));
  return zb_launch_check();
}

}  // namespace zb

using namespace zb;

extern "C" {

const char* zb_version(void) { return "libzb 0.1 (sm_100a)"; }

size_t zb_swe2d_workspace_bytes(const zb_swe2d_cfg* cfg) {
  if (!valid_cfg(cfg)) return 0;
  const size_t es = cfg->dtype == ZB_F64 ? 8 : 4;
  return 3 * (size_t)cfg->nx * cfg->ny * es + 256;
}

size_t zb_swe2d_bed_bytes(const zb_swe2d_cfg* cfg) {
  if (!valid_cfg(cfg) || !bed_scheme(cfg)) return 0;
  return 3 * (size_t)cfg->nx * cfg->ny * (cfg->dtype == ZB_F64 ? 8 : 4);
}

int zb_swe2d_bed_prepare(const zb_swe2d_cfg* cfg, const void* Q, void* bed, size_t bed_bytes,
                         zb_stream_t stream) {
  if (!valid_cfg(cfg) || !bed_scheme(cfg) || !Q || !bed) return ZB_E_ARG;
  if (bed_bytes < zb_swe2d_bed_bytes(cfg) || ((uintptr_t)bed & 7u)) return ZB_E_ARG;
  const size_t n = (size_t)cfg->nx * cfg->ny;
  const int grid = (int)std::min<size_t>((n + NT - 1) / NT, (size_t)148 * 16);
  if (cfg->dtype == ZB_F64) {
    const SweParams<double> p = make_params<double>(cfg, 0.0, 1.0);
    swe2d_bed_kernel<double><<<grid, NT, 0, (cudaStream_t)stream>>>((const double*)Q,
                                                                     (double*)bed, p);
  } else {
    const SweParams<float> p = make_params<float>(cfg, 0.0, 1.0);
    swe2d_bed_kernel<float><<<grid, NT, 0, (cudaStream_t)stream>>>((const float*)Q,
                                                                   (float*)bed, p);
  }
  return zb_launch_check();
}

int zb_swe2d_init(const zb_swe2d_cfg* cfg, const void* Q, zb_ctrl* ctrl, int phase,
                  double t0, zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !ctrl || phase < 0 || phase > 2) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  swe2d_ctrl_init_kernel<<<1, 32, 0, st>>>(ctrl, phase, t0);
  if (cfg->dtype == ZB_F32) return amax_into<float>(cfg, (const float*)Q, &ctrl->amax[phase], st);
  return amax_into<double>(cfg, (const double*)Q, &ctrl->amax[phase], st);
}

int zb_swe2d_dt(const zb_swe2d_cfg* cfg, const void* Q, zb_ctrl* ctrl, double t,
                zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !ctrl) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = cfg->dtype == ZB_F32
               ? amax_into<float>(cfg, (const float*)Q, &ctrl->reserved[0], st)
               : amax_into<double>(cfg, (const double*)Q, &ctrl->reserved[0], st);
  if (rc) return rc;
  const double r_in = cfg->dx * cfg->dy / (cfg->dx + cfg->dy);
  swe2d_dt_finalize_kernel<<<1, 32, 0, st>>>(
      ctrl, t, cfg->cfl * 2.0 * r_in,
      (double)cfg->dim_factor * (double)(2 * cfg->degree + 1), cfg->dt_max, cfg->t_end);
  return zb_launch_check();
}

int zb_swe2d_step_part(const zb_swe2d_cfg* cfg, void* Q, void* workspace,
                       size_t workspace_bytes, zb_ctrl* ctrl, int phase, int part,
                       zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !ctrl || phase < 0 || phase > 2) return ZB_E_ARG;
  if (part < -1 || part > 1) return ZB_E_ARG;
  if (!workspace || workspace_bytes < zb_swe2d_workspace_bytes(cfg)) return ZB_E_ARG;
  if (cfg->recon == ZB_RECON_ETA && cfg->riemann == ZB_RIEMANN_RUSANOV) return ZB_E_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  if (cfg->dtype == ZB_F32) {
    return dispatch<float>(cfg, [&](auto O, auto R, auto M) {
      return run_step<float, decltype(O)::value, decltype(R)::value, decltype(M)::value>(
          cfg, (float*)Q, (float*)workspace, ctrl, phase, part, st);
    });
  }
  return dispatch<double>(cfg, [&](auto O, auto R, auto M) {
    return run_step<double, decltype(O)::value, decltype(R)::value, decltype(M)::value>(
        cfg, (double*)Q, (double*)workspace, ctrl, phase, part, st);
  });
}

int zb_swe2d_step(const zb_swe2d_cfg* cfg, void* Q, void* workspace, size_t workspace_bytes,
                  zb_ctrl* ctrl, int phase, zb_stream_t stream) {
  return zb_swe2d_step_part(cfg, Q, workspace, workspace_bytes, ctrl, phase, -1, stream);
}

int zb_swe2d_stage(const zb_swe2d_cfg* cfg, const void* Qk, const void* Q0, void* Q_out,
                   double alpha, double beta, double dt, const void* hinv_src,
                   const uint8_t* force_o1, uint8_t* trouble_out, zb_ctrl* ctrl,
                   zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Qk || !Q_out || !ctrl) return ZB_E_ARG;
  if (Q_out == Qk) return ZB_E_ARG;
  if (!(dt >= 0.0) && !(dt < 0.0)) return ZB_E_ARG;
  if (alpha != 0.0 && !Q0) return ZB_E_ARG;
  if (cfg->recon == ZB_RECON_ETA && cfg->riemann == ZB_RIEMANN_RUSANOV) return ZB_E_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  if (cfg->dtype == ZB_F32) {
    return dispatch<float>(cfg, [&](auto O, auto R, auto M) {
      return run_generic_stage<float, decltype(O)::value, decltype(R)::value, decltype(M)::value>(
          cfg, (const float*)Qk, (const float*)Q0, (float*)Q_out, alpha, beta, dt, ctrl,
          (const float*)hinv_src, force_o1, trouble_out, st);
    });
  }
  return dispatch<double>(cfg, [&](auto O, auto R, auto M) {
    return run_generic_stage<double, decltype(O)::value, decltype(R)::value, decltype(M)::value>(
        cfg, (const double*)Qk, (const double*)Q0, (double*)Q_out, alpha, beta, dt, ctrl,
        (const double*)hinv_src, force_o1, trouble_out, st);
  });
}

int zb_swe2d_source(const zb_swe2d_cfg* cfg, void* Q, const void* hinv0, double dt,
                    zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !hinv0 || !(dt >= 0.0)) return ZB_E_ARG;
  if (cfg->manning_n == 0.0) return ZB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t C = (size_t)cfg->nx * cfg->ny;
  const int blocks = (int)std::min<size_t>((C + NT - 1) / NT, 148 * 16);
  if (cfg->dtype == ZB_F32)
    swe2d_source_kernel<float><<<blocks, NT, 0, st>>>(
        (float*)Q + 2 * C, (float*)Q + 3 * C, (const float*)hinv0, C, (float)cfg->g,
        (float)cfg->manning_n, (float)dt, cfg->implicit_source);
  else
    swe2d_source_kernel<double><<<blocks, NT, 0, st>>>(
        (double*)Q + 2 * C, (double*)Q + 3 * C, (const double*)hinv0, C, cfg->g,
        cfg->manning_n, dt, cfg->implicit_source);
  return zb_launch_check();
}

size_t zb_swe2d_mass_partials(const zb_swe2d_cfg* cfg) {
  (void)cfg;
  return MASS_BLOCKS;
}

int zb_swe2d_mass(const zb_swe2d_cfg* cfg, const void* Q, double* partial, zb_ctrl* ctrl,
                  zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !partial || !ctrl) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t C = (size_t)cfg->nx * cfg->ny;
  const double vol = cfg->dx * cfg->dy;
  if (cfg->dtype == ZB_F32)
    mass_partial_kernel<float><<<MASS_BLOCKS, NT, 0, st>>>((const float*)Q + C, C, vol, partial);
  else
    mass_partial_kernel<double><<<MASS_BLOCKS, NT, 0, st>>>((const double*)Q + C, C, vol, partial);
  mass_final_kernel<<<1, NT, 0, st>>>(partial, MASS_BLOCKS, ctrl);
  return zb_launch_check();
}

int zb_swe2d_aux(const zb_swe2d_cfg* cfg, const void* Q, void* Qaux, zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !Qaux) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t C = (size_t)cfg->nx * cfg->ny;
  const int blocks = (int)std::min<size_t>((C + NT - 1) / NT, 148 * 16);
  if (cfg->dtype == ZB_F32)
    swe2d_aux_kernel<float><<<blocks, NT, 0, st>>>((const float*)Q, (float*)Qaux, cfg->nx,
                                                   cfg->ny, (float)cfg->wet_dry_eps,
                                                   make_lsq<float>(cfg->dx, cfg->dy));
  else
    swe2d_aux_kernel<double><<<blocks, NT, 0, st>>>((const double*)Q, (double*)Qaux, cfg->nx,
                                                    cfg->ny, cfg->wet_dry_eps,
                                                    make_lsq<double>(cfg->dx, cfg->dy));
  return zb_launch_check();
}

int zb_newton_check_f64(const double* a, const double* b, double* out, int64_t n,
                        zb_stream_t stream) {
  if (!a || !b || !out || n < 0) return ZB_E_ARG;
  if (n == 0) return ZB_OK;
  const int blocks = (int)std::min<long long>((n + NT - 1) / NT, 148 * 8);
  newton_check_kernel<<<blocks, NT, 0, (cudaStream_t)stream>>>(a, b, out, (long long)n);
  return zb_launch_check();
}

// ── allocation-free step ────────────────────────────────────────────────────
// Some callers cannot call cudaMalloc: a framework that owns every device
// byte hands a plugin only its operands (an XLA / JAX FFI custom call
// declared without a scratch buffer, an inference-engine plugin at enqueue
// time), and the plugin has no way to ask for more.  For them the stage-1
// state of the fused step lives in this file-scope device array instead of a
// caller workspace: three planes of up to ZB_NOALLOC_MAX_CELLS cells in
// float64 (float32 uses the first half), 24 MiB plus 256 bytes of padding.
// Every GPU that loads libzb holds the array until the process exits.
static __device__ __align__(256) double g_noalloc_scratch[3 * ZB_NOALLOC_MAX_CELLS + 32];

// The array's name in host code is only a host-side stand-in; the kernels
// need its device address, fetched once per device with that device current.
static std::mutex g_noalloc_mu;
static void* g_noalloc_ptr[64] = {};

static int noalloc_scratch(void** out) {
  int dev = -1;
  ZB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return ZB_E_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return ZB_E_CUDA;
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return ZB_OK;
}

int zb_swe2d_step_noalloc(const zb_swe2d_cfg* cfg, void* Q, zb_ctrl* ctrl, int phase,
                          zb_stream_t stream) {
  if (!valid_cfg(cfg) || !Q || !ctrl || phase < 0 || phase > 2) return ZB_E_ARG;
  if ((size_t)cfg->nx * (size_t)cfg->ny > (size_t)ZB_NOALLOC_MAX_CELLS) return ZB_E_TOO_LARGE;
  void* ws = nullptr;
  const int rc = noalloc_scratch(&ws);
  if (rc != ZB_OK) return rc;
  return zb_swe2d_step(cfg, Q, ws, sizeof(g_noalloc_scratch), ctrl, phase, stream);
}


// ── ensemble C ABI ──────────────────────────────────────────────────────────
size_t zb_ens_table_bytes_tuned(const zb_swe2d_cfg* common, const zb_ens_instance* inst,
                                int n_inst, const zb_ens_tuning* tuning) {
  if (!ens_tuning_valid(common, tuning)) return 0;
  if (!ens_valid(common, inst, n_inst, tuning->tile_x)) return 0;
  const size_t strips = ens_count(inst, n_inst, *tuning);
  const size_t d = common->dtype == ZB_F64 ? ens_desc_bytes<double>(n_inst)
                                           : ens_desc_bytes<float>(n_inst);
  return d + (1 + strips) * sizeof(int4);
}

size_t zb_ens_table_bytes(const zb_swe2d_cfg* common, const zb_ens_instance* inst, int n_inst,
                          int tile_x) {
  if (!common) return 0;
  const zb_ens_tuning t = ens_default_tuning(common, tile_x);
  return zb_ens_table_bytes_tuned(common, inst, n_inst, &t);
}

int zb_ens_prepare(const zb_swe2d_cfg* common, const zb_ens_instance* inst, int n_inst,
                   int tile_x, void* table, size_t table_bytes, int* n_items_out) {
  if (!common) return ZB_E_ARG;
  const zb_ens_tuning t = ens_default_tuning(common, tile_x);
  return zb_ens_prepare_tuned(common, inst, n_inst, &t, table, table_bytes, n_items_out);
}

int zb_ens_prepare_tuned(const zb_swe2d_cfg* common, const zb_ens_instance* inst, int n_inst,
                         const zb_ens_tuning* tuning, void* table, size_t table_bytes,
                         int* n_items_out) {
  if (!ens_tuning_valid(common, tuning)) return ZB_E_ARG;
  const int tile_x = tuning->tile_x;
  if (!ens_valid(common, inst, n_inst, tile_x) || !table || !n_items_out) return ZB_E_ARG;
  if (table_bytes < zb_ens_table_bytes_tuned(common, inst, n_inst, tuning)) return ZB_E_ARG;
  auto build = [&](auto tag) -> int {
    using T = decltype(tag);
    std::vector<EnsDesc<T>> desc(n_inst);
    // items[0]: {interior items, boundary items}
    std::vector<int4> items(1), strips, estrips;
    for (int i = 0; i < n_inst; ++i) {
      zb_swe2d_cfg c = *common;
      c.bed = nullptr;   // instances read their own b; no prepared bed planes
      c.nx = inst[i].nx;
      c.ny = inst[i].ny;
      c.dx = inst[i].dx;
      c.dy = inst[i].dy;
      c.manning_n = inst[i].manning_n;
      c.t_end = inst[i].t_end;
      std::memset(&desc[i], 0, sizeof(EnsDesc<T>));
      desc[i].p = make_params<T>(&c, 0.0, 1.0);
      desc[i].q_off = inst[i].q_offset;
      desc[i].ws_off = inst[i].ws_offset;
      ens_strip_items(inst[i], *tuning, [&](int st, int r0, int r1, int kind, bool lead) {
        (kind ? estrips : strips).push_back(make_int4(i, st, r0, (lead ? 1 : 0) | (r1 << 1)));
      });
    }
    // longest items first: the block scheduler hands out CTAs in order, so the
    // short ones fill the tail of the long ones
    auto longest_first = [](std::vector<int4>& v) {
      std::stable_sort(v.begin(), v.end(), [](const int4& a, const int4& b) {
        return (a.w >> 1) - a.z > (b.w >> 1) - b.z;
      });
    };
    longest_first(strips);
    longest_first(estrips);
    items[0] = make_int4((int)strips.size(), (int)estrips.size(), 0, 0);
    items.insert(items.end(), strips.begin(), strips.end());
    items.insert(items.end(), estrips.begin(), estrips.end());
    const size_t db = ens_desc_bytes<T>(n_inst);
    // the table may still be read by steps in flight on any stream: wait for
    // the device, copy, and return only once the copy has landed
    ZB_CUDA_TRY(cudaDeviceSynchronize());
    ZB_CUDA_TRY(cudaMemcpy(table, desc.data(), desc.size() * sizeof(EnsDesc<T>),
                           cudaMemcpyHostToDevice));
    ZB_CUDA_TRY(cudaMemcpy((char*)table + db, items.data(), items.size() * sizeof(int4),
                           cudaMemcpyHostToDevice));
    ZB_CUDA_TRY(cudaDeviceSynchronize());
    *n_items_out = (int)items.size() - 1;
    return ZB_OK;
  };
  return common->dtype == ZB_F64 ? build(double()) : build(float());
}

int zb_ens_init(const zb_swe2d_cfg* common, const void* table, int n_inst, const void* Q,
                zb_ctrl* ctrls, int phase, double t0, zb_stream_t stream) {
  if (!common || !table || !Q || !ctrls || n_inst < 1 || phase < 0 || phase > 2) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  ens_ctrl_init_kernel<<<(n_inst + NT - 1) / NT, NT, 0, st>>>(ctrls, n_inst, phase, t0);
  const int grid = n_inst * AMAX_PARTS;
  if (common->dtype == ZB_F64)
    ens_amax_kernel<double><<<grid, NT, 0, st>>>((const EnsDesc<double>*)table, (const double*)Q,
                                                 ctrls, n_inst, phase, common->g,
                                                 common->wet_dry_eps);
  else
    ens_amax_kernel<float><<<grid, NT, 0, st>>>((const EnsDesc<float>*)table, (const float*)Q,
                                                ctrls, n_inst, phase, (float)common->g,
                                                (float)common->wet_dry_eps);
  return zb_launch_check();
}

int zb_ens_step_part_tuned(const zb_swe2d_cfg* common, const void* table, int n_inst,
                           int n_items, const zb_ens_tuning* tuning, int grid, void* Q, void* W,
                           zb_ctrl* ctrls, int phase, int part, zb_stream_t stream) {
  if (!common || !table || !Q || !W || !ctrls || n_inst < 1 || n_items < 1) return ZB_E_ARG;
  if (phase < 0 || phase > 2 || part < -1 || part > 1) return ZB_E_ARG;
  if (!ens_tuning_valid(common, tuning)) return ZB_E_ARG;
  (void)grid;
  cudaStream_t st = (cudaStream_t)stream;
  for (int pt = (part == 1 ? 1 : 0); pt <= (part == 0 ? 0 : 1); ++pt) {
    const int rc = common->dtype == ZB_F64
                       ? ens_launch<double>(pt, table, n_inst, n_items, Q, W, ctrls, phase, st)
                       : ens_launch<float>(pt, table, n_inst, n_items, Q, W, ctrls, phase, st);
    if (rc) return rc;
  }
  return ZB_OK;
}

int zb_ens_step_part(const zb_swe2d_cfg* common, const void* table, int n_inst, int n_items,
                     int tile_x, int grid, void* Q, void* W, zb_ctrl* ctrls, int phase,
                     int part, zb_stream_t stream) {
  if (!common || (tile_x != 8 && tile_x != 16)) return ZB_E_ARG;
  const zb_ens_tuning t = ens_default_tuning(common, tile_x);
  return zb_ens_step_part_tuned(common, table, n_inst, n_items, &t, grid, Q, W, ctrls, phase,
                                part, stream);
}

}  // extern "C"
