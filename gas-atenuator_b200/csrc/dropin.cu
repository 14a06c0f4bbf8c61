// dropin.cu - CUDA drop-ins for the reference driver's MATLAB functions:
//   find_CS0, free_motion, particle_density, electricmagneticfield6
//   (EM2 + EM7 + EM3_1 + EM3 + EM4), electron_collision (electron_transport).
// Plain FP64 on the MATLAB column-major arrays; compiled with -fmad=false so
// the arithmetic follows the reference expression by expression, but for
// electricmagneticfield6, whose particle step multiplies by reciprocals and
// uses explicit FMAs.
#include <cub/device/device_scan.cuh>
#include <cmath>
#include <cstring>
#include <string>
#include "fdtd.cuh"
#include "gasatt_internal.h"

using namespace gasatt;

namespace {

constexpr int kBlock = 256;

// ------------------------------------------------------------- find_CS0
struct XsRaw {            // device copies of the raw find_CS0 tables
  const double *t_el; int n_el;
  const double *t_sel; int n_sel;
  const double *t_ion; int n_ion;
  const double *t_exc; int n_exc;
};

__device__ double d_interp1(const double *x, int sx, const double *y, int sy, int n, double xq) {
  if (!(xq >= x[0] && xq <= x[(int64_t)(n - 1) * sx])) return nan("");
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (x[(int64_t)mid * sx] <= xq) lo = mid; else hi = mid;
  }
  const double x0 = x[(int64_t)lo * sx], x1 = x[(int64_t)hi * sx];
  const double y0 = y[(int64_t)lo * sy], y1 = y[(int64_t)hi * sy];
  return y0 + (xq - x0) * (y1 - y0) / (x1 - x0);
}

__device__ double d_loglog(const double *x, int sx, const double *y, int sy, int n, double xq) {
  const double x0 = x[(int64_t)(n - 2) * sx], x1 = x[(int64_t)(n - 1) * sx];
  const double y0 = y[(int64_t)(n - 2) * sy], y1 = y[(int64_t)(n - 1) * sy];
  const double s = log(y1 / y0) / log(x1 / x0);
  return y1 * pow(xq / x1, s);
}

// x^e; the excitation table's exponents are 1, 3 and 3/4, whose powers need no
// logarithm (200,000 energies: 53 us with pow throughout, 18 us so).  Below 0 sqrt
// is no number, but pow(-infinity, 3/4), of an energy of 0, is infinite.
__device__ __forceinline__ double pow_table(double x, double e) {
  if (e == 1) return x;
  if (e == 3) return x * x * x;
  if (e == 0.75 && x >= 0) {
    const double r = sqrt(x);
    return r * sqrt(r);
  }
  return pow(x, e);
}

// find_CS0.m:100-146 on one energy E [keV]
__global__ void k_find_cs0(XsRaw t, const double *__restrict__ E, int64_t n, double *se,
                           double *si, double *sx, unsigned flags) {
  const bool faithful = (flags & GASATT_Q_XS_NAN) != 0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const double e = E[p];
    double sel = 0.0;
    if (e >= 0.05) {
      sel = d_interp1(&t.t_el[0], 2, &t.t_el[1], 2, t.n_el, e);
      if (!faithful && e > t.t_el[2 * (t.n_el - 1)]) sel = d_loglog(&t.t_el[0], 2, &t.t_el[1], 2, t.n_el, e);
      sel = sel * GASATT_A0SQ * 2;
    } else if (e < 0.05) {
      double Ev = e * 1000;
      if (!faithful && Ev < t.t_sel[0]) Ev = t.t_sel[0];
      sel = d_interp1(&t.t_sel[0], 1, &t.t_sel[t.n_sel], 1, t.n_sel, Ev) * 1e-20;
    }
    se[p] = sel;
    const double T = e * 1000;
    double sion;
    if (!faithful && T <= t.t_ion[0]) sion = 0.0;
    else if (!faithful && T > t.t_ion[t.n_ion - 1])
      sion = d_loglog(&t.t_ion[0], 1, &t.t_ion[t.n_ion], 1, t.n_ion, T) * 1e-20;
    else sion = d_interp1(&t.t_ion[0], 1, &t.t_ion[t.n_ion], 1, t.n_ion, T) * 1e-20;
    si[p] = sion;
    double s = 0.0;
    for (int i = 0; i < t.n_exc; ++i) {
      const double k = t.t_exc[i], A = t.t_exc[t.n_exc + i], om = t.t_exc[2 * t.n_exc + i];
      const double nu = t.t_exc[3 * t.n_exc + i], ga = t.t_exc[4 * t.n_exc + i];
      if (!faithful && !(T > k)) continue;
      const double a = GASATT_CS_Q0 * A / (k * k);
      const double b = pow_table(k / T, om);
      const double c = pow_table(1 - pow_table(k / T, ga), nu);
      s = s + a * b * c;
    }
    sx[p] = s * 1e-4;
  }
}

// ---------------------------------------------------------- free_motion
__global__ void k_free_motion(const double *vx, const double *vy, const double *vz,
                              const double *x, const double *y, const double *z, int64_t n,
                              double dt, double *xn, double *yn, double *zn, double *rn,
                              double *phin) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double X = x[i] + vx[i] * dt, Y = y[i] + vy[i] * dt, Z = z[i] + vz[i] * dt;
    xn[i] = X; yn[i] = Y; zn[i] = Z;
    rn[i] = sqrt(X * X + Y * Y);
    phin[i] = atan2(Y, X);
  }
}

// ---------------------------------------------------------------- REBOND
// REBOND.m:6-66: an azimuth below 0 is raised by PHIp, with (v1, v2) turned
// by +PHIp, until it is not; the wrapped particle's x, y are rebuilt from r
// and the new azimuth; the same downwards above PHIp; then specular
// reflection at z = Lp and at z = 0.  Each wrap or reflection is one boundary
// event (count[0]).  The reference loops until every azimuth is inside; here a
// particle stops after kRebondMaxWraps wraps and raises count[1] (the call
// then fails) instead of looping without end on a wild azimuth.
constexpr int kRebondMaxWraps = 4096;

__global__ void k_rebond(double *pos, int64_t ldp, const double *r, const double *phi,
                         double *vel, int64_t ldv, int64_t n, double Lp, double PHIp, double cP,
                         double sP, unsigned long long *count) {
  unsigned long long ev = 0, bad = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double ph = phi[i], v1 = vel[i], v2 = vel[ldv + i];
    int k = 0;
    if (ph < 0) {
      while (ph < 0 && k < kRebondMaxWraps) {
        ph = ph + PHIp;
        const double w = v1 * cP - v2 * sP;
        v2 = v1 * sP + v2 * cP;
        v1 = w;
        ++k;
      }
      pos[i] = r[i] * cos(ph);
      pos[ldp + i] = r[i] * sin(ph);
    }
    if (ph > PHIp) {
      while (ph > PHIp && k < kRebondMaxWraps) {
        ph = ph - PHIp;
        const double w = v1 * cP + v2 * sP;
        v2 = -v1 * sP + v2 * cP;
        v1 = w;
        ++k;
      }
      pos[i] = r[i] * cos(ph);
      pos[ldp + i] = r[i] * sin(ph);
    }
    if (ph < 0 || ph > PHIp) bad++;
    vel[i] = v1;
    vel[ldv + i] = v2;
    double z = pos[2 * ldp + i], vz = vel[2 * ldv + i];
    if (z > Lp) { z = 2 * Lp - z; vz = -vz; ++k; }
    if (z < 0) { z = -z; vz = -vz; ++k; }
    pos[2 * ldp + i] = z;
    vel[2 * ldv + i] = vz;
    ev += (unsigned long long)k;
  }
  for (int o = 16; o; o >>= 1) {
    ev += __shfl_down_sync(0xFFFFFFFFu, ev, o);
    bad += __shfl_down_sync(0xFFFFFFFFu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (ev) atomicAdd(count, ev);
    if (bad) atomicAdd(count + 1, bad);
  }
}

// ------------------------------------------------------ particle_density
// particle_density.m:24-28: 1-based cell index via MATLAB round(x/d + 0.5)
__global__ void k_density_count(double dr, double dz, const double *dphi, int rmax,
                                const double *r, const double *phi, const double *z, int64_t n,
                                int cellnumxy, const double *sum_cell, int64_t ncell,
                                unsigned long long *count) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const double iz = round(z[p] / dz + 0.5), ir = round(r[p] / dr + 0.5);
    if (!(ir >= 1 && ir <= rmax)) continue;
    const double ip = round(phi[p] / dphi[(int)ir - 1] + 0.5);
    const double base = ((int)ir != 1) ? sum_cell[(int)ir - 2] : 0.0;
    const double idx = (iz - 1) * cellnumxy + base + ip;
    if (!(idx >= 1 && idx <= (double)ncell)) continue;
    atomicAdd(count + ((int64_t)idx - 1), 1ull);
  }
}

__global__ void k_density_finish(const unsigned long long *count, int64_t ncell, int cellnumxy,
                                 const double *VC, double FN, double *density) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncell;
       c += (int64_t)gridDim.x * blockDim.x)
    density[c] = FN * (double)count[c] / VC[c % cellnumxy];
}

// Per-cell counters of gasatt_particle_density_noalloc: a fixed array in the
// library's device image, so that call needs no device allocation.  In host
// code the name g_density_counts stands for a host-side shadow, not a device
// address; the device address comes from cudaGetSymbolAddress with the
// device current.
static __device__ __align__(256) unsigned long long
    g_density_counts[GASATT_DENSITY_NOALLOC_MAX_CELLS];

// Device address of g_density_counts on the current device, looked up on
// every call: a cached address would go stale when the device's primary
// context is reset (cudaDeviceReset, or MATLAB's reset(gpuDevice)) and the
// module is loaded again elsewhere.  Once the module is loaded the lookup is
// a table read.
int density_counts_on_device(gasatt_ctx *ctx, unsigned long long **out) {
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_density_counts);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaGetSymbolAddress(g_density_counts)");
  *out = static_cast<unsigned long long *>(p);
  return GASATT_OK;
}

// -------------------------------------------- electricmagneticfield6 path
// Per particle step one field sub-cycle (k_em_fields) and one particle kernel
// (k_em_push: kick and second half drift of the step, first half drift and
// deposit of the next), where one launch per reference kernel took 26.  The
// push multiplies by reciprocals and takes the sine and cosine of the azimuth
// from x / r and y / r.  It waits on its gathers and global atomics.  100 x 500
// cells, 260,000 particles: push 20 us sorted by cell (27 as they come),
// fields 11 us; in 26 launches a step took 165 us.
struct Species {
  double *pos[3], *vel[3];
  int64_t n[3];
  int64_t start[3];
};

struct EmState {
  double *x, *y, *z, *vx, *vy, *vz;
  int *of;                                // o: particle o of the inputs is in this slot; ~o: it was, and has left
};

// From kEmSortParticles on the particles are sorted by cell before the first
// step and every kEmSortPeriod steps, where kEmSortLeast steps are still to
// come: a sort costs about eight steps' gain.  20 steps without -> with the
// sort: 25,000 particles 596 -> 678 us, 65,000 670 -> 673, 260,000 1069 -> 989,
// 750,000 1975 -> 1671.
constexpr int kEmSortPeriod = 25, kEmSortLeast = 10;
constexpr int64_t kEmSortParticles = 100000;

struct EmParams {
  double Rp, Lp, PHIp, cP, sP, hdt;       // hdt: half the particle step
  double id, mu, c, ic2, FN, scale;       // id: 1 / cell size
  double q[3], m[3], qm_dt[3];            // per species: charge, mass, q/m x particle step
  int nr, nz;
  int wrap;                               // azimuth: 0 full ring, 1 wedge of at most pi/2, 2 any other wedge
  bool atan_phi, euler, fast_fx;          // fast_fx: |fixed-point contribution| <= 2^50
  unsigned long long *Jr, *Jz;            // deposit target
};

__device__ __forceinline__ int species_of(const Species &s, int64_t o) {
  return o >= s.start[2] ? 2 : (o >= s.start[1] ? 1 : 0);
}

// EM2.cu:26-57 / EM4.cu:146-177: drift by half a step, delete beyond Rp, wrap
// the azimuth into the wedge turning the velocity with it, reflect at z = 0
// and Lp.  (c, s): cosine and sine of the new azimuth.  On a wedge of at most
// pi/2 the tests phi < 0 and phi > PHIp are the signs of sin(phi) and
// sin(phi - PHIp); atan(y/x) (atan_phi) is the azimuth of (|x|, y sign(x)).
__device__ __forceinline__ void em_halfdrift(const EmParams &g, double &x, double &y, double &z, double &vx,
                                             double &vy, double &vz, double &r, double &c, double &s,
                                             bool &del) {
  const double X = fma(g.hdt, vx, x), Y = fma(g.hdt, vy, y);
  double Z = fma(g.hdt, vz, z);
  r = sqrt(fma(X, X, Y * Y));
  const double ir = 1 / r;
  if (r > g.Rp) del = true;
  if (g.wrap == 2) {
    double phi = g.atan_phi ? atan(Y / X) : atan2(Y, X);
    // bounded: a wrap count above 2^20 means phi is not finite-sized
    for (int it = 0; phi < 0 && it < (1 << 20); ++it) {
      phi = phi + g.PHIp;
      const double w = vx * g.cP - vy * g.sP;
      vy = vx * g.sP + vy * g.cP;
      vx = w;
    }
    for (int it = 0; phi > g.PHIp && it < (1 << 20); ++it) {
      phi = phi - g.PHIp;
      const double w = vx * g.cP + vy * g.sP;
      vy = -vx * g.sP + vy * g.cP;
      vx = w;
    }
    sincos(phi, &s, &c);
  } else {
    if (g.atan_phi) {
      c = fabs(X) * ir;
      s = (signbit(X) ? -Y : Y) * ir;
    } else {
      c = r > 0 ? X * ir : 1.0;
      s = r > 0 ? Y * ir : 0.0;
    }
    if (g.wrap) {
      const double s0 = s;
      for (int it = 0; s < 0 && it < (1 << 20); ++it) {
        const double k = c * g.cP - s * g.sP;
        s = c * g.sP + s * g.cP;
        c = k;
        const double w = vx * g.cP - vy * g.sP;
        vy = vx * g.sP + vy * g.cP;
        vx = w;
      }
      for (int it = 0; s * g.cP - c * g.sP > 0 && it < (1 << 20); ++it) {
        const double k = c * g.cP + s * g.sP;
        s = -c * g.sP + s * g.cP;
        c = k;
        const double w = vx * g.cP + vy * g.sP;
        vy = -vx * g.sP + vy * g.cP;
        vx = w;
      }
      // the turns' roundings off the length of (c, s), which would become the radius
      // (thousands of turns into a narrow wedge: 1e-13)
      if (s != s0) {
        const double k = fma(-0.5, fma(c, c, s * s), 1.5);
        c *= k;
        s *= k;
      }
    }
  }
  x = r * c;
  y = r * s;
  if (Z > g.Lp) { Z = 2 * g.Lp - Z; vz = -vz; }
  if (Z < 0) { Z = -Z; vz = -vz; }
  z = Z;
}

// k b rounded to a whole number.  In one FMA where it is known to be at most
// 2^50 (fast) - but for velocities or positions that are not finite (on the axis atan(y/x) is
// none) or far beyond the speed of light: the sum has then left the binade of
// 1.5 2^52, and the conversion's rules hold.
__device__ __forceinline__ long long em_fixed(bool fast, double k, double b) {
  if (fast) {
    const double v = fma(k, b, 6755399441055744.0);
    if ((__double2hiint(v) >> 20) == 0x433) return __double_as_longlong(v) - 0x4338000000000000LL;
  }
  return __double2ll_rn(k * b);
}

// EM7.cu:51-202: q FN v w of a particle at (r, z) into its four nodes, in fixed point
__device__ __forceinline__ void em_deposit(const EmParams &g, double r, double z, double vr, double vz,
                                           double q) {
  const Axis64 R = axis64(r * g.id, g.nr), Z = axis64(z * g.id, g.nz);
  const double k = g.FN * q * g.scale, kr = k * vr, kz = k * vz;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int64_t a = (n & 1 ? R.hi : R.lo) + (int64_t)(n & 2 ? Z.hi : Z.lo) * g.nr;
    const double b = (n & 1 ? R.w : 1 - R.w) * (n & 2 ? Z.w : 1 - Z.w);
    const long long vr_fx = em_fixed(g.fast_fx, kr, b), vz_fx = em_fixed(g.fast_fx, kz, b);
    if (vr_fx) atomicAdd(g.Jr + a, (unsigned long long)vr_fx);
    if (vz_fx) atomicAdd(g.Jz + a, (unsigned long long)vz_fx);
  }
}

// the first half drift of a step and its deposit (EM2.cu, EM7.cu)
__device__ __forceinline__ void em_first_half(const EmParams &g, double &x, double &y, double &z, double &vx,
                                              double &vy, double &vz, double q, bool &del) {
  double r, c, s;
  em_halfdrift(g, x, y, z, vx, vy, vz, r, c, s, del);
  if (!del) em_deposit(g, r, z, fma(vx, c, vy * s), vz, q);
}

// electricmagneticfield6.m:65-73, 113-118: concatenate the three species; with
// steps to take, the first half drift and deposit
__global__ void k_em_load(Species sp, EmState st, EmParams g, int64_t N, bool cyl, bool steps) {
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < N;
       o += (int64_t)gridDim.x * blockDim.x) {
    const int k = species_of(sp, o);
    const int64_t i = o - sp.start[k], ld = sp.n[k];
    double x = sp.pos[k][i], y = sp.pos[k][ld + i], z = sp.pos[k][2 * ld + i];
    if (cyl) {
      double c, s;
      sincos(y, &s, &c);
      y = x * s;
      x = x * c;
    }
    double vx = sp.vel[k][i], vy = sp.vel[k][ld + i], vz = sp.vel[k][2 * ld + i];
    bool del = false;
    if (steps) em_first_half(g, x, y, z, vx, vy, vz, g.q[k], del);
    st.x[o] = x; st.y[o] = y; st.z[o] = z;
    st.vx[o] = vx; st.vy[o] = vy; st.vz[o] = vz;
    st.of[o] = del ? ~(int)o : (int)o;
  }
}

// Counting sort of the slots by grid cell (the departed last), so that
// neighbouring threads gather from and deposit to neighbouring nodes.  Two
// passes, the second from one set of slots to the other; both work the cell
// out, to the same bits (an explicit fma).  Bound by scattered stores: 23 us
// for 260,000 particles.  The deposits are whole numbers, so the order leaves
// the results as they are.
__device__ __forceinline__ int em_cell(const EmState &st, const EmParams &g, int64_t p) {
  if (st.of[p] < 0) return g.nr * g.nz;
  const double x = st.x[p], y = st.y[p];
  const int i = (int)(sqrt(fma(x, x, y * y)) * g.id), j = (int)(st.z[p] * g.id);
  return min(max(i, 0), g.nr - 1) + min(max(j, 0), g.nz - 1) * g.nr;
}

__global__ void k_em_count(EmState st, EmParams g, int64_t N, int *count, int *rank) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x)
    rank[p] = atomicAdd(count + em_cell(st, g, p), 1);
}

__global__ void k_em_scatter(EmState a, EmState b, EmParams g, int64_t N, const int *__restrict__ offset,
                             const int *__restrict__ rank) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t d = offset[em_cell(a, g, p)] + (int64_t)rank[p];
    b.x[d] = a.x[p]; b.y[d] = a.y[p]; b.z[d] = a.z[p];
    b.vx[d] = a.vx[p]; b.vy[d] = a.vy[p]; b.vz[d] = a.vz[p];
    b.of[d] = a.of[p];
  }
}

// EM4.cu:33-177, then (more steps to come) EM2.cu and EM7.cu of the next step
template <bool LAST>
__global__ void __launch_bounds__(kBlock) k_em_push(Species sp, EmState st, EmParams g, int64_t N,
                                                    const double *Er, const double *Ez,
                                                    const double *H, double *E) {
  wait_for_previous();
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < N;
       o += (int64_t)gridDim.x * blockDim.x) {
    const int of = st.of[o];
    if (of < 0) continue;
    const int k = species_of(sp, of);
    double x = st.x[o], y = st.y[o], z = st.z[o], vx = st.vx[o], vy = st.vy[o], vz = st.vz[o];
    double r = sqrt(fma(x, x, y * y));
    const double ir = 1 / r;
    double c = x * ir, s = y * ir;
    if (!g.atan_phi && !(r > 0)) { c = 1; s = 0; }
    // the staggered bilinear gather (EM4.cu:41-122), one-sided at the edges
    const Axis64 R = axis64(r * g.id, g.nr), Z = axis64(z * g.id, g.nz);
    const double *e0 = Er + (int64_t)Z.i * g.nr, *e1 = e0 + g.nr;
    const double *z0 = Ez + (int64_t)Z.lo * (g.nr + 1) + R.i, *z1 = Ez + (int64_t)Z.hi * (g.nr + 1) + R.i;
    const double *h0 = H + (int64_t)Z.lo * g.nr, *h1 = H + (int64_t)Z.hi * g.nr;
    const double Er0 = lerp64(lerp64(e0[R.lo], e0[R.hi], R.w), lerp64(e1[R.lo], e1[R.hi], R.w), Z.f);
    const double Ez0 = lerp64(lerp64(z0[0], z0[1], R.f), lerp64(z1[0], z1[1], R.f), Z.w);
    const double H0 = lerp64(lerp64(h0[R.lo], h0[R.hi], R.w), lerp64(h1[R.lo], h1[R.hi], R.w), Z.w);
    const double g0 = rsqrt(1 - (vx * vx + vy * vy + vz * vz) * g.ic2);
    double ux = g0 * vx, uy = g0 * vy, uz = g0 * vz;
    if (g.euler) {
      const double B = H0 * g.mu, vr = vx * c + vy * s;
      const double fr = g.qm_dt[k] * (Er0 - vz * B);
      ux = fma(fr, c, ux);
      uy = fma(fr, s, uy);
      uz = fma(g.qm_dt[k], Ez0 + vr * B, uz);
    } else {
      const double B = g.mu * H0;
      boris(ux, uy, uz, Er0 * c, Er0 * s, Ez0, -B * s, B * c, 0.0, 0.5 * g.qm_dt[k], g.c);
    }
    const double u2 = 1 + (ux * ux + uy * uy + uz * uz) * g.ic2;
    if (LAST) E[of] = (sqrt(u2) - 1) * g.m[k] * g.c * g.c;
    const double ig = rsqrt(u2);
    vx = ux * ig; vy = uy * ig; vz = uz * ig;
    bool del = false;
    em_halfdrift(g, x, y, z, vx, vy, vz, r, c, s, del);
    if (!LAST && !del) em_first_half(g, x, y, z, vx, vy, vz, g.q[k], del);
    st.x[o] = x; st.y[o] = y; st.z[o] = z;
    st.vx[o] = vx; st.vy[o] = vy; st.vz[o] = vz;
    if (del) st.of[o] = ~of;
  }
  let_next_start();
}

// `pairs` H and E updates of the field sub-cycle (EM3_1.cu:2-17, EM3.cu:2-43;
// electricmagneticfield6.m:146-151 calls ten pairs between a first and a last
// H update of dt/4) in one launch, from one set of fields to another: a block
// of kEmWarps warps owns a patch of 32 columns (a lane each) x kEmRows rows,
// each warp kEmSeg consecutive rows in registers.  Horizontal neighbours are
// shuffles, vertical ones registers, and between warps one row in shared
// memory per update.  An E update reads one column and row below, an H update one above,
// so `pairs` columns and rows on the low side and pairs + 1 on the high side of
// a patch are recomputed by its neighbours instead of exchanged.  Points outside the grid
// take the same expressions on zeros; no point inside reads them
// (fdtd_block_body has the same rules).  The first H update takes h_first, the
// others dt/2; a last one takes h_last (0: none).
constexpr int kEmWarps = 8, kEmSeg = 8, kEmRows = kEmWarps * kEmSeg;

struct EmFields { const double *Er, *Ez, *H; double *oEr, *oEz, *oH; };

struct EmFieldParams {
  int nr, nz, pairs;
  int tiles_x;                            // tiles across (one block per tile, a row of tiles after the other)
  double delta, PHIp, inv_scale, dt_eps, dt_eps_dz, axis;
  double h_first, h_mid, h_last;          // h / (mu delta)
  bool endcopy, jsign, rshift;
};

__host__ __device__ inline int em_tile_cols(int pairs) { return 32 - 2 * pairs - 1; }
__host__ __device__ inline int em_tile_rows(int pairs) { return kEmRows - 2 * pairs - 1; }

__global__ void __launch_bounds__(32 * kEmWarps) k_em_fields(EmFields f, EmFieldParams P,
                                                             const unsigned long long *Jr,
                                                             const unsigned long long *Jz,
                                                             unsigned long long *Jr_next,
                                                             unsigned long long *Jz_next) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int S = kEmSeg;
  // the rows of a segment its neighbours read: first and last Er, last H
  // (the Er rows in two buffers by turns: an E update reads one while others write the other)
  __shared__ double s_first[2][kEmWarps][32], s_last[2][kEmWarps][32], s_h[kEmWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nr = P.nr, nz = P.nz;
  const int ty = (int)blockIdx.x / P.tiles_x, tx = (int)blockIdx.x - ty * P.tiles_x;
  const int col = tx * em_tile_cols(P.pairs) - P.pairs + lane;
  const int y0 = ty * em_tile_rows(P.pairs) - P.pairs + w * S;     // the segment's first row
  const bool in = col >= 0 && col < nr;
  double iv = 0, ezp = 0, ezm = 0;        // coefficients of EM3.cu; Ez at column n_r stays as it is
  if (in) {
    iv = P.inv_scale / shell_volume(col, P.delta, P.delta, P.PHIp);
    const double ri = (P.rshift ? col + 1 : col) * P.delta, id = 1 / P.delta;
    ezp = col == 0 ? P.axis : P.dt_eps * (1 / (2 * ri) + id);
    ezm = col == 0 ? 0.0 : P.dt_eps * (1 / (2 * ri) - id);
  }
  double er[S], ez[S], h[S], jr[S], jz[S];
  wait_for_previous();
  {
    auto current = [&](const unsigned long long *J, int j) {
      return in && j >= 0 && j < nz ? (double)(long long)J[col + (int64_t)j * nr] * iv : 0.0;
    };
    double below = current(Jr, y0 - 1);
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const int j = y0 + r;
      const bool row = j >= 0 && j < nz;
      er[r] = in && j >= 0 && j <= nz ? f.Er[col + (int64_t)j * nr] : 0.0;
      ez[r] = col >= 0 && col <= nr && row ? f.Ez[col + (int64_t)j * (nr + 1)] : 0.0;
      h[r] = in && row ? f.H[col + (int64_t)j * nr] : 0.0;
      const double a = current(Jr, j);
      jr[r] = P.dt_eps * (below + a) / 2;
      below = a;
      jz[r] = current(Jz, j);
    }
  }
#pragma unroll
  for (int r = 0; r < S; ++r) {
    const double left = __shfl_up_sync(FULL, jz[r], 1);
    jz[r] = col == 0 ? (P.jsign ? -(P.dt_eps * jz[r]) : P.dt_eps * jz[r]) : in ? P.dt_eps * (left + jz[r]) / 2 : 0.0;
  }
  const int up = min(w + 1, kEmWarps - 1), dn = max(w - 1, 0);
  const int r0 = -y0, rn = nz - y0;       // the end rows 0 and n_z of Er in this segment
  auto publish_e = [&](int b) {
    s_first[b][w][lane] = er[0];
    s_last[b][w][lane] = er[S - 1];
    __syncthreads();
  };
  auto h_update = [&](double k, int b) {
    const double above = s_first[b][up][lane];
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const double right = __shfl_down_sync(FULL, ez[r], 1);
      const double e1 = r + 1 < S ? er[r + 1 < S ? r + 1 : r] : above;
      h[r] = fma(k, (right - ez[r]) - (e1 - er[r]), h[r]);
    }
  };
  auto e_update = [&](int b) {
    const double below = s_h[dn][lane], er_up = s_first[b][up][lane], er_dn = s_last[b][dn][lane];
    double ne[S];
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const double left = __shfl_up_sync(FULL, h[r], 1), hl = col > 0 ? left : 0.0;
      const double hb = r > 0 ? h[r > 0 ? r - 1 : 0] : below;
      ne[r] = fma(-P.dt_eps_dz, h[r] - hb, er[r] - jr[r]);
      if (in) ez[r] = fma(ezm, hl, fma(ezp, h[r], ez[r] - jz[r]));
    }
    if ((r0 >= 0 && r0 < S) || (rn >= 0 && rn < S)) {
#pragma unroll
      for (int r = 0; r < S; ++r) {
        if (r == r0) ne[r] = P.endcopy ? (r + 1 < S ? er[r + 1 < S ? r + 1 : r] : er_up) : 0.0;
        if (r == rn) ne[r] = P.endcopy ? (r > 0 ? er[r > 0 ? r - 1 : 0] : er_dn) : 0.0;
      }
    }
#pragma unroll
    for (int r = 0; r < S; ++r) er[r] = ne[r];
  };
  publish_e(0);
  for (int p = 0; p < P.pairs; ++p) {
    h_update(p == 0 ? P.h_first : P.h_mid, p & 1);
    s_h[w][lane] = h[S - 1];
    __syncthreads();
    e_update(p & 1);
    publish_e((p & 1) ^ 1);
  }
  if (P.h_last != 0) h_update(P.h_last, P.pairs & 1);
  // write the tile back, and clear it in the next deposit's current
  if (lane < P.pairs || lane >= 32 - P.pairs - 1 || col > nr) return;
#pragma unroll
  for (int r = 0; r < S; ++r) {
    const int j = y0 + r, pr = w * S + r;
    if (pr < P.pairs || pr >= kEmRows - P.pairs - 1 || j > nz) continue;
    const int64_t a = col + (int64_t)j * nr;
    if (in) f.oEr[a] = er[r];
    if (j < nz) {
      f.oEz[col + (int64_t)j * (nr + 1)] = ez[r];
      if (in) {
        f.oH[a] = h[r];
        Jr_next[a] = 0;
        Jz_next[a] = 0;
      }
    }
  }
  let_next_start();                     // (a lane that returned has signalled by that)
}

// counts[0..3]: the scan at the species' starts and the end; electricmagneticfield6.m:168-188
// with each species compacted by its own delete flags; pos[] is the exclusive
// scan of the keep flags (N+1 entries)
__global__ void k_em_store(Species sp, EmState st, int64_t N, const int *pos, const double *E, double *kin,
                           double e, int *counts) {
  if (blockIdx.x == 0 && threadIdx.x < 4) counts[threadIdx.x] = pos[threadIdx.x < 3 ? sp.start[threadIdx.x] : N];
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int o = st.of[p];
    if (o < 0) continue;
    const int s = species_of(sp, o);
    const int64_t w = pos[o] - pos[sp.start[s]], ld = sp.n[s];
    sp.pos[s][w] = st.x[p]; sp.pos[s][ld + w] = st.y[p]; sp.pos[s][2 * ld + w] = st.z[p];
    sp.vel[s][w] = st.vx[p]; sp.vel[s][ld + w] = st.vy[p]; sp.vel[s][2 * ld + w] = st.vz[p];
    if (s == 0 && kin) kin[w] = (E ? E[o] : 0.0) / (1000 * e);
  }
}

// keep[o]: particle o is still there (N + 1 entries, the last 0)
__global__ void k_keep_flags(EmState st, int64_t N, int *keep) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p <= N;
       p += (int64_t)gridDim.x * blockDim.x)
    if (p < N) {
      const int o = st.of[p];
      keep[o < 0 ? ~o : o] = o >= 0;
    } else {
      keep[N] = 0;
    }
}

// ------------------------------------------------------- electron_collision
// The table set-up, the test of every electron
// (k_collision_select: density cell, collision test, branch), and the
// collisions alone (k_collision_elastic, k_collision_other), compacted by branch.  One thread per
// electron that ran whatever befell it took 461 us for 200,000 electrons: an
// elastic angle evaluates the 181-angle PDF up to three times, and most lanes
// of a warp wait for the few that collide.
struct MccTables {
  const double *xI, *yI, *V;  int ne;
  const double *exc;  int n_exc;     // n_exc x 5 column-major
  const double *dphi; const int *sum_cell0; int rmax; int cellnumxy;
  const double *density, *temperature; int64_t ncell;
};

// the raw tables packed in one upload (offsets in doubles)
struct MccRaw {
  const double *sel1, *el, *sdel, *del;
  int n_sel1, n_el, sdel_cols, del_cols;
};

// electron_collision.m:12-33 as build_elastic_tables (tables.cpp): combined
// cross-sections and the logarithms of the energies and DCS columns
__global__ void k_collision_tables(MccRaw t, double *xI, double *yI, double *V) {
  const int m1 = t.n_sel1 - 1, ns = t.sdel_cols - 1, ne = ns + t.del_cols - 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ne * 182; i += gridDim.x * blockDim.x) {
    const int c = i / 182, k = i - c * 182;
    const double v = log(c < ns ? t.sdel[(int64_t)(c + 1) * 182 + k] : t.del[(int64_t)(c - ns + 1) * 182 + k]);
    if (k == 0) {
      xI[c] = v;
      yI[c] = c < m1 ? t.sel1[t.n_sel1 + c] * 1e-20 / GASATT_A0SQ / 2 : t.el[2 * (c - m1) + 1];
    } else {
      V[(int64_t)c * 181 + k - 1] = v;
    }
  }
}

__device__ __forceinline__ double pow_sel(double a, double b, unsigned flags) {
  if (flags & GASATT_Q_EXC_POWF) return (double)powf((float)a, (float)b);
  return pow(a, b);
}

struct MccOut {
  int *sec;                          // 1: a secondary is born (n + 1 entries, the last 0)
  double *svx, *svy, *svz, *sample, *ivx, *ivy, *ivz;
};

// colliding electrons by branch: elastic ones, and the others (an ionization
// as ~index); n[0], n[1]: how many
struct MccLists { int *elastic, *other; unsigned *n; };

__device__ __forceinline__ void list_push(bool want, int v, unsigned *n, int *list) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(n, (unsigned)__popc(m));
  base = __shfl_sync(0xFFFFFFFFu, base, leader);
  if (want) list[base + __popc(m & ((1u << lane) - 1))] = v;
}

// electron_transport.cu:64-87, 127-128, 139: the density cell, the collision
// test and the branch of every electron
__global__ void k_collision_select(const double *__restrict__ pos, const double *__restrict__ vel, int64_t cap,
                                   int64_t n, const double *__restrict__ sig_el,
                                   const double *__restrict__ sig_ion, const double *__restrict__ sig_exc,
                                   const double *__restrict__ energy, MccTables t, MccOut out, MccLists ls,
                                   double dr, double dz, double dt, const double *__restrict__ draws,
                                   uint64_t seed, int64_t call, unsigned flags) {
  const double I = GASATT_ION_I_EV;
  const int lane = threadIdx.x & 31;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base <= n;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = base + lane;
    bool elastic = false, other = false, ion = false;
    if (p <= n) out.sec[p] = 0;
    if (p < n) {
      double U0, U1;
      if (draws) {
        U0 = draws[p * GASATT_MCC_NDRAW];
        U1 = draws[p * GASATT_MCC_NDRAW + 1];
      } else {
        const U2 a = draw2(seed, (uint64_t)p, call, 0);
        U0 = a.a; U1 = a.b;
      }
      const double vx = vel[p], vy = vel[cap + p], vz = vel[2 * cap + p];
      const double x = pos[p], y = pos[cap + p], z = pos[2 * cap + p];
      const double v_e = sqrt(vx * vx + vy * vy + vz * vz);
      const double dx = v_e * dt;
      const double r = sqrt(x * x + y * y);
      const double phi = atan(y / x);
      int iz = (int)floor(z / dz), ir = (int)floor(r / dr);
      if (ir > t.rmax - 1) ir = t.rmax - 1;
      if (ir < 0) ir = 0;
      int iphi = (int)floor(phi / t.dphi[ir]);
      const int nphi = t.sum_cell0[ir + 1] - t.sum_cell0[ir];
      if (iphi > nphi - 1) iphi = nphi - 1;
      if (iphi < 0) iphi = 0;
      int64_t index = (int64_t)iz * t.cellnumxy + t.sum_cell0[ir] + iphi;
      if (index < 0) index = 0;
      if (index > t.ncell - 1) index = t.ncell - 1;
      const double den = t.density[index];
      const double p_el = dx * den * sig_el[p];
      const double p_io = dx * den * sig_ion[p];
      const double p_ex = dx * den * sig_exc[p];
      double p_tot = p_el + p_io + p_ex;
      const double a = p_el / p_tot;
      const double b = a + p_io / p_tot;
      if (!(flags & GASATT_Q_COLL_LINEAR_P)) p_tot = -expm1(-p_tot);
      if (U0 < p_tot) {
        elastic = U1 < a;
        other = !elastic;
        ion = other && U1 < b && energy[p] > I / 1000;
        if (ion) out.sample[p] = (double)index;
      }
    }
    list_push(elastic, (int)p, ls.n, ls.elastic);
    list_push(other, ion ? ~(int)p : (int)p, ls.n + 1, ls.other);
  }
}

// Elastic angles, kElGroup electrons per block: its warps evaluate the PDF of
// each at the 181 angles, a lane per angle, into shared memory; then a lane
// per electron forms the CDF in the reference's order and inverts it.  Bound
// by instruction issue (the exponentials: 181 an electron); 107,000 elastic
// collisions take 97 us.
constexpr int kElGroup = 32, kElThreads = 256;
constexpr int kElSmem = (kElGroup + 1) * 181 * 8;    // the PDFs (181 apart: no bank conflicts), and the sines

struct ElasticAt { int i; double a0, b0, inv_tcs; };

// electron_transport.cu:88-102: the energy columns around an electron's energy
// (by a whole warp: the first column whose upper end is not below it)
__device__ __forceinline__ ElasticAt elastic_at(double energy, const MccTables &t, unsigned flags) {
  const double *xI = t.xI;
  double Ee = (flags & GASATT_Q_XS_LINEAR_E) ? energy : log(energy);
  if (!(flags & GASATT_Q_XS_LINEAR_E)) {
    if (Ee < xI[0]) Ee = xI[0];
    if (Ee > xI[t.ne - 1]) Ee = xI[t.ne - 1];
  }
  ElasticAt e;
  const int lane = threadIdx.x & 31;
  e.i = t.ne - 2;
  for (int k = 0; k < t.ne - 2; k += 32) {
    const unsigned stop = __ballot_sync(0xFFFFFFFFu, k + lane < t.ne - 2 && !(Ee > xI[k + lane + 1]));
    if (stop) { e.i = k + __ffs(stop) - 1; break; }
  }
  e.a0 = (xI[e.i + 1] - Ee) / (xI[e.i + 1] - xI[e.i]);
  e.b0 = (Ee - xI[e.i]) / (xI[e.i + 1] - xI[e.i]);
  e.inv_tcs = 1 / ((e.a0 * t.yI[e.i] + e.b0 * t.yI[e.i + 1]) * 2);
  return e;
}

// The angle from f[k] = PDF(k degrees) pi / 180, k = 0..180 (the rectangles of
// the reference's CDF): electron_transport.cu:103-121 (GASATT_Q_CDF_NEXTBIN) or
// get_ElasticSc_sub1.m.  The running sums, added in the reference's order,
// replace f, and its walk up the CDF becomes a bisection (it stops at once
// where the sums are not above 0, else they rise).
__device__ double elastic_theta(double *f, const ElasticAt &e, const MccTables &t, double U, double pi,
                                unsigned flags) {
  double sum = 0, last = f[0];
  if (flags & GASATT_Q_CDF_NEXTBIN) {
#pragma unroll 8
    for (int k = 0; k <= 180; ++k) {
      sum = sum + f[k];
      f[k] = sum;                          // the first k + 1 rectangles
    }
    const double rnd = U * sum;
    int k = 0;                             // the first k with rnd <= the first k rectangles
    if (rnd > 0) {
      int lo = 0, hi = 181;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (rnd > f[mid - 1]) lo = mid; else hi = mid;
      }
      k = hi;
    }
    const double i1 = k > 0 ? f[k - 1] : 0.0;
    double i2;
    if (k < 181) {
      i2 = f[k];
    } else {             // the reference goes on into the next column (clamped to the table)
      const int64_t end = (int64_t)t.ne * 181 - 1, i1k = (int64_t)e.i * 181 + k, i2k = i1k + 181;
      const double vI = e.a0 * t.V[i1k < end ? i1k : end] + e.b0 * t.V[i2k < end ? i2k : end];
      i2 = i1 + e.inv_tcs * (2 * pi * sin(k * pi / 180) * exp(vI) * 2) * pi / 180;
    }
    const double aa = (i2 - rnd) / (i2 - i1), bb = (rnd - i1) / (i2 - i1);
    return (aa * (k - 1) + bb * k) * pi / 180;
  }
  // trapezoid CDF and linear inverse (cumtrapz + interp1)
  f[0] = 0;
#pragma unroll 4
  for (int k = 1; k <= 180; ++k) {
    const double fk = f[k];
    sum = sum + (last + fk) / 2;
    f[k] = sum;
    last = fk;
  }
  const double rn = U * sum;
  int lo = 0, hi = 180;                    // the first k with CDF(k) > rn, at most 180
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (f[mid] > rn) hi = mid; else lo = mid;
  }
  return ((hi - 1) + (rn - f[hi - 1]) / (f[hi] - f[hi - 1])) * (pi / 180);
}

__device__ __forceinline__ void late_draws(const double *draws, int64_t p, uint64_t seed, int64_t call, double &u2,
                                           double &u3) {
  if (draws) {
    u2 = draws[p * GASATT_MCC_NDRAW + 2];
    u3 = draws[p * GASATT_MCC_NDRAW + 3];
  } else {
    const U2 b = draw2(seed, (uint64_t)p, call, 1);
    u2 = b.a; u3 = b.b;
  }
}

// An ionization or excitation of electron p (electron_transport.cu:139-227)
__device__ __forceinline__ void collide_other(int64_t p, bool ion, double *vel, int64_t cap, double en,
                                              const MccTables &t, const MccOut &out, const double *draws,
                                              uint64_t seed, int64_t call, double pi, unsigned flags) {
  const double e = GASATT_MCC_E, c = GASATT_MCC_C, m = GASATT_MCC_ME, m_ion = GASATT_MCC_MION;
  const double kb = GASATT_MCC_KB, E_e = m * c * c / e, I = GASATT_ION_I_EV;
  double vx = vel[p], vy = vel[cap + p], vz = vel[2 * cap + p];
  const double v_e = sqrt(vx * vx + vy * vy + vz * vz);
  const double T = en * 1000;
  if (ion) {
    double u2, u3;
    late_draws(draws, p, seed, call, u2, u3);
    const double T_a = 1000, T_b = 2 * I, t_b = I, T_s = 4.17, t_s = 13.8;
    const double T_0 = T_s - T_a / (T + T_b);
    const double tt = t_s * T / (T + t_b);
    const double T_m = (T - I) / 2;
    const double k_1 = atan((T_m - T_0) / tt);
    const double k_2 = atan(T_0 / tt);
    const double k0 = T_0 + tt * tan(u2 * (k_1 + k_2) - k_2);
    const double E_1 = k0, E_2 = T - E_1 - I;
    double E_p, E_s;
    if (E_2 > E_1) { E_p = E_2; E_s = E_1; } else { E_p = E_1; E_s = E_2; }
    const double kk = (flags & GASATT_Q_SEC_LAB_FRAME) ? k0 : E_s;
    E_p = E_p * e;
    E_s = E_s * e;
    const double phi_p = 2 * pi * u3;
    const double phi_s = phi_p - pi;
    const double th_p = asin(sqrt((kk / T) / ((1 - kk / T) * T / (2 * E_e) + 1)));
    const double th_s = asin(sqrt((1 - kk / T) / (1 + kk / (2 * E_e))));
    const double ix = vx / v_e, iy = vy / v_e, iz_ = vz / v_e;
    double gamma = 1 + E_p / (m * c * c);
    const double v_p = c * sqrt(1 - 1 / (gamma * gamma));
    const double ratio = v_p / v_e;
    vx = ratio * vx; vy = ratio * vy; vz = ratio * vz;
    rotate_v(vx, vy, vz, th_p, phi_p, true);
    gamma = 1 + E_s / (m * c * c);
    const double v_s = c * sqrt(1 - 1 / (gamma * gamma));
    out.sec[p] = 1;
    if (flags & GASATT_Q_SEC_LAB_FRAME) {
      out.svx[p] = v_s * sin(th_s) * cos(phi_s);
      out.svy[p] = v_s * sin(th_s) * sin(phi_s);
      out.svz[p] = v_s * cos(th_s);
    } else {
      double sx = ix * v_s, sy = iy * v_s, sz = iz_ * v_s;
      rotate_v(sx, sy, sz, th_s, phi_s, true);
      out.svx[p] = sx; out.svy[p] = sy; out.svz[p] = sz;
    }
    double g[3];
    if (draws) {
      for (int k = 0; k < 3; ++k) g[k] = draws[p * GASATT_MCC_NDRAW + 4 + k];
    } else {
      const U2 g1 = draw2(seed, (uint64_t)p, call, 2), g2 = draw2(seed, (uint64_t)p, call, 3);
      const double rad1 = sqrt(-2 * log(g1.a)), rad2 = sqrt(-2 * log(g2.a));
      g[0] = rad1 * cos(2 * GASATT_PI * g1.b);
      g[1] = rad1 * sin(2 * GASATT_PI * g1.b);
      g[2] = rad2 * cos(2 * GASATT_PI * g2.b);
    }
    const double sd = sqrt(m_ion / (kb * t.temperature[(int64_t)out.sample[p]]));
    out.ivx[p] = (double)(float)g[0] / sd;
    out.ivy[p] = (double)(float)g[1] / sd;
    out.ivz[p] = (double)(float)g[2] / sd;
  } else {
    double k1 = 0, k2 = 0;
    for (int i = 0; i < t.n_exc; ++i) {
      const double k = t.exc[i], A = t.exc[t.n_exc + i], om = t.exc[2 * t.n_exc + i];
      const double nu = t.exc[3 * t.n_exc + i], ga = t.exc[4 * t.n_exc + i];
      if (!(flags & GASATT_Q_EXC_POWF) && !(T > k)) continue;
      const double aE = GASATT_MCC_Q0 * A / (k * k);
      const double bE = pow_sel(k / T, om, flags);
      const double cE = pow_sel(pow_sel(1 - k / T, ga, flags), nu, flags);
      k1 = k1 + aE * bE * cE * k;
      k2 = k2 + aE * bE * cE;
    }
    if (k2 == 0) return;
    const double E_dep = k1 / k2;
    const double E_p = T - E_dep;
    const double gamma = 1 + E_p * e / (m * c * c);
    const double v_p = c * sqrt(1 - 1 / (gamma * gamma));
    const double ratio = v_p / v_e;
    vx = ratio * vx; vy = ratio * vy; vz = ratio * vz;
  }
  vel[p] = vx; vel[cap + p] = vy; vel[2 * cap + p] = vz;
}

// the ionizations and excitations (electron_transport.cu:139-227), one per thread
__global__ void k_collision_other(double *vel, int64_t cap, const double *__restrict__ energy, MccTables t,
                                  MccOut out, MccLists ls, const double *__restrict__ draws, uint64_t seed,
                                  int64_t call, unsigned flags) {
  const double pi = (flags & GASATT_Q_PI7) ? GASATT_MCC_PI7 : GASATT_PI;
  const unsigned n = ls.n[1];
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int v = ls.other[k], p = v < 0 ? ~v : v;
    collide_other(p, v < 0, vel, cap, energy[p], t, out, draws, seed, call, pi, flags);
  }
}

// the elastic collisions (electron_transport.cu:88-135), in groups
__global__ void __launch_bounds__(kElThreads) k_collision_elastic(double *vel, int64_t cap,
                                                                  const double *__restrict__ energy, MccTables t,
                                                                  MccLists ls, const double *__restrict__ draws,
                                                                  uint64_t seed, int64_t call, unsigned flags) {
  extern __shared__ double el_smem[];
  __shared__ ElasticAt at[kElGroup];
  const double pi = (flags & GASATT_Q_PI7) ? GASATT_MCC_PI7 : GASATT_PI;
  const unsigned n = ls.n[0];
  double *sines = el_smem + kElGroup * 181;
  for (int k = threadIdx.x; k < 181; k += kElThreads) sines[k] = 4 * pi * sin(k * pi / 180) * (pi / 180);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned g = blockIdx.x * kElGroup; g < n; g += gridDim.x * kElGroup) {
    const int m = min(n - g, (unsigned)kElGroup);
    __syncthreads();                      // the last group's PDFs are no longer read
    for (int j = warp; j < m; j += kElThreads / 32) {
      const ElasticAt e = elastic_at(energy[ls.elastic[g + j]], t, flags);
      if (lane == 0) at[j] = e;
      // electron_transport.cu:103-109
      const double *V = t.V + e.i * 181 + lane;
      double *f = el_smem + j * 181 + lane;
#pragma unroll
      for (int k = 0; k < 181; k += 32)
        if (k + lane < 181) f[k] = e.inv_tcs * sines[k + lane] * exp(e.a0 * V[k] + e.b0 * V[k + 181]);
    }
    __syncthreads();
    if ((int)threadIdx.x < m) {
      const int64_t p = ls.elastic[g + threadIdx.x];
      double u2, u3;
      late_draws(draws, p, seed, call, u2, u3);
      const double th = elastic_theta(el_smem + threadIdx.x * 181, at[threadIdx.x], t, u2, pi, flags);
      double vx = vel[p], vy = vel[cap + p], vz = vel[2 * cap + p];
      rotate_v(vx, vy, vz, th, 2 * pi * u3, true);
      vel[p] = vx; vel[cap + p] = vy; vel[2 * cap + p] = vz;
    }
  }
}

// electron_collision.m:63-75: append secondaries and ions in parent order
__global__ void k_append(double *e_pos, double *e_vel, int64_t cap_e, int64_t n_e,
                         double *i_pos, double *i_vel, int64_t cap_i, int64_t n_i,
                         const int *pos, MccOut out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n_e;
       p += (int64_t)gridDim.x * blockDim.x) {
    if (!out.sec[p]) continue;
    const int64_t we = n_e + pos[p], wi = n_i + pos[p];
    for (int d = 0; d < 3; ++d) {
      const double v = e_pos[d * cap_e + p];
      e_pos[d * cap_e + we] = v;
      i_pos[d * cap_i + wi] = v;
    }
    e_vel[we] = out.svx[p]; e_vel[cap_e + we] = out.svy[p]; e_vel[2 * cap_e + we] = out.svz[p];
    i_vel[wi] = out.ivx[p]; i_vel[cap_i + wi] = out.ivy[p]; i_vel[2 * cap_i + wi] = out.ivz[p];
  }
}

int exclusive_scan(gasatt_ctx *ctx, const int *in, int *out, int64_t n, void *tmp, size_t tmp_bytes) {
  size_t need = 0;
  GASATT_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, need, in, out, (int)n, ctx->stream));
  if (need > tmp_bytes) return fail(ctx, GASATT_E_ARG, "scan scratch too small");
  GASATT_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, need, in, out, (int)n, ctx->stream));
  ctx->launches++;
  return GASATT_OK;
}

size_t scan_tmp_bytes(int64_t n) {
  size_t need = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, need, (const int *)nullptr, (int *)nullptr, (int)n);
  return need + 256;
}

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// device copy of a host array into a carved scratch region
struct Carver {
  char *base; size_t off = 0;
  template <typename T> T *take(size_t n) {
    T *p = (T *)(base + off);
    off += align256(n * sizeof(T));
    return p;
  }
};

}  // namespace

// ====================================================================== C ABI
extern "C" {

int gasatt_find_CS0(gasatt_ctx *ctx, const gasatt_tables *tab, const double *E_keV, int64_t n,
                    double *sig_el, double *sig_ion, double *sig_exc, unsigned flags) {
  if (!ctx) return GASATT_E_ARG;
  std::string err;
  int st = check_tables(tab, err);
  if (st) return fail(ctx, st, err);
  if (n < 0 || (n > 0 && (!E_keV || !sig_el || !sig_ion || !sig_exc)))
    return fail(ctx, GASATT_E_ARG, "find_CS0: bad arrays");
  if (n == 0) return GASATT_OK;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t ne = 2 * (size_t)tab->n_el, ns = 2 * (size_t)tab->n_sel, ni = 2 * (size_t)tab->n_ion,
               nx = 5 * (size_t)tab->n_exc;
  void *buf;
  st = scratch(ctx, (ne + ns + ni + nx) * 8, &buf);
  if (st) return st;
  // one upload of the four tables
  std::vector<double> host(ne + ns + ni + nx);
  std::memcpy(host.data(), tab->t_el, ne * 8);
  std::memcpy(host.data() + ne, tab->t_sel, ns * 8);
  std::memcpy(host.data() + ne + ns, tab->t_ion, ni * 8);
  std::memcpy(host.data() + ne + ns + ni, tab->t_exc, nx * 8);
  const double *d = (const double *)buf;
  GASATT_CUDA(ctx, cudaMemcpyAsync(buf, host.data(), host.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  XsRaw t{d, tab->n_el, d + ne, tab->n_sel, d + ne + ns, tab->n_ion, d + ne + ns + ni, tab->n_exc};
  k_find_cs0<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(t, E_keV, n, sig_el, sig_ion, sig_exc, flags);
  GASATT_LAUNCHED(ctx);
  GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GASATT_OK;
}

int gasatt_free_motion(gasatt_ctx *ctx, const double *vx, const double *vy, const double *vz,
                       const double *x, const double *y, const double *z, int64_t n, double dt,
                       double *xn, double *yn, double *zn, double *rn, double *phin) {
  if (!ctx || n < 0) return GASATT_E_ARG;
  if (n == 0) return GASATT_OK;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  k_free_motion<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(vx, vy, vz, x, y, z, n, dt, xn, yn, zn, rn, phin);
  GASATT_LAUNCHED(ctx);
  return GASATT_OK;
}

int gasatt_rebond(gasatt_ctx *ctx, double *pos, int64_t ld_pos, const double *r,
                  const double *phi, double *vel, int64_t ld_vel, int64_t n, double Lp,
                  double PHIp, int64_t *n_boundary) {
  if (!ctx || n < 0 || ld_pos < n || ld_vel < n || !(PHIp > 0) || !(Lp > 0))
    return fail(ctx, GASATT_E_ARG, "REBOND: bad sizes");
  if (n_boundary) *n_boundary = 0;
  if (n == 0) return GASATT_OK;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  void *buf;
  int st = scratch(ctx, 16, &buf);
  if (st) return st;
  unsigned long long *cnt = (unsigned long long *)buf, h[2] = {0, 0};
  GASATT_CUDA(ctx, cudaMemsetAsync(cnt, 0, 16, ctx->stream));
  // cos and sin of the wedge angle on the host, once, like the reference's
  // cos(PHIp) and sin(PHIp) of every wrap
  k_rebond<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(pos, ld_pos, r, phi, vel, ld_vel, n, Lp,
                                                             PHIp, std::cos(PHIp), std::sin(PHIp), cnt);
  GASATT_LAUNCHED(ctx);
  GASATT_CUDA(ctx, cudaMemcpyAsync(h, cnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
  GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (h[1]) return fail(ctx, GASATT_E_ARG, "REBOND: an azimuth lies more than 4096 wedges outside");
  if (n_boundary) *n_boundary = (int64_t)h[0];
  return GASATT_OK;
}

int gasatt_particle_density(gasatt_ctx *ctx, double dr, double dz, const double *dphi, int rmax,
                            const double *r, const double *phi, const double *z, int64_t n,
                            int cellnumxy, const double *sum_cell, const double *VC, int64_t ncell,
                            double FN, double *density) {
  if (!ctx || n < 0 || ncell <= 0 || rmax <= 0 || cellnumxy <= 0)
    return fail(ctx, GASATT_E_ARG, "particle_density: bad sizes");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  void *buf;
  int st = scratch(ctx, (size_t)ncell * 8, &buf);
  if (st) return st;
  unsigned long long *cnt = (unsigned long long *)buf;
  GASATT_CUDA(ctx, cudaMemsetAsync(cnt, 0, (size_t)ncell * 8, ctx->stream));
  if (n > 0) {
    k_density_count<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(dr, dz, dphi, rmax, r, phi, z, n,
                                                                     cellnumxy, sum_cell, ncell, cnt);
    GASATT_LAUNCHED(ctx);
  }
  k_density_finish<<<grid_for(ncell, kBlock), kBlock, 0, ctx->stream>>>(cnt, ncell, cellnumxy, VC, FN, density);
  GASATT_LAUNCHED(ctx);
  return GASATT_OK;
}

int gasatt_particle_density_noalloc(gasatt_ctx *ctx, double dr, double dz, const double *dphi,
                                    int rmax, const double *r, const double *phi, const double *z,
                                    int64_t n, int cellnumxy, const double *sum_cell,
                                    const double *VC, int64_t ncell, double FN, double *density) {
  if (!ctx || n < 0 || ncell <= 0 || rmax <= 0 || cellnumxy <= 0)
    return fail(ctx, GASATT_E_ARG, "particle_density_noalloc: bad sizes");
  if (ncell > (int64_t)GASATT_DENSITY_NOALLOC_MAX_CELLS)
    return fail(ctx, GASATT_E_CAPACITY,
                "particle_density_noalloc: ncell = " + std::to_string(ncell) +
                    " exceeds its fixed scratch of " +
                    std::to_string((long long)GASATT_DENSITY_NOALLOC_MAX_CELLS) +
                    " cells (use gasatt_particle_density)");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  unsigned long long *cnt = nullptr;
  int st = density_counts_on_device(ctx, &cnt);
  if (st) return st;
  // the array keeps the previous call's counts: clear the cells used now
  GASATT_CUDA(ctx, cudaMemsetAsync(cnt, 0, (size_t)ncell * 8, ctx->stream));
  if (n > 0) {
    k_density_count<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(dr, dz, dphi, rmax, r, phi, z, n,
                                                                     cellnumxy, sum_cell, ncell, cnt);
    GASATT_LAUNCHED(ctx);
  }
  k_density_finish<<<grid_for(ncell, kBlock), kBlock, 0, ctx->stream>>>(cnt, ncell, cellnumxy, VC, FN, density);
  GASATT_LAUNCHED(ctx);
  return GASATT_OK;
}

int gasatt_electricmagneticfield6(gasatt_ctx *ctx, double *e_pos, double *e_vel, int64_t n_e,
                                  double *i1_pos, double *i1_vel, int64_t n_i1, double *i2_pos,
                                  double *i2_vel, int64_t n_i2, double *Er, double *Ez,
                                  double *Hphi, int n_r, int n_z, double delta, double dt,
                                  double Rp, double Lp, double PHIp, double FN, int cycle_time,
                                  double *electron_kinetic, int64_t *n_e_out, int64_t *n_i1_out,
                                  int64_t *n_i2_out, unsigned flags) {
  if (!ctx) return GASATT_E_ARG;
  if (n_e < 0 || n_i1 < 0 || n_i2 < 0 || n_r < 1 || n_z < 2 || !(delta > 0) || cycle_time < 0)
    return fail(ctx, GASATT_E_ARG, "electricmagneticfield6: bad sizes");
  if (std::fabs(Rp / delta - n_r) > 1e-6 * n_r || std::fabs(Lp / delta - n_z) > 1e-6 * n_z)
    return fail(ctx, GASATT_E_ARG, "electricmagneticfield6: grid must be Rp/delta x Lp/delta");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  const int64_t N = n_e + n_i1 + n_i2;
  const size_t ncel = (size_t)n_r * n_z, nEr = (size_t)n_r * (n_z + 1), nEz = (size_t)(n_r + 1) * n_z;
  const int ratio = 5, steps = cycle_time / ratio;
  const bool sorted = steps >= kEmSortLeast && N >= kEmSortParticles;
  const int64_t nscan = (int64_t)ncel + 2 > N + 1 ? (int64_t)ncel + 2 : N + 1;
  const size_t sc = scan_tmp_bytes(nscan);
  // sorted: a second set of slots, which holds E and the scan once the sorts are done
  const size_t bytes = (sorted ? 12 : 7) * align256((size_t)(N + 1) * 8) + 3 * align256((size_t)(N + 1) * 4) +
                       (sorted ? 2 * align256((ncel + 2) * 4) : 0) + 4 * align256(ncel * 8) +
                       align256(nEr * 8) + align256(nEz * 8) + align256(ncel * 8) + align256(16) + align256(sc);
  void *buf;
  int st = scratch(ctx, bytes, &buf);
  if (st) return st;
  Carver cv{(char *)buf};
  EmState slots[2] = {};
  for (int i = 0; i < (sorted ? 2 : 1); ++i) {
    double **f[6] = {&slots[i].x, &slots[i].y, &slots[i].z, &slots[i].vx, &slots[i].vy, &slots[i].vz};
    for (double **d : f) *d = cv.take<double>(N + 1);
    slots[i].of = cv.take<int>(N + 1);
  }
  int *keep = cv.take<int>(N + 1);
  double *E = sorted ? nullptr : cv.take<double>(N + 1);
  int *scanned = sorted ? nullptr : cv.take<int>(N + 1);
  int *cell_count = sorted ? cv.take<int>(ncel + 2) : nullptr, *cell_first = sorted ? cv.take<int>(ncel + 2) : nullptr;
  int cur = 0;                                          // the slots in use
  unsigned long long *J[2][2];                          // [buffer][r, z]
  for (int i = 0; i < 4; ++i) J[i >> 1][i & 1] = cv.take<unsigned long long>(ncel);
  double *Er2 = cv.take<double>(nEr), *Ez2 = cv.take<double>(nEz), *H2 = cv.take<double>(ncel);
  int *counts = cv.take<int>(4);
  void *tmp = cv.take<char>(sc);
  Species sp;
  sp.pos[0] = e_pos; sp.pos[1] = i1_pos; sp.pos[2] = i2_pos;
  sp.vel[0] = e_vel; sp.vel[1] = i1_vel; sp.vel[2] = i2_vel;
  sp.n[0] = n_e; sp.n[1] = n_i1; sp.n[2] = n_i2;
  sp.start[0] = 0; sp.start[1] = n_e; sp.start[2] = n_e + n_i1;
  const double e = GASATT_EM_E, c = GASATT_EM_C, mu = GASATT_EM_MU, eps = GASATT_EM_EPS;
  const unsigned g = grid_for(N, kBlock);
  // fixed-point scale: |q FN v w| <= 2e FN c per particle, N particles per node at most
  const double bound = (double)(N > 0 ? N : 1) * 2 * e * std::fabs(FN) * c;
  const int S = (int)std::floor(std::log2(std::ldexp(1.0, 62) / bound));
  const double ddt = ratio * dt;                       // electricmagneticfield6.m:134-135
  EmParams ep;
  ep.Rp = Rp; ep.Lp = Lp; ep.PHIp = PHIp; ep.cP = std::cos(PHIp); ep.sP = std::sin(PHIp);
  ep.hdt = 0.5 * ddt;
  ep.id = 1 / delta; ep.mu = mu; ep.c = c; ep.ic2 = 1 / (c * c); ep.FN = FN; ep.scale = std::ldexp(1.0, S);
  for (int k = 0; k < 3; ++k) {
    ep.q[k] = k == 0 ? -e : k * e;
    ep.m[k] = k == 0 ? GASATT_EM_ME : GASATT_EM_MION;
    ep.qm_dt[k] = ep.q[k] / ep.m[k] * ddt;
  }
  ep.nr = n_r; ep.nz = n_z;
  ep.atan_phi = (flags & GASATT_Q_ATAN_PHI) != 0;
  ep.euler = (flags & GASATT_Q_EULER_KICK) != 0;
  ep.fast_fx = N >= 4096;
  ep.wrap = !ep.atan_phi && !(PHIp < 2 * GASATT_PI - 1e-12) ? 0 : PHIp > 0 && PHIp <= GASATT_PI / 2 ? 1 : 2;
  EmFieldParams fp;
  fp.nr = n_r; fp.nz = n_z; fp.delta = delta; fp.PHIp = PHIp; fp.inv_scale = std::ldexp(1.0, -S);
  fp.dt_eps = (dt / 2) / eps;
  fp.dt_eps_dz = (dt / 2) / (eps * delta);
  fp.axis = 4 * (dt / 2) / (eps * delta);
  fp.endcopy = (flags & GASATT_Q_ER_END_COPY) != 0;
  fp.jsign = (flags & GASATT_Q_EZ_AXIS_JSIGN) != 0;
  fp.rshift = (flags & GASATT_Q_EZ_RSHIFT) != 0;
  fp.h_mid = (dt / 2) / (mu * delta);
  // One launch of all ten pairs where its tiles (11 columns of 32) still fit
  // the GPU at once, else two of five (21 columns of 32).  A call of 20 steps
  // with one launch / two: 100 x 500 cells 1069 / 1188 us, 200 x 1000 cells
  // 1956 / 1916, 400 x 2000 cells 2837 / 2574.
  const int whole = 2 * ratio;
  auto tiles_x = [&](int pairs) { return (n_r + em_tile_cols(pairs)) / em_tile_cols(pairs); };
  auto tiles = [&](int pairs) { return (int64_t)tiles_x(pairs) * ((n_z + em_tile_rows(pairs)) / em_tile_rows(pairs)); };
  const bool single = tiles(whole) <= ctx->sms;
  const EmFields there{Er, Ez, Hphi, Er2, Ez2, H2}, back{Er2, Ez2, H2, Er, Ez, Hphi};
  bool away = false;                                   // the fields are in the scratch set
  // (every kernel of the loop starts while the one before it drains)
  auto launch_fields = [&](int pairs, bool first, bool last, int b) {
    fp.pairs = pairs;
    fp.tiles_x = tiles_x(pairs);
    fp.h_first = first ? (dt / 4) / (mu * delta) : fp.h_mid;      // dt/2 after the -dt/4 that opens the sub-cycle
    fp.h_last = last ? (dt / 4) / (mu * delta) : 0;
    const cudaError_t err = launch_early(true, k_em_fields, dim3((unsigned)tiles(pairs)), dim3(32 * kEmWarps), 0, ctx->stream,
                                         away ? back : there, fp, J[b][0], J[b][1], J[1 - b][0], J[1 - b][1]);
    away = !away;
    return err;
  };
  if (steps > 0)
    for (int i = 0; i < (N > 0 ? 2 : 4); ++i)
      GASATT_CUDA(ctx, cudaMemsetAsync(J[i >> 1][i & 1], 0, ncel * 8, ctx->stream));
  if (N > 0) {
    ep.Jr = J[0][0]; ep.Jz = J[0][1];
    k_em_load<<<g, kBlock, 0, ctx->stream>>>(sp, slots[0], ep, N, (flags & GASATT_POS_IN_CYL) != 0, steps > 0);
    GASATT_LAUNCHED(ctx);
  }
  for (int k = 0; k < steps; ++k) {                    // :138-166
    const int b = k & 1;
    if (sorted && k % kEmSortPeriod == 0 && steps - k >= kEmSortLeast) {
      GASATT_CUDA(ctx, cudaMemsetAsync(cell_count, 0, (ncel + 2) * 4, ctx->stream));
      k_em_count<<<g, kBlock, 0, ctx->stream>>>(slots[cur], ep, N, cell_count, keep);
      GASATT_LAUNCHED(ctx);
      st = exclusive_scan(ctx, cell_count, cell_first, ncel + 2, tmp, sc);
      if (st) return st;
      k_em_scatter<<<g, kBlock, 0, ctx->stream>>>(slots[cur], slots[1 - cur], ep, N, cell_first, keep);
      GASATT_LAUNCHED(ctx);
      cur = 1 - cur;
    }
    // (an odd number of single launches would leave the fields in the scratch set)
    if (single && !(k == steps - 1 && !away)) {
      GASATT_CUDA(ctx, launch_fields(whole, true, true, b));
      ctx->launches++;
    } else {
      GASATT_CUDA(ctx, launch_fields(ratio, true, false, b));
      GASATT_CUDA(ctx, launch_fields(ratio, false, true, b));
      ctx->launches += 2;
    }
    if (N > 0) {
      ep.Jr = J[1 - b][0]; ep.Jz = J[1 - b][1];
      if (sorted) E = slots[1 - cur].x;                 // (written in the last step)
      auto push = k == steps - 1 ? k_em_push<true> : k_em_push<false>;
      GASATT_CUDA(ctx, launch_early(true, push, dim3(g), dim3(kBlock), 0, ctx->stream, sp, slots[cur], ep, N,
                                    away ? Er2 : Er, away ? Ez2 : Ez, away ? H2 : Hphi, E));
      ctx->launches++;
    }
  }
  int64_t outs[3] = {0, 0, 0};
  if (N > 0) {
    if (sorted) scanned = slots[1 - cur].of;
    k_keep_flags<<<grid_for(N + 1, kBlock), kBlock, 0, ctx->stream>>>(slots[cur], N, keep);
    GASATT_LAUNCHED(ctx);
    st = exclusive_scan(ctx, keep, scanned, N + 1, tmp, sc);
    if (st) return st;
    k_em_store<<<g, kBlock, 0, ctx->stream>>>(sp, slots[cur], N, scanned, steps > 0 ? E : nullptr, electron_kinetic, e,
                                            counts);
    GASATT_LAUNCHED(ctx);
    int h[4];
    GASATT_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, counts, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    std::memcpy(h, ctx->pinned, sizeof(h));
    outs[0] = h[1] - h[0]; outs[1] = h[2] - h[1]; outs[2] = h[3] - h[2];
  } else {
    GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  if (n_e_out) *n_e_out = outs[0];
  if (n_i1_out) *n_i1_out = outs[1];
  if (n_i2_out) *n_i2_out = outs[2];
  return GASATT_OK;
}

int gasatt_electron_collision(gasatt_ctx *ctx, double *e_pos, double *e_vel, int64_t n_e,
                              int64_t cap_e, double *i1_pos, double *i1_vel, int64_t n_i1,
                              int64_t cap_i1, const gasatt_tables *tab,
                              const double *electron_kinetic, const double *sum_cell, int rmax,
                              int cellnumxy, const double *density, const double *temperature,
                              int64_t ncell, double PHIp, const double *phimax, double dr,
                              double dz, const double *sig_el, const double *sig_ion,
                              const double *sig_exc, double dt_transport, const double *draws,
                              int64_t *n_e_out, int64_t *n_i1_out, unsigned flags) {
  if (!ctx) return GASATT_E_ARG;
  if (n_e < 0 || cap_e < n_e || n_i1 < 0 || cap_i1 < n_i1 || rmax < 1 || cellnumxy < 1 || ncell < 1)
    return fail(ctx, GASATT_E_ARG, "electron_collision: bad sizes");
  std::string err;
  int st = check_tables(tab, err);
  if (st) return fail(ctx, st, err);
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  const int64_t n = n_e;
  const int ne = tab->n_sel1 - 1 + tab->n_el;
  // one upload: the raw tables, the azimuthal cell widths and the rings' first
  // cells (electron_collision.m:53-54)
  const size_t len[6] = {2 * (size_t)tab->n_sel1, 2 * (size_t)tab->n_el, 182 * (size_t)tab->sdel_cols,
                         182 * (size_t)tab->del_cols, 5 * (size_t)tab->n_exc, (size_t)rmax};
  size_t off[7] = {0};
  for (int i = 0; i < 6; ++i) off[i + 1] = off[i] + len[i];
  std::vector<double> host(off[6] + (size_t)(rmax + 2) / 2);
  const double *src[5] = {tab->t_sel_1, tab->t_el, tab->t_sdel, tab->t_del, tab->t_exc};
  for (int i = 0; i < 5; ++i) std::memcpy(host.data() + off[i], src[i], len[i] * 8);
  int *sc0 = reinterpret_cast<int *>(host.data() + off[6]);
  sc0[0] = 0;
  for (int i = 0; i < rmax; ++i) {
    sc0[i + 1] = (int)sum_cell[i];
    host[off[5] + i] = PHIp * 1 / phimax[i];
  }
  const size_t sc = scan_tmp_bytes(n + 1);
  const size_t bytes = align256(host.size() * 8) + 2 * align256((size_t)ne * 8) + align256((size_t)ne * 181 * 8) +
                       align256(8) + 7 * align256((size_t)(n + 1) * 8) + 4 * align256((size_t)(n + 1) * 4) +
                       align256(sc);
  void *buf;
  st = scratch(ctx, bytes, &buf);
  if (st) return st;
  Carver cv{(char *)buf};
  double *d_host = cv.take<double>(host.size());
  double *d_xI = cv.take<double>(ne), *d_yI = cv.take<double>(ne), *d_V = cv.take<double>((size_t)ne * 181);
  MccLists ls;
  ls.n = cv.take<unsigned>(2);
  MccOut out;
  double **o7[7] = {&out.svx, &out.svy, &out.svz, &out.sample, &out.ivx, &out.ivy, &out.ivz};
  for (int i = 0; i < 7; ++i) *o7[i] = cv.take<double>(n + 1);
  out.sec = cv.take<int>(n + 1);
  int *posb = cv.take<int>(n + 1);
  ls.elastic = cv.take<int>(n + 1);
  ls.other = cv.take<int>(n + 1);
  void *tmp = cv.take<char>(sc);
  cudaStream_t s = ctx->stream;
  GASATT_CUDA(ctx, cudaMemcpyAsync(d_host, host.data(), host.size() * 8, cudaMemcpyHostToDevice, s));
  GASATT_CUDA(ctx, cudaMemsetAsync(ls.n, 0, 8, s));
  MccTables t{d_xI, d_yI, d_V, ne, d_host + off[4], tab->n_exc, d_host + off[5],
              reinterpret_cast<const int *>(d_host + off[6]), rmax, cellnumxy, density, temperature, ncell};
  const int64_t call = ctx->mcc_calls++;
  if (n > 0) {
    k_collision_tables<<<(ne * 182 + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        MccRaw{d_host, d_host + off[1], d_host + off[2], d_host + off[3], tab->n_sel1, tab->n_el, tab->sdel_cols,
               tab->del_cols}, d_xI, d_yI, d_V);
    GASATT_LAUNCHED(ctx);
    k_collision_select<<<grid_for(n + 1, kBlock), kBlock, 0, s>>>(
        e_pos, e_vel, cap_e, n, sig_el, sig_ion, sig_exc, electron_kinetic, t, out, ls, dr, dz, dt_transport, draws,
        ctx->seed, call, flags);
    GASATT_LAUNCHED(ctx);
    k_collision_other<<<grid_for(n, kElThreads), kElThreads, 0, s>>>(e_vel, cap_e, electron_kinetic, t, out, ls, draws,
                                                                    ctx->seed, call, flags);
    GASATT_LAUNCHED(ctx);
    k_collision_elastic<<<grid_for(n, kElGroup, 4u * ctx->sms), kElThreads, kElSmem, s>>>(
        e_vel, cap_e, electron_kinetic, t, ls, draws, ctx->seed, call, flags);
    GASATT_LAUNCHED(ctx);
  } else {
    GASATT_CUDA(ctx, cudaMemsetAsync(out.sec, 0, 4, s));
  }
  st = exclusive_scan(ctx, out.sec, posb, n + 1, tmp, sc);
  if (st) return st;
  GASATT_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, posb + n, 4, cudaMemcpyDeviceToHost, s));
  GASATT_CUDA(ctx, cudaStreamSynchronize(s));
  int nb;
  std::memcpy(&nb, ctx->pinned, 4);
  if (n_e + nb > cap_e || n_i1 + nb > cap_i1)
    return fail(ctx, GASATT_E_CAPACITY, "electron_collision: no room for the secondaries");
  if (n > 0 && nb > 0) {
    k_append<<<grid_for(n, kBlock), kBlock, 0, s>>>(e_pos, e_vel, cap_e, n_e, i1_pos, i1_vel,
                                                    cap_i1, n_i1, posb, out);
    GASATT_LAUNCHED(ctx);
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(s));
  if (n_e_out) *n_e_out = n_e + nb;
  if (n_i1_out) *n_i1_out = n_i1 + nb;
  return GASATT_OK;
}

}  // extern "C"
