// sim.cu - the resident PIC-MCC simulation (the hot path).
//
// One step s = FDTD sub-cycle (fields t^s -> t^{s+1}) followed by one fused
// particle pass:
//   gather (EM4.cu:41-122) -> relativistic Boris kick -> drift over the step
//   with the wall / end rules (EM2.cu:26-57, EM4.cu:146-177) -> current
//   deposit (EM7.cu:56-202) into 64-bit fixed point -> null-collision
//   candidate test,
// and then the null-collision MCC of the candidates against the tabulated N2
// cross-sections (electron_transport.cu:64-227, corrected) with secondary
// birth, at the end of the step (operator splitting: push, then collide, as
// the reference's driver alternates its push and electron_collision calls).
// That collision kernel touches neither fields nor current, so the step graph
// runs it beside the next field update; observations of the state (read,
// diagnostics, sort, end of a run) first apply any collisions still queued.
// Particles never leave HBM; the per-step sequence is replayed from CUDA graphs.
//
// Two state forms:
//   FP64      r, z [m]; u_r, u_theta, u_z = gamma v [m/s]; id.  Dead: r < 0.
//   FP32      key = (iz << 16) | ir, fr, fz in-cell offsets [cells], u / c
//             (gamma beta) in float; id.  Dead: key = 0xFFFFFFFF.
// The collision test, branch selection, energy sharing and threshold
// subtraction run in FP64 in both forms.
//
// Deposit: each particle's four node contributions (q FN v w) are rounded to
// integers first, so the grid sum is exact and independent of order: a
// shared-memory window per chunk of sorted particles, then one 64-bit atomic
// per touched node.
//
// Both forms drift the whole step at once (the reference's two half drifts
// joined).
#include <cmath>
#include <cstring>
#include <vector>
#include <cudaTypedefs.h>
#include "fdtd.cuh"
#include "fdtd_tma.cuh"
#include "gasatt_internal.h"

using namespace gasatt;

namespace {

constexpr uint32_t kDead = 0xFFFFFFFFu;
constexpr int kBlock = 256;
constexpr int kMccBlock = 64;             // collision kernels: two warps per block

// Device counters.  Fields that every thread reads when a kernel starts share
// the first 128-byte line; the counters that take atomics during a pass get
// lines of their own, so those atomics do not hold up the reads.
struct SimCounters {
  unsigned long long n_total;    // committed slots
  long long step;                // FP32: index of the current (last) particle pass
  unsigned long long cap;        // slot capacity
  unsigned long long sorted_total;
  long long step64[2];           // FP64: index of the last pass of parity 0 / 1 (it queued that queue)
  int pad0_;
  int chunk;                     // FP32: particles per chunk of the next pass
  int chunk_fixed, pass_blocks;  // FP32: the configured chunk (0: by population), blocks of a pass
  unsigned long long pad1_[8];
  unsigned long long n_births;   // slots claimed by births since the last commit
  unsigned long long pad2_[15];
  unsigned long long n_cand[2];  // collision candidates queued, per queue parity
  unsigned long long pad3_[14];
  unsigned long long chunk_next; // FP32 pass: next chunk to hand out
  unsigned long long pad4_[15];
  unsigned long long ion, ela, exc, nul, lost, cap_overflow;
  unsigned long long kin_fx;     // diagnostic: sum E_kin * 2^16 [eV]
  unsigned long long alive;      // diagnostic
  unsigned long long exc_loss_fx; // diagnostic: excitation energy losses * 2^16 [eV]
  unsigned long long wall_loss_fx;// diagnostic: kinetic energy absorbed at r = Rp * 2^16 [eV]
  unsigned fdtd_err;             // a field-update block gave up waiting for its tile copy
  unsigned scan_err;             // a sort's scan gave up waiting for a predecessor tile
  unsigned long long pad5_[5];
  unsigned long long n_ions;     // ion slots claimed (loads and births; may pass the capacity)
  unsigned long long ion_overflow, ion_lost;
  unsigned long long ion_alive, ion_charge, ion_kin_fx;   // diagnostics; kinetic: E * 2^32 [eV]
};

// slots holding particles, including births since the last commit or sort
__device__ __forceinline__ long long slots_in_use(const SimCounters *cnt) {
  const unsigned long long nt = cnt->n_total + cnt->n_births;
  return (long long)(nt < cnt->cap ? nt : cnt->cap);
}

// Chunk size that gives every one of `blocks` blocks the same number of
// chunks, as few as `most` particles a chunk allow: a multiple of the block
// size.  A small population is spread over all blocks: with chunks of 1792 the
// FP32 pass ran 4,000 electrons on 3 blocks (step 33 us, now 21) and 300,000 on
// 168 of the 592 that fit (41 us, now 32); 2M electrons fill the blocks either way.
__host__ __device__ inline int even_chunk(unsigned n, unsigned blocks, int most) {
  const unsigned per = n / blocks + 1;
  const unsigned k = (per + most - 1) / most;
  return (int)(((per + k - 1) / k + kBlock - 1) / kBlock) * kBlock;
}
constexpr int kChunkMax = 7 * kBlock;     // FP32 pass: 1792 particles a chunk at most

// N2+ ions (FP64 in both forms): (r, z), (u_r, u_theta), u_z, id, charge number
struct IonState { double2 *rz; double2 *urt; double *uz; uint64_t *id; int8_t *q; };

struct SimParams {
  int nr, nz;
  int ldf, ldj;             // row strides (elements) of the field grids and of the current grids
  double dr, dz, dt, c, qe, me, mu0, FN, PHIp, n_gas, nu_max, P_null, Rp, Lp, kb, m_ion, T_gas;
  const double *gas;        // per-cell N2 density [m^-3] (n_r x n_z), or null: n_gas everywhere
  const double *ion_sig;    // per-cell sqrt(kT/m_ion) of newborn ions (n_r x n_z), or null: ion_sigma
  uint64_t seed;
  PhiloxKeys pk;            // Philox round keys of seed
  int secondaries;
  long long cap;
  double qm_dt2;            // -q_e/m_e dt/2
  double idr, idz, ic2;     // 1/dr, 1/dz, 1/c^2
  double mc2_ev, imc2_ev, idlnE;   // m_e c^2 [eV] and its inverse; 1 / dlnE
  double mu_qm;             // mu0 q_e/m_e dt/2 with the sign of qm_dt2 (FP64 form)
  double dep_q;             // FP64 form: fixed-point factor of the electrons' current (x v)
  float aE, aB, hdr, hdz;   // FP32 form: impulse per (V/m), per (A/m); c dt/(2 dr), c dt/(2 dz)
  double dep;               // fixed-point factor: FP64 q FN scale (x v)
  float depf;               // FP32: q FN c scale (x beta)
  uint64_t cand_below;      // null-collision candidate iff the 52-bit draw is below this
  int chunk;                // FP32 pass: particles per chunk (a multiple of the block, <= kChunkMax; 0: chosen by population)
  // tables
  const double *sig;        // 3 x G (el, ion, exc)
  const double *cdf;        // G x 181
  const double *edep;       // G: mean excitation energy loss [eV]
  double exc_kmin;          // lowest excitation threshold [eV]
  int G;
  double lnEmin, dlnE;
  int n_exc;
  double exc[5][16];
  unsigned long long *Jr, *Jz;
  const float4 *qEr, *qEz, *qH;   // FP32 form: packed gather quads (FieldQuads)
  IonState ion;             // ion store (ion_cap > 0)
  long long ion_cap;        // ions stored at most; 0: no ion species
  double ion_sigma;         // spread of a newborn ion's velocity components sqrt(kT/m) [m/s]
};

template <typename Real>
struct Fields { Real *Er, *Ez, *H; };

// FP64: (r, z), (u_r, u_theta), u_z, id.   FP32: (key, fr, fz, u_r), (u_theta, u_z), id.
struct State64 { double2 *rz; double2 *urt; double *uz; uint64_t *id; };
struct State32 { uint4 *a; float2 *b; uint64_t *id; };

// ------------------------------------------------------------------- MCC
struct Birth { bool born; double ux, uy, uz; double eloss; };   // eloss: excitation loss [eV]

__device__ __forceinline__ void xs_lookup(const SimParams &P, double Eev, double &se, double &si,
                                          double &sx, double &L) {
  L = (log(Eev) - P.lnEmin) * P.idlnE;
  int i;
  double f;
  if (!(L > 0)) { i = 0; f = 0; }
  else if (L >= P.G - 1) { i = P.G - 2; f = 1; }
  else { i = (int)L; f = L - i; }
  const double *s0 = P.sig, *s1 = P.sig + P.G, *s2 = P.sig + 2 * P.G;
  se = s0[i] + f * (s0[i + 1] - s0[i]);
  si = s1[i] + f * (s1[i + 1] - s1[i]);
  sx = s2[i] + f * (s2[i + 1] - s2[i]);
}

// Inverse CDF: the largest k in [0, 179] with C[k] <= U, then linear in
// between (interp1 of the cumtrapz, get_ElasticSc_sub1.m:16-19).  Found in two
// rounds of independent loads (every 12th entry, then the 12 in the bracket)
// instead of eight dependent ones; same k as a bisection.
__device__ __forceinline__ double cdf_theta(const SimParams &P, double L, double U) {
  const double Lr = floor(L + 0.5);
  const int g = Lr < 0 ? 0 : (Lr > P.G - 1 ? P.G - 1 : (int)Lr);
  const double *C = P.cdf + (int64_t)g * 181;
  double coarse[15];
#pragma unroll
  for (int m = 0; m < 15; ++m) coarse[m] = C[12 * (m + 1)];
  int seg = 0;                                     // C[12 seg] <= U
#pragma unroll
  for (int m = 0; m < 15; ++m) seg += coarse[m] <= U ? 1 : 0;
  const int base = 12 * seg;
  double fine[12];
#pragma unroll
  for (int m = 0; m < 12; ++m) fine[m] = C[min(base + 1 + m, 180)];
  int lo = base;
#pragma unroll
  for (int m = 0; m < 12; ++m) lo += (base + 1 + m <= 179 && fine[m] <= U) ? 1 : 0;
  const double c0 = lo == base ? C[base] : fine[lo - base - 1];
  const double c1 = fine[lo - base];
  return (lo + (U - c0) / (c1 - c0)) * (GASATT_PI / 180);
}

// gamma v of an electron of kinetic energy E [eV]
__device__ __forceinline__ double u_of_energy(const SimParams &P, double E) {
  const double e = E * P.imc2_ev;
  return P.c * sqrt(e * (2 + e));
}

// Null-collision candidate test U1 < P_null on the integer draw: with
// U1 = (2b+1) 2^-53 (b the top 52 bits of the first two words) this is
// exactly b < P.cand_below.
__device__ __forceinline__ bool null_candidate(const SimParams &P, uint64_t id, long long step) {
  uint32_t c[4] = {(uint32_t)id, (uint32_t)(id >> 32), (uint32_t)step, 0u};
  philox4x32_10(c, P.pk);
  const uint64_t b = ((((uint64_t)c[0]) << 32) | c[1]) >> 12;
  return b < P.cand_below;
}

// Turn (vx, vy, vz) by the polar angle th and the azimuth ph about its own
// direction, from their sines and cosines (the rotation of
// electron_transport.cu:118-135 in the corrected frame, p2 = vx^2 + vy^2).
template <typename R>
__device__ __forceinline__ void rotate_sc(R &vx, R &vy, R &vz, R st, R ct, R sp, R cp) {
  const R v = sqrt(vx * vx + vy * vy + vz * vz);
  const R p2 = vx * vx + vy * vy;
  R x0, y0, z0;
  if (p2 > R(0.0001)) {
    const R s = sqrt(p2);
    const R f = st / s;
    x0 = vx * ct + f * (vx * vz * cp - v * vy * sp);
    y0 = vy * ct + f * (vy * vz * cp + v * vx * sp);
    z0 = vz * ct - s * st * cp;
  } else {
    x0 = v * st * cp;
    y0 = v * st * sp;
    z0 = v * ct;
  }
  vx = x0; vy = y0; vz = z0;
}

// Apply the rotation with (st, ct) given and azimuth 2 pi b (sign = -1: the
// opposite azimuth, phi - pi).  FAST (the FP32 form): float arithmetic with
// the hardware sine and cosine on the azimuth folded into [-pi, pi].
template <bool FAST>
__device__ __forceinline__ void turn(double &ux, double &uy, double &uz, double st, double ct,
                                     double b, double sign) {
  if (FAST) {
    float sp, cp;
    const float ph = (float)(2 * GASATT_PI * (b > 0.5 ? b - 1 : b));
    __sincosf(ph, &sp, &cp);
    float x = (float)ux, y = (float)uy, z = (float)uz;
    rotate_sc<float>(x, y, z, (float)st, (float)ct, (float)sign * sp, (float)sign * cp);
    ux = x; uy = y; uz = z;
  } else {
    double sp, cp;
    sincos(2 * GASATT_PI * b, &sp, &cp);
    rotate_sc<double>(ux, uy, uz, st, ct, sign * sp, sign * cp);
  }
}

// Collision of a candidate electron at step `step` (corrected form of
// electron_transport.cu:74-227).  u in m/s, local (r, theta, z) frame.
// Returns 1 elastic, 2 ionization, 3 excitation, 4 null.  The collision test,
// the branch choice, the ionization energy sharing and the threshold
// subtractions are FP64 in both forms; FAST (the FP32 form) turns the
// velocity in float.  The code is kept short: one candidate runs it alone,
// mostly from a cold instruction cache.
// gas density of cell (ir, iz), the neutral background of the collisions
__device__ __forceinline__ double gas_density(const SimParams &P, int ir, int iz) {
  if (!P.gas) return P.n_gas;
  ir = min(max(ir, 0), P.nr - 1);
  iz = min(max(iz, 0), P.nz - 1);
  return P.gas[ir + (int64_t)iz * P.nr];
}

// velocity spread sqrt(kT/m_ion) of an ion born in cell (ir, iz): the gas
// temperature of that cell (electron_transport.cu:202-204 reads
// temperature[index]) or the uniform one
__device__ __forceinline__ double ion_spread(const SimParams &P, int ir, int iz) {
  if (!P.ion_sig) return P.ion_sigma;
  ir = min(max(ir, 0), P.nr - 1);
  iz = min(max(iz, 0), P.nz - 1);
  return P.ion_sig[ir + (int64_t)iz * P.nr];
}

template <bool FAST>
__device__ __forceinline__ int mcc_event(const SimParams &P, uint64_t id, long long step, double &ux,
                                      double &uy, double &uz, Birth &b, double n_gas) {
  b.born = false;
  b.eloss = 0;
  const U2 d0 = draw2(P.seed, id, step, 0);
  const double I = GASATT_ION_I_EV;
  const double u2 = ux * ux + uy * uy + uz * uz;
  const double w2 = u2 * P.ic2, ig = rsqrt(1 + w2);
  const double Eev = P.mc2_ev * (w2 / ((1 + w2) * ig + 1));
  const double ium = u2 > 0 ? rsqrt(u2) : 0.0, um = u2 * ium, v = um * ig;
  double se, si, sx, L;
  xs_lookup(P, Eev, se, si, sx, L);
  const double nu_el = n_gas * se * v, nu_io = n_gas * si * v, nu_ex = n_gas * sx * v;
  const double X = d0.b * P.nu_max;
  if (X < nu_el) {
    const U2 d1 = draw2(P.seed, id, step, 1);
    const double th = cdf_theta(P, L, d1.a);
    double st, ct;
    if (FAST) {
      float sf, cf;
      __sincosf((float)th, &sf, &cf);
      st = sf; ct = cf;
    } else {
      sincos(th, &st, &ct);
    }
    turn<FAST>(ux, uy, uz, st, ct, d1.b, 1.0);
    return 1;
  }
  if (X < nu_el + nu_io && Eev > I) {
    const U2 d1 = draw2(P.seed, id, step, 1);
    const double T = Eev;
    const double T_a = 1000, T_b = 2 * I, t_b = I, T_s = 4.17, t_s = 13.8;
    const double T_0 = T_s - T_a / (T + T_b);
    const double t = t_s * T / (T + t_b);
    const double T_m = (T - I) / 2;
    // E_1 = T_0 + t tan(U (k_1 + k_2) - k_2), k_1 = atan((T_m - T_0)/t),
    // k_2 = atan(T_0/t): with k_1 + k_2 from one atan2 and
    // tan(x - k_2) = (tan x - tan k_2) / (1 + tan x tan k_2)
    const double it = 1 / t, a1 = (T_m - T_0) * it, a2 = T_0 * it;
    const double tx = tan(d1.a * atan2(a1 + a2, 1 - a1 * a2));
    const double k0 = T_0 + t * ((tx - a2) / (1 + a2 * tx));
    const double E_1 = k0, E_2 = T - E_1 - I;
    double E_p, E_s;
    if (E_2 > E_1) { E_p = E_2; E_s = E_1; } else { E_p = E_1; E_s = E_2; }
    // polar angles as sines (the reference's asin arguments) and cosines
    const double h = 0.5 * P.imc2_ev, es = E_s / T;
    const double sp2 = es / ((T - E_s) * h + 1);
    const double ss2 = (1 - es) / (E_s * h + 1);
    const double ix = ux * ium, iy = uy * ium, iz = uz * ium;
    const double up = u_of_energy(P, E_p), us = u_of_energy(P, E_s);
    ux = ix * up; uy = iy * up; uz = iz * up;
    turn<FAST>(ux, uy, uz, sqrt(sp2), sqrt(1 - sp2), d1.b, 1.0);
    if (P.secondaries) {
      double sx_ = ix * us, sy_ = iy * us, sz_ = iz * us;
      turn<FAST>(sx_, sy_, sz_, sqrt(ss2), sqrt(1 - ss2), d1.b, -1.0);
      b.born = true; b.ux = sx_; b.uy = sy_; b.uz = sz_;
    }
    return 2;
  }
  if (X < nu_el + nu_io + nu_ex) {
    // tabulated mean energy loss, interpolated like the cross-sections
    if (!(Eev > P.exc_kmin)) return 4;
    int i;
    double f;
    if (!(L > 0)) { i = 0; f = 0; }
    else if (L >= P.G - 1) { i = P.G - 2; f = 1; }
    else { i = (int)L; f = L - i; }
    const double E_dep = P.edep[i] + f * (P.edep[i + 1] - P.edep[i]);
    if (!(E_dep > 0) || !(E_dep < Eev)) return 4;
    const double up = u_of_energy(P, Eev - E_dep) * ium;
    ux *= up; uy *= up; uz *= up;
    b.eloss = E_dep;
    return 3;
  }
  return 4;
}

// kinetic energy of a particle absorbed at the wall, u2 = |u / c|^2 and
// mc2 = m c^2 / q_e [eV] (rare: taken only on the step it leaves)
__device__ __forceinline__ void count_wall_loss(SimCounters *cnt, double u2, double mc2) {
  const double E = mc2 * (u2 / (sqrt(1 + u2) + 1));
  atomicAdd(&cnt->wall_loss_fx, (unsigned long long)__double2ll_rn(E * 65536.0));
}

__device__ __forceinline__ void count_event(SimCounters *cnt, int ev, const Birth &b) {
  if (ev == 1) atomicAdd(&cnt->ela, 1ull);
  else if (ev == 2) atomicAdd(&cnt->ion, 1ull);
  else if (ev == 3) {
    atomicAdd(&cnt->exc, 1ull);
    atomicAdd(&cnt->exc_loss_fx, (unsigned long long)__double2ll_rn(b.eloss * 65536.0));
  } else if (ev == 4) atomicAdd(&cnt->nul, 1ull);
}

// The N2+ ion of an ionization of electron `id` at step `step`, at the
// parent's position (r, z), singly charged, with a Maxwellian velocity at the
// gas temperature: each component normal with spread sqrt(kT/m)
// (electron_transport.cu:202-204).  The three normals are the Box-Muller
// transforms of the Philox draws (id, step) blocks 2 and 3; the ion takes the
// id of the secondary electron.  Takes no SimParams: a reference to a kernel
// parameter handed to a call would copy the whole block to the stack.
__device__ __noinline__ void ion_birth(IonState I, long long cap, double sigma, uint64_t seed,
                                       SimCounters *cnt, uint64_t id, long long step, double r,
                                       double z) {
  const unsigned long long k = atomicAdd(&cnt->n_ions, 1ull);
  if (k >= (unsigned long long)cap) { atomicAdd(&cnt->ion_overflow, 1ull); return; }
  const U2 a = draw2(seed, id, step, 2), b = draw2(seed, id, step, 3);
  double sa, ca, sb, cb;
  sincos(2 * GASATT_PI * a.b, &sa, &ca);
  sincos(2 * GASATT_PI * b.b, &sb, &cb);
  const double ra = sigma * sqrt(-2 * log(a.a)), rb = sigma * sqrt(-2 * log(b.a));
  I.rz[k] = make_double2(r, z);
  I.urt[k] = make_double2(ra * ca, ra * sa);
  I.uz[k] = rb * cb;
  I.id[k] = child_id(id, step);
  I.q[k] = 1;
}

// warp-aggregated append of candidate slots to the collision queue
__device__ __forceinline__ void queue_push(bool want, long long p, unsigned long long *n_cand,
                                           int *queue) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(n_cand, (unsigned long long)__popc(m));
  base = __shfl_sync(0xFFFFFFFFu, base, leader);
  if (want) queue[base + __popc(m & ((1u << lane) - 1))] = (int)p;
}

// FP64 bookkeeping.  The pass of parity q runs one step after the pass of the
// other parity (step64), and births go on counting from the slots of the last
// sort, so nothing has to be committed between a pass and the collisions it
// queued - a one-thread kernel in between lengthened the collision branch, the
// critical path of a small cell's step, by 3 us.  Only the queue that the next
// pass fills has to be empty: the pass itself does that for a cell on its own
// (the other queue was consumed before it), and one kernel for all cells of a batch.
__device__ __forceinline__ void clear_next_queue(SimCounters *cnt, int q) { cnt->n_cand[1 - q] = 0; }
__global__ void k_clear_next_queue(SimCounters *cnt, int q) { clear_next_queue(cnt, q); }

// ------------------------------------------------------ deposit
// The ions' deposit.  Each one's four node contributions (q FN v w, both
// components) are integers, so every summation order gives the same grid.  The lanes of a warp
// that share a node quad (the sort key; the quad fixes the four node indices)
// are summed with redux.sync, one quad per round, and the first lane of the
// quad adds the eight sums with 64-bit atomics.  Sorted particles put one to
// three quads in a warp; after kDepRounds rounds the lanes left add their own
// contributions.
constexpr int kDepRounds = 4;

// FP64-form contribution, |v| <= 2^48, summed as hi 2^24 + lo with lo in
// [0, 2^24): both 32-lane partial sums fit int32, the recombination is exact
__device__ __forceinline__ long long warp_sum(long long v) {
  const int lo = (int)(v & 0xFFFFFFLL), hi = (int)(v >> 24);
  const long long slo = __reduce_add_sync(0xFFFFFFFFu, lo);
  const long long shi = __reduce_add_sync(0xFFFFFFFFu, hi);
  return shi * (1LL << 24) + slo;
}

template <typename VT>
__device__ __forceinline__ void deposit_atomic(const int64_t a[4], const VT vr[4],
                                               const VT vz[4], unsigned long long *Jr,
                                               unsigned long long *Jz) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (vr[k]) atomicAdd(Jr + a[k], (unsigned long long)(long long)vr[k]);
    if (vz[k]) atomicAdd(Jz + a[k], (unsigned long long)(long long)vz[k]);
  }
}

template <typename VT>
__device__ __forceinline__ void warp_deposit(bool act, unsigned key, const int64_t a[4],
                                             const VT vr[4], const VT vz[4],
                                             unsigned long long *Jr, unsigned long long *Jz) {
  const int lane = threadIdx.x & 31;
  unsigned pending = __ballot_sync(0xFFFFFFFFu, act);
#pragma unroll 1
  for (int round = 0; round < kDepRounds && pending; ++round) {
    const int leader = __ffs(pending) - 1;
    const unsigned lk = __shfl_sync(0xFFFFFFFFu, key, leader);
    const bool mine = act && key == lk;
    pending &= ~__ballot_sync(0xFFFFFFFFu, mine);
    long long sr[4], sz[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      sr[q] = warp_sum(mine ? vr[q] : (VT)0);
      sz[q] = warp_sum(mine ? vz[q] : (VT)0);
    }
    if (lane == leader) deposit_atomic<long long>(a, sr, sz, Jr, Jz);
  }
  if ((pending >> lane) & 1u) deposit_atomic<VT>(a, vr, vz, Jr, Jz);
}


// ----------------------------------------------------------- FP64 form
__device__ __forceinline__ void halfdrift64(double &r, double &z, double &ur, double &ut,
                                            double &uz, bool &alive, const SimParams &P) {
  const double g = sqrt(1 + (ur * ur + ut * ut + uz * uz) / (P.c * P.c));
  const double X = r + 0.5 * (ur / g) * P.dt;
  const double Y = 0.5 * (ut / g) * P.dt;
  double Z = z + 0.5 * (uz / g) * P.dt;
  const double rn = sqrt(X * X + Y * Y);
  const double cs = rn > 0 ? X / rn : 1.0, sn = rn > 0 ? Y / rn : 0.0;
  const double nur = cs * ur + sn * ut, nut = -sn * ur + cs * ut;
  ur = nur; ut = nut;
  if (rn > P.Rp) alive = false;
  if (Z > P.Lp) { Z = 2 * P.Lp - Z; uz = -uz; }
  if (Z < 0) { Z = -Z; uz = -uz; }
  r = rn; z = Z;
}

__device__ __forceinline__ void deposit_values64(const SimParams &P, double r, double z,
                                                 double ur, double ut, double uz, double q,
                                                 int64_t a[4], long long vr[4], long long vz[4],
                                                 unsigned &key) {
  const double g = sqrt(1 + (ur * ur + ut * ut + uz * uz) / (P.c * P.c));
  const double vrr = ur / g, vzz = uz / g;
  double b[4];
  const int ar = em7_weights_ld(r, z, P.nr, P.nz, P.ldj, P.dr, P.dz, a, b);
  const int az = (int)floor(z / P.dz - 0.5);
  key = (unsigned)((ar + 1) + (az + 1) * (P.nr + 1));
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    vr[k] = __double2ll_rn(P.FN * b[k] * q * vrr * P.dep);
    vz[k] = __double2ll_rn(P.FN * b[k] * q * vzz * P.dep);
  }
}

// FP64 pass.  Bound by instruction issue and the shared-memory pipe (the
// deposit's atomics).  2M electrons on 256 x 1024 cells: 36M warp
// instructions, 64 us a pass.  With a division and a square root wherever
// the formulas have one (some forty an electron), the drift in two halves and
// the deposit summed by redux.sync over the lanes of each node quad it was
// 108M and 169 us.  So the push multiplies by reciprocals (SimParams), takes
// three rsqrt's and one division, forms floors and fixed-point roundings in
// the FP64 adder, and deposits through a window in shared memory.  Three
// blocks of 256 threads per SM: at four (64 registers) the step is 8 us
// longer.  Chunks of up to 4608 particles: 1024 / 1536 / 2560 are 5 / 2 / 1 us
// longer (more flushes).

// Boris kick in E = (Er, 0, Ez), B = (0, mu0 H, 0) with the fields of the
// staggered bilinear gather (EM4.cu:41-122).
__device__ __forceinline__ void kick64(const SimParams &P, const Fields<double> &F, double r,
                                       double z, double &ur, double ut, double &uz) {
  const Axis64 R = axis64(__dmul_rn(r, P.idr), P.nr), Z = axis64(__dmul_rn(z, P.idz), P.nz);
  const double *e0 = F.Er + (int64_t)Z.i * P.ldf, *e1 = e0 + P.ldf;
  const double *z0 = F.Ez + (int64_t)Z.lo * P.ldf + R.i, *z1 = F.Ez + (int64_t)Z.hi * P.ldf + R.i;
  const double *h0 = F.H + (int64_t)Z.lo * P.ldf, *h1 = F.H + (int64_t)Z.hi * P.ldf;
  const double a0 = __ldg(e0 + R.lo), a1 = __ldg(e0 + R.hi), a2 = __ldg(e1 + R.lo), a3 = __ldg(e1 + R.hi);
  const double b0 = __ldg(z0), b1 = __ldg(z0 + 1), b2 = __ldg(z1), b3 = __ldg(z1 + 1);
  const double c0 = __ldg(h0 + R.lo), c1 = __ldg(h0 + R.hi), c2 = __ldg(h1 + R.lo), c3 = __ldg(h1 + R.hi);
  const double Er = lerp64(lerp64(a0, a1, R.w), lerp64(a2, a3, R.w), Z.f);
  const double Ez = lerp64(lerp64(b0, b1, R.f), lerp64(b2, b3, R.f), Z.w);
  const double H = lerp64(lerp64(c0, c1, R.w), lerp64(c2, c3, R.w), Z.w);
  const double umr = fma(P.qm_dt2, Er, ur), umz = fma(P.qm_dt2, Ez, uz);
  const double u2 = fma(umr, umr, fma(ut, ut, __dmul_rn(umz, umz)));
  const double t = __dmul_rn(__dmul_rn(P.mu_qm, H), rsqrt(fma(u2, P.ic2, 1.0)));
  const double upr = fma(-umz, t, umr), upz = fma(umr, t, umz);
  const double s = __ddiv_rn(__dadd_rn(t, t), fma(t, t, 1.0));
  ur = fma(P.qm_dt2, Er, fma(-upz, s, umr));
  uz = fma(P.qm_dt2, Ez, fma(upr, s, umz));
}

// Straight-line drift over the time dt (a whole step: the reference's two
// half drifts joined - the same line, the radius along a line is convex, the
// end reflection specular), EM2.cu:26-57.  ig: 1/gamma, kept by the turn.
__device__ __forceinline__ void drift64(const SimParams &P, double dt, double &r, double &z, double &ur,
                                        double &ut, double &uz, double &ig, bool &alive) {
  ig = rsqrt(fma(fma(ur, ur, fma(ut, ut, __dmul_rn(uz, uz))), P.ic2, 1.0));
  const double h = __dmul_rn(ig, dt);
  const double X = fma(ur, h, r), Y = __dmul_rn(ut, h);
  double Z = fma(uz, h, z);
  const double r2 = fma(X, X, __dmul_rn(Y, Y));
  const bool off = r2 > 0;
  const double irn = off ? rsqrt(r2) : 0.0;
  const double rn = __dmul_rn(r2, irn);
  const double cs = off ? __dmul_rn(X, irn) : 1.0, sn = __dmul_rn(Y, irn);
  const double nur = fma(cs, ur, __dmul_rn(sn, ut)), nut = fma(cs, ut, -__dmul_rn(sn, ur));
  ur = nur; ut = nut;
  if (rn > P.Rp) alive = false;
  if (Z > P.Lp) { Z = __dsub_rn(2 * P.Lp, Z); uz = -uz; }
  if (Z < 0) { Z = -Z; uz = -uz; }
  r = rn; z = Z;
}

// FP64-form deposit window: 64-bit sums of one chunk of particles on a box of
// the grid in shared memory, each sum as two 32-bit words - shared memory has
// no native 64-bit add.  The low word's add returns its old value, which
// tells whether this add carried; every carry is seen exactly once, so the two
// words hold the sum modulo 2^64 whatever the order (|contribution| <= 2^48
// keeps the high word's sum far inside 32 bits).  The four words of the
// nodes (r low, r high, z low, z high) sit in four planes, so neighbouring
// nodes are in neighbouring banks; rows are ws = 3 (mod 32) nodes apart, so the
// 3 x 3 nodes around a warp's particles are in nine.
constexpr int kWin64Nodes = 3072;
constexpr int kWin64Bytes = kWin64Nodes * 16;
constexpr int kWinCols = 256;             // columns of a deposit box at most (wide grids)
constexpr int kChunk64 = 4608;            // particles per chunk at most

struct Win64 {
  unsigned *w;
  int row0, rows, col0, cols, ws;
};

__host__ __device__ inline int win_cols(int nr) { return nr < kWinCols ? nr : kWinCols; }
__host__ __device__ inline int win_stride(int cols) { return cols + ((3 - cols % 32) + 32) % 32; }

// Box of a chunk: the rows of its first and last live particles (row_lo..row_hi;
// row_hi < 0: none live) plus up to three rows either side for the drift
// since the last sort; all columns, or on a grid wider than the box those
// from a little below the first particle's when the chunk sits in one row (the
// particles are sorted by row, then column), else from the axis.
__device__ __forceinline__ void chunk_box(int nr, int nz, int cols, int maxrows, int row_lo, int row_hi,
                                          int col_lo, int &row0, int &rows, int &col0) {
  row0 = 0; rows = maxrows; col0 = 0;
  if (row_hi < 0) return;
  const int core = row_hi - row_lo + 3;
  const int below = maxrows >= core + 6 ? 3 : max(1, 1 + (maxrows - core) / 2);
  row0 = min(max(0, row_lo - below), nz - maxrows);
  rows = min(maxrows, row_hi + 4 - row0);
  if (row_lo == row_hi) col0 = min(max(0, col_lo - 8), nr - cols);
}

__device__ __forceinline__ void box64(const SimParams &P, const State64 &S, long long beg, long long end,
                                      int maxrows, int &row0, int &rows, int &col0) {
  const double2 a = S.rz[beg], b = S.rz[end - 1];
  int lo = P.nz, hi = -1, col = 0;
  if (a.x >= 0) {
    lo = hi = min(max((int)(a.y * P.idz), 0), P.nz - 1);
    col = min(max((int)(a.x * P.idr), 0), P.nr - 1);
  }
  if (b.x >= 0) {
    const int k = min(max((int)(b.y * P.idz), 0), P.nz - 1);
    lo = min(lo, k);
    hi = max(hi, k);
  }
  chunk_box(P.nr, P.nz, win_cols(P.nr), maxrows, lo, hi, col, row0, rows, col0);
}

__device__ __forceinline__ void win64_add(unsigned *w, double v) {
  const unsigned lo = (unsigned)__double2loint(v);
  const int hi = __double2hiint(v) - 0x43380000;      // v = 1.5 2^52 + contribution
  const unsigned old = atomicAdd(w, lo);
  const int up = hi + (old + lo < lo ? 1 : 0);
  if (up) atomicAdd(w + kWin64Nodes, (unsigned)up);
}

// One particle's current into its four nodes (EM7.cu:56-202 weights, clamped
// one-sided at the edges): q FN v w in fixed point, rounded to nearest in one
// FMA.  The lanes visit the nodes in an order permuted by lane & 3, so lanes on
// the same quad hit four different nodes.  Nodes outside the box go to the grid.
__device__ __forceinline__ void deposit64(const SimParams &P, const Win64 &w, double r, double z, double ur,
                                          double uz, double ig) {
  const Axis64 R = axis64(__dmul_rn(r, P.idr), P.nr), Z = axis64(__dmul_rn(z, P.idz), P.nz);
  const double k = __dmul_rn(P.dep_q, ig), kr = __dmul_rn(k, ur), kz = __dmul_rn(k, uz);
  const bool sc = threadIdx.x & 1, sr = threadIdx.x & 2;
  const int ca = sc ? R.hi : R.lo, cb = sc ? R.lo : R.hi, ra = sr ? Z.hi : Z.lo, rb = sr ? Z.lo : Z.hi;
  const double om = __dsub_rn(1.0, R.w), on = __dsub_rn(1.0, Z.w);
  const double wa = sc ? R.w : om, wb = sc ? om : R.w, va = sr ? Z.w : on, vb = sr ? on : Z.w;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int col = n & 1 ? cb : ca, row = n & 2 ? rb : ra;
    const double b = __dmul_rn(n & 1 ? wb : wa, n & 2 ? vb : va);
    const double vr = fma(kr, b, 6755399441055744.0), vz = fma(kz, b, 6755399441055744.0);
    const unsigned lr = (unsigned)(row - w.row0), lc = (unsigned)(col - w.col0);
    if (lr < (unsigned)w.rows && lc < (unsigned)w.cols) {
      unsigned *m = w.w + ((int)lr * w.ws + (int)lc);
      win64_add(m, vr);
      win64_add(m + 2 * kWin64Nodes, vz);
    } else {
      const int64_t g = col + (int64_t)row * P.ldj;
      const long long ir = __double_as_longlong(vr) - 0x4338000000000000LL;
      const long long iz = __double_as_longlong(vz) - 0x4338000000000000LL;
      if (ir) atomicAdd(P.Jr + g, (unsigned long long)ir);
      if (iz) atomicAdd(P.Jz + g, (unsigned long long)iz);
    }
  }
}

// add the box to the grid (one 64-bit atomic per nonzero sum) and zero it:
// its first bw columns, the ones the chunk touched
__device__ __forceinline__ void flush64(const SimParams &P, const Win64 &w, int bw) {
  const int nb = bw > 0 ? bw * w.rows : 0;
  for (int i = threadIdx.x; i < nb; i += kBlock) {
    const int row = i / bw, col = i - row * bw;
    unsigned *m = w.w + row * w.ws + col;
    const uint4 v = make_uint4(m[0], m[kWin64Nodes], m[2 * kWin64Nodes], m[3 * kWin64Nodes]);
    if (v.x | v.y | v.z | v.w) {
      const int64_t g = (int64_t)(w.row0 + row) * P.ldj + w.col0 + col;
      if (v.x | v.y) atomicAdd(P.Jr + g, ((unsigned long long)v.y << 32) + v.x);
      if (v.z | v.w) atomicAdd(P.Jz + g, ((unsigned long long)v.w << 32) + v.z);
      m[0] = m[kWin64Nodes] = m[2 * kWin64Nodes] = m[3 * kWin64Nodes] = 0;
    }
  }
}

// Bring the state of particles [beg, end) into L2 ahead of their chunk (one
// thread; cp.async.bulk.prefetch.L2, a hint that completes on its own).  beg
// is a multiple of the chunk size, hence even, so every range starts on a
// 16-byte boundary; the sizes are rounded down to 16 bytes.
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
  if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_chunk64(const State64 &S, long long beg, long long end) {
  const long long n = end - beg;
  if (n <= 0) return;
  prefetch_l2(S.rz + beg, (uint32_t)(n * 16));
  prefetch_l2(S.urt + beg, (uint32_t)(n * 16));
  prefetch_l2(S.uz + beg, (uint32_t)((n * 8) & ~15ll));
  prefetch_l2(S.id + beg, (uint32_t)((n * 8) & ~15ll));
}

// The particles [beg, end) of one chunk of the FP64 pass of step `step`
// (executed by the whole block).  MODE 0: full step - kick, drift, deposit;
// collision candidates go to queue q for k_mcc64; MODE 1: half drift +
// deposit only (start of a run); MODE 2: kick + half drift only, ending at
// integer time (end of a run).  The highest box column touched is merged
// into *box_cmax.
template <int MODE>
__device__ __forceinline__ void chunk64(const SimParams &P, const State64 &S, const Fields<double> &F,
                                        SimCounters *cnt, int *queue, int q, long long step, int beg,
                                        int end, const Win64 &w, int *box_cmax) {
  const int lane = threadIdx.x & 31;
  unsigned lost = 0;
  int cmax = -1;
  int base = beg + (int)(threadIdx.x & ~31);
  double2 rzn = make_double2(-1.0, 0.0), urtn = rzn;
  double uzn = 0;
  uint64_t idn = 0;
  // the next iteration's particle is loaded one iteration ahead, so its latency
  // overlaps the current particle's arithmetic
  auto load = [&](int k) {
    rzn = S.rz[k];
    urtn = S.urt[k];
    uzn = S.uz[k];
    if (MODE == 0) idn = S.id[k];
  };
  if (base + lane < end) load(base + lane);
  for (; base < end; base += kBlock) {
    const int p = base + lane;
    const double2 rz = rzn, urt = urtn;
    double uz = uzn;
    const uint64_t id = idn;
    bool act = rz.x >= 0;
    rzn.x = -1.0;
    if (p + kBlock < end) load(p + kBlock);
    bool cand = false;
    if (act) {
      double ur = urt.x, ut = urt.y, r = rz.x, z = rz.y, ig;
      if (MODE == 0) cand = null_candidate(P, id, step);
      if (MODE != 1) kick64(P, F, r, z, ur, ut, uz);
      drift64(P, MODE == 0 ? P.dt : 0.5 * P.dt, r, z, ur, ut, uz, ig, act);
      if (!act) {
        lost++;
        cand = false;
        r = -1.0;
        count_wall_loss(cnt, (ur * ur + ut * ut + uz * uz) * P.ic2, P.me * P.c * P.c / P.qe);
      }
      S.rz[p] = make_double2(r, z);
      S.urt[p] = make_double2(ur, ut);
      S.uz[p] = uz;
      if (MODE != 2 && act) {
        deposit64(P, w, r, z, ur, uz, ig);
        cmax = max(cmax, min((int)(r * P.idr) + 1, P.nr - 1) - w.col0);
      }
    }
    if (MODE == 0) queue_push(cand, p, &cnt->n_cand[q], queue + (long long)q * P.cap);
  }
  if (MODE != 2) {
    cmax = __reduce_max_sync(0xFFFFFFFFu, cmax);
    if (lane == 0 && cmax >= 0) atomicMax(box_cmax, min(cmax, w.cols - 1));
  }
  lost = __reduce_add_sync(0xFFFFFFFFu, lost);
  if (lane == 0 && lost) atomicAdd(&cnt->lost, (unsigned long long)lost);
}

template <int MODE>
__global__ void __launch_bounds__(kBlock, 3) k_pass64(SimParams P, State64 S, Fields<double> F,
                                                      SimCounters *cnt, int *queue, int q) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int box_row0[2], box_rows[2], box_col0[2], box_cmax[2];   // of this chunk and the next
  // the window starts zeroed; each chunk's flush leaves it zeroed again
  for (int i = threadIdx.x; i < kWin64Nodes; i += kBlock) reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
  // (never started early: it follows the field update and the collisions)
  const long long n0 = slots_in_use(cnt);
  const long long step = cnt->step64[1 - q] + 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cnt->step64[q] = step;
    clear_next_queue(cnt, q);
  }
  const int chunk = even_chunk((unsigned)n0, gridDim.x, kChunk64);
  const int cols = win_cols(P.nr), ws = win_stride(cols), maxrows = min(kWin64Nodes / ws, P.nz);
  // the blocks take the chunks in turn, so neighbouring blocks work on
  // neighbouring grid rows; thread 0 brings the block's next chunk into L2
  // and, at the end of this one, places its box
  const long long stride = (long long)gridDim.x * chunk;
  long long beg = (long long)blockIdx.x * chunk;
  if (threadIdx.x == 0) {
    box_cmax[0] = -1;
    if (MODE != 2 && beg < n0) box64(P, S, beg, min(beg + chunk, n0), maxrows, box_row0[0], box_rows[0], box_col0[0]);
  }
  int b = 0;
  __syncthreads();
  for (; beg < n0; beg += stride, b ^= 1) {
    const Win64 w{reinterpret_cast<unsigned *>(smem), box_row0[b], box_rows[b], box_col0[b], cols, ws};
    const long long nb = beg + stride;
    if (threadIdx.x == 0 && nb < n0) prefetch_chunk64(S, nb, min(nb + chunk, n0));
    chunk64<MODE>(P, S, F, cnt, queue, q, step, (int)beg, (int)min(beg + chunk, n0), w, &box_cmax[b]);
    if (MODE == 2) continue;
    if (threadIdx.x == 0) {
      box_cmax[b ^ 1] = -1;
      if (nb < n0) box64(P, S, nb, min(nb + chunk, n0), maxrows, box_row0[b ^ 1], box_rows[b ^ 1], box_col0[b ^ 1]);
    }
    __syncthreads();
    flush64(P, w, box_cmax[b] + 1);
    __syncthreads();
  }
  let_next_start();
}

// The collision of candidate slot p queued at step `step` (FP64 form): MCC,
// the ion and the secondary's birth at the parent's position.  n0: the
// slots of the last sort (births land beyond).
__device__ __forceinline__ void mcc64_one(const SimParams &P, const State64 &S, SimCounters *cnt,
                                          long long p, long long step, long long n0) {
  const double2 rz = S.rz[p], urt = S.urt[p];
  double ur = urt.x, ut = urt.y, uz = S.uz[p];
  const uint64_t id = S.id[p];
  Birth b;
  const double ng = gas_density(P, (int)floor(rz.x / P.dr), (int)floor(rz.y / P.dz));
  const int ev = mcc_event<false>(P, id, step, ur, ut, uz, b, ng);
  count_event(cnt, ev, b);
  if (ev == 2 && P.ion_cap > 0)
    ion_birth(P.ion, P.ion_cap, ion_spread(P, (int)floor(rz.x / P.dr), (int)floor(rz.y / P.dz)),
              P.seed, cnt, id, step, rz.x, rz.y);
  if (b.born) {
    const unsigned long long kb = atomicAdd(&cnt->n_births, 1ull);
    const long long slot = n0 + (long long)kb;
    if (slot < P.cap) {
      S.rz[slot] = rz;
      S.urt[slot] = make_double2(b.ux, b.uy);
      S.uz[slot] = b.uz;
      S.id[slot] = child_id(id, step);
    } else {
      atomicAdd(&cnt->cap_overflow, 1ull);
    }
  }
  S.urt[p] = make_double2(ur, ut); S.uz[p] = uz;
}

// The collisions of the pass that filled queue q, at the end of its step
// (after the drift and the deposit): the MCC changes the velocity, and an
// ionization appends its secondary at the parent's position.  Nothing here
// reads or writes the fields or the current, so it can run beside the next
// field update.
__global__ void __launch_bounds__(kMccBlock) k_mcc64(SimParams P, State64 S, SimCounters *cnt,
                                                     const int *queue, int q) {
  // one candidate per warp (lane 0): the collision branches differ a lot in
  // length, and lanes on different branches would run them one after another
  if ((threadIdx.x & 31) != 0) return;
  const long long n0 = (long long)cnt->n_total;
  const long long step = cnt->step64[q];
  const long long nq = (long long)cnt->n_cand[q];
  const int *qu = queue + (long long)q * P.cap;
  const long long nwarps = (long long)gridDim.x * (kMccBlock / 32);
  for (long long k = (blockIdx.x * (long long)kMccBlock + threadIdx.x) >> 5; k < nq; k += nwarps)
    mcc64_one(P, S, cnt, qu[k], step, n0);
}

constexpr int kMaxBatch = 256;               // cells a batch holds at most

// the cell of work item k: the last c with prefix[c] <= k (prefix ascending,
// prefix[0] = 0, n cells)
__device__ __forceinline__ int cell_of_item(const long long *prefix, int n, long long k) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------- batched FP64 step
struct BatchCell64 {
  SimParams P[2];             // deposit into current buffer 0 / 1
  State64 S[2];
  SimCounters *cnt;
  int *queue;
  Fields<double> F[2];        // field buffers 0 / 1 (the pass into current buffer jb reads F[jb])
};
// empties every cell's queue that the pass after the one of parity q fills
__global__ void k_batch_clear_next64(const BatchCell64 *__restrict__ cells, int ncell, int q) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x)
    clear_next_queue(cells[c].cnt, q);
}

// the collisions queued (parity q) by every cell's last pass, one per warp
__global__ void __launch_bounds__(kMccBlock) k_batch_mcc64(const BatchCell64 *__restrict__ cells,
                                                           int ncell, int cur, int q) {
  __shared__ long long pre[kMaxBatch + 1];
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) pre[c + 1] = (long long)cells[c].cnt->n_cand[q];
  __syncthreads();
  if (threadIdx.x == 0) {
    pre[0] = 0;
    for (int c = 0; c < ncell; ++c) pre[c + 1] += pre[c];
  }
  __syncthreads();
  if ((threadIdx.x & 31) != 0) return;
  const long long nq = pre[ncell];
  const long long nwarps = (long long)gridDim.x * (kMccBlock / 32);
  for (long long k = (blockIdx.x * (long long)kMccBlock + threadIdx.x) >> 5; k < nq; k += nwarps) {
    const int c = cell_of_item(pre, ncell, k);
    const BatchCell64 &C = cells[c];
    SimCounters *cc = C.cnt;
    const int *qu = C.queue + (long long)q * C.P[0].cap;
    mcc64_one(C.P[0], C.S[cur], cc, qu[k - pre[c]], cc->step64[q], (long long)cc->n_total);
  }
}

// The FP64 pass of every cell of a batch: (cell, chunk) work items from one
// counter (*chunk_next, zeroed by the field kernel), the cell's parameters
// copied into shared memory when the cell changes.
__global__ void __launch_bounds__(kBlock, 3) k_batch_pass64(const BatchCell64 *__restrict__ cells,
                                                            int ncell, int cur, int jb, int q,
                                                            unsigned long long *chunk_next) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ long long pre[kMaxBatch + 1];
  __shared__ long long item_at;
  __shared__ int chunk_s, cell_at, box_row0, box_rows, box_col0, box_cmax;
  __shared__ __align__(16) unsigned char sP_raw[sizeof(SimParams)];
  SimParams &sP = *reinterpret_cast<SimParams *>(sP_raw);
  for (int i = threadIdx.x; i < kWin64Nodes; i += kBlock) reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) pre[c + 1] = slots_in_use(cells[c].cnt);
  __syncthreads();
  if (threadIdx.x == 0) {
    long long total = 0;
    for (int c = 0; c < ncell; ++c) total += pre[c + 1];
    // a few chunks per block, so that the counter evens out the cells
    const int chunk = even_chunk((unsigned)min((total + 3) / 4, 0x7FFFFFFFll), gridDim.x, kChunk64);
    chunk_s = chunk;
    cell_at = -1;
    pre[0] = 0;
    for (int c = 0; c < ncell; ++c) pre[c + 1] = pre[c] + (pre[c + 1] + chunk - 1) / chunk;
    if (blockIdx.x == 0)
      for (int c = 0; c < ncell; ++c) cells[c].cnt->step64[q] = cells[c].cnt->step64[1 - q] + 1;
  }
  __syncthreads();
  const long long nitem = pre[ncell];
  const int chunk = chunk_s;
  // thread 0 claims the block's next item while one is worked on, brings its
  // state into L2 and, at the end of this one, places its box
  long long next = 0;
  int next_row0 = 0, next_rows = 0, next_col0 = 0;
  auto span = [&](long long g, const BatchCell64 *&C, long long &beg, long long &end) {
    const int c = cell_of_item(pre, ncell, g);
    C = cells + c;
    beg = (g - pre[c]) * chunk;
    end = min(beg + chunk, slots_in_use(C->cnt));
  };
  auto resolve = [&]() {
    if (next >= nitem) return;
    const BatchCell64 *C;
    long long beg, end;
    span(next, C, beg, end);
    const SimParams &Pc = C->P[jb];
    prefetch_chunk64(C->S[cur], beg, end);
    box64(Pc, C->S[cur], beg, end, min(kWin64Nodes / win_stride(win_cols(Pc.nr)), Pc.nz), next_row0,
          next_rows, next_col0);
  };
  if (threadIdx.x == 0) {
    next = (long long)atomicAdd(chunk_next, 1ull);
    resolve();
  }
  for (;;) {
    if (threadIdx.x == 0) {
      item_at = next;
      box_row0 = next_row0;
      box_rows = next_rows;
      box_col0 = next_col0;
      box_cmax = -1;
    }
    __syncthreads();
    const long long g = item_at;
    if (g >= nitem) break;
    if (threadIdx.x == 0) next = (long long)atomicAdd(chunk_next, 1ull);
    const BatchCell64 *C;
    long long beg, end;
    span(g, C, beg, end);
    const int c = (int)(C - cells);
    if (c != cell_at) {          // this block's first chunk of cell c: its parameters
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&C->P[jb]);
      uint32_t *dst = reinterpret_cast<uint32_t *>(sP_raw);
      for (int i = threadIdx.x; i < (int)(sizeof(SimParams) / 4); i += kBlock) dst[i] = src[i];
      __syncthreads();
      if (threadIdx.x == 0) cell_at = c;
    }
    const int cols = win_cols(sP.nr);
    const Win64 w{reinterpret_cast<unsigned *>(smem), box_row0, box_rows, box_col0, cols, win_stride(cols)};
    chunk64<0>(sP, C->S[cur], C->F[jb], C->cnt, C->queue, q, C->cnt->step64[1 - q] + 1, (int)beg, (int)end, w, &box_cmax);
    if (threadIdx.x == 0) resolve();
    __syncthreads();
    flush64(sP, w, box_cmax + 1);
    __syncthreads();
  }

}

// ----------------------------------------------------------- ions
// Before each push the ions are sorted by deposit node quad (the electrons'
// sort key) from the store into a scratch store, dropping the dead; the push
// reads the scratch and writes the store back in that order.  Ions hardly
// move between pushes, so only those born since the last push are out of
// place, and the lanes of a warp then share their deposit nodes (the warp
// sums replace most of the atomics on the crowded cells near the axis).
__device__ __forceinline__ int ion_cell(const IonState &I, long long p, int nr, int nz, double dr,
                                        double dz) {
  const double2 rz = I.rz[p];
  if (rz.x < 0) return -1;
  int ar = (int)floor(rz.x / dr - 0.5) + 1, az = (int)floor(rz.y / dz - 0.5) + 1;
  ar = min(max(ar, 0), nr);
  az = min(max(az, 0), nz);
  return ar + az * (nr + 1);
}

__device__ __forceinline__ long long ions_in_use(const SimCounters *cnt, long long cap) {
  const unsigned long long nc = cnt->n_ions;
  return (long long)(nc < (unsigned long long)cap ? nc : cap);
}

__global__ void k_ion_hist(IonState I, const SimCounters *cnt, long long cap, int nr, int nz,
                           double dr, double dz, int *count) {
  const long long n = ions_in_use(cnt, cap);
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * blockDim.x) {
    const long long p = base + (threadIdx.x & 31);
    const int c = p < n ? ion_cell(I, p, nr, nz, dr, dz) : -1;
    const unsigned live = __ballot_sync(0xFFFFFFFFu, c >= 0);
    if (c < 0) continue;
    const unsigned mask = __match_any_sync(live, c);
    if ((__ffs(mask) - 1) == (int)(threadIdx.x & 31)) atomicAdd(count + c, __popc(mask));
  }
}

__global__ void k_ion_scatter(IonState A, IonState B, const SimCounters *cnt, long long cap,
                              int nr, int nz, double dr, double dz, const int *offset,
                              int *cursor) {
  const long long n = ions_in_use(cnt, cap);
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * blockDim.x) {
    const long long p = base + lane;
    const int c = p < n ? ion_cell(A, p, nr, nz, dr, dz) : -1;
    const unsigned live = __ballot_sync(0xFFFFFFFFu, c >= 0);
    if (c < 0) continue;
    const unsigned mask = __match_any_sync(live, c);
    const int leader = __ffs(mask) - 1;
    int basepos = 0;
    if (lane == leader) basepos = atomicAdd(cursor + c, __popc(mask));
    basepos = __shfl_sync(mask, basepos, leader);
    const long long dst = (long long)offset[c] + basepos + __popc(mask & ((1u << lane) - 1));
    B.rz[dst] = A.rz[p]; B.urt[dst] = A.urt[p]; B.uz[dst] = A.uz[p];
    B.id[dst] = A.id[p]; B.q[dst] = A.q[p];
  }
}

// the live ions are now the first offset[nbin] slots
__global__ void k_ion_sort_finish(SimCounters *cnt, const int *offset, int nbin) {
  cnt->n_ions = (unsigned long long)offset[nbin];
}

// Ion push, once every ion_subcycle electron steps: P is the simulation's
// parameter block with dt = the ion step, qm_dt2 = q_e/m_ion dt/2 and the
// ion current buffers as Jr/Jz (cleared before the launch), dep = the
// fixed-point factor of the ion current.  Per ion of the sorted scratch
// store src: gather, Boris kick with charge Z q_e, two half drifts (the
// electrons' walls: absorbed beyond Rp, reflected at z = 0 and Lp), deposit
// of Z q_e FN v at the new position; the ion goes back to the store P.ion at
// the same index.  The field update adds the ion current to the electrons'
// until the next push (charge moved over the ion step = the held current x
// the ion step).
template <typename T>
__global__ void __launch_bounds__(kBlock) k_ion_push(SimParams P, Fields<T> F, SimCounters *cnt,
                                                     IonState src) {
  const long long n = ions_in_use(cnt, P.ion_cap);
  const IonState I = P.ion;
  unsigned lost = 0;
  for (long long base = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * blockDim.x) {
    const long long p = base + (threadIdx.x & 31);
    bool act = p < n;
    double2 rz = make_double2(-1.0, 0.0), urt = make_double2(0.0, 0.0);
    double uz = 0, Zq = 0;
    if (act) {
      rz = src.rz[p];
      act = rz.x >= 0;
    }
    if (act) {
      urt = src.urt[p]; uz = src.uz[p];
      const int8_t q = src.q[p];
      Zq = (double)q;
      I.id[p] = src.id[p]; I.q[p] = q;
      double r = rz.x, z = rz.y, ur = urt.x, ut = urt.y;
      bool alive = true;
      double E_r, E_z, Hp;
      gather3s<T>(F.Er, F.Ez, F.H, P.nr, P.nz, P.ldf, P.ldf, P.ldf, P.dr, P.dz, r, z, E_r, E_z, Hp);
      boris(ur, ut, uz, E_r, 0.0, E_z, 0.0, P.mu0 * Hp, 0.0, Zq * P.qm_dt2, P.c);
      halfdrift64(r, z, ur, ut, uz, alive, P);
      if (alive) halfdrift64(r, z, ur, ut, uz, alive, P);
      if (!alive) {
        lost++;
        r = -1.0;
        count_wall_loss(cnt, (ur * ur + ut * ut + uz * uz) / (P.c * P.c), P.m_ion * P.c * P.c / P.qe);
      }
      rz = make_double2(r, z); urt = make_double2(ur, ut);
      I.rz[p] = rz; I.urt[p] = urt; I.uz[p] = uz;
      act = alive;
    }
    int64_t a[4] = {0, 0, 0, 0};
    long long vr[4] = {0, 0, 0, 0}, vz[4] = {0, 0, 0, 0};
    unsigned key = 0;
    if (act) deposit_values64(P, rz.x, rz.y, urt.x, urt.y, uz, Zq * P.qe, a, vr, vz, key);
    warp_deposit<long long>(act, key, a, vr, vz, P.Jr, P.Jz);
  }
  lost = __reduce_add_sync(0xFFFFFFFFu, lost);
  if ((threadIdx.x & 31) == 0 && lost) atomicAdd(&cnt->ion_lost, (unsigned long long)lost);
}

// ion diagnostics: alive, sum of charge numbers, kinetic energy (fixed point)
__global__ void k_ion_diag(IonState I, long long cap, SimCounters *cnt, double c, double m_ion,
                           double qe) {
  const unsigned long long nc = cnt->n_ions;
  const long long n = (long long)(nc < (unsigned long long)cap ? nc : cap);
  unsigned long long kin = 0, alive = 0, charge = 0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    if (I.rz[p].x < 0) continue;
    const double2 a = I.urt[p];
    const double w = I.uz[p];
    const double u2 = (a.x * a.x + a.y * a.y + w * w) / (c * c);
    const double g = sqrt(1 + u2);
    kin += (unsigned long long)__double2ll_rn(m_ion * c * c * (u2 / (g + 1)) / qe * 4294967296.0);
    alive++;
    charge += (unsigned long long)I.q[p];
  }
  for (int o = 16; o; o >>= 1) {
    kin += __shfl_down_sync(0xFFFFFFFFu, kin, o);
    alive += __shfl_down_sync(0xFFFFFFFFu, alive, o);
    charge += __shfl_down_sync(0xFFFFFFFFu, charge, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&cnt->ion_kin_fx, kin);
    atomicAdd(&cnt->ion_alive, alive);
    atomicAdd(&cnt->ion_charge, charge);
  }
}

__global__ void k_ion_load(IonState I, const double *r, const double *z, const double *ur,
                           const double *ut, const double *uz, const uint64_t *id,
                           const int8_t *q, long long n) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    I.rz[p] = make_double2(r[p], z[p]);
    I.urt[p] = make_double2(ur[p], ut[p]);
    I.uz[p] = uz[p];
    I.id[p] = id[p];
    I.q[p] = q ? q[p] : (int8_t)1;
  }
}

__global__ void k_ion_read(IonState I, double *r, double *z, double *ur, double *ut, double *uz,
                           uint64_t *id, int8_t *q, long long n) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    const double2 a = I.rz[p], b = I.urt[p];
    r[p] = a.x; z[p] = a.y; ur[p] = b.x; ut[p] = b.y; uz[p] = I.uz[p];
    id[p] = I.id[p];
    q[p] = I.q[p];
  }
}

// ----------------------------------------------------------- FP32 form
// 1/sqrt(x) refined by one Newton step: the hardware estimate is biased, and
// a biased rotation normaliser or gamma makes the FP32 energy drift steadily
__device__ __forceinline__ float rsqrt_nr(float x) {
  const float y = rsqrtf(x);
  return y * fmaf(-0.5f * x * y, y, 1.5f);
}

// Packed pairs: Blackwell issues two FP32 operations of a float2 as one
// instruction (__fadd2/__fmul2/__ffma2, sm_100); the FP32 push pairs its
// independent r/z (or column/row) operations this way.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// a + d with stochastic rounding.  The per-step velocity changes of the FP32
// form (a drift rotation by a small angle, a kick in a weak field) are often
// below one float ulp of u; rounding them to nearest would bias |u| steadily.
// With h the spacing of the floats in a's binade and U uniform in [0, 1), the
// sum a + d + sign(a) U h rounded toward zero is a + d rounded to one of its
// two neighbours on that grid, the far one with probability equal to the
// distance from the near one in units of h: unbiased as long as a + d stays
// in a's binade (within |d| of a power of two the grid changes and the split
// is off by up to a factor 2; there |d| << |a| makes that a rare, tiny
// error).  a + d + U h is formed exactly enough in one FMA (d and U h are
// both small against a) and rounded once.  U = (k + 1/2) 2^-16, k a 16-bit
// random number, is built as a float in [1, 2) minus 1; a = 0 gives h = 0
// and the exact d.  Done on a pair of components: k from the low 16 bits of r
// for x, from the high 16 for y.
__device__ __forceinline__ float2 sround_add2(float2 a, float2 d, uint32_t r) {
  const float2 h = __fmul2_rn(f2(__int_as_float(__float_as_int(a.x) & 0x7F800000),
                                 __int_as_float(__float_as_int(a.y) & 0x7F800000)),
                              f2(1.1920928955078125e-07f));
  const float2 u = __fadd2_rn(f2(__uint_as_float(0x3F800040u | ((r & 0xFFFFu) << 7)),
                                 __uint_as_float(0x3F800040u | ((r >> 16) << 7))),
                              f2(-1.0f));
  return __fadd2_rz(a, __ffma2_rn(f2(copysignf(u.x, a.x), copysignf(u.y, a.y)), h, d));
}

// Floors and nearest integers in FP32 without conversions: for |x| < 2^22,
// x + 1.5 2^23 lies where the floats are one apart, so rounding that sum
// down (or to nearest) gives 1.5 2^23 + floor(x) (or + rint(x)) exactly and
// its bit pattern minus 0x4B400000 is the integer.

// half-cell staggered index/weight: position ic + f measured from node ic-1/2
__device__ __forceinline__ void half_shift(int ic, float f, int &a, float &w) {
  const bool up = f >= 0.5f;
  a = up ? ic : ic - 1;
  w = up ? f - 0.5f : f + 0.5f;
}

// specular reflection of the cell coordinate (iz, fz) into [0, nz)
__device__ __forceinline__ void reflect_z(int &iz, float &fz, float &uz, int nz) {
  if (iz < 0 || iz >= nz) {
    iz = iz < 0 ? -iz - 1 : 2 * nz - iz - 1;
    fz = 1.f - fz;
    uz = -uz;
    if (fz >= 1.f) { fz = 0.f; iz += 1; }
    if (iz > nz - 1) { iz = nz - 1; fz = 0.99999994f; }
    if (iz < 0) { iz = 0; fz = 0.f; }
  }
}

// Straight-line drift in cell units over (hr, hz) cells per unit beta:
// (P.hdr, P.hdz) is a half step, twice that a full step.  Two half drifts at
// the same velocity are one full drift: the Cartesian path is the same line,
// the radius along a line is convex (a particle inside the wall at both ends
// is inside at the midpoint), and the end reflection is specular.  The new
// radius comes from the exact difference r' - rc = (dx (2 rc + dx) + dy^2) /
// (r' + rc) (no cancellation at large rc); (u_r, u_theta) turn by the drift
// angle a, written with the small quantities sin a and 1 - cos a = sin^2 a /
// (1 + cos a) and added to u with stochastic rounding (rb: two 16-bit random
// numbers).
__device__ __forceinline__ void drift32(int &ir, int &iz, float &fr, float &fz, float &ur,
                                        float &ut, float &uz, bool &alive, const SimParams &P,
                                        uint32_t rb, float hr, float hz, float &ig) {
  // 1/gamma, kept by the turn.  (The hardware estimate is enough here: it only
  // scales the displacement and the current, and the turn keeps |u| whatever
  // it is; the kick's 1/gamma is refined.)
  ig = rsqrtf(fmaf(ur, ur, fmaf(ut, ut, fmaf(uz, uz, 1.0f))));
  const float2 dxy = __fmul2_rn(__fmul2_rn(f2(ur, ut), f2(ig)), f2(hr));   // (dx, dy)
  const float dx = dxy.x, dy = dxy.y, dzz = uz * ig * hz;
  const float rc = (float)ir + fr;
  const float X = rc + dx;
  const float r2 = fmaf(X, X, dy * dy);
  // (products that feed a sum are __fmul_rn: never contracted into an FMA,
  // so every kernel that inlines this rounds the same way)
  const float irn = rsqrt_nr(r2);                    // 1/r' (inf at r' = 0)
  const float rn = __fmul_rn(r2, irn);
  const float sn = r2 > 0.f ? dy * irn : 0.f;
  const float s2 = __fmul_rn(sn, sn);
  const float cs = r2 > 0.f ? X * irn : 1.f;         // cos a
  const float c1 = X >= 0.f ? __fdividef(s2, 1.f + cs) : 1.f - cs;   // 1 - cos a
  // (du_r, du_theta) = (sn ut - c1 ur, -sn ur - c1 ut)
  const float2 du = __ffma2_rn(f2(sn, -sn), f2(ut, ur), __fmul2_rn(f2(ur, ut), f2(-c1)));
  const float2 u2 = sround_add2(f2(ur, ut), du, rb);
  ur = u2.x;
  ut = u2.y;
  const float den = rn + rc;
  const float drr = den > 0.f ? __fdividef(fmaf(dx, 2.f * rc + dx, dy * dy), den) : 0.f;
  // floor of both offsets at once (take_floor on a pair)
  const float2 f = __fadd2_rn(f2(fr, fz), f2(drr, dzz));
  const float2 t = __fadd2_rd(f, f2(12582912.0f));
  const float2 g = __fadd2_rn(f, neg2(__fadd2_rn(t, f2(-12582912.0f))));
  fr = g.x;
  fz = g.y;
  ir += __float_as_int(t.x) - 0x4B400000;
  iz += __float_as_int(t.y) - 0x4B400000;
  if (ir < 0) { ir = 0; fr = 0.f; }
  alive = alive && ir < P.nr;
  reflect_z(iz, fz, uz, P.nz);
}

// The fixed-point contributions to the four deposit nodes (columns ar, ar + 1,
// rows az, az + 1; clamped one-sided at the edges as EM7.cu:56-202, see
// clamp_nodes).  perm (0..7) permutes them: bit 2 swaps the components (vr then
// holds z, vz r), bit 0 the columns, bit 1 the rows, so the node order is (c0,r0), (c1,r0), (c0,r1), (c1,r1) with (c0,
// c1) = (ar, ar + 1) or (ar + 1, ar) and likewise rows; each node's integer is the same
// whatever the order (its weight is the same product of the same two factors).  The
// weights sum to 1, so one particle adds at most 2^20 in magnitude to any
// node, even where clamped nodes merge.  ig: 1/gamma of u (the drift's,
// which turns u without changing |u|).
__device__ __forceinline__ void deposit_values32(const SimParams &P, int ir, int iz, float fr, float fz,
                                                 float ur, float uz, float ig, int perm, int &ar, int &az,
                                                 int vr[4], int vz[4]) {
  float wr, wz;
  half_shift(ir, fr, ar, wr);
  half_shift(iz, fz, az, wz);
  const bool sc = perm & 1, sr = perm & 2;
  const float2 om = __fadd2_rn(f2(1.f), f2(-wr, -wz));        // (1 - wr, 1 - wz)
  const float2 A = sc ? f2(wr, om.x) : f2(om.x, wr);         // column factors of c0, c1
  const float B0 = sr ? wz : om.y, B1 = sr ? om.y : wz;       // row factors of r0, r1
  const float2 w01 = __fmul2_rn(A, f2(B0)), w23 = __fmul2_rn(A, f2(B1));
  const bool sw = perm & 4;
  const float2 k = __fmul2_rn(__fmul2_rn(f2(P.depf), sw ? f2(uz, ur) : f2(ur, uz)), f2(ig));   // (kr, kz)
  const float2 C = f2(12582912.0f);
  const float2 v0 = __ffma2_rn(k, f2(w01.x), C), v1 = __ffma2_rn(k, f2(w01.y), C);
  const float2 v2 = __ffma2_rn(k, f2(w23.x), C), v3 = __ffma2_rn(k, f2(w23.y), C);
  vr[0] = __float_as_int(v0.x) - 0x4B400000; vz[0] = __float_as_int(v0.y) - 0x4B400000;
  vr[1] = __float_as_int(v1.x) - 0x4B400000; vz[1] = __float_as_int(v1.y) - 0x4B400000;
  vr[2] = __float_as_int(v2.x) - 0x4B400000; vz[2] = __float_as_int(v2.y) - 0x4B400000;
  vr[3] = __float_as_int(v3.x) - 0x4B400000; vz[3] = __float_as_int(v3.y) - 0x4B400000;
}

__device__ __forceinline__ void clamp_nodes(const SimParams &P, int ar, int az, int perm, int &c0, int &c1,
                                            int &r0, int &r1) {
  const int ca = max(ar, 0), cb = min(ar + 1, P.nr - 1);
  const int ra = max(az, 0), rb = min(az + 1, P.nz - 1);
  const bool sc = perm & 1, sr = perm & 2;
  c0 = sc ? cb : ca; c1 = sc ? ca : cb;
  r0 = sr ? rb : ra; r1 = sr ? ra : rb;
}

// FP32-form deposit window: int32 sums of one chunk of particles on a box of
// the grid in shared memory (chunk_box).  A chunk holds at most kChunkMax
// particles, so a node's window sum stays below kChunkMax * 2^20 < 2^31.  A
// node's two sums (r, z) are adjacent words, so one address serves both
// atomics; rows are ws >= cols nodes apart with ws = 3 (mod 32), so the 3 x 3
// nodes around a warp's particles sit in 9 different bank pairs.  Nodes
// outside the window go straight to the grid with 64-bit atomics; the window
// is added to the grid with one 64-bit atomic per touched node.
// WIDE: the grid has more than kWinCols columns and the box only a part of
// them, but 15 rows.  With all columns a 1024-wide grid had 3 rows, which the
// electrons leave between two sorts: 16M electrons, step 495 us, now 423.  A
// box of all columns needs no column test (on 256 columns the test and the
// register for the box's first column cost 0.7 us of 55).
constexpr int kWinNodes = 4096;           // nodes (two int32 sums each)
constexpr int64_t kQuadCells = 1300000;   // cells of a grid with gather quads at most: 62 MB, half of L2

struct Win32 {
  int *rz;                  // node k: r at rz[2k], z at rz[2k + 1]
  int row0, rows, col0, cols, ws;
};

template <bool WIDE>
__device__ __forceinline__ void win_node(const Win32 &w, const SimParams &P, int col, int row,
                                         int vr, int vz) {
  const unsigned lr = (unsigned)(row - w.row0), lc = (unsigned)(col - w.col0);
  if (lr < (unsigned)w.rows && (!WIDE || lc < (unsigned)w.cols)) {
    const int k = (int)lr * w.ws + (int)lc;
    atomicAdd(w.rz + 2 * k, vr);
    atomicAdd(w.rz + 2 * k + 1, vz);
  } else {
    const int64_t g = col + (int64_t)row * P.ldj;
    if (vr) atomicAdd(P.Jr + g, (unsigned long long)(long long)vr);
    if (vz) atomicAdd(P.Jz + g, (unsigned long long)(long long)vz);
  }
}

// FP32 state flags.  The in-cell offsets fr, fz are >= 0, so their sign bits
// are free: the sign of fr marks a pending collision (the particle sits in the
// collision queue of the pass that pushed it last), the sign of fz is the
// parity of the step in which the particle was pushed last.
constexpr uint32_t kSign = 0x80000000u;

__device__ __forceinline__ uint4 pack32(int ir, int iz, float fr, float fz, float ur, bool alive,
                                        bool pending = false, int par = 0) {
  return make_uint4(alive ? (((uint32_t)iz << 16) | (uint32_t)ir) : kDead,
                    __float_as_uint(fr) | (pending ? kSign : 0u),
                    __float_as_uint(fz) | (par ? kSign : 0u), __float_as_uint(ur));
}

// One particle's push in step `step`.  mode 0: gather, Boris kick, drift of
// the whole step, null-collision candidate test; mode 1: half drift (start of
// a run); mode 2: gather, kick, half drift to integer time (end of a run).
// Returns whether the particle is a collision candidate (alive, mode 0).
template <int MODE>
__device__ __forceinline__ bool push32(const SimParams &P, const Fields<float> &F, uint64_t id,
                                       long long step, int &ir, int &iz, float &fr,
                                       float &fz, float &ur, float &ut, float &uz, bool &alive,
                                       float &ig) {
  // block 0 of this particle's stream: words 0-1 decide the null-collision
  // candidate, words 2-3 drive the stochastic rounding of the kick and the turn
  uint32_t c[4] = {(uint32_t)id, (uint32_t)(id >> 32), (uint32_t)step, 0u};
  if (MODE == 1) {
    philox4x32_10(c, P.pk);
    drift32(ir, iz, fr, fz, ur, ut, uz, alive, P, c[3], P.hdr, P.hdz, ig);
    return false;
  }
  int ar, az;
  float wr, wz;
  half_shift(ir, fr, ar, wr);
  half_shift(iz, fz, az, wz);
  // the field loads go out first, their latency hidden behind Philox: one
  // packed quad per field (corners already clamped at the edges), or the
  // same four corners from the fields themselves (the same floats).  Ordinary
  // loads: the field update may still be writing when this kernel starts, so the
  // arrays are not read-only for its whole life, as __ldg requires.
  float4 a4, b4, c4;
  if (P.qEr) {
    a4 = P.qEr[(ar + 1) + iz * (P.nr + 1)];
    b4 = P.qEz[ir + (az + 1) * P.nr];
    c4 = P.qH[(ar + 1) + (az + 1) * (P.nr + 1)];
  } else {
    const int c0 = max(ar, 0), c1 = min(ar + 1, P.nr - 1);
    const int ra = max(az, 0), rb = min(az + 1, P.nz - 1);
    const float *e0 = F.Er + iz * P.ldf, *e1 = e0 + P.ldf;
    a4 = make_float4(e0[c0], e0[c1], e1[c0], e1[c1]);
    const float *z0 = F.Ez + ra * P.ldf + ir, *z1 = F.Ez + rb * P.ldf + ir;
    b4 = make_float4(z0[0], z0[1], z1[0], z1[1]);
    const float *h0 = F.H + ra * P.ldf, *h1 = F.H + rb * P.ldf;
    c4 = make_float4(h0[c0], h0[c1], h1[c0], h1[c1]);
  }
  philox4x32_10(c, P.pk);
  // bilinear mixes from the quads' corners (c0,r0), (c1,r0), (c0,r1), (c1,r1)
  // = (x, y, z, w), paired: the low and high rows of each quad along its
  // columns, then Er and Ez along their rows
  const float2 cE = __ffma2_rn(f2(wr), __fadd2_rn(f2(a4.y, a4.w), f2(-a4.x, -a4.z)), f2(a4.x, a4.z));
  const float2 cZ = __ffma2_rn(f2(fr), __fadd2_rn(f2(b4.y, b4.w), f2(-b4.x, -b4.z)), f2(b4.x, b4.z));
  const float2 cH = __ffma2_rn(f2(wr), __fadd2_rn(f2(c4.y, c4.w), f2(-c4.x, -c4.z)), f2(c4.x, c4.z));
  const float2 E = __ffma2_rn(f2(fz, wz), __fadd2_rn(f2(cE.y, cZ.y), f2(-cE.x, -cZ.x)), f2(cE.x, cZ.x));
  const float H = fmaf(wz, cH.y - cH.x, cH.x);
  // Boris in gamma*beta units: E = (Er, 0, Ez), B = (0, mu0 H, 0); the
  // increment u+ - u is formed first, then added with stochastic rounding
  // (random bits: Philox words 2 and 3)
  const float2 he = __fmul2_rn(f2(P.aE), E);                  // (her, hez)
  const float2 um = __fadd2_rn(f2(ur, uz), he);               // (umr, umz)
  const float igm = rsqrt_nr(fmaf(um.x, um.x, fmaf(ut, ut, fmaf(um.y, um.y, 1.0f))));
  const float t = P.aB * H * igm;
  const float s = __fdividef(2.f * t, fmaf(t, t, 1.f));
  const float2 up = __ffma2_rn(f2(-um.y, um.x), f2(t), um);   // (upr, upz)
  const float2 du = __ffma2_rn(f2(-up.y, up.x), f2(s), __fadd2_rn(he, he));
  const float2 uk = sround_add2(f2(ur, uz), du, c[2]);
  ur = uk.x;
  uz = uk.y;
  const float h = MODE == 0 ? 2.f : 1.f;
  drift32(ir, iz, fr, fz, ur, ut, uz, alive, P, c[3], h * P.hdr, h * P.hdz, ig);
  return alive && MODE == 0 && (((((uint64_t)c[0]) << 32) | c[1]) >> 12) < P.cand_below;
}

// ig: the drift's 1/gamma, as in the chunk loop, so that a particle deposits
// the same integers whichever path pushed it
__device__ __forceinline__ void deposit_global32(const SimParams &P, int ir, int iz, float fr,
                                                 float fz, float ur, float uz, float ig) {
  int ar, az, ca, cb, ra, rb, vr[4], vz[4];
  deposit_values32(P, ir, iz, fr, fz, ur, uz, ig, 0, ar, az, vr, vz);
  clamp_nodes(P, ar, az, 0, ca, cb, ra, rb);
  const int64_t a[4] = {ca + (int64_t)ra * P.ldj, cb + (int64_t)ra * P.ldj,
                        ca + (int64_t)rb * P.ldj, cb + (int64_t)rb * P.ldj};
  deposit_atomic<int>(a, vr, vz, P.Jr, P.Jz);
}

__device__ __forceinline__ void queue_one(SimCounters *cnt, int *queue, const SimParams &P,
                                          int par, long long p) {
  const unsigned long long k = atomicAdd(&cnt->n_cand[par], 1ull);
  queue[(long long)par * P.cap + (long long)k] = (int)p;
}

// A collision candidate of the previous step (FP32 form), taken by two lanes:
// the MCC at the end of step `step` - 1 (FP64 test, branch, energy sharing;
// float turn) by both, then the first lane goes on with the electron and the
// second (kid) with its secondary, born at the parent's position.  PUSH: each
// is pushed in step `step` (MODE as push32), its current deposited by global
// atomics, with its own candidate test; otherwise nothing more.  The two pushes
// share their instructions: one after the other in one lane, with the push of
// every mode inlined, a pass whose chains are its critical path was 2 us
// longer.  The chunk loop of the pass skips these particles (pending flag set,
// or pushed-parity = this step's).
// P: the launch's parameters in global memory (a reference to the kernel's
// own parameter block would make every thread copy it to its stack).
template <int MODE, bool PUSH>
__device__ __noinline__ void candidate32(const SimParams *__restrict__ Pg, Fields<float> F,
                                         State32 S, SimCounters *cnt, int *queue, long long p,
                                         long long step, bool kid, long long n0, unsigned &lost) {
  const SimParams &P = *Pg;
  const int par = (int)(step & 1);
  const long long cstep = PUSH ? step - 1 : step;      // step whose collision this is
  const uint4 A = S.a[p];
  const float2 B = S.b[p];
  uint64_t id = S.id[p];
  __syncwarp(3u << (threadIdx.x & 30));   // both lanes have read p before the first one writes it
  int ir = (int)(A.x & 0xFFFFu), iz = (int)(A.x >> 16);
  float fr = __uint_as_float(A.y & ~kSign), fz = __uint_as_float(A.z & ~kSign);
  double dux = (double)__uint_as_float(A.w) * P.c, duy = (double)B.x * P.c, duz = (double)B.y * P.c;
  Birth b;
  const int ev = mcc_event<true>(P, id, cstep, dux, duy, duz, b, gas_density(P, ir, iz));
  if (kid) {
    if (!b.born) return;
    const unsigned long long kb = atomicAdd(&cnt->n_births, 1ull);
    p = n0 + (long long)kb;
    if (p >= P.cap) {
      atomicAdd(&cnt->cap_overflow, 1ull);
      return;
    }
    id = child_id(id, cstep);
    dux = b.ux; duy = b.uy; duz = b.uz;
  } else {
    count_event(cnt, ev, b);
    if (ev == 2 && P.ion_cap > 0)
      ion_birth(P.ion, P.ion_cap, ion_spread(P, ir, iz), P.seed, cnt, id, cstep, ((double)ir + (double)fr) * P.dr,
                ((double)iz + (double)fz) * P.dz);
  }
  float ur = (float)(dux / P.c), ut = (float)(duy / P.c), uz = (float)(duz / P.c);
  bool alive = true, cand = false;
  if (PUSH) {
    float ig;
    cand = push32<MODE>(P, F, id, step, ir, iz, fr, fz, ur, ut, uz, alive, ig);
    if (alive && MODE != 2) deposit_global32(P, ir, iz, fr, fz, ur, uz, ig);
    if (!alive) {
      lost++;
      count_wall_loss(cnt, (double)ur * ur + (double)ut * ut + (double)uz * uz, P.me * P.c * P.c / P.qe);
    }
    if (cand) queue_one(cnt, queue, P, par, p);
  }
  S.a[p] = pack32(ir, iz, fr, fz, ur, alive, cand, PUSH ? par : (int)(cstep & 1));
  S.b[p] = make_float2(ut, uz);
  if (kid) S.id[p] = id;
}

// Box of the particles [beg, end) (chunk_box) from the cells of the first and last one
__device__ __forceinline__ void box32(const SimParams &P, const State32 &S, long long beg, long long end,
                                      int cols, int maxrows, int &row0, int &rows, int &col0) {
  const uint32_t k0 = reinterpret_cast<const uint32_t *>(S.a + beg)[0];
  const uint32_t k1 = reinterpret_cast<const uint32_t *>(S.a + end - 1)[0];
  int lo = P.nz, hi = -1, col = 0;
  if (k0 != kDead) { lo = hi = (int)(k0 >> 16); col = (int)(k0 & 0xFFFFu); }
  if (k1 != kDead) { lo = min(lo, (int)(k1 >> 16)); hi = max(hi, (int)(k1 >> 16)); }
  chunk_box(P.nr, P.nz, cols, maxrows, lo, hi, col, row0, rows, col0);
}

__device__ __forceinline__ void prefetch_chunk32(const State32 &S, long long beg, long long end) {
  const long long n = end - beg;
  if (n <= 0) return;
  prefetch_l2(S.a + beg, (uint32_t)(n * 16));
  prefetch_l2(S.b + beg, (uint32_t)((n * 8) & ~15ll));
  prefetch_l2(S.id + beg, (uint32_t)((n * 8) & ~15ll));
}

// The particles [beg, end) of one chunk of the FP32 pass of step `step`:
// push (push32), collision candidates queued, deposit into the window w
// (nodes outside the window straight to the grid).  The highest window column touched is merged
// into *box_cmax; electrons absorbed at the wall are counted into cnt.
template <int MODE, bool WIDE>
__device__ __forceinline__ void chunk32(const SimParams &P, const State32 &S, const Fields<float> &F,
                                        SimCounters *cnt, int *queue, long long step,
                                        int beg, int end, const Win32 &w, int *box_cmax) {
  const int par = (int)(step & 1);
  const uint32_t parbit = par ? kSign : 0u;
  const int lane = threadIdx.x & 31;
  unsigned lost = 0;
  int wc_max = -1;                 // highest window column this lane touched
  // the next iteration's particle is loaded one iteration ahead, so its
  // HBM latency overlaps the current particle's arithmetic
  int base = beg + (int)(threadIdx.x & ~31);
  uint4 An = make_uint4(kDead, 0, 0, 0);
  float2 Bn = make_float2(0.f, 0.f);
  uint64_t idn = 0;
  if (base + lane < end) { An = S.a[base + lane]; Bn = S.b[base + lane]; idn = S.id[base + lane]; }
  for (; base < end; base += kBlock) {
    const int p = base + lane;
    uint4 A = An;
    const float2 B = Bn;
    const uint64_t id = idn;
    {
      const int pn = p + kBlock;
      An = make_uint4(kDead, 0, 0, 0);
      if (pn < end) { An = S.a[pn]; Bn = S.b[pn]; idn = S.id[pn]; }
    }
    // skip the dead, the pending collisions and those already pushed in
    // this step (the candidates the pass has taken)
    bool act = p < end && A.x != kDead && !(A.y & kSign) && (A.z & kSign) != parbit;
    int ir = (int)(A.x & 0xFFFFu), iz = (int)(A.x >> 16);
    float fr = __uint_as_float(A.y & ~kSign), fz = __uint_as_float(A.z & ~kSign);
    float ur = __uint_as_float(A.w), ut = B.x, uz = B.y, ig = 1.f;
    bool cand = false;
    if (act) {
      bool alive = true;
      cand = push32<MODE>(P, F, id, step, ir, iz, fr, fz, ur, ut, uz, alive, ig);
      if (!alive) {
        lost++;
        count_wall_loss(cnt, (double)ur * ur + (double)ut * ut + (double)uz * uz, P.me * P.c * P.c / P.qe);
      }
      S.a[p] = pack32(ir, iz, fr, fz, ur, alive, cand, par);
      S.b[p] = make_float2(ut, uz);
      act = alive && MODE != 2;
    }
    queue_push(cand, p, &cnt->n_cand[par], queue + (long long)par * P.cap);
    // Deposit: each lane adds its own eight contributions to the window,
    // visiting its four nodes in an order permuted by lane & 3 (columns
    // swapped on bit 0, rows on bit 1) and at each node r and z in an order by
    // bit 2, so lanes on the same node quad - sorted particles put one to a few
    // quads in a warp - hit eight different words in each atomic, in even and
    // odd banks.  (With r always first the batched pass of 16 cells, whose
    // shared-memory pipe is 70% busy, was 10 us of 200 longer.  Summing the lanes of a quad first with
    // match.any / redux.sync made this pass two to four times slower on B200.)
    if (act) {
      int ar, az, vr[4], vz[4];
      deposit_values32(P, ir, iz, fr, fz, ur, uz, ig, lane & 7, ar, az, vr, vz);
      const int a = ar - (WIDE ? w.col0 : 0), b = az - w.row0;
      int c0, c1, r0, r1;
      if ((unsigned)a < (unsigned)(w.cols - 1) && (unsigned)b < (unsigned)(w.rows - 1)) {
        // all four nodes in the box and on the grid (no clamping)
        const int k = 2 * (b * w.ws + a), dr = lane & 2 ? 2 * w.ws : 0, e = 2 * (lane & 1) + ((lane >> 2) & 1);
        int *n0 = w.rz + (k + dr), *n1 = w.rz + (k + 2 * w.ws - dr);
        atomicAdd(n0 + e, vr[0]); atomicAdd(n0 + (e ^ 1), vz[0]);
        atomicAdd(n0 + (e ^ 2), vr[1]); atomicAdd(n0 + (e ^ 3), vz[1]);
        atomicAdd(n1 + e, vr[2]); atomicAdd(n1 + (e ^ 1), vz[2]);
        atomicAdd(n1 + (e ^ 2), vr[3]); atomicAdd(n1 + (e ^ 3), vz[3]);
      } else {
        clamp_nodes(P, ar, az, lane & 3, c0, c1, r0, r1);
        if (lane & 4) {
#pragma unroll
          for (int n = 0; n < 4; ++n) { const int t = vr[n]; vr[n] = vz[n]; vz[n] = t; }
        }
        win_node<WIDE>(w, P, c0, r0, vr[0], vz[0]);
        win_node<WIDE>(w, P, c1, r0, vr[1], vz[1]);
        win_node<WIDE>(w, P, c0, r1, vr[2], vz[2]);
        win_node<WIDE>(w, P, c1, r1, vr[3], vz[3]);
      }
      wc_max = max(wc_max, a + 1);   // (win_node may use the window for one row or column)
    }
  }
  // the window columns this warp touched, merged into the block's; the wall
  // losses of the warp
  wc_max = __reduce_max_sync(0xFFFFFFFFu, wc_max);
  if (lane == 0 && wc_max >= 0) atomicMax(box_cmax, min(wc_max, w.cols - 1));
  lost = __reduce_add_sync(0xFFFFFFFFu, lost);
  if (lane == 0 && lost) atomicAdd(&cnt->lost, (unsigned long long)lost);
}

// Add the window columns [0, bw) of every window row to the grid (one 64-bit
// atomic per nonzero node) and zero them for the next chunk.
__device__ __forceinline__ void flush32(const SimParams &P, const Win32 &w, int bw) {
  const int nb = bw > 0 ? bw * w.rows : 0;
  for (int i = threadIdx.x; i < nb; i += kBlock) {
    const int row = i / bw, col = i - row * bw;
    const int k = row * w.ws + col;
    const int2 v = reinterpret_cast<const int2 *>(w.rz)[k];
    const int vr = v.x, vz = v.y;
    if (vr | vz) {
      const int64_t g = (int64_t)(w.row0 + row) * P.ldj + w.col0 + col;
      if (vr) atomicAdd(P.Jr + g, (unsigned long long)(long long)vr);
      if (vz) atomicAdd(P.Jz + g, (unsigned long long)(long long)vz);
      reinterpret_cast<int2 *>(w.rz)[k] = make_int2(0, 0);
    }
  }
}

constexpr int kCandLanes = 8;     // collision candidates a warp of the pass takes at once

// FP32 particle pass of step `step` (modes as push32).  Its blocks first take
// the collision candidates queued by the previous pass, kCandLanes per warp,
// two lanes each (a long serial chain; a warp's chains share its issue but
// serialise their different collision branches, so a few per warp, not 32,
// keep the longest warp short), then all other particles in chunks of
// P.chunk handed out in order, so the blocks that ran candidates simply take
// fewer chunks.  Counters are committed by the field
// kernel of the next step.
template <int MODE, bool WIDE>
__global__ void __launch_bounds__(kBlock, 4) k_pass32(SimParams P, State32 S, Fields<float> F,
                                                      SimCounters *cnt, int *queue,
                                                      const SimParams *__restrict__ Pg) {
  constexpr int mode = MODE;
  __shared__ __align__(16) int win_rz[2 * kWinNodes];
  __shared__ int win_row0, win_rows, win_col0;
  __shared__ int box_cmax;                       // highest window column the chunk touched
  __shared__ long long chunk_at;
  // the window starts zeroed; each chunk's flush leaves it zeroed again
  for (int i = threadIdx.x; i < kWinNodes; i += kBlock) reinterpret_cast<int2 *>(win_rz)[i] = make_int2(0, 0);
  wait_for_previous();
  const long long n0 = (long long)cnt->n_total;   // births of this pass land beyond
  const long long step = cnt->step;
  const int par = (int)(step & 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = win_cols(P.nr), ws = win_stride(cols);
  const int maxrows = min(kWinNodes / ws, P.nz);
  const int chunk = max(cnt->chunk, kBlock);      // chosen with the commit (no division here)
  if (mode != 1) {
    // The candidates go to the last blocks, kCandLanes per warp, two lanes each;
    // where there are fewer chunks than blocks, to the warps of all blocks that
    // would otherwise be idle, fewer per warp.  A block takes its chunks after
    // its candidates.
    const long long nq = (long long)cnt->n_cand[par ^ 1];
    const int *qin = queue + (long long)(par ^ 1) * P.cap;
    int lanes = kCandLanes;
    if (n0 <= (long long)chunk * (gridDim.x - 1)) {
      const unsigned idle = (gridDim.x - ((unsigned)n0 + chunk - 1) / chunk) * (kBlock / 32);
      lanes = (int)min(((unsigned)nq + idle - 1) / idle, (unsigned)kCandLanes);
    }
    unsigned lost = 0;
    if (lane < 2 * lanes)
      for (long long k = ((long long)(gridDim.x - 1 - blockIdx.x) * (kBlock / 32) + warp) * lanes + (lane >> 1); k < nq;
           k += (long long)gridDim.x * (kBlock / 32) * lanes)
        candidate32<MODE, true>(Pg, F, S, cnt, queue, qin[k], step, lane & 1, n0, lost);
    if (lost) atomicAdd(&cnt->lost, (unsigned long long)lost);
  }
  // thread 0 claims the block's next chunk (index and window rows) a chunk
  // ahead and has its state brought into L2 meanwhile
  long long next_ch = 0;
  int next_row0 = 0, next_rows = 0, next_col0 = 0;
  if (threadIdx.x == 0) {
    next_ch = (long long)atomicAdd(&cnt->chunk_next, 1ull);
    if (next_ch * chunk < n0) prefetch_chunk32(S, next_ch * chunk, min((next_ch + 1) * chunk, n0));
  }
  if (threadIdx.x == 0 && next_ch * chunk < n0)
    box32(P, S, next_ch * chunk, min((next_ch + 1) * chunk, n0), cols, maxrows, next_row0, next_rows, next_col0);
  for (;;) {
    if (threadIdx.x == 0) {
      chunk_at = next_ch;
      win_row0 = next_row0;
      win_rows = next_rows;
      if (WIDE) win_col0 = next_col0;
      box_cmax = -1;
    }
    __syncthreads();
    const long long ch = chunk_at;
    if (ch * chunk >= n0) break;
    // thread 0 claims the next chunk now; the claim's result is first used
    // after this chunk, so its round trip overlaps the chunk's work instead
    // of holding the block at the barrier above
    if (threadIdx.x == 0) next_ch = (long long)atomicAdd(&cnt->chunk_next, 1ull);
    // 32-bit slot indices: the capacity is below 2^31
    const int beg = (int)(ch * chunk), end = (int)min((long long)beg + chunk, n0);
    const Win32 w{win_rz, win_row0, win_rows, WIDE ? win_col0 : 0, WIDE ? cols : P.nr, ws};
    chunk32<MODE, WIDE>(P, S, F, cnt, queue, step, beg, end, w, &box_cmax);
    if (threadIdx.x == 0 && next_ch * chunk < n0) {
      prefetch_chunk32(S, next_ch * chunk, min((next_ch + 1) * chunk, n0));
      box32(P, S, next_ch * chunk, min((next_ch + 1) * chunk, n0), cols, maxrows, next_row0, next_rows, next_col0);
    }
    __syncthreads();
    flush32(P, w, box_cmax + 1);
    __syncthreads();
  }
  let_next_start();
}

// ------------------------------------------------------- batched FP32 pass
// One cell of a batch as the batched FP32 pass sees it (global memory): its
// parameters with the current buffer 0 / 1 as the deposit target, its two
// state buffers, counters, candidate queues and fields.
struct BatchCell32 {
  SimParams P[2];
  State32 S[2];
  SimCounters *cnt;
  int *queue;
  Fields<float> F[2];         // field buffers 0 / 1 (the pass into current buffer jb reads F[jb])
};

// The FP32 pass of one step for every cell of a batch in one launch: each
// block reads the cells' counters and forms the prefix sums of their
// collision candidates and chunks; the candidates of all cells go first, two
// lanes each, then the blocks take (cell, chunk) work items from one counter
// (*chunk_next, zeroed by the field kernel), copying the cell's parameters into
// shared memory when the cell changes.  Every cell gives what its own
// k_pass32 gives.
template <bool WIDE>
__global__ void __launch_bounds__(kBlock, 4) k_batch_pass32(const BatchCell32 *__restrict__ cells,
                                                            int ncell, int cur, int jb,
                                                            unsigned long long *chunk_next) {
  constexpr int mode = 0;        // a batch only takes whole steps
  __shared__ __align__(16) int win_rz[2 * kWinNodes];
  __shared__ int win_row0, win_rows, win_col0, box_cmax, cell_at;
  __shared__ long long chunk_at;
  __shared__ long long cand_pre[kMaxBatch + 1], chunk_pre[kMaxBatch + 1];
  __shared__ int cell_chunk[kMaxBatch];
  __shared__ unsigned long long total;
  __shared__ __align__(16) unsigned char sP_raw[sizeof(SimParams)];
  SimParams &sP = *reinterpret_cast<SimParams *>(sP_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kWinNodes; i += kBlock) reinterpret_cast<int2 *>(win_rz)[i] = make_int2(0, 0);
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  wait_for_previous();
  // per-cell candidates (of the previous pass) and chunks, then prefix sums
  for (int c = threadIdx.x; c < ncell; c += kBlock) {
    const SimCounters *cc = cells[c].cnt;
    const long long step = cc->step;
    cand_pre[c + 1] = mode != 1 ? (long long)cc->n_cand[(int)(step & 1) ^ 1] : 0;
    chunk_pre[c + 1] = (long long)cc->n_total;
    atomicAdd(&total, (unsigned long long)cc->n_total);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < ncell; c += kBlock) {
    const int fixed = cells[c].P[jb].chunk;
    const int chunk = fixed ? fixed : even_chunk((unsigned)min(total, 0x7FFFFFFFull), gridDim.x, kChunkMax);
    cell_chunk[c] = chunk;
    chunk_pre[c + 1] = ((unsigned)chunk_pre[c + 1] + chunk - 1) / chunk;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    cand_pre[0] = 0; chunk_pre[0] = 0;
    for (int c = 0; c < ncell; ++c) {
      cand_pre[c + 1] += cand_pre[c];
      chunk_pre[c + 1] += chunk_pre[c];
    }
  }
  __syncthreads();
  const long long nq = cand_pre[ncell], nchunk = chunk_pre[ncell];
  // (cell, chunk) work items; the block's first one is claimed (and its state
  // brought into L2) before the candidates
  long long next = 0;
  int next_c = -1, next_row0 = 0, next_rows = 0, next_col0 = 0;
  auto resolve = [&]() {         // thread 0: the cell and window rows of the claimed item
    if (next < nchunk) {
      next_c = cell_of_item(chunk_pre, ncell, next);
      const BatchCell32 &C = cells[next_c];
      const SimParams &Pc = C.P[jb];
      const int cols = win_cols(Pc.nr), maxrows = min(kWinNodes / win_stride(cols), Pc.nz);
      const long long n0c = (long long)C.cnt->n_total, chc = next - chunk_pre[next_c];
      const int chunk = cell_chunk[next_c];
      prefetch_chunk32(C.S[cur], chc * chunk, min((chc + 1) * chunk, n0c));
      box32(Pc, C.S[cur], chc * chunk, min((chc + 1) * chunk, n0c), cols, maxrows, next_row0, next_rows, next_col0);
    }
  };
  if (threadIdx.x == 0) {
    next = (long long)atomicAdd(chunk_next, 1ull);
    resolve();
    cell_at = -1;
  }
  // one candidate per two lanes (the chains of a warp share its instruction issue)
  for (long long k = (((long long)blockIdx.x * (kBlock / 32) + warp) * 32 + lane) >> 1; k < nq;
       k += (long long)gridDim.x * (kBlock / 2)) {
    const int c = cell_of_item(cand_pre, ncell, k);
    const BatchCell32 &C = cells[c];
    SimCounters *cc = C.cnt;
    const long long step = cc->step;
    const int *qin = C.queue + (long long)((int)(step & 1) ^ 1) * C.P[jb].cap;
    unsigned lost = 0;
    candidate32<mode, true>(&C.P[jb], C.F[jb], C.S[cur], cc, C.queue, qin[k - cand_pre[c]], step, lane & 1,
                            (long long)cc->n_total, lost);
    if (lost) atomicAdd(&cc->lost, (unsigned long long)lost);
  }
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      chunk_at = next;
      win_row0 = next_row0;
      win_rows = next_rows;
      win_col0 = next_col0;
      box_cmax = -1;
    }
    __syncthreads();
    const long long g = chunk_at;
    if (g >= nchunk) break;
    const int c = cell_of_item(chunk_pre, ncell, g);
    if (c != cell_at) {          // this block's first chunk of cell c: its parameters
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&cells[c].P[jb]);
      uint32_t *dst = reinterpret_cast<uint32_t *>(sP_raw);
      for (int i = threadIdx.x; i < (int)(sizeof(SimParams) / 4); i += kBlock) dst[i] = src[i];
      __syncthreads();
      if (threadIdx.x == 0) cell_at = c;
    }
    // the next item is claimed now and resolved after this one, so the
    // claim's round trip and the loads it leads to overlap the chunk's work
    if (threadIdx.x == 0 && next < nchunk) next = (long long)atomicAdd(chunk_next, 1ull);
    const BatchCell32 &C = cells[c];
    SimCounters *cc = C.cnt;
    const long long n0 = (long long)cc->n_total, step = cc->step;
    const int chunk = cell_chunk[c];
    const long long ch = g - chunk_pre[c];
    const int beg = (int)(ch * chunk), end = (int)min((long long)beg + chunk, n0);
    const int cols = WIDE ? win_cols(sP.nr) : sP.nr;
    const Win32 w{win_rz, win_row0, win_rows, WIDE ? win_col0 : 0, cols, win_stride(cols)};
    chunk32<0, WIDE>(sP, C.S[cur], C.F[jb], cc, C.queue, step, beg, end, w, &box_cmax);
    if (threadIdx.x == 0) resolve();
    __syncthreads();
    flush32(sP, w, box_cmax + 1);
  }
  let_next_start();
}

// The collisions still queued by the last FP32 pass, without the next push
// (before an observation of the state): MCC at the end of that step and the
// secondaries' birth; the pending flags are cleared.
__global__ void __launch_bounds__(kMccBlock) k_collide32(const SimParams *__restrict__ Pg,
                                                         State32 S, Fields<float> F,
                                                         SimCounters *cnt, int *queue) {
  const SimParams &P = *Pg;
  const long long n0 = (long long)cnt->n_total;
  const long long step = cnt->step;
  const int par = (int)(step & 1);
  const long long nq = (long long)cnt->n_cand[par];
  const int *qu = queue + (long long)par * P.cap;
  unsigned lost = 0;              // (no push here: nothing reaches the wall)
  for (long long k = (blockIdx.x * (long long)kMccBlock + threadIdx.x) >> 1; k < nq;
       k += (long long)gridDim.x * (kMccBlock / 2))
    candidate32<0, false>(Pg, F, S, cnt, queue, qu[k], step, threadIdx.x & 1, n0, lost);
}

// k_collide32 for every cell of a batch in one launch (before the batch's
// sort): the cells' queued collisions in one range by prefix sums, two lanes
// each; each cell's are those its own k_collide32 would apply.
__global__ void __launch_bounds__(kMccBlock) k_batch_collide32(const BatchCell32 *__restrict__ cells,
                                                               int ncell, int cur) {
  __shared__ long long pre[kMaxBatch + 1];
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
    const SimCounters *cc = cells[c].cnt;
    pre[c + 1] = (long long)cc->n_cand[(int)(cc->step & 1)];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    pre[0] = 0;
    for (int c = 0; c < ncell; ++c) pre[c + 1] += pre[c];
  }
  __syncthreads();
  const long long nq = pre[ncell];
  for (long long k = (blockIdx.x * (long long)kMccBlock + threadIdx.x) >> 1; k < nq;
       k += (long long)gridDim.x * (kMccBlock / 2)) {
    const int c = cell_of_item(pre, ncell, k);
    const BatchCell32 &C = cells[c];
    SimCounters *cc = C.cnt;
    const long long step = cc->step;
    const int *qu = C.queue + (long long)(int)(step & 1) * C.P[0].cap;
    unsigned lost = 0;
    candidate32<0, false>(&C.P[0], C.F[0], C.S[cur], cc, C.queue, qu[k - pre[c]], step, threadIdx.x & 1,
                          (long long)cc->n_total, lost);
  }
}

// every cell's collision queue of parity q (q < 0: both) emptied, after its
// collisions ran
template <typename Cell>
__global__ void k_batch_clear_cand(const Cell *__restrict__ cells, int ncell, int q) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
    if (q != 1) cells[c].cnt->n_cand[0] = 0;
    if (q != 0) cells[c].cnt->n_cand[1] = 0;
  }
}

// ------------------------------------------------------------- FDTD
// FP32 form (cnt given): commit the previous pass and open step s - the
// births of the last pass join the slots, the queue that pass consumed is
// emptied, the chunk counter rewinds; no other kernel runs meanwhile
__device__ __forceinline__ void commit_pass32(SimCounters *cnt) {
  const long long ns = cnt->step + 1;
  const unsigned long long nt = cnt->n_total + cnt->n_births;
  cnt->n_total = nt < cnt->cap ? nt : cnt->cap;
  cnt->n_births = 0;
  cnt->n_cand[ns & 1] = 0;
  cnt->chunk_next = 0;
  cnt->chunk = cnt->chunk_fixed ? cnt->chunk_fixed : even_chunk((unsigned)cnt->n_total, (unsigned)cnt->pass_blocks, kChunkMax);
  cnt->step = ns;
}

// the same before a pass that no field update precedes (sim_prime)
__global__ void k_commit32(SimCounters *cnt) { commit_pass32(cnt); }

// The field sub-cycle of one step for fdtd_ratio 1: one block per patch of
// shape K (fdtd_tma.cuh).
template <typename T, int K>
__global__ void __launch_bounds__(32 * tma_warps(K), tma_blocks(K)) k_sim_fdtd_tma(
    const __grid_constant__ FdtdInst I, SimCounters *cnt) {
  wait_for_previous();
  if (cnt && blockIdx.x == 0 && threadIdx.x == 0) commit_pass32(cnt);
  fdtd_block_body<T, K>(FdtdWork{&I, nullptr, I.ntiles});
  let_next_start();
}

// The field update of every cell of a batch in one launch: the blocks walk a
// table of (cell, tile) work items; FP32 form (commit given): they first
// commit the previous pass of every cell.
template <typename T, int K>
__global__ void __launch_bounds__(32 * tma_warps(K), tma_blocks(K)) k_batch_fdtd_tma(
    const FdtdInst *insts, const int2 *table, int nitems, SimCounters *const *commit, int ninst,
    unsigned long long *chunk_next) {
  wait_for_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) *chunk_next = 0;        // the pass's, which runs next
  if (commit && threadIdx.x == 0)
    for (int i = blockIdx.x; i < ninst; i += gridDim.x) commit_pass32(commit[i]);
  fdtd_block_body<T, K>(FdtdWork{insts, table, nitems});
  let_next_start();
}

using SimFdtdTmaFn = void (*)(const FdtdInst, SimCounters *);
using BatchFdtdTmaFn = void (*)(const FdtdInst *, const int2 *, int, SimCounters *const *, int, unsigned long long *);

// the instance of each kernel, and its dynamic shared memory, for knob value `rows`
template <typename T>
SimFdtdTmaFn sim_fdtd_tma_fn(int rows) {
  return rows == 12 ? k_sim_fdtd_tma<T, 12> : rows == 20 ? k_sim_fdtd_tma<T, 20> : k_sim_fdtd_tma<T, 16>;
}
template <typename T>
BatchFdtdTmaFn batch_fdtd_tma_fn(int rows) {
  return rows == 12 ? k_batch_fdtd_tma<T, 12> : rows == 20 ? k_batch_fdtd_tma<T, 20> : k_batch_fdtd_tma<T, 16>;
}
template <typename T>
size_t tma_block_bytes(int rows) {
  return rows == 12 ? TmaStage<T, tma_rows(12)>::block_bytes
                    : rows == 20 ? TmaStage<T, tma_rows(20)>::block_bytes : TmaStage<T, tma_rows(16)>::block_bytes;
}

// The general sub-cycle (fdtd_ratio > 1): one 32 x 32 patch per block
// (fdtd_tiled), from the fields `in` to the fields `out`.
template <typename T>
__global__ void __launch_bounds__(32 * kFdtdRows, 3) k_sim_fdtd(Fields<T> in, Fields<T> out,
                                                  const unsigned long long *Jr,
                                                  const unsigned long long *Jz,
                                                  unsigned long long *Jr_next,
                                                  unsigned long long *Jz_next, int nr, int nz,
                                                  int ldf, int ldj, FdtdCoef c, const double *invV, double mu,
                                                  double dt, int R, unsigned flags,
                                                  SimCounters *cnt, ExtraCurrent ion,
                                                  FieldQuads quads) {
  wait_for_previous();
  if (cnt && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0)
    commit_pass32(cnt);
  fdtd_tiled<T>(in.Er, in.Ez, in.H, out.Er, out.Ez, out.H, Jr, Jz, Jr_next, Jz_next, nr, nz, ldf, ldj,
                c, invV, mu, dt, R, flags, ion, quads);
  let_next_start();
}

// ---------------------------------------------------------- load/read

// one particle in SI (r, z [m], u = gamma v [m/s]) into the FP32 state; mark:
// the pushed-parity flag (the opposite of the parity of the pass that will
// push it first)
__device__ __forceinline__ void store32(State32 S, long long p, double r, double z, double ur,
                                        double ut, double uz, uint64_t id, int nr, int nz,
                                        double dr, double dz, double c, int mark) {
  const double R = r / dr, Z = z / dz;
  int ir = (int)floor(R), iz = (int)floor(Z);
  float fr = (float)(R - ir), fz = (float)(Z - iz);
  if (fr >= 1.f) { fr = 0.f; ir++; }
  if (fz >= 1.f) { fz = 0.f; iz++; }
  if (iz >= nz) { iz = nz - 1; fz = 0.99999994f; }
  const bool alive = r >= 0 && ir < nr && iz >= 0;
  S.a[p] = pack32(ir, iz, fr, fz, (float)(ur / c), alive, false, mark);
  S.b[p] = make_float2((float)(ut / c), (float)(uz / c));
  S.id[p] = id;
}

__device__ __forceinline__ void store64(State64 S, long long p, double r, double z, double ur,
                                        double ut, double uz, uint64_t id) {
  S.rz[p] = make_double2(r, z);
  S.urt[p] = make_double2(ur, ut);
  S.uz[p] = uz;
  S.id[p] = id;
}

__global__ void k_load64(State64 S, const double *r, const double *z, const double *ur,
                         const double *ut, const double *uz, const uint64_t *id, long long n) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x)
    store64(S, p, r[p], z[p], ur[p], ut[p], uz[p], id[p]);
}

__global__ void k_load32(State32 S, const double *r, const double *z, const double *ur,
                         const double *ut, const double *uz, const uint64_t *id, long long n,
                         int nr, int nz, double dr, double dz, double c, int mark) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x)
    store32(S, p, r[p], z[p], ur[p], ut[p], uz[p], id[p], nr, nz, dr, dz, c, mark);
}

// ------------------------------------------------------------ births
// Photoionization births on the device: per photon a photoelectron (photon
// energy minus the N K-shell binding, 410 eV as EB_14.csv's 409.9; direction
// density ~ (d . x)^2 about the polarisation x) and an isotropic 360 eV Auger
// electron, both at a Rayleigh(sigma_r) radius (inside the wall), uniform
// azimuth and uniform z; the state keeps the local (r, theta, z) frame of that
// azimuth.  The reference draws its births on the host (INCIDENCE1.m:51-158,
// with a Sauter photoelectron and a 383 eV Auger line); these are the
// workload's laws.  Draws: Philox keyed on (seed, photon index) with the
// reserved step word kBirthStream, apart from every simulation draw.
constexpr long long kBirthStream = -2;
constexpr double kKShellEv = 410.0, kAugerEv = 360.0;

template <int FORM>
__global__ void k_birth_photo(State64 S64, State32 S32, long long n_photo, double u_pe,
                              double u_au, double sigma_r, double r_max, double Lp,
                              uint64_t seed, uint64_t id_base, int nr, int nz, double dr,
                              double dz, double c) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n_photo;
       k += (long long)gridDim.x * blockDim.x) {
    const U2 d0 = draw2(seed, (uint64_t)k, kBirthStream, 0), d1 = draw2(seed, (uint64_t)k, kBirthStream, 1);
    const U2 d2 = draw2(seed, (uint64_t)k, kBirthStream, 2), d3 = draw2(seed, (uint64_t)k, kBirthStream, 3);
    const double r = fmin(sigma_r * sqrt(-2.0 * log1p(-d0.a)), r_max);
    const double z = d0.b * Lp;
    double sp, cp;
    sincos(2 * GASATT_PI * d1.a, &sp, &cp);                // azimuth of the birth point
    // photoelectron: mu = cos(angle to x), p(mu) ~ mu^2 -> mu = cbrt(2U - 1)
    const double mu = cbrt(2 * d1.b - 1), s = sqrt(fmax(0.0, 1 - mu * mu));
    double sps, cps;
    sincos(2 * GASATT_PI * d2.a, &sps, &cps);
    const double px = mu, py = s * cps, pz = s * sps;
    // Auger: isotropic
    const double ct = 2 * d2.b - 1, st = sqrt(fmax(0.0, 1 - ct * ct));
    double spa, cpa;
    sincos(2 * GASATT_PI * d3.a, &spa, &cpa);
    const double ax = st * cpa, ay = st * spa, az = ct;
    const double pr = u_pe * (px * cp + py * sp), pt = u_pe * (-px * sp + py * cp), pzz = u_pe * pz;
    const double ar = u_au * (ax * cp + ay * sp), at = u_au * (-ax * sp + ay * cp), azz = u_au * az;
    const long long p = 2 * k;
    if (FORM == 0) {
      store64(S64, p, r, z, pr, pt, pzz, id_base + (uint64_t)p);
      store64(S64, p + 1, r, z, ar, at, azz, id_base + (uint64_t)p + 1);
    } else {
      store32(S32, p, r, z, pr, pt, pzz, id_base + (uint64_t)p, nr, nz, dr, dz, c, 0);
      store32(S32, p + 1, r, z, ar, at, azz, id_base + (uint64_t)p + 1, nr, nz, dr, dz, c, 0);
    }
  }
}

__global__ void k_read64(State64 S, double *r, double *z, double *ur, double *ut, double *uz,
                         uint64_t *id, long long n) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    const double2 a = S.rz[p], b = S.urt[p];
    r[p] = a.x; z[p] = a.y; ur[p] = b.x; ut[p] = b.y; uz[p] = S.uz[p];
    id[p] = S.id[p];
  }
}

__global__ void k_read32(State32 S, double *r, double *z, double *ur, double *ut, double *uz,
                         uint64_t *id, long long n, double dr, double dz, double c) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    const uint4 A = S.a[p];
    const float2 B = S.b[p];
    if (A.x == kDead) { r[p] = -1.0; z[p] = 0; }
    else {
      r[p] = ((double)(A.x & 0xFFFFu) + (double)__uint_as_float(A.y & ~kSign)) * dr;
      z[p] = ((double)(A.x >> 16) + (double)__uint_as_float(A.z & ~kSign)) * dz;
    }
    ur[p] = (double)__uint_as_float(A.w) * c; ut[p] = (double)B.x * c; uz[p] = (double)B.y * c;
    id[p] = S.id[p];
  }
}

// ---------------------------------------------------------------- sort
// Counting sort by cell (z-major), dropping dead slots.  Order inside a cell
// is arbitrary; nothing downstream depends on it (random streams are keyed
// on particle ids and the deposit is an exact integer sum).
// sort key: the deposit node quad (ar, az) = cell shifted by half a cell, so
// that lanes of a warp share their four deposit nodes right after a sort;
// (nr + 1) x (nz + 1) bins
__device__ __forceinline__ int cell_of64(const State64 &S, long long p, int nr, int nz,
                                         double dr, double dz) {
  const double2 rz = S.rz[p];
  if (rz.x < 0) return -1;
  int ar = (int)floor(rz.x / dr - 0.5) + 1, az = (int)floor(rz.y / dz - 0.5) + 1;
  ar = min(max(ar, 0), nr);
  az = min(max(az, 0), nz);
  return ar + az * (nr + 1);
}
__device__ __forceinline__ int cell_of32(const State32 &S, long long p, int nr) {
  const uint4 A = S.a[p];
  if (A.x == kDead) return -1;
  const int ar = (int)(A.x & 0xFFFFu) + (__uint_as_float(A.y & ~kSign) >= 0.5f ? 1 : 0);
  const int az = (int)(A.x >> 16) + (__uint_as_float(A.z & ~kSign) >= 0.5f ? 1 : 0);
  return ar + az * (nr + 1);
}

// Runs of equal keys among the lanes of a warp (the particles are nearly in
// key order, so a warp holds few runs): a lane heads a run when its key
// differs from the lane below's; dead lanes (key -1) end runs.  For each lane:
// its run's head lane h and, at the head, the run's length.
__device__ __forceinline__ void key_runs(int c, int lane, int &h, int &len) {
  const int below = __shfl_up_sync(0xFFFFFFFFu, c, 1);
  const bool head = c >= 0 && (lane == 0 || below != c);
  const unsigned heads = __ballot_sync(0xFFFFFFFFu, head);
  const unsigned ends = __ballot_sync(0xFFFFFFFFu, head || c < 0);
  const unsigned up = lane == 31 ? 0u : ends & (0xFFFFFFFFu << (lane + 1));
  len = (up ? __ffs(up) - 1 : 32) - lane;
  const unsigned le = heads & (lane == 31 ? 0xFFFFFFFFu : ((2u << lane) - 1));
  h = le ? 31 - __clz(le) : lane;
}

// Each warp takes segments of kSortSeg particles (kSortSeg / 32 per lane,
// consecutive groups of 32), loading all of a segment's keys before using
// them, so that several loads per thread are in flight.
constexpr int kSortSeg = 128;

template <int FORM>
__global__ void k_sort_hist(State64 S64, State32 S32, const SimCounters *cnt, int nr, int nz,
                            double dr, double dz, int *count) {
  constexpr int G = kSortSeg / 32;
  const long long n0 = slots_in_use(cnt);
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long seg = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
       seg * kSortSeg < n0; seg += warps) {
    int c[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const long long p = seg * kSortSeg + g * 32 + lane;
      c[g] = -1;
      if (p < n0) c[g] = FORM == 0 ? cell_of64(S64, p, nr, nz, dr, dz) : cell_of32(S32, p, nr);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      int h, len;
      key_runs(c[g], lane, h, len);
      if (c[g] >= 0 && h == lane) atomicAdd(count + c[g], len);
    }
  }
}

template <int FORM>
__global__ void k_sort_scatter(State64 A64, State64 B64, State32 A32, State32 B32,
                               SimCounters *cnt, int nr, int nz, double dr, double dz,
                               const int *offset, int *cursor) {
  constexpr int G = kSortSeg / 32;
  const long long n0 = slots_in_use(cnt);
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long seg = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
       seg * kSortSeg < n0; seg += warps) {
    int c[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const long long p = seg * kSortSeg + g * 32 + lane;
      c[g] = -1;
      if (p < n0) c[g] = FORM == 0 ? cell_of64(A64, p, nr, nz, dr, dz) : cell_of32(A32, p, nr);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const long long p = seg * kSortSeg + g * 32 + lane;
      int h, len;
      key_runs(c[g], lane, h, len);
      // the head claims its run's slots in the bin and hands the first one out
      long long first = 0;
      if (c[g] >= 0 && h == lane) first = (long long)offset[c[g]] + atomicAdd(cursor + c[g], len);
      first = __shfl_sync(0xFFFFFFFFu, first, h);
      if (c[g] < 0) continue;
      const long long dst = first + (lane - h);
      if (FORM == 0) {
        B64.rz[dst] = A64.rz[p]; B64.urt[dst] = A64.urt[p]; B64.uz[dst] = A64.uz[p];
        B64.id[dst] = A64.id[p];
      } else {
        B32.a[dst] = A32.a[p]; B32.b[dst] = A32.b[p]; B32.id[dst] = A32.id[p];
      }
    }
  }
}

// ------------------------------------------------------------ scan
// Exclusive prefix sum of n ints in one pass (decoupled look-back): each
// block takes a tile of kScanTile counts by ticket, so a tile's predecessors
// are always running or done; it publishes its tile total (flag 1), looks
// back over the predecessors' published totals until it meets an inclusive
// prefix (flag 2), publishes its own inclusive prefix and writes its tile.
// The look-back reads 32 predecessors at a time, one per lane of a warp.
// A published word is (flag << 62) | value, written in one 64-bit store.
// The look-back wait on a tile that has published nothing yet is bounded;
// past the bound the scan sets *err and takes 0 for the tiles it waited on.
constexpr int kScanThreads = 256, kScanItems = 16, kScanTile = kScanThreads * kScanItems;
constexpr unsigned kScanWaitLimit = 1u << 24;

struct ScanState {
  unsigned long long *tile;   // ceil(n / kScanTile) published words, zeroed before each scan
  unsigned *ticket;           // tile ticket, zeroed before each scan
  unsigned *err;
};

__device__ __forceinline__ unsigned long long ld_volatile_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan(const int *in, int *out, int n, ScanState S) {
  __shared__ int warp_sum[kScanThreads / 32];
  __shared__ unsigned tile_s;
  __shared__ long long excl_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) tile_s = atomicAdd(S.ticket, 1u);
  __syncthreads();
  const unsigned t = tile_s;
  const long long base = (long long)t * kScanTile + (long long)threadIdx.x * kScanItems;
  int v[kScanItems];
  int sum = 0;
  if (base + kScanItems <= n) {            // whole: four 16-byte loads (base is a multiple of 16)
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4) {
      const int4 q = *reinterpret_cast<const int4 *>(in + base + k);
      v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0;
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) sum += v[k];
  // block scan of the thread sums
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int wbase = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    wbase += w < warp ? warp_sum[w] : 0;
    total += warp_sum[w];
  }
  if (warp == 0) {
    // warp-parallel look-back: lane i reads the word of tile p - i; the
    // aggregates up to the nearest inclusive prefix are summed in one go
    constexpr unsigned long long kVal = (1ull << 62) - 1;
    long long excl = 0;
    if (t == 0) {
      if (lane == 0) atomicExch(S.tile, (2ull << 62) | (unsigned long long)total);
    } else {
      if (lane == 0) atomicExch(S.tile + t, (1ull << 62) | (unsigned long long)total);
      bool failed = false;
      for (long long p = (long long)t - 1; p >= 0; p -= 32) {
        const long long q = p - lane;
        // before tile 0: an inclusive prefix of 0
        unsigned long long w = q >= 0 ? ld_volatile_u64(S.tile + q) : (2ull << 62);
        unsigned it = 0;
        while (__any_sync(0xFFFFFFFFu, (w >> 62) == 0) && ++it < kScanWaitLimit)
          if ((w >> 62) == 0) w = ld_volatile_u64(S.tile + q);
        if (__any_sync(0xFFFFFFFFu, (w >> 62) == 0)) { failed = true; break; }
        const unsigned inc = __ballot_sync(0xFFFFFFFFu, (w >> 62) == 2);
        const int stop = inc ? __ffs(inc) - 1 : 31;
        long long v = lane <= stop ? (long long)(w & kVal) : 0;
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
        excl += v;
        if (inc) break;
      }
      if (lane == 0) {
        if (failed) atomicOr(S.err, 1u);
        atomicExch(S.tile + t, (2ull << 62) | (unsigned long long)(excl + total));
      }
    }
    if (lane == 0) excl_s = excl;
  }
  __syncthreads();
  int run = (int)excl_s + wbase + incl - sum;
  if (base + kScanItems <= n) {
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4) {
      int4 o;
      o.x = run; run += v[k];
      o.y = run; run += v[k + 1];
      o.z = run; run += v[k + 2];
      o.w = run; run += v[k + 3];
      *reinterpret_cast<int4 *>(out + base + k) = o;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < n) out[base + k] = run;
      run += v[k];
    }
  }
}

__global__ void k_sort_finish(SimCounters *cnt, const int *offset, int ncell) {
  cnt->n_total = (unsigned long long)offset[ncell];
  cnt->n_births = 0;
  cnt->sorted_total = cnt->n_total;
}

// ---------------------------------------------------------- diagnostics
template <int FORM>
__global__ void k_diag(State64 S64, State32 S32, SimCounters *cnt, double c, double me,
                       double qe) {
  const long long n0 = slots_in_use(cnt);
  unsigned long long kin = 0, alive = 0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n0;
       p += (long long)gridDim.x * blockDim.x) {
    double u2;
    if (FORM == 0) {
      if (S64.rz[p].x < 0) continue;
      const double2 a = S64.urt[p];
      const double w = S64.uz[p];
      u2 = (a.x * a.x + a.y * a.y + w * w) / (c * c);
    } else {
      const uint4 A = S32.a[p];
      if (A.x == kDead) continue;
      const float2 B = S32.b[p];
      const double a = __uint_as_float(A.w), b = B.x, d = B.y;
      u2 = a * a + b * b + d * d;
    }
    const double g = sqrt(1 + u2);
    const double Eev = me * c * c * (u2 / (g + 1)) / qe;
    kin += (unsigned long long)__double2ll_rn(Eev * 65536.0);
    alive++;
  }
  for (int o = 16; o; o >>= 1) {
    kin += __shfl_down_sync(0xFFFFFFFFu, kin, o);
    alive += __shfl_down_sync(0xFFFFFFFFu, alive, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&cnt->kin_fx, kin);
    atomicAdd(&cnt->alive, alive);
  }
}

// trapezoid-weighted field energy (electricmagneticfield6.m:153-154),
// per-block partial sums in a fixed order
template <typename T>
__global__ void k_field_energy(const T *Er, const T *Ez, const T *H, int nr, int nz, int ld,
                               double dr, double dz, double *partial) {
  __shared__ double sh[kBlock];
  const int64_t nE = (int64_t)nr * (nz + 1), nZ = (int64_t)(nr + 1) * nz, nH = (int64_t)nr * nz;
  double acc[3] = {0, 0, 0};
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < nE + nZ + nH;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int f, ncol, nrow;
    int64_t k;
    double r0;
    const T *A;
    if (idx < nE) { f = 0; k = idx; ncol = nr; nrow = nz + 1; r0 = dr / 2; A = Er; }
    else if (idx < nE + nZ) { f = 0; k = idx - nE; ncol = nr + 1; nrow = nz; r0 = 0; A = Ez; }
    else { f = 1; k = idx - nE - nZ; ncol = nr; nrow = nz; r0 = dr / 2; A = H; }
    const int i = (int)(k % ncol), j = (int)(k / ncol);
    const double wi = (i == 0 || i == ncol - 1) ? 0.5 : 1.0;
    const double wj = (j == 0 || j == nrow - 1) ? 0.5 : 1.0;
    const double v = (double)A[i + (int64_t)j * ld];
    acc[f] += wi * wj * v * v * (r0 + i * dr) * dr * dz;
  }
  for (int f = 0; f < 2; ++f) {
    sh[threadIdx.x] = acc[f];
    __syncthreads();
    for (int s = kBlock / 2; s; s >>= 1) {
      if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x * 2 + f] = sh[0];
    __syncthreads();
  }
}

}  // namespace

// Steps that one graph launch takes where no sort, ion push or odd start falls
// between them.  A graph of one step each leaves the GPU idle for a launch's
// time between steps: 2 to 3 us of every step (64 x 256 cells FP64 16.8 us a step
// with graphs of one step, 14.1 with ten; 2M electrons FP32 55.2 and 53.1).  Ten
// divides the usual sort periods.
constexpr int kGraphSteps = 10;

// ================================================================ sim object
struct gasatt_sim {
  gasatt_ctx *ctx = nullptr;
  gasatt_sim_config cfg{};
  SimTables tabs;
  SimParams P{};
  int form = 0;
  // state (double-buffered for the sort)
  State64 s64[2]{};
  State32 s32[2]{};
  int cur = 0;
  // fields, double-buffered: the step of parity q reads buffer q and writes
  // buffer 1 - q (the field update keeps patches of the old fields while
  // others are written), so the fields of the current time are in buffer
  // host_step & 1
  void *Er[2] = {nullptr, nullptr}, *Ez[2] = {nullptr, nullptr}, *H[2] = {nullptr, nullptr};
  // field update of fdtd_ratio 1: the cell's descriptor for the steps of
  // parity 0 / 1 (tensor maps of the fields and current read, write-back
  // targets, tiles), the patch rows, the grid and its shared memory
  FdtdInst fdtd_inst[2];
  int tma_rows = 0;
  unsigned tma_grid = 0;
  size_t tma_smem = 0;
  // Internal grid layout: column-major like the reference's arrays, with row
  // strides padded so that every row starts on a 16-byte boundary (the field
  // update stages its tiles with TMA).  Er(i, j) at i + j ldf (j <= n_z),
  // Ez(i, j) at i + j ldf (i <= n_r), H(i, j) at i + j ldf; currents
  // J(i, j) at i + j ldj.  The padding stays zero.
  int ldf = 0, ldj = 0;
  // current accumulators, double-buffered: the field update of step s reads
  // buffer s & 1 and clears the other one, which the pass of step s fills
  unsigned long long *Jr[2] = {nullptr, nullptr}, *Jz[2] = {nullptr, nullptr};
  double *d_tab = nullptr;
  double *invV = nullptr;         // per column: 2^-S / shell volume
  double *fdtd_colc = nullptr;    // per column: {invV, Ez coefficients} (fdtd_column_table)
  SimCounters *cnt = nullptr;
  SimCounters *h_cnt = nullptr;   // pinned
  int *cell_count = nullptr, *cell_offset = nullptr, *cell_cursor = nullptr;
  // the sort's scan: one published word per tile of counts, then the tile ticket
  unsigned long long *scan_tiles = nullptr;
  int scan_ntiles_max = 0;
  double *partial = nullptr;
  int partial_blocks = 0;
  std::vector<void *> allocs;
  bool primed = false;
  int64_t host_step = 0;          // particle passes completed
  int64_t since_sort = 0;
  cudaGraphExec_t g_step[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [state buffer][step parity]
  cudaGraph_t gr_step[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};     // the same, not instantiated
  cudaGraphExec_t g_steps[2] = {nullptr, nullptr};   // kGraphSteps steps from parity 0 on [state buffer]
  cudaGraph_t gr_steps[2] = {nullptr, nullptr};      // the same, not instantiated
  cudaGraphExec_t g_sort[2] = {nullptr, nullptr};
  cudaGraph_t gr_sort[2] = {nullptr, nullptr};       // the same, not instantiated
  double scale = 1.0;
  unsigned pass_grid = 0, mcc_grid = 0;
  int *queue = nullptr;           // collision candidates, two queues of capacity slots
  SimParams *d_P = nullptr;       // device copies of P with the current of buffer 0 / 1
  double *d_gas = nullptr;        // per-cell gas density (gasatt_sim_set_gas_density)
  double *d_ion_sig = nullptr;    // per-cell newborn-ion spread (gasatt_sim_set_gas_temperature)
  // ions (cfg.ion_capacity > 0): the store lives in P.ion; the ion current,
  // deposited by each ion push and held until the next, in fixed point with
  // the factor ion_scale (2^48 per q_e FN c, in both forms)
  unsigned long long *Jir = nullptr, *Jiz = nullptr;
  double ion_scale = 1.0;
  IonState ion_tmp{};             // scratch store the ions are sorted into before a push
  FieldQuads quads{};             // FP32 form: gather quads, written with the fields
  bool mcc_pending = false;       // the last pass's collisions are not applied yet
  bool batch_pass = false;        // FP64: the last pass was a batch's (clear_after_batch)
  bool uncommitted = false;       // FP32: gasatt_sim_run_host's last pass, which no field update has committed
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;   // graph capture fork/join
  bool timing = false;
  // field update start/end, particle pass start/end, collision kernel start/end
  cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
};

namespace {

template <typename T>
int sim_alloc(gasatt_sim *s, T **p, size_t n) {
  cudaError_t e = cudaMalloc((void **)p, (n ? n : 1) * sizeof(T));
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "cudaMalloc");
  s->allocs.push_back((void *)*p);
  return GASATT_OK;
}

#define SIM_TRY(x) do { int rc__ = (x); if (rc__) return rc__; } while (0)

// bytes of one current grid (n_z rows of ldj 64-bit counters)
size_t jbytes(const gasatt_sim *s) { return (size_t)s->ldj * s->cfg.n_z * 8; }

FdtdCoef fdtd_coef(const gasatt_sim *s) {
  const auto &c = s->cfg;
  const double dt = c.dt / c.fdtd_ratio, eps = c.eps0;
  FdtdCoef fc;
  fc.dr = c.dr; fc.dz = c.dz; fc.PHIp = c.PHIp; fc.inv_scale = 1.0 / s->scale;
  fc.dt_eps = (dt / 2) / eps;
  fc.dt_eps_dz = (dt / 2) / (eps * c.dz);
  fc.axis = 4 * (dt / 2) / (eps * c.dr);
  fc.chr = fc.chz = 0;
  return fc;
}

// field sub-cycle of step with parity q: reads current buffer q, clears 1 - q
// field buffer k as the kernels take it
template <typename T>
Fields<T> fields_of(const gasatt_sim *s, int k) {
  return Fields<T>{(T *)s->Er[k], (T *)s->Ez[k], (T *)s->H[k]};
}
// the field buffer that holds the fields of the current time
inline int fcur(const gasatt_sim *s) { return (int)(s->host_step & 1); }

// field update of a step of parity q: reads field buffer q and current
// buffer q, writes field buffer 1 - q and clears current buffer 1 - q
int launch_fdtd(gasatt_sim *s, cudaStream_t st, int q, bool early = false) {
  const auto &c = s->cfg;
  const int nr = c.n_r, nz = c.n_z, R = c.fdtd_ratio;
  const FdtdCoef fc = fdtd_coef(s);
  const double dt = c.dt / R;
  // the held ion current, in the electron current's fixed-point units
  const ExtraCurrent ion{s->Jir, s->Jiz, s->scale / s->ion_scale};
  if (R == 1) {
    const dim3 block(32 * tma_warps(s->tma_rows));
    const cudaError_t e =
        launch_early(early, s->form == 0 ? sim_fdtd_tma_fn<double>(s->tma_rows) : sim_fdtd_tma_fn<float>(s->tma_rows),
                     dim3(s->tma_grid), block, s->tma_smem, st, s->fdtd_inst[q], s->form == 0 ? nullptr : s->cnt);
    s->ctx->launches++;
    if (e != cudaSuccess) return cuda_fail(s->ctx, e, "fdtd launch");
    return GASATT_OK;
  }
  const int tile = fdtd_tile(R);
  const dim3 grid((nr + 1 + tile - 1) / tile, (nz + 1 + tile - 1) / tile);
  const dim3 block(32, kFdtdRows);
  cudaError_t e;
  if (s->form == 0)
    e = launch_early(early, k_sim_fdtd<double>, grid, block, 0, st, fields_of<double>(s, q), fields_of<double>(s, 1 - q),
                     s->Jr[q], s->Jz[q], s->Jr[1 - q], s->Jz[1 - q], nr, nz, s->ldf, s->ldj, fc, s->invV, c.mu0, dt, R,
                     c.flags, nullptr, ion, FieldQuads{});
  else
    e = launch_early(early, k_sim_fdtd<float>, grid, block, 0, st, fields_of<float>(s, q), fields_of<float>(s, 1 - q),
                     s->Jr[q], s->Jz[q], s->Jr[1 - q], s->Jz[1 - q], nr, nz, s->ldf, s->ldj, fc, s->invV, c.mu0, dt, R,
                     c.flags, s->cnt, ion, s->quads);
  s->ctx->launches++;
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "fdtd launch");
  return GASATT_OK;
}

// particle pass; its collision candidates (mode 0) go to queue q, its
// current to buffer jb; it gathers from field buffer fb
int launch_pass(gasatt_sim *s, cudaStream_t st, int mode, int jb, int q, int fb, bool early = false) {
  SimParams P = s->P;
  P.Jr = s->Jr[jb];
  P.Jz = s->Jz[jb];
  const int b = s->cur;
  cudaError_t e;
  if (s->form == 0) {
    auto kern = mode == 0 ? k_pass64<0> : mode == 1 ? k_pass64<1> : k_pass64<2>;
    // (never early: two kernels are before it)
    e = launch_early(false, kern, dim3(s->pass_grid), dim3(kBlock), kWin64Bytes, st, P, s->s64[b],
                     fields_of<double>(s, fb), s->cnt, s->queue, q);
  } else {
    auto kern = win_cols(P.nr) < P.nr
                    ? (mode == 0 ? k_pass32<0, true> : mode == 1 ? k_pass32<1, true> : k_pass32<2, true>)
                    : (mode == 0 ? k_pass32<0, false> : mode == 1 ? k_pass32<1, false> : k_pass32<2, false>);
    e = launch_early(early, kern, dim3(s->pass_grid), dim3(kBlock), 0, st, P, s->s32[b], fields_of<float>(s, fb),
                     s->cnt, s->queue, s->d_P + jb);
  }
  s->ctx->launches++;
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "particle pass launch");
  return GASATT_OK;
}

// FP64: before a pass of a cell on its own that follows a batch's (of parity q)
int clear_after_batch(gasatt_sim *s, cudaStream_t st, int q) {
  if (s->form != 0 || !s->batch_pass) return GASATT_OK;
  s->batch_pass = false;
  k_clear_next_queue<<<1, 1, 0, st>>>(s->cnt, q);
  s->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "queue clear launch");
  return GASATT_OK;
}

// the collisions queued (parity q) by the last pass that used that parity
int launch_mcc(gasatt_sim *s, cudaStream_t st, int q) {
  const int b = s->cur;
  if (s->form == 0)
    k_mcc64<<<s->mcc_grid, kMccBlock, 0, st>>>(s->P, s->s64[b], s->cnt, s->queue, q);
  else
    k_collide32<<<s->mcc_grid, kMccBlock, 0, st>>>(s->d_P, s->s32[b], fields_of<float>(s, fcur(s)),
                                                   s->cnt, s->queue);
  s->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "collision launch");
  return GASATT_OK;
}

// Apply the collisions still queued by the last pass, so that the particle
// state and the counters are complete (before a sort, a read, diagnostics or
// the end of a run).  The queue is emptied afterwards, so the collision kernel
// of the next step graph finds nothing to redo.
int flush_collisions(gasatt_sim *s) {
  if (!s->mcc_pending) return GASATT_OK;
  const int q = (int)((s->host_step - 1) & 1);
  cudaStream_t st = s->ctx->stream;
  SIM_TRY(launch_mcc(s, st, q));
  // The FP32 kernels pick their queue by the parity of the device's step
  // counter, which gasatt_sim_run_host moves against host_step's, so both
  // queues are emptied (the other one was consumed by the last pass); the
  // FP64 kernels are told the parity q.
  if (s->form == 1)
    GASATT_CUDA(s->ctx, cudaMemsetAsync(s->cnt->n_cand, 0, sizeof(s->cnt->n_cand), st));
  else
    GASATT_CUDA(s->ctx, cudaMemsetAsync(&s->cnt->n_cand[q], 0, sizeof(unsigned long long), st));
  s->mcc_pending = false;
  return GASATT_OK;
}

// exclusive prefix sum of n counts (k_scan), its tile words and ticket cleared first
int launch_scan(gasatt_sim *s, cudaStream_t st, const int *in, int *out, int n) {
  const int ntiles = (n + kScanTile - 1) / kScanTile;
  if (ntiles > s->scan_ntiles_max) return fail(s->ctx, GASATT_E_ARG, "scan longer than its tile words");
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->scan_tiles, 0, ((size_t)ntiles + 1) * 8, st));
  k_scan<<<ntiles, kScanThreads, 0, st>>>(
      in, out, n, ScanState{s->scan_tiles, reinterpret_cast<unsigned *>(s->scan_tiles + ntiles), &s->cnt->scan_err});
  s->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "scan launch");
  return GASATT_OK;
}

// Ion push after step host_step when it completes a sub-cycle.  Collisions
// still queued are applied first, so that the ions born in the step just
// taken are pushed with the others.
int launch_ion_push(gasatt_sim *s, cudaStream_t st) {
  SIM_TRY(flush_collisions(s));
  const auto &c = s->cfg;
  const int nbin = (c.n_r + 1) * (c.n_z + 1);
  const unsigned g = grid_for(c.ion_capacity, kBlock) < s->pass_grid ? grid_for(c.ion_capacity, kBlock) : s->pass_grid;
  // sort the store into the scratch store (the electrons' sort buffers are free here)
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->cell_count, 0, (size_t)(nbin + 1) * 4, st));
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->cell_cursor, 0, (size_t)nbin * 4, st));
  k_ion_hist<<<g, kBlock, 0, st>>>(s->P.ion, s->cnt, c.ion_capacity, c.n_r, c.n_z, c.dr, c.dz, s->cell_count);
  SIM_TRY(launch_scan(s, st, s->cell_count, s->cell_offset, nbin + 1));
  k_ion_scatter<<<g, kBlock, 0, st>>>(s->P.ion, s->ion_tmp, s->cnt, c.ion_capacity, c.n_r, c.n_z, c.dr,
                                      c.dz, s->cell_offset, s->cell_cursor);
  k_ion_sort_finish<<<1, 1, 0, st>>>(s->cnt, s->cell_offset, nbin);
  s->ctx->launches += 3;
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->Jir, 0, jbytes(s), st));
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->Jiz, 0, jbytes(s), st));
  SimParams PI = s->P;
  PI.dt = c.dt * c.ion_subcycle;
  PI.qm_dt2 = c.q_e / c.m_ion * PI.dt / 2;
  PI.dep = s->ion_scale;
  PI.Jr = s->Jir; PI.Jz = s->Jiz;
  if (s->form == 0)
    k_ion_push<double><<<g, kBlock, 0, st>>>(PI, fields_of<double>(s, fcur(s)), s->cnt, s->ion_tmp);
  else
    k_ion_push<float><<<g, kBlock, 0, st>>>(PI, fields_of<float>(s, fcur(s)), s->cnt, s->ion_tmp);
  s->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "ion push launch");
  return GASATT_OK;
}

bool ion_push_due(const gasatt_sim *s) {
  return s->cfg.ion_capacity > 0 && s->host_step % s->cfg.ion_subcycle == 0;
}

// whether kGraphSteps more steps end at the latest with the step before the
// next sort, and with the next ion push
bool steps_fit(const gasatt_sim *s, int sort_period) {
  const auto &c = s->cfg;
  return (sort_period <= 0 || sort_period - s->since_sort >= kGraphSteps) &&
         (c.ion_capacity <= 0 || c.ion_subcycle - s->host_step % c.ion_subcycle >= kGraphSteps);
}

// sort from buffer `from` into 1 - from
int launch_sort(gasatt_sim *s, cudaStream_t st, int from) {
  const auto &c = s->cfg;
  const int ncell = (c.n_r + 1) * (c.n_z + 1);    // sort bins
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->cell_count, 0, (size_t)(ncell + 1) * 4, st));
  GASATT_CUDA(s->ctx, cudaMemsetAsync(s->cell_cursor, 0, (size_t)ncell * 4, st));
  const unsigned g = s->pass_grid;
  if (s->form == 0)
    k_sort_hist<0><<<g, kBlock, 0, st>>>(s->s64[from], s->s32[from], s->cnt, c.n_r, c.n_z, c.dr, c.dz, s->cell_count);
  else
    k_sort_hist<1><<<g, kBlock, 0, st>>>(s->s64[from], s->s32[from], s->cnt, c.n_r, c.n_z, c.dr, c.dz, s->cell_count);
  s->ctx->launches++;
  SIM_TRY(launch_scan(s, st, s->cell_count, s->cell_offset, ncell + 1));
  if (s->form == 0)
    k_sort_scatter<0><<<g, kBlock, 0, st>>>(s->s64[from], s->s64[1 - from], s->s32[from], s->s32[1 - from],
                                            s->cnt, c.n_r, c.n_z, c.dr, c.dz, s->cell_offset, s->cell_cursor);
  else
    k_sort_scatter<1><<<g, kBlock, 0, st>>>(s->s64[from], s->s64[1 - from], s->s32[from], s->s32[1 - from],
                                            s->cnt, c.n_r, c.n_z, c.dr, c.dz, s->cell_offset, s->cell_cursor);
  s->ctx->launches++;
  k_sort_finish<<<1, 1, 0, st>>>(s->cnt, s->cell_offset, ncell);
  s->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(s->ctx, e, "sort launch");
  return GASATT_OK;
}

void drop_step_graphs(gasatt_sim *s) {
  for (int i = 0; i < 2; ++i)
    for (int q = 0; q < 2; ++q) {
      if (s->g_step[i][q]) cudaGraphExecDestroy(s->g_step[i][q]);
      s->g_step[i][q] = nullptr;
      if (s->gr_step[i][q]) cudaGraphDestroy(s->gr_step[i][q]);
      s->gr_step[i][q] = nullptr;
    }
}

void drop_graphs(gasatt_sim *s) {
  drop_step_graphs(s);
  for (int i = 0; i < 2; ++i) {
    if (s->g_steps[i]) cudaGraphExecDestroy(s->g_steps[i]);
    s->g_steps[i] = nullptr;
    if (s->gr_steps[i]) cudaGraphDestroy(s->gr_steps[i]);
    s->gr_steps[i] = nullptr;
    if (s->g_sort[i]) cudaGraphExecDestroy(s->g_sort[i]);
    s->g_sort[i] = nullptr;
    if (s->gr_sort[i]) cudaGraphDestroy(s->gr_sort[i]);
    s->gr_sort[i] = nullptr;
  }
}

// host_step starts over at 0: the fields of the current time move to field
// buffer 0 (they are in buffer host_step & 1)
int restart_steps(gasatt_sim *s, cudaStream_t st) {
  if (fcur(s) != 0) {
    const size_t esz = s->form == 0 ? 8 : 4, nz = (size_t)s->cfg.n_z, ld = (size_t)s->ldf;
    GASATT_CUDA(s->ctx, cudaMemcpyAsync(s->Er[0], s->Er[1], ld * (nz + 1) * esz, cudaMemcpyDeviceToDevice, st));
    GASATT_CUDA(s->ctx, cudaMemcpyAsync(s->Ez[0], s->Ez[1], ld * nz * esz, cudaMemcpyDeviceToDevice, st));
    GASATT_CUDA(s->ctx, cudaMemcpyAsync(s->H[0], s->H[1], ld * nz * esz, cudaMemcpyDeviceToDevice, st));
  }
  s->host_step = 0;
  return GASATT_OK;
}

// the pass's chunk for the population in h (FP32; later the commits choose it)
void set_chunk(const gasatt_sim *s, SimCounters &h) {
  h.chunk_fixed = s->P.chunk;
  h.pass_blocks = (int)s->pass_grid;
  h.chunk = h.chunk_fixed ? h.chunk_fixed : even_chunk((unsigned)h.n_total, s->pass_grid, kChunkMax);
}

// A fresh population of n particles sits in state buffer 0: counters, current
// buffers and the step bookkeeping start over.
int sim_reset(gasatt_sim *s, int64_t n) {
  gasatt_ctx *ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  SimCounters zc{};
  zc.n_total = (unsigned long long)n;
  zc.step = -1;
  zc.step64[0] = zc.step64[1] = -2;          // the prologue (parity 1) runs as step -1
  zc.cap = (unsigned long long)s->cfg.capacity;
  set_chunk(s, zc);
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->cnt, &zc, sizeof(zc), cudaMemcpyHostToDevice, st));
  for (int q = 0; q < 2; ++q) {
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jr[q], 0, jbytes(s), st));
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jz[q], 0, jbytes(s), st));
  }
  if (s->Jir) {                    // a new run: no ions, no ion current
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jir, 0, jbytes(s), st));
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jiz, 0, jbytes(s), st));
  }
  SIM_TRY(restart_steps(s, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  s->primed = false;
  s->mcc_pending = false;
  s->batch_pass = false;
  s->uncommitted = false;
  s->since_sort = 0;
  return GASATT_OK;
}

// Null-collision bound for a peak gas density n_max: nu_max = n_max *
// max(sigma_tot v), P_null = 1 - exp(-nu_max dt), and the integer threshold
// of the candidate test on the 52-bit draw.
void set_collision_bound(gasatt_sim *s, double n_max) {
  SimParams &P = s->P;
  P.nu_max = n_max * s->tabs.sigv_max;
  P.P_null = -std::expm1(-P.nu_max * s->cfg.dt);
  // largest count of 52-bit draws b with (2b+1) 2^-53 < P_null (exact in double)
  uint64_t t = (uint64_t)std::floor(P.P_null * 0x1.0p52);
  while ((2.0 * (double)t + 1.0) * 0x1.0p-53 < P.P_null) ++t;
  while (t > 0 && !((2.0 * (double)(t - 1) + 1.0) * 0x1.0p-53 < P.P_null)) --t;
  P.cand_below = t;
}

// cuTensorMapEncodeTiled from the driver (looked up once)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// A 2D tensor map over a w x h grid of elements with row stride ld_bytes
// (a multiple of 16), box bw x bh; out-of-bounds boxes fill with zeros.
int encode_map(gasatt_sim *s, CUtensorMap *m, CUtensorMapDataType type, void *base, int w, int h,
               size_t ld_bytes, int bw, int bh) {
  auto enc = tensor_map_encoder();
  if (!enc) return fail(s->ctx, GASATT_E_CUDA, "cuTensorMapEncodeTiled not available from the driver");
  const cuuint64_t dims[2] = {(cuuint64_t)w, (cuuint64_t)h};
  const cuuint64_t strides[1] = {(cuuint64_t)ld_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = enc(m, type, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(s->ctx, GASATT_E_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return GASATT_OK;
}

// The patch shape for cells of the given numbers of tiles in the three shapes
// (fdtd_tile_rows 0): the smallest patches (short segments, so the shortest
// chain) while they leave half of the GPU's block slots (nsm SMs) free, the middle ones
// while their tiles are one wave of blocks, beyond that the tallest (the least
// halo recomputed).  FP32 step with shape 12 / 16 / 20: 32 x 64 cells 18.4 / 19.2
// / 21.2 us; 256 x 1024 54.3 / 54.4 / 56.7 (FP64 79.7 / 78.5 / 78.4); 1024 x
// 4096 423 / 417 / 405; 16 batched cells 328 / 314 / 301.
int tma_auto(long long tiles12, long long tiles16, int nsm) {
  return tiles12 <= 4 * nsm ? 12 : tiles16 <= 4 * nsm ? 16 : 20;
}

// The field update's descriptor of a cell for the steps of parity q with patch
// shape k: tensor maps of the fields and of the current read, where the
// tiles are written.
template <typename T>
int fdtd_inst_of(gasatt_sim *s, int k, int q, FdtdInst &I) {
  const auto &c = s->cfg;
  const int rows = tma_rows(k);
  const CUtensorMapDataType ft = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const size_t ldb = (size_t)s->ldf * sizeof(T), ldjb = (size_t)s->ldj * 8;
  const int bw = TmaBox<T>::w;
  std::memset(&I, 0, sizeof(I));
  TmaMaps &M = I.maps;
  SIM_TRY(encode_map(s, &M.er, ft, s->Er[q], c.n_r, c.n_z + 1, ldb, bw, rows));
  SIM_TRY(encode_map(s, &M.ez, ft, s->Ez[q], c.n_r + 1, c.n_z, ldb, bw, rows));
  SIM_TRY(encode_map(s, &M.h, ft, s->H[q], c.n_r, c.n_z, ldb, bw, rows));
  SIM_TRY(encode_map(s, &M.jr, CU_TENSOR_MAP_DATA_TYPE_INT64, s->Jr[q], c.n_r, c.n_z, ldjb, 34, rows));
  SIM_TRY(encode_map(s, &M.jz, CU_TENSOR_MAP_DATA_TYPE_INT64, s->Jz[q], c.n_r, c.n_z, ldjb, 34, rows));
  I.Er = s->Er[1 - q]; I.Ez = s->Ez[1 - q]; I.H = s->H[1 - q];
  I.Jr_next = s->Jr[1 - q]; I.Jz_next = s->Jz[1 - q];
  I.colc = s->fdtd_colc;
  I.xj = ExtraCurrent{s->Jir, s->Jiz, s->scale / s->ion_scale};
  I.q = sizeof(T) == 4 ? s->quads : FieldQuads{};
  I.c = fdtd_coef(s);
  const double h4 = c.dt / 4, h2 = c.dt / 2;
  I.chr4 = h4 / (c.mu0 * I.c.dr);
  I.chz4 = h4 / (c.mu0 * I.c.dz);
  I.chr2 = h2 / (c.mu0 * I.c.dr);
  I.chz2 = h2 / (c.mu0 * I.c.dz);
  I.nr = c.n_r; I.nz = c.n_z; I.ldf = s->ldf; I.ldj = s->ldj;
  I.flags = c.flags;
  I.tiles_x = tma_tiles_x(c.n_r);
  I.ntiles = tma_tiles(k, c.n_r, c.n_z);
  I.err = &s->cnt->fdtd_err;
  return GASATT_OK;
}

// The field update of fdtd_ratio 1: patch shape, descriptors, grid and shared memory.
template <typename T>
int setup_fdtd_tma(gasatt_sim *s, int nsm) {
  const auto &c = s->cfg;
  const int k = c.fdtd_tile_rows > 0 ? c.fdtd_tile_rows
                                     : tma_auto(tma_tiles(12, c.n_r, c.n_z), tma_tiles(16, c.n_r, c.n_z), nsm);
  if (!tma_rows_ok(k)) return fail(s->ctx, GASATT_E_ARG, "fdtd_tile_rows: 12, 16 or 20");
  s->tma_rows = k;
  s->tma_smem = tma_block_bytes<T>(k);
  const int ntiles = tma_tiles(k, c.n_r, c.n_z);
  const SimFdtdTmaFn kern = sim_fdtd_tma_fn<T>(k);
  GASATT_CUDA(s->ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)s->tma_smem));
  int occ = 0;
  GASATT_CUDA(s->ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * tma_warps(k), s->tma_smem));
  if (occ < 1) return fail(s->ctx, GASATT_E_ARG, "field update: patch does not fit in shared memory");
  const long long slots = (long long)nsm * occ;
  s->tma_grid = (unsigned)(slots < ntiles ? slots : ntiles);
  for (int q = 0; q < 2; ++q) SIM_TRY(fdtd_inst_of<T>(s, k, q, s->fdtd_inst[q]));
  return GASATT_OK;
}

// device copies of P (current buffers 0 and 1) for the kernels that read it
// from global memory
int upload_params(gasatt_sim *s) {
  SimParams Pq[2] = {s->P, s->P};
  Pq[0].Jr = s->Jr[0]; Pq[0].Jz = s->Jz[0];
  Pq[1].Jr = s->Jr[1]; Pq[1].Jz = s->Jz[1];
  GASATT_CUDA(s->ctx, cudaMemcpy(s->d_P, Pq, sizeof(Pq), cudaMemcpyHostToDevice));
  return GASATT_OK;
}

// Start of a run: the particles at x^0 move to x^{1/2} and deposit j^{1/2}
// (no collision candidates; queue parity 1 is the one step 0 reads).
int sim_prime(gasatt_sim *s) {
  if (s->primed) return GASATT_OK;
  cudaStream_t st = s->ctx->stream;
  if (s->cfg.sort_period > 0) SIM_TRY(gasatt_sim_sort(s));
  // The prologue runs as parity 1, one step after the last pass (after a new
  // population both indices are equal).  A run that goes on after
  // gasatt_sim_run_host may have had its last pass on parity 1, or go on with
  // parity 1: the other parity's index then takes over the last one's, before or after.
  auto catch_up = [&]() {
    return cudaMemcpyAsync(&s->cnt->step64[0], &s->cnt->step64[1], sizeof(long long), cudaMemcpyDeviceToDevice, st);
  };
  const bool odd = s->host_step & 1;
  if (s->form == 0 && !odd) GASATT_CUDA(s->ctx, catch_up());
  // FP32: as a step of its own, else it would find the chunks of the last pass
  // handed out and its electrons marked as pushed
  if (s->form == 1 && s->uncommitted) {
    k_commit32<<<1, 1, 0, st>>>(s->cnt);
    GASATT_LAUNCHED(s->ctx);
  }
  s->uncommitted = false;
  // The current goes to the buffer that the next step reads: buffer host_step & 1,
  // which the last field update left empty (both are empty in a new run).  (A half drift
  // reads no field.)
  SIM_TRY(launch_pass(s, st, 1, (int)odd, 1, fcur(s)));
  if (s->form == 0 && odd) GASATT_CUDA(s->ctx, catch_up());
  s->primed = true;
  return GASATT_OK;
}

// Capture one step for state buffer b and step parity q:
//
//    [field update of step s]  ||  [collisions queued by pass s-1 (parity 1-q)]
//                      \\               /
//                   [particle pass s: kick, drift, deposit, queue q]
//
// The field update needs only the current of pass s-1 and the collisions only
// the particles, so the two run side by side.  Also one sort b -> 1-b.
// early: where a kernel has one other before it, it may start early (but for
// the first of a graph).  FP64: the field update after the pass only.
int capture_step(gasatt_sim *s, cudaStream_t cs, cudaStream_t side, int q, bool first, bool early) {
  int rc = GASATT_OK;
  cudaError_t e = cudaSuccess;
  auto mark = [&](int k, cudaStream_t st) {
    if (e == cudaSuccess && !rc && s->timing) e = cudaEventRecordWithFlags(s->ev[k], st, cudaEventRecordExternal);
  };
  if (s->form == 1) {
    // FP32: the field kernel commits the previous pass, the pass runs the
    // previous step's collisions itself.  Timing: one event before, one
    // between and one after the two kernels (the pass's collisions have
    // no kernel of their own)
    mark(0, cs);
    if (e == cudaSuccess) rc = launch_fdtd(s, cs, q, early && !first);
    mark(1, cs);
    if (e == cudaSuccess && !rc) rc = launch_pass(s, cs, 0, 1 - q, q, 1 - q, early);
    mark(3, cs);
  } else {
    e = cudaEventRecord(s->fork_ev, cs);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side, s->fork_ev, 0);
    mark(4, side);
    if (e == cudaSuccess) rc = launch_mcc(s, side, 1 - q);
    mark(5, side);
    if (e == cudaSuccess && !rc) e = cudaEventRecord(s->join_ev, side);
    mark(0, cs);
    if (e == cudaSuccess && !rc) rc = launch_fdtd(s, cs, q, early && !first);
    mark(1, cs);
    if (e == cudaSuccess && !rc) e = cudaStreamWaitEvent(cs, s->join_ev, 0);
    mark(2, cs);
    if (e == cudaSuccess && !rc) rc = launch_pass(s, cs, 0, 1 - q, q, 1 - q);
    mark(3, cs);
  }
  if (!rc && e != cudaSuccess) rc = cuda_fail(s->ctx, e, "capture step");
  return rc;
}

// `count` steps, the first of parity q, as one graph, instantiated and as it
// is.  No early starts in a graph of one step: it is also a child of a batch's graph.
int capture_steps(gasatt_sim *s, cudaStream_t cs, cudaStream_t side, int q, int count, cudaGraphExec_t *exec,
                  cudaGraph_t *keep) {
  cudaGraph_t g;
  GASATT_CUDA(s->ctx, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
  int rc = GASATT_OK;
  for (int k = 0; k < count && !rc; ++k) rc = capture_step(s, cs, side, (q + k) & 1, k == 0, count > 1);
  cudaError_t e = cudaStreamEndCapture(cs, &g);
  const bool captured = e == cudaSuccess;
  if (!rc && !captured) rc = cuda_fail(s->ctx, e, "capture step");
  if (!rc) {
    e = cudaGraphInstantiate(exec, g, 0);
    if (e != cudaSuccess) rc = cuda_fail(s->ctx, e, "instantiate step");
  }
  if (captured) {
    if (!rc) *keep = g; else cudaGraphDestroy(g);
  }
  return rc;
}

// copies of the arguments that v points to, of a kernel such as this one
template <typename... K>
std::vector<std::vector<char>> copy_args(void (*)(K...), void **v) {
  std::vector<std::vector<char>> c;
  for (size_t size : {sizeof(K)...}) {
    const char *p = static_cast<const char *>(*v++);
    c.emplace_back(p, p + size);
  }
  return c;
}

// Changed launch parameters (s->P) into the kernel nodes of a step graph that
// hold them: the pass and the FP64 collisions, each with SimParams first.
int renew_params(gasatt_sim *s, cudaGraph_t g, cudaGraphExec_t exec) {
  if (!g) return GASATT_OK;
  size_t n = 0;
  GASATT_CUDA(s->ctx, cudaGraphGetNodes(g, nullptr, &n));
  std::vector<cudaGraphNode_t> nodes(n);
  GASATT_CUDA(s->ctx, cudaGraphGetNodes(g, nodes.data(), &n));
  for (cudaGraphNode_t node : nodes) {
    cudaGraphNodeType type;
    GASATT_CUDA(s->ctx, cudaGraphNodeGetType(node, &type));
    if (type != cudaGraphNodeTypeKernel) continue;
    cudaKernelNodeParams k;
    GASATT_CUDA(s->ctx, cudaGraphKernelNodeGetParams(node, &k));
    std::vector<std::vector<char>> c;
    if (k.func == (void *)k_pass64<0>) c = copy_args(k_pass64<0>, k.kernelParams);
    else if (k.func == (void *)k_mcc64) c = copy_args(k_mcc64, k.kernelParams);
    else if (k.func == (void *)k_pass32<0, false> || k.func == (void *)k_pass32<0, true>)
      c = copy_args(k_pass32<0, false>, k.kernelParams);
    else continue;
    SimParams P = s->P, old;
    std::memcpy(&old, c[0].data(), sizeof(old));
    P.Jr = old.Jr;                         // the node's current buffer
    P.Jz = old.Jz;
    std::memcpy(c[0].data(), &P, sizeof(P));
    void *args[8];
    for (size_t i = 0; i < c.size(); ++i) args[i] = c[i].data();
    k.kernelParams = args;
    GASATT_CUDA(s->ctx, cudaGraphExecKernelNodeSetParams(exec, node, &k));
    GASATT_CUDA(s->ctx, cudaGraphKernelNodeSetParams(node, &k));
  }
  return GASATT_OK;
}

// The same for all step graphs.  Building them anew instead took 3.8 ms of
// gasatt_sim_set_gas_density in the FP64 form and 1.2 ms in the FP32 form, most of
// it for the forks of the graphs of ten steps; now 0.16 and 0.13 ms.
int renew_params(gasatt_sim *s) {
  for (int b = 0; b < 2; ++b) {
    for (int q = 0; q < 2; ++q) SIM_TRY(renew_params(s, s->gr_step[b][q], s->g_step[b][q]));
    SIM_TRY(renew_params(s, s->gr_steps[b], s->g_steps[b]));
  }
  return GASATT_OK;
}

// the graphs that there are not yet (with the timing on, those of one step
// hold its events, and those of ten are not used)
int build_graphs(gasatt_sim *s) {
  // the field update goes on a higher-priority stream than the collision
  // branch, so its blocks are placed first when both are ready
  int lo_prio = 0, hi_prio = 0;
  cudaDeviceGetStreamPriorityRange(&lo_prio, &hi_prio);
  cudaStream_t cs, side;
  GASATT_CUDA(s->ctx, cudaStreamCreateWithPriority(&cs, cudaStreamNonBlocking, hi_prio));
  GASATT_CUDA(s->ctx, cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, lo_prio));
  const int save = s->cur;
  const int64_t save_launch = s->ctx->launches;
  int rc = GASATT_OK;
  for (int b = 0; b < 2 && !rc; ++b) {
    cudaGraph_t g;
    s->cur = b;
    for (int q = 0; q < 2 && !rc; ++q) rc = capture_steps(s, cs, side, q, 1, &s->g_step[b][q], &s->gr_step[b][q]);
    if (!rc && !s->timing && !s->g_steps[b]) rc = capture_steps(s, cs, side, 0, kGraphSteps, &s->g_steps[b], &s->gr_steps[b]);
    if (rc) break;
    if (s->g_sort[b]) continue;
    GASATT_CUDA(s->ctx, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    rc = launch_sort(s, cs, b);
    cudaError_t e = cudaStreamEndCapture(cs, &g);
    const bool captured = e == cudaSuccess;
    if (!rc && !captured) rc = cuda_fail(s->ctx, e, "capture sort");
    if (!rc) {
      e = cudaGraphInstantiate(&s->g_sort[b], g, 0);
      if (e != cudaSuccess) rc = cuda_fail(s->ctx, e, "instantiate sort");
    }
    if (captured) {
      if (!rc) s->gr_sort[b] = g; else cudaGraphDestroy(g);
    }
  }
  s->cur = save;
  s->ctx->launches = save_launch;
  cudaStreamDestroy(side);
  cudaStreamDestroy(cs);
  return rc;
}

}  // namespace

extern "C" {

int gasatt_sim_default_config(gasatt_sim_config *c) {
  if (!c) return GASATT_E_ARG;
  std::memset(c, 0, sizeof(*c));
  c->n_r = 256; c->n_z = 1024; c->dr = 5e-6; c->dz = 5e-6; c->dt = 1e-14;
  c->fdtd_ratio = 1;
  c->PHIp = 2 * GASATT_PI;
  c->FN = 1.0;
  c->gas_temperature = 300.0;
  c->kb = 1.380649e-23;
  c->gas_density = 133.322368 / (c->kb * 300.0);     // 1 Torr
  c->q_e = 1.602176634e-19; c->m_e = 9.1093837015e-31; c->c = 299792458.0;
  c->eps0 = 8.8541878128e-12; c->mu0 = 1.25663706212e-6;
  c->m_ion = 28.0134 * 1.66053906660e-27;
  c->precision = GASATT_FP32_SPLIT;
  c->capacity = 1 << 20;
  c->ion_capacity = 0;
  c->ion_subcycle = 50;
  c->seed = 0;
  c->flags = 0;
  c->sort_period = 20;
  c->secondaries = 1;
  c->table_n = 2048; c->table_emin_ev = 0.1; c->table_emax_ev = 30000.0;
  return GASATT_OK;
}

int gasatt_sim_create(gasatt_ctx *ctx, const gasatt_sim_config *cfg, const gasatt_tables *tab,
                      gasatt_sim **out) {
  if (!ctx || !cfg || !out) return GASATT_E_ARG;
  *out = nullptr;
  const gasatt_sim_config &c = *cfg;
  if (c.n_r < 2 || c.n_z < 2 || c.n_r > 65535 || c.n_z > 65535 ||
      (int64_t)(c.n_r + 1) * (c.n_z + 1) > 0x7FFFFFFFLL || !(c.dr > 0) || !(c.dz > 0) ||
      !(c.dt > 0) || c.fdtd_ratio < 1 || c.capacity < 1 || c.capacity > 0x7FFFFFFFLL ||
      (c.precision != GASATT_FP64 && c.precision != GASATT_FP32_SPLIT))
    return fail(ctx, GASATT_E_ARG, "sim config out of range");
  if (c.flags & ~(unsigned)(GASATT_Q_ER_END_COPY | GASATT_Q_EZ_AXIS_JSIGN | GASATT_Q_EZ_RSHIFT))
    return fail(ctx, GASATT_E_ARG, "the resident simulation accepts only the field quirk flags");
  if (c.pass_chunk < 0 || c.pass_chunk > kChunkMax || c.pass_chunk % kBlock)
    return fail(ctx, GASATT_E_ARG, "pass_chunk: a multiple of 256 in [256, 1792] (0: by population)");
  if (c.fdtd_tile_rows < 0) return fail(ctx, GASATT_E_ARG, "fdtd_tile_rows: >= 0");
  if (c.gather < 0 || c.gather > 2) return fail(ctx, GASATT_E_ARG, "gather: 0 (auto), 1 (quads) or 2 (fields)");
  if (c.ion_capacity < 0 || (c.ion_capacity > 0 && (c.ion_subcycle < 1 || !(c.m_ion > 0) ||
                                                     !(c.gas_temperature >= 0))))
    return fail(ctx, GASATT_E_ARG, "ion species: ion_capacity >= 0, ion_subcycle >= 1, m_ion > 0");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  gasatt_sim *s = new gasatt_sim();
  s->ctx = ctx;
  s->cfg = c;
  s->form = c.precision;
  std::string err;
  int rc = build_sim_tables(tab, c.table_n, c.table_emin_ev, c.table_emax_ev, c.gas_density, c.c,
                            c.m_e, c.q_e, s->tabs, err);
  if (rc) { delete s; return fail(ctx, rc, err); }
  const int64_t cap = c.capacity;
  const int nr = c.n_r, nz = c.n_z, nbin = (nr + 1) * (nz + 1);
  s->ldf = (nr + 1 + 3) & ~3;       // 16-byte rows for float and double
  s->ldj = (nr + 1) & ~1;           // 16-byte rows of 64-bit counters
  const size_t ncur = (size_t)s->ldj * nz;
  auto cleanup = [&](int code) { gasatt_sim_destroy(s); return code; };
  for (int b = 0; b < 2; ++b) {
    if (s->form == 0) {
      State64 &S = s->s64[b];
      if ((rc = sim_alloc(s, &S.rz, cap)) || (rc = sim_alloc(s, &S.urt, cap)) ||
          (rc = sim_alloc(s, &S.uz, cap)) || (rc = sim_alloc(s, &S.id, cap)))
        return cleanup(rc);
    } else {
      State32 &S = s->s32[b];
      if ((rc = sim_alloc(s, &S.a, cap)) || (rc = sim_alloc(s, &S.b, cap)) || (rc = sim_alloc(s, &S.id, cap)))
        return cleanup(rc);
    }
  }
  if ((rc = sim_alloc(s, &s->queue, 2 * (size_t)cap))) return cleanup(rc);
  if (c.ion_capacity > 0) {
    IonState &I = s->P.ion;
    const size_t ic = (size_t)c.ion_capacity;
    if ((rc = sim_alloc(s, &I.rz, ic)) || (rc = sim_alloc(s, &I.urt, ic)) ||
        (rc = sim_alloc(s, &I.uz, ic)) || (rc = sim_alloc(s, &I.id, ic)) ||
        (rc = sim_alloc(s, &I.q, ic)) || (rc = sim_alloc(s, &s->ion_tmp.rz, ic)) ||
        (rc = sim_alloc(s, &s->ion_tmp.urt, ic)) || (rc = sim_alloc(s, &s->ion_tmp.uz, ic)) ||
        (rc = sim_alloc(s, &s->ion_tmp.id, ic)) || (rc = sim_alloc(s, &s->ion_tmp.q, ic)) ||
        (rc = sim_alloc(s, &s->Jir, ncur)) || (rc = sim_alloc(s, &s->Jiz, ncur)))
      return cleanup(rc);
  }
  const size_t esz = s->form == 0 ? 8 : 4;
  double *tmpd;
  const size_t nfE = (size_t)s->ldf * (nz + 1), nfZ = (size_t)s->ldf * nz, nfH = (size_t)s->ldf * nz;
  if ((rc = sim_alloc(s, (char **)&s->Er[0], nfE * esz)) ||
      (rc = sim_alloc(s, (char **)&s->Ez[0], nfZ * esz)) ||
      (rc = sim_alloc(s, (char **)&s->H[0], nfH * esz)) ||
      (rc = sim_alloc(s, (char **)&s->Er[1], nfE * esz)) ||
      (rc = sim_alloc(s, (char **)&s->Ez[1], nfZ * esz)) ||
      (rc = sim_alloc(s, (char **)&s->H[1], nfH * esz)) ||
      (rc = sim_alloc(s, &s->Jr[0], ncur)) || (rc = sim_alloc(s, &s->Jz[0], ncur)) ||
      (rc = sim_alloc(s, &s->Jr[1], ncur)) || (rc = sim_alloc(s, &s->Jz[1], ncur)) ||
      (rc = sim_alloc(s, &s->cnt, 1)) || (rc = sim_alloc(s, &s->cell_count, (size_t)nbin + 1)) ||
      (rc = sim_alloc(s, &s->cell_offset, (size_t)nbin + 1)) ||
      (rc = sim_alloc(s, &s->cell_cursor, (size_t)nbin)) ||
      (rc = sim_alloc(s, &tmpd, (size_t)4 * c.table_n + (size_t)181 * c.table_n)))
    return cleanup(rc);
  s->d_tab = tmpd;
  if ((rc = sim_alloc(s, &s->invV, (size_t)nr)) || (rc = sim_alloc(s, &s->fdtd_colc, (size_t)3 * nr)))
    return cleanup(rc);
  // FP32 gather quads: 48 bytes more per cell written by every field update,
  // against nine fewer loads per electron; worth it where electrons are dense
  // and the quads stay in L2 between the field update and the pass.  256 x 1024
  // cells, 2M electrons: step 56.7 us with quads, 58.2 with the fields; 1024 x
  // 4096 cells (200 MB of quads), 16M electrons: 525 and 493.
  const bool quads = s->form == 1 &&
                     (c.gather == 1 || (c.gather == 0 && (int64_t)(nr + 1) * (nz + 1) <= kQuadCells &&
                                        c.capacity >= 4 * (int64_t)(nr + 1) * (nz + 1)));
  if (quads) {
    if ((rc = sim_alloc(s, &s->quads.er, (size_t)(nr + 1) * nz)) ||
        (rc = sim_alloc(s, &s->quads.ez, (size_t)nr * (nz + 1))) ||
        (rc = sim_alloc(s, &s->quads.h, (size_t)(nr + 1) * (nz + 1))))
      return cleanup(rc);
    cudaMemset(s->quads.er, 0, (size_t)(nr + 1) * nz * 16);
    cudaMemset(s->quads.ez, 0, (size_t)nr * (nz + 1) * 16);
    cudaMemset(s->quads.h, 0, (size_t)(nr + 1) * (nz + 1) * 16);
  }
  s->scan_ntiles_max = (nbin + 1 + kScanTile - 1) / kScanTile;
  if ((rc = sim_alloc(s, &s->scan_tiles, (size_t)s->scan_ntiles_max + 1))) return cleanup(rc);
  s->partial_blocks = 296;
  if ((rc = sim_alloc(s, &s->partial, (size_t)2 * s->partial_blocks))) return cleanup(rc);
  if (cudaMallocHost((void **)&s->h_cnt, sizeof(SimCounters)) != cudaSuccess)
    return cleanup(fail(ctx, GASATT_E_CUDA, "cudaMallocHost"));
  // tables
  std::vector<double> host((size_t)4 * c.table_n + (size_t)181 * c.table_n);
  std::memcpy(host.data(), s->tabs.sig_el.data(), c.table_n * 8);
  std::memcpy(host.data() + c.table_n, s->tabs.sig_ion.data(), c.table_n * 8);
  std::memcpy(host.data() + 2 * c.table_n, s->tabs.sig_exc.data(), c.table_n * 8);
  std::memcpy(host.data() + 3 * c.table_n, s->tabs.edep.data(), c.table_n * 8);
  std::memcpy(host.data() + 4 * c.table_n, s->tabs.cdf.data(), (size_t)181 * c.table_n * 8);
  if (cudaMemcpy(s->d_tab, host.data(), host.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
    return cleanup(fail(ctx, GASATT_E_CUDA, "table upload"));
  // parameters
  SimParams &P = s->P;
  P.nr = nr; P.nz = nz; P.ldf = s->ldf; P.ldj = s->ldj; P.dr = c.dr; P.dz = c.dz; P.dt = c.dt; P.c = c.c; P.qe = c.q_e;
  P.me = c.m_e; P.mu0 = c.mu0; P.FN = c.FN; P.PHIp = c.PHIp; P.n_gas = c.gas_density;
  P.gas = nullptr;
  P.ion_sig = nullptr;
  P.Rp = nr * c.dr; P.Lp = nz * c.dz; P.kb = c.kb; P.m_ion = c.m_ion; P.T_gas = c.gas_temperature;
  P.chunk = c.pass_chunk;
  P.seed = c.seed; P.pk = philox_keys(c.seed); P.secondaries = c.secondaries; P.cap = cap;
  P.ion_cap = c.ion_capacity;
  P.ion_sigma = c.ion_capacity > 0 ? std::sqrt(c.kb * c.gas_temperature / c.m_ion) : 0.0;
  P.qm_dt2 = -c.q_e / c.m_e * c.dt / 2;
  P.idr = 1 / c.dr; P.idz = 1 / c.dz; P.ic2 = 1 / (c.c * c.c);
  P.mu_qm = c.mu0 * P.qm_dt2;
  P.aE = (float)(-c.q_e * c.dt / (2 * c.m_e * c.c));
  P.aB = (float)(-c.q_e * c.dt * c.mu0 / (2 * c.m_e));
  P.hdr = (float)(c.c * c.dt / (2 * c.dr));
  P.hdz = (float)(c.c * c.dt / (2 * c.dz));
  // fixed point: FP64 |q FN v w| * scale <= 2^48; FP32 <= 2^20 (the int32
  // deposit window of a chunk of particles cannot overflow)
  const double qfc = c.q_e * std::fabs(c.FN) * c.c;
  s->scale = s->form == 0 ? std::ldexp(1.0, 48) / qfc : std::ldexp(1.0, 20) / qfc;
  P.dep = s->scale;
  P.dep_q = -c.q_e * c.FN * s->scale;
  P.depf = (float)(-c.q_e * c.FN * c.c * s->scale);
  s->ion_scale = std::ldexp(1.0, 48) / qfc;
  set_collision_bound(s, c.gas_density);
  P.sig = s->d_tab;
  P.edep = s->d_tab + 3 * c.table_n;
  P.cdf = s->d_tab + 4 * c.table_n;
  P.exc_kmin = s->tabs.exc_kmin;
  P.G = c.table_n; P.lnEmin = s->tabs.lnEmin; P.dlnE = s->tabs.dlnE;
  P.mc2_ev = c.m_e * c.c * c.c / c.q_e; P.imc2_ev = 1 / P.mc2_ev; P.idlnE = 1 / P.dlnE;
  P.n_exc = s->tabs.n_exc;
  std::memcpy(P.exc, s->tabs.exc, sizeof(P.exc));
  P.Jr = s->Jr[0]; P.Jz = s->Jz[0];
  P.qEr = s->quads.er; P.qEz = s->quads.ez; P.qH = s->quads.h;
  {
    std::vector<double> iv(nr);
    for (int i = 0; i < nr; ++i) iv[i] = (1.0 / s->scale) / shell_volume(i, c.dr, c.dz, c.PHIp);
    std::vector<double> colc((size_t)3 * nr);
    fdtd_column_table(nr, fdtd_coef(s), iv.data(), c.flags, colc.data());
    if (cudaMemcpy(s->invV, iv.data(), (size_t)nr * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(s->fdtd_colc, colc.data(), (size_t)3 * nr * 8, cudaMemcpyHostToDevice) != cudaSuccess)
      return cleanup(fail(ctx, GASATT_E_CUDA, "volume table upload"));
  }
  if ((rc = sim_alloc(s, &s->d_P, 2)) || (rc = upload_params(s))) return cleanup(rc);
  if (fdtd_tile(c.fdtd_ratio) < 4)
    return cleanup(fail(ctx, GASATT_E_ARG, "fdtd_ratio too large for the fused field update (max 6)"));
  const int nsm = ctx->sms;
  if (c.fdtd_ratio == 1) {
    if ((rc = s->form == 0 ? setup_fdtd_tma<double>(s, nsm) : setup_fdtd_tma<float>(s, nsm)))
      return cleanup(rc);
  }
  int occ = 4;
  if (s->form == 0) {
    for (auto k : {k_pass64<0>, k_pass64<1>, k_pass64<2>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kWin64Bytes) != cudaSuccess)
        return cleanup(fail(ctx, GASATT_E_CUDA, "FP64 pass: shared memory"));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_pass64<0>, kBlock, kWin64Bytes);
  }
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (k_pass32<0, false>), kBlock, 0);
  s->pass_grid = (unsigned)(nsm * (occ > 0 ? occ : 1));
  if (s->form == 1) {
    // FP32 blocks take chunks from a counter: no more blocks than chunks the
    // capacity can hold (small instances then leave the GPU to others)
    const int least = P.chunk > 0 ? P.chunk : kBlock;
    const long long chunks = (cap + least - 1) / least;
    if ((long long)s->pass_grid > chunks) s->pass_grid = (unsigned)(chunks > 0 ? chunks : 1);
  }
  // as many collision warps as fit on the device at once
  int occ_mcc = 1;
  if (s->form == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_mcc, k_mcc64, kMccBlock, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_mcc, k_collide32, kMccBlock, 0);
  s->mcc_grid = (unsigned)(nsm * (occ_mcc > 0 ? occ_mcc : 1));
  // zero state
  SimCounters z{};
  z.step = -1;
  z.step64[0] = z.step64[1] = -2;
  z.cap = (unsigned long long)cap;
  set_chunk(s, z);
  if (cudaMemcpy(s->cnt, &z, sizeof(z), cudaMemcpyHostToDevice) != cudaSuccess)
    return cleanup(fail(ctx, GASATT_E_CUDA, "counter init"));
  for (int k = 0; k < 2; ++k) {
    cudaMemset(s->Er[k], 0, nfE * esz);
    cudaMemset(s->Ez[k], 0, nfZ * esz);
    cudaMemset(s->H[k], 0, nfH * esz);
  }
  for (int q = 0; q < 2; ++q) {
    cudaMemset(s->Jr[q], 0, ncur * 8);
    cudaMemset(s->Jz[q], 0, ncur * 8);
  }
  if (s->Jir) {
    cudaMemset(s->Jir, 0, ncur * 8);
    cudaMemset(s->Jiz, 0, ncur * 8);
  }
  for (int i = 0; i < 6; ++i)
    if (cudaEventCreate(&s->ev[i]) != cudaSuccess) return cleanup(fail(ctx, GASATT_E_CUDA, "event"));
  if (cudaEventCreateWithFlags(&s->fork_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&s->join_ev, cudaEventDisableTiming) != cudaSuccess)
    return cleanup(fail(ctx, GASATT_E_CUDA, "event"));
  rc = build_graphs(s);
  if (rc) return cleanup(rc);
  if (cudaDeviceSynchronize() != cudaSuccess) return cleanup(fail(ctx, GASATT_E_CUDA, "sim init"));
  *out = s;
  return GASATT_OK;
}

int gasatt_sim_get_config(const gasatt_sim *s, gasatt_sim_config *cfg) {
  if (!s || !cfg) return GASATT_E_ARG;
  *cfg = s->cfg;
  return GASATT_OK;
}

int gasatt_sim_destroy(gasatt_sim *s) {
  if (!s) return GASATT_OK;
  cudaSetDevice(s->ctx->device);
  cudaDeviceSynchronize();
  drop_graphs(s);
  for (int i = 0; i < 6; ++i)
    if (s->ev[i]) cudaEventDestroy(s->ev[i]);
  if (s->fork_ev) cudaEventDestroy(s->fork_ev);
  if (s->join_ev) cudaEventDestroy(s->join_ev);
  for (void *p : s->allocs) cudaFree(p);
  if (s->h_cnt) cudaFreeHost(s->h_cnt);
  delete s;
  return GASATT_OK;
}

int gasatt_sim_load(gasatt_sim *s, const double *r, const double *z, const double *ur,
                    const double *ut, const double *uz, const uint64_t *id, int64_t n,
                    int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  if (n < 0 || n > s->cfg.capacity) return fail(ctx, GASATT_E_CAPACITY, "load exceeds capacity");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const double *src[5] = {r, z, ur, ut, uz};
  const double *d[5];
  const uint64_t *did = id;
  void *buf = nullptr;
  if (!on_device && n > 0) {
    int rc = scratch(ctx, (size_t)n * 48, &buf);
    if (rc) return rc;
    for (int i = 0; i < 5; ++i) {
      d[i] = (double *)buf + (size_t)i * n;
      GASATT_CUDA(ctx, cudaMemcpyAsync((void *)d[i], src[i], (size_t)n * 8, cudaMemcpyHostToDevice, st));
    }
    did = (uint64_t *)((double *)buf + 5 * (size_t)n);
    GASATT_CUDA(ctx, cudaMemcpyAsync((void *)did, id, (size_t)n * 8, cudaMemcpyHostToDevice, st));
  } else {
    for (int i = 0; i < 5; ++i) d[i] = src[i];
  }
  s->cur = 0;
  if (n > 0) {
    if (s->form == 0)
      k_load64<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s64[0], d[0], d[1], d[2], d[3], d[4], did, n);
    else
      k_load32<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s32[0], d[0], d[1], d[2], d[3], d[4], did, n,
                                                       s->cfg.n_r, s->cfg.n_z, s->cfg.dr, s->cfg.dz, s->cfg.c,
                                                       0);   // the first pass runs at step -1
    GASATT_LAUNCHED(ctx);
  }
  return sim_reset(s, n);
}

int gasatt_sim_set_gas_density(gasatt_sim *s, const double *density, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t ncell = (size_t)s->cfg.n_r * s->cfg.n_z;
  std::vector<double> h;
  if (density) {
    h.resize(ncell);
    GASATT_CUDA(ctx, cudaMemcpy(h.data(), density, ncell * 8,
                                on_device ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost));
    for (double v : h)
      if (!(v >= 0) || !std::isfinite(v)) return fail(ctx, GASATT_E_ARG, "gas density: negative or not finite");
  }
  // collisions still queued were drawn against the old bound: apply them first
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double n_max = s->cfg.gas_density;
  if (density) {
    if (!s->d_gas) {
      int rc = sim_alloc(s, &s->d_gas, ncell);
      if (rc) return rc;
    }
    GASATT_CUDA(ctx, cudaMemcpy(s->d_gas, h.data(), ncell * 8, cudaMemcpyHostToDevice));
    n_max = 0;
    for (double v : h) n_max = v > n_max ? v : n_max;
    s->P.gas = s->d_gas;
  } else {
    s->P.gas = nullptr;
  }
  set_collision_bound(s, n_max);
  SIM_TRY(upload_params(s));
  return renew_params(s);          // the step graphs hold the launch parameters
}

int gasatt_sim_set_gas_temperature(gasatt_sim *s, const double *temperature, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t ncell = (size_t)s->cfg.n_r * s->cfg.n_z;
  std::vector<double> h;
  if (temperature) {
    h.resize(ncell);
    GASATT_CUDA(ctx, cudaMemcpy(h.data(), temperature, ncell * 8,
                                on_device ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost));
    for (double &v : h) {
      if (!(v >= 0) || !std::isfinite(v))
        return fail(ctx, GASATT_E_ARG, "gas temperature: negative or not finite");
      v = std::sqrt(s->cfg.kb * v / s->cfg.m_ion);    // the spread the births use
    }
  }
  // ions of the collisions still queued are born at the old temperature
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (temperature) {
    if (!s->d_ion_sig) {
      int rc = sim_alloc(s, &s->d_ion_sig, ncell);
      if (rc) return rc;
    }
    GASATT_CUDA(ctx, cudaMemcpy(s->d_ion_sig, h.data(), ncell * 8, cudaMemcpyHostToDevice));
    s->P.ion_sig = s->d_ion_sig;
  } else {
    s->P.ion_sig = nullptr;
  }
  SIM_TRY(upload_params(s));
  return renew_params(s);          // the step graphs hold the launch parameters
}

int gasatt_sim_birth_photo(gasatt_sim *s, int64_t n_photo, double photon_keV, double sigma_r,
                           uint64_t seed, uint64_t id_base) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  if (n_photo < 0 || !(sigma_r > 0) || !(photon_keV * 1000 > kKShellEv))
    return fail(ctx, GASATT_E_ARG, "birth_photo: bad arguments");
  if (2 * n_photo > s->cfg.capacity) return fail(ctx, GASATT_E_CAPACITY, "birth_photo exceeds capacity");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const auto &c = s->cfg;
  auto speed = [&](double E_ev) {                      // u = gamma v of kinetic energy E
    const double e = E_ev * c.q_e / (c.m_e * c.c * c.c);
    return c.c * std::sqrt(e * (2 + e));
  };
  const double Rp = c.n_r * c.dr, Lp = c.n_z * c.dz;
  const double r_max = std::nextafter(Rp, 0.0);
  s->cur = 0;
  if (n_photo > 0) {
    const unsigned g = grid_for(n_photo, kBlock);
    if (s->form == 0)
      k_birth_photo<0><<<g, kBlock, 0, st>>>(s->s64[0], s->s32[0], n_photo,
                                             speed(photon_keV * 1000 - kKShellEv), speed(kAugerEv),
                                             sigma_r, r_max, Lp, seed, id_base, c.n_r, c.n_z,
                                             c.dr, c.dz, c.c);
    else
      k_birth_photo<1><<<g, kBlock, 0, st>>>(s->s64[0], s->s32[0], n_photo,
                                             speed(photon_keV * 1000 - kKShellEv), speed(kAugerEv),
                                             sigma_r, r_max, Lp, seed, id_base, c.n_r, c.n_z,
                                             c.dr, c.dz, c.c);
    GASATT_LAUNCHED(ctx);
  }
  return sim_reset(s, 2 * n_photo);
}

int gasatt_sim_read(gasatt_sim *s, double *r, double *z, double *ur, double *ut, double *uz,
                    uint64_t *id, int64_t cap, int64_t *n_out, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  const unsigned long long nt = s->h_cnt->n_total + s->h_cnt->n_births;
  const int64_t n = (int64_t)(nt < s->h_cnt->cap ? nt : s->h_cnt->cap);
  if (n_out) *n_out = n;
  if (n > cap) return fail(ctx, GASATT_E_CAPACITY, "read buffer too small");
  if (n == 0) return GASATT_OK;
  double *d[5] = {r, z, ur, ut, uz};
  uint64_t *did = id;
  void *buf = nullptr;
  if (!on_device) {
    int rc = scratch(ctx, (size_t)n * 48, &buf);
    if (rc) return rc;
    for (int i = 0; i < 5; ++i) d[i] = (double *)buf + (size_t)i * n;
    did = (uint64_t *)((double *)buf + 5 * (size_t)n);
  }
  if (s->form == 0)
    k_read64<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s64[s->cur], d[0], d[1], d[2], d[3], d[4], did, n);
  else
    k_read32<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s32[s->cur], d[0], d[1], d[2], d[3], d[4], did, n,
                                                     s->cfg.dr, s->cfg.dz, s->cfg.c);
  GASATT_LAUNCHED(ctx);
  if (!on_device) {
    double *h[5] = {r, z, ur, ut, uz};
    for (int i = 0; i < 5; ++i)
      GASATT_CUDA(ctx, cudaMemcpyAsync(h[i], d[i], (size_t)n * 8, cudaMemcpyDeviceToHost, st));
    GASATT_CUDA(ctx, cudaMemcpyAsync(id, did, (size_t)n * 8, cudaMemcpyDeviceToHost, st));
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  return GASATT_OK;
}

int gasatt_sim_load_ions(gasatt_sim *s, const double *r, const double *z, const double *ur,
                         const double *ut, const double *uz, const uint64_t *id,
                         const int8_t *charge, int64_t n, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  if (s->cfg.ion_capacity <= 0) return fail(ctx, GASATT_E_STATE, "load_ions: no ion species (ion_capacity 0)");
  if (n < 0 || n > s->cfg.ion_capacity) return fail(ctx, GASATT_E_CAPACITY, "load_ions exceeds ion_capacity");
  if (n > 0 && (!r || !z || !ur || !ut || !uz || !id)) return fail(ctx, GASATT_E_ARG, "load_ions: null array");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  SIM_TRY(flush_collisions(s));
  const double *src[5] = {r, z, ur, ut, uz};
  const double *d[5] = {r, z, ur, ut, uz};
  const uint64_t *did = id;
  const int8_t *dq = charge;
  if (!on_device && n > 0) {
    void *buf = nullptr;
    int rc = scratch(ctx, (size_t)n * 49, &buf);
    if (rc) return rc;
    for (int i = 0; i < 5; ++i) {
      d[i] = (double *)buf + (size_t)i * n;
      GASATT_CUDA(ctx, cudaMemcpyAsync((void *)d[i], src[i], (size_t)n * 8, cudaMemcpyHostToDevice, st));
    }
    did = (uint64_t *)((double *)buf + 5 * (size_t)n);
    GASATT_CUDA(ctx, cudaMemcpyAsync((void *)did, id, (size_t)n * 8, cudaMemcpyHostToDevice, st));
    if (charge) {
      dq = (int8_t *)(did + n);
      GASATT_CUDA(ctx, cudaMemcpyAsync((void *)dq, charge, (size_t)n, cudaMemcpyHostToDevice, st));
    }
  }
  if (n > 0) {
    k_ion_load<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->P.ion, d[0], d[1], d[2], d[3], d[4], did, dq, n);
    GASATT_LAUNCHED(ctx);
  }
  const unsigned long long zc[3] = {(unsigned long long)n, 0ull, 0ull};   // n_ions, overflow, lost
  GASATT_CUDA(ctx, cudaMemcpyAsync((char *)s->cnt + offsetof(SimCounters, n_ions), zc, sizeof(zc),
                                   cudaMemcpyHostToDevice, st));
  GASATT_CUDA(ctx, cudaMemsetAsync(s->Jir, 0, jbytes(s), st));
  GASATT_CUDA(ctx, cudaMemsetAsync(s->Jiz, 0, jbytes(s), st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));    // the host arrays zc and charge go out of scope
  return GASATT_OK;
}

int gasatt_sim_read_ions(gasatt_sim *s, double *r, double *z, double *ur, double *ut, double *uz,
                         uint64_t *id, int8_t *charge, int64_t cap, int64_t *n_out, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  if (s->cfg.ion_capacity <= 0) {
    if (n_out) *n_out = 0;
    return GASATT_OK;
  }
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  const unsigned long long nc = s->h_cnt->n_ions;
  const int64_t n = (int64_t)(nc < (unsigned long long)s->cfg.ion_capacity ? nc : s->cfg.ion_capacity);
  if (n_out) *n_out = n;
  if (n > cap) return fail(ctx, GASATT_E_CAPACITY, "read_ions buffer too small");
  if (n == 0) return GASATT_OK;
  if (!r || !z || !ur || !ut || !uz || !id || !charge) return fail(ctx, GASATT_E_ARG, "read_ions: null array");
  double *d[5] = {r, z, ur, ut, uz};
  uint64_t *did = id;
  int8_t *dq = charge;
  if (!on_device) {
    void *buf = nullptr;
    int rc = scratch(ctx, (size_t)n * 49, &buf);
    if (rc) return rc;
    for (int i = 0; i < 5; ++i) d[i] = (double *)buf + (size_t)i * n;
    did = (uint64_t *)((double *)buf + 5 * (size_t)n);
    dq = (int8_t *)(did + n);
  }
  k_ion_read<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->P.ion, d[0], d[1], d[2], d[3], d[4], did, dq, n);
  GASATT_LAUNCHED(ctx);
  if (!on_device) {
    double *h[5] = {r, z, ur, ut, uz};
    for (int i = 0; i < 5; ++i)
      GASATT_CUDA(ctx, cudaMemcpyAsync(h[i], d[i], (size_t)n * 8, cudaMemcpyDeviceToHost, st));
    GASATT_CUDA(ctx, cudaMemcpyAsync(id, did, (size_t)n * 8, cudaMemcpyDeviceToHost, st));
    GASATT_CUDA(ctx, cudaMemcpyAsync(charge, dq, (size_t)n, cudaMemcpyDeviceToHost, st));
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  return GASATT_OK;
}

namespace {
// the gather quads of whole float fields (after the fields are set from outside)
__global__ void k_build_quads(const float *Er, const float *Ez, const float *H, int nr, int nz,
                              int ld, FieldQuads q) {
  const int64_t nE = (int64_t)nr * (nz + 1), nZ = (int64_t)(nr + 1) * nz, nH = (int64_t)nr * nz;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nE + nZ + nH;
       k += (int64_t)gridDim.x * blockDim.x) {
    if (k < nE) {
      const int i = (int)(k % nr), j = (int)(k / nr);
      quad_put(q.er, nr + 1, quad_axis_shifted(i, nr), quad_axis_plain(j, nz), Er[i + (int64_t)j * ld]);
    } else if (k < nE + nZ) {
      const int64_t m = k - nE;
      const int i = (int)(m % (nr + 1)), j = (int)(m / (nr + 1));
      quad_put(q.ez, nr, quad_axis_plain(i, nr), quad_axis_shifted(j, nz), Ez[i + (int64_t)j * ld]);
    } else {
      const int64_t m = k - nE - nZ;
      const int i = (int)(m % nr), j = (int)(m / nr);
      quad_put(q.h, nr + 1, quad_axis_shifted(i, nr), quad_axis_shifted(j, nz), H[i + (int64_t)j * ld]);
    }
  }
}

// dense column-major double (ncol x nrow, the reference's layout) <-> the
// padded internal float layout (row stride ld)
__global__ void k_dense_to_strided(const double *src, float *dst, int ncol, int nrow, int ld) {
  const int64_t n = (int64_t)ncol * nrow;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(k % ncol), j = (int)(k / ncol);
    dst[i + (int64_t)j * ld] = (float)src[k];
  }
}
__global__ void k_strided_to_dense(const float *src, double *dst, int ncol, int nrow, int ld) {
  const int64_t n = (int64_t)ncol * nrow;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(k % ncol), j = (int)(k / ncol);
    dst[k] = (double)src[i + (int64_t)j * ld];
  }
}
__global__ void k_j_to_density(const unsigned long long *J, int nr, int nz, int ldj,
                               double inv_scale, double dr, double dz, double PHIp, double *out) {
  const int64_t n = (int64_t)nr * nz;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(k % nr), j = (int)(k / nr);
    out[k] = (double)(long long)J[i + (int64_t)j * ldj] * inv_scale / shell_volume(i, dr, dz, PHIp);
  }
}

int fields_io(gasatt_sim *s, double *Er, double *Ez, double *H, int on_device, bool set) {
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const int nr = s->cfg.n_r, nz = s->cfg.n_z, ld = s->ldf;
  const int ncol[3] = {nr, nr + 1, nr}, nrow[3] = {nz + 1, nz, nz};
  double *u[3] = {Er, Ez, H};
  void *dev[3] = {s->Er[fcur(s)], s->Ez[fcur(s)], s->H[fcur(s)]};
  if (s->form == 0) {
    // FP64: a pitched copy between the caller's dense array and the padded grid
    for (int f = 0; f < 3; ++f) {
      const size_t w = (size_t)ncol[f] * 8;
      if (set)
        GASATT_CUDA(ctx, cudaMemcpy2DAsync(dev[f], (size_t)ld * 8, u[f], w, w, nrow[f],
                                           on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, st));
      else
        GASATT_CUDA(ctx, cudaMemcpy2DAsync(u[f], w, dev[f], (size_t)ld * 8, w, nrow[f],
                                           on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
    }
    GASATT_CUDA(ctx, cudaStreamSynchronize(st));
    return GASATT_OK;
  }
  // FP32: through a dense double stage on the device when the caller's
  // arrays are host memory
  void *buf = nullptr;
  if (!on_device) {
    int rc = scratch(ctx, (size_t)((int64_t)ncol[0] * nrow[0] + (int64_t)ncol[1] * nrow[1] +
                                   (int64_t)ncol[2] * nrow[2]) * 8, &buf);
    if (rc) return rc;
  }
  int64_t off = 0;
  for (int f = 0; f < 3; ++f) {
    const int64_t n = (int64_t)ncol[f] * nrow[f];
    double *stage = on_device ? u[f] : (double *)buf + off;
    if (set) {
      if (!on_device) GASATT_CUDA(ctx, cudaMemcpyAsync(stage, u[f], n * 8, cudaMemcpyHostToDevice, st));
      k_dense_to_strided<<<grid_for(n, kBlock), kBlock, 0, st>>>(stage, (float *)dev[f], ncol[f], nrow[f], ld);
      GASATT_LAUNCHED(ctx);
    } else {
      k_strided_to_dense<<<grid_for(n, kBlock), kBlock, 0, st>>>((const float *)dev[f], stage, ncol[f], nrow[f], ld);
      GASATT_LAUNCHED(ctx);
      if (!on_device) GASATT_CUDA(ctx, cudaMemcpyAsync(u[f], stage, n * 8, cudaMemcpyDeviceToHost, st));
    }
    off += n;
  }
  if (set && s->quads.er) {
    const int64_t n = (int64_t)nr * (nz + 1) + (int64_t)(nr + 1) * nz + (int64_t)nr * nz;
    k_build_quads<<<grid_for(n, kBlock), kBlock, 0, st>>>(
        (const float *)s->Er[fcur(s)], (const float *)s->Ez[fcur(s)], (const float *)s->H[fcur(s)], nr, nz, ld,
        s->quads);
    GASATT_LAUNCHED(ctx);
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  return GASATT_OK;
}
}  // namespace

int gasatt_sim_set_fields(gasatt_sim *s, const double *Er, const double *Ez, const double *H,
                          int on_device) {
  if (!s) return GASATT_E_ARG;
  return fields_io(s, (double *)Er, (double *)Ez, (double *)H, on_device, true);
}

int gasatt_sim_get_fields(gasatt_sim *s, double *Er, double *Ez, double *H, int on_device) {
  if (!s) return GASATT_E_ARG;
  return fields_io(s, Er, Ez, H, on_device, false);
}

int gasatt_sim_get_current(gasatt_sim *s, double *jr, double *jz, int on_device) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const int nr = s->cfg.n_r, nz = s->cfg.n_z;
  const int64_t n = (int64_t)nr * nz;
  double *d[2] = {jr, jz};
  void *buf = nullptr;
  if (!on_device) {
    int rc = scratch(ctx, (size_t)n * 16, &buf);
    if (rc) return rc;
    d[0] = (double *)buf; d[1] = (double *)buf + n;
  }
  const int q = (int)(s->host_step & 1);   // buffer of the most recent deposit
  const unsigned long long *J[2] = {s->Jr[q], s->Jz[q]};
  for (int f = 0; f < 2; ++f) {
    k_j_to_density<<<grid_for(n, kBlock), kBlock, 0, st>>>(J[f], nr, nz, s->ldj, 1.0 / s->scale,
                                                           s->cfg.dr, s->cfg.dz, s->cfg.PHIp, d[f]);
    GASATT_LAUNCHED(ctx);
  }
  if (!on_device) {
    GASATT_CUDA(ctx, cudaMemcpyAsync(jr, d[0], n * 8, cudaMemcpyDeviceToHost, st));
    GASATT_CUDA(ctx, cudaMemcpyAsync(jz, d[1], n * 8, cudaMemcpyDeviceToHost, st));
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  return GASATT_OK;
}

int gasatt_sim_sort(gasatt_sim *s) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  SIM_TRY(flush_collisions(s));            // the queue holds slot indices
  GASATT_CUDA(ctx, cudaGraphLaunch(s->g_sort[s->cur], ctx->stream));
  ctx->launches += 4;
  s->cur = 1 - s->cur;
  s->since_sort = 0;
  return GASATT_OK;
}

int gasatt_sim_step(gasatt_sim *s, int nsteps) {
  if (!s || nsteps < 0) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  SIM_TRY(sim_prime(s));
  // field update, (FP64: collision kernel,) particle pass
  const int per_step = s->form == 0 ? 3 : 2;
  if (nsteps > 0) SIM_TRY(clear_after_batch(s, st, (int)((s->host_step - 1) & 1)));
  for (int k = 0; k < nsteps; ++k) {
    if (s->cfg.sort_period > 0 && s->since_sort >= s->cfg.sort_period) SIM_TRY(gasatt_sim_sort(s));
    // several steps by one launch: from an even step, up to the next sort and ion push
    int many = 1;
    if (!s->timing && !(s->host_step & 1) && nsteps - k >= kGraphSteps && steps_fit(s, s->cfg.sort_period))
      many = kGraphSteps;
    GASATT_CUDA(ctx, cudaGraphLaunch(many > 1 ? s->g_steps[s->cur] : s->g_step[s->cur][s->host_step & 1], st));
    ctx->launches += many * per_step;
    s->host_step += many;
    s->since_sort += many;
    k += many - 1;
    s->mcc_pending = true;
    if (ion_push_due(s)) SIM_TRY(launch_ion_push(s, st));
  }
  return GASATT_OK;
}

int gasatt_sim_diag(gasatt_sim *s, gasatt_diag *d) {
  if (!s || !d) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaMemsetAsync((char *)s->cnt + offsetof(SimCounters, kin_fx), 0, 16, st));
  if (s->form == 0) k_diag<0><<<s->pass_grid, kBlock, 0, st>>>(s->s64[s->cur], s->s32[s->cur], s->cnt, s->cfg.c, s->cfg.m_e, s->cfg.q_e);
  else k_diag<1><<<s->pass_grid, kBlock, 0, st>>>(s->s64[s->cur], s->s32[s->cur], s->cnt, s->cfg.c, s->cfg.m_e, s->cfg.q_e);
  GASATT_LAUNCHED(ctx);
  if (s->cfg.ion_capacity > 0) {
    GASATT_CUDA(ctx, cudaMemsetAsync((char *)s->cnt + offsetof(SimCounters, ion_alive), 0, 24, st));
    k_ion_diag<<<s->pass_grid, kBlock, 0, st>>>(s->P.ion, s->cfg.ion_capacity, s->cnt, s->cfg.c,
                                                  s->cfg.m_ion, s->cfg.q_e);
    GASATT_LAUNCHED(ctx);
  }
  const int nr = s->cfg.n_r, nz = s->cfg.n_z;
  if (s->form == 0)
    k_field_energy<double><<<s->partial_blocks, kBlock, 0, st>>>((double *)s->Er[fcur(s)], (double *)s->Ez[fcur(s)], (double *)s->H[fcur(s)], nr, nz, s->ldf, s->cfg.dr, s->cfg.dz, s->partial);
  else
    k_field_energy<float><<<s->partial_blocks, kBlock, 0, st>>>((float *)s->Er[fcur(s)], (float *)s->Ez[fcur(s)], (float *)s->H[fcur(s)], nr, nz, s->ldf, s->cfg.dr, s->cfg.dz, s->partial);
  GASATT_LAUNCHED(ctx);
  std::vector<double> part(2 * s->partial_blocks);
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaMemcpyAsync(part.data(), s->partial, part.size() * 8, cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  const SimCounters &h = *s->h_cnt;
  double we = 0, wm = 0;
  for (int b = 0; b < s->partial_blocks; ++b) { we += part[2 * b]; wm += part[2 * b + 1]; }
  d->n_alive = (int64_t)h.alive;
  d->n_total = (int64_t)(h.n_total + h.n_births < h.cap ? h.n_total + h.n_births : h.cap);
  d->n_ionizations = (int64_t)h.ion;
  d->n_elastic = (int64_t)h.ela;
  d->n_excitation = (int64_t)h.exc;
  d->n_null = (int64_t)h.nul;
  d->n_lost_wall = (int64_t)h.lost;
  d->n_ions = (int64_t)h.ion_alive;
  d->kinetic_ev = (double)h.kin_fx / 65536.0;
  d->field_energy_j = s->cfg.PHIp * 0.5 * s->cfg.eps0 * we + s->cfg.PHIp * 0.5 * s->cfg.mu0 * wm;
  d->steps = s->host_step;
  d->status_flags = (h.cap_overflow ? 2 : 0) | (h.ion_overflow ? 4 : 0) |
                    (h.fdtd_err || h.scan_err ? 8 : 0);
  d->n_ion_lost_wall = (int64_t)h.ion_lost;
  d->ion_kinetic_ev = (double)h.ion_kin_fx / 4294967296.0;
  d->net_charge_c = s->cfg.q_e * s->cfg.FN * ((double)h.ion_charge - (double)h.alive);
  d->collision_loss_ev = GASATT_ION_I_EV * (double)h.ion + (double)h.exc_loss_fx / 65536.0;
  d->wall_loss_ev = (double)h.wall_loss_fx / 65536.0;
  return GASATT_OK;
}

int gasatt_sim_counts(gasatt_sim *s, int64_t *n_slots, int64_t *n_ion, int64_t *n_lost) {
  if (!s) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  SIM_TRY(flush_collisions(s));
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, ctx->stream));
  GASATT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const SimCounters &h = *s->h_cnt;
  const unsigned long long nt = h.n_total + h.n_births;
  if (n_slots) *n_slots = (int64_t)(nt < h.cap ? nt : h.cap);
  if (n_ion) *n_ion = (int64_t)h.ion;
  if (n_lost) *n_lost = (int64_t)h.lost;
  return GASATT_OK;
}

int gasatt_sim_enable_timing(gasatt_sim *s, int enable) {
  if (!s) return GASATT_E_ARG;
  if ((bool)enable == s->timing) return GASATT_OK;
  GASATT_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  GASATT_CUDA(s->ctx, cudaStreamSynchronize(s->ctx->stream));
  drop_step_graphs(s);
  s->timing = enable != 0;
  return build_graphs(s);
}

int gasatt_sim_last_timing(gasatt_sim *s, float *fdtd_ms, float *pass_ms, float *mcc_ms) {
  if (!s) return GASATT_E_ARG;
  if (!s->timing) return fail(s->ctx, GASATT_E_STATE, "timing not enabled");
  GASATT_CUDA(s->ctx, cudaEventSynchronize(s->ev[3]));
  float a = 0, b = 0, m = 0;
  GASATT_CUDA(s->ctx, cudaEventElapsedTime(&a, s->ev[0], s->ev[1]));
  if (s->form == 1) {
    // FP32: the pass runs the collisions itself; no separate collision kernel
    GASATT_CUDA(s->ctx, cudaEventElapsedTime(&b, s->ev[1], s->ev[3]));
  } else {
    GASATT_CUDA(s->ctx, cudaEventElapsedTime(&b, s->ev[2], s->ev[3]));
    GASATT_CUDA(s->ctx, cudaEventElapsedTime(&m, s->ev[4], s->ev[5]));
  }
  if (fdtd_ms) *fdtd_ms = a;
  if (pass_ms) *pass_ms = b;
  if (mcc_ms) *mcc_ms = m;
  return GASATT_OK;
}

}  // extern "C"

namespace {

// Cartesian (x, y, z, v) columns -> axisymmetric state (r, z, u = gamma v local), id = slot
__global__ void k_cart_in(const double *pos, const double *vel, int64_t ld, int64_t n, double c,
                          double *r, double *z, double *ur, double *ut, double *uz, uint64_t *id,
                          uint64_t id_base) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const double x = pos[p], y = pos[ld + p];
    const double vx = vel[p], vy = vel[ld + p], vz = vel[2 * ld + p];
    const double rr = sqrt(x * x + y * y);
    const double cp = rr > 0 ? x / rr : 1.0, sp = rr > 0 ? y / rr : 0.0;
    const double g = 1 / sqrt(1 - (vx * vx + vy * vy + vz * vz) / (c * c));
    r[p] = rr; z[p] = pos[2 * ld + p];
    ur[p] = g * (vx * cp + vy * sp); ut[p] = g * (-vx * sp + vy * cp); uz[p] = g * vz;
    id[p] = id_base + (uint64_t)p;
  }
}

// axisymmetric state -> Cartesian columns at azimuth 0, velocity v = u / gamma
__global__ void k_cart_out(const double *r, const double *z, const double *ur, const double *ut,
                           const double *uz, int64_t n, double c, double *pos, double *vel,
                           int64_t ld) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const double g = sqrt(1 + (ur[p] * ur[p] + ut[p] * ut[p] + uz[p] * uz[p]) / (c * c));
    pos[p] = r[p]; pos[ld + p] = 0.0; pos[2 * ld + p] = z[p];
    vel[p] = ur[p] / g; vel[ld + p] = ut[p] / g; vel[2 * ld + p] = uz[p] / g;
  }
}

}  // namespace

extern "C" {

int gasatt_sim_run_host(gasatt_sim *s, double *pos, double *vel, int64_t *n_io, int64_t cap,
                        int nsteps) {
  if (!s || !n_io || nsteps < 1) return GASATT_E_ARG;
  gasatt_ctx *ctx = s->ctx;
  const int64_t n = *n_io;
  if (n < 0 || n > cap || n > s->cfg.capacity) return fail(ctx, GASATT_E_ARG, "run_host: bad count");
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  // device staging: 6 columns in, reused for the way out; plus state scratch
  void *buf;
  const int64_t m = s->cfg.capacity;
  int rc = scratch(ctx, (size_t)m * 8 * 12, &buf);
  if (rc) return rc;
  double *dpos = (double *)buf, *dvel = dpos + 3 * m;
  double *sr = dvel + 3 * m, *sz = sr + m, *sur = sz + m, *sut = sur + m, *suz = sut + m;
  uint64_t *sid = (uint64_t *)(suz + m);
  for (int d = 0; d < 3; ++d) {
    GASATT_CUDA(ctx, cudaMemcpyAsync(dpos + d * m, pos + d * cap, (size_t)n * 8, cudaMemcpyHostToDevice, st));
    GASATT_CUDA(ctx, cudaMemcpyAsync(dvel + d * m, vel + d * cap, (size_t)n * 8, cudaMemcpyHostToDevice, st));
  }
  // the step counter keeps running across calls, so (id = slot, step) never repeats
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  if (n > 0) {
    k_cart_in<<<grid_for(n, kBlock), kBlock, 0, st>>>(dpos, dvel, m, n, s->cfg.c, sr, sz, sur, sut, suz, sid, 0);
    GASATT_LAUNCHED(ctx);
    if (s->form == 0)
      k_load64<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s64[s->cur], sr, sz, sur, sut, suz, sid, n);
    else
      k_load32<<<grid_for(n, kBlock), kBlock, 0, st>>>(s->s32[s->cur], sr, sz, sur, sut, suz, sid, n,
                                                       s->cfg.n_r, s->cfg.n_z, s->cfg.dr, s->cfg.dz, s->cfg.c,
                                                       (int)(((s->h_cnt->step + 1) & 1) ^ 1));
    GASATT_LAUNCHED(ctx);
  }
  SimCounters h = *s->h_cnt;
  h.n_total = (unsigned long long)n;
  h.n_births = 0;
  h.n_cand[0] = h.n_cand[1] = 0;
  h.chunk_next = 0;
  set_chunk(s, h);
  h.step += 1;                               // never reuse the last pass's step
  h.step64[0] = h.step64[1] = (h.step64[0] > h.step64[1] ? h.step64[0] : h.step64[1]) + 1;   // the prologue runs one later
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->cnt, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  for (int q = 0; q < 2; ++q) {
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jr[q], 0, jbytes(s), st));
    GASATT_CUDA(ctx, cudaMemsetAsync(s->Jz[q], 0, jbytes(s), st));
  }
  s->primed = false;
  s->mcc_pending = false;
  s->batch_pass = false;
  s->uncommitted = false;
  SIM_TRY(restart_steps(s, st));             // the prologue deposits into buffer 0
  s->since_sort = s->cfg.sort_period;       // sort the fresh population first
  SIM_TRY(gasatt_sim_step(s, nsteps - 1));
  // last step: the pending collisions, the fields, then a push that ends at
  // integer time
  SIM_TRY(flush_collisions(s));
  SIM_TRY(launch_fdtd(s, st, (int)(s->host_step & 1)));
  SIM_TRY(launch_pass(s, st, 2, (int)((s->host_step + 1) & 1), (int)(s->host_step & 1),
                      (int)((s->host_step + 1) & 1)));
  SIM_TRY(gasatt_sim_sort(s));               // compacts away the dead
  s->host_step++;
  s->primed = false;
  s->uncommitted = true;
  GASATT_CUDA(ctx, cudaMemcpyAsync(s->h_cnt, s->cnt, sizeof(SimCounters), cudaMemcpyDeviceToHost, st));
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  const int64_t nout = (int64_t)s->h_cnt->n_total;
  const int64_t nw = nout < cap ? nout : cap;
  if (nw > 0) {
    if (s->form == 0)
      k_read64<<<grid_for(nw, kBlock), kBlock, 0, st>>>(s->s64[s->cur], sr, sz, sur, sut, suz, sid, nw);
    else
      k_read32<<<grid_for(nw, kBlock), kBlock, 0, st>>>(s->s32[s->cur], sr, sz, sur, sut, suz, sid, nw,
                                                        s->cfg.dr, s->cfg.dz, s->cfg.c);
    GASATT_LAUNCHED(ctx);
    k_cart_out<<<grid_for(nw, kBlock), kBlock, 0, st>>>(sr, sz, sur, sut, suz, nw, s->cfg.c, dpos, dvel, m);
    GASATT_LAUNCHED(ctx);
    for (int d = 0; d < 3; ++d) {
      GASATT_CUDA(ctx, cudaMemcpyAsync(pos + d * cap, dpos + d * m, (size_t)nw * 8, cudaMemcpyDeviceToHost, st));
      GASATT_CUDA(ctx, cudaMemcpyAsync(vel + d * cap, dvel + d * m, (size_t)nw * 8, cudaMemcpyDeviceToHost, st));
    }
  }
  GASATT_CUDA(ctx, cudaStreamSynchronize(st));
  *n_io = nw;
  if (nout > cap) return fail(ctx, GASATT_E_CAPACITY, "run_host: more electrons than cap rows");
  return GASATT_OK;
}

// ================================================================ batches
// Many independent gas cells stepped together.  Cells of the same precision
// form and field patch (fdtd_ratio 1) form a group that runs each step as a
// few launches for the whole group - the field update over every cell's
// tiles (k_batch_fdtd_tma), (FP64: the emptying of the next queues and the collisions beside it,)
// then the particle pass over every cell's candidates and chunks
// (k_batch_pass32 / k_batch_pass64) - instead of one set of launches per
// cell, so the blocks of each launch share all cells' work and small cells
// do not leave the GPU idle.  Groups, and any cell that fits no group
// (fdtd_ratio > 1), run side by side as branches of one graph.  The cells
// share a sort period, so they swap state buffers in lockstep; if one is
// ever out of step (stepped on its own in between), the batch steps each
// cell with its own graph.
struct BatchGroup {
  int form = 0, ph = 0;                  // ph: patch shape (0 until set up: chosen for the group)
  std::vector<gasatt_sim *> sims;
  void *cells = nullptr;                 // BatchCell32 / BatchCell64 per cell
  FdtdInst *insts[2] = {nullptr, nullptr};   // per step parity (the current buffer read)
  int2 *table = nullptr;                 // (cell, tile) work items of the field update
  int nitems = 0;
  SimCounters **commit = nullptr;        // FP32: counters the field update commits
  unsigned long long *chunk_next = nullptr;
  unsigned fdtd_grid = 0, pass_grid = 0, mcc_grid = 0;
  size_t fdtd_smem = 0;
  bool wide = false;                     // a cell's grid is wider than a deposit box
};

struct gasatt_batch {
  gasatt_ctx *ctx = nullptr;
  std::vector<gasatt_sim *> sims;
  std::vector<BatchGroup> groups;
  std::vector<gasatt_sim *> singles;     // cells stepped by their own step graph
  std::vector<void *> allocs;
  int sort_period = 0;
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
  cudaGraphExec_t g[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [state buffer][parity]
  cudaGraphExec_t g_steps[2] = {nullptr, nullptr};  // kGraphSteps steps from parity 0 on [state buffer]
  int64_t lone[2] = {0, 0}, worth = 0;   // steps taken without g_steps that it fits, and how many of them it is worth
  cudaGraphExec_t g_sort[2] = {nullptr, nullptr};   // every cell's sort side by side [state buffer]
};

int gasatt_batch_destroy(gasatt_batch *b) {
  if (!b) return GASATT_OK;
  cudaSetDevice(b->ctx->device);
  cudaStreamSynchronize(b->ctx->stream);
  for (int i = 0; i < 2; ++i) {
    for (int q = 0; q < 2; ++q)
      if (b->g[i][q]) cudaGraphExecDestroy(b->g[i][q]);
    if (b->g_steps[i]) cudaGraphExecDestroy(b->g_steps[i]);
    if (b->g_sort[i]) cudaGraphExecDestroy(b->g_sort[i]);
  }
  if (b->fork_ev) cudaEventDestroy(b->fork_ev);
  if (b->join_ev) cudaEventDestroy(b->join_ev);
  for (void *p : b->allocs) cudaFree(p);
  delete b;
  return GASATT_OK;
}

extern "C++" {
namespace {

template <typename T>
int batch_alloc(gasatt_batch *b, T **p, size_t n) {
  cudaError_t e = cudaMalloc((void **)p, (n ? n : 1) * sizeof(T));
  if (e != cudaSuccess) return cuda_fail(b->ctx, e, "cudaMalloc (batch)");
  b->allocs.push_back((void *)*p);
  return GASATT_OK;
}

// device tables of a group: the cells' pass and field-update descriptors,
// the field update's work items, the commit list, the chunk counter, grids
int batch_group_setup(gasatt_batch *b, BatchGroup &G) {
  gasatt_ctx *ctx = b->ctx;
  const int n = (int)G.sims.size();
  if (G.form == 1) {
    std::vector<BatchCell32> h(n);
    std::vector<SimCounters *> cm(n);
    for (int i = 0; i < n; ++i) {
      gasatt_sim *s = G.sims[i];
      for (int jb = 0; jb < 2; ++jb) {
        h[i].P[jb] = s->P;
        h[i].P[jb].Jr = s->Jr[jb]; h[i].P[jb].Jz = s->Jz[jb];
      }
      h[i].S[0] = s->s32[0]; h[i].S[1] = s->s32[1];
      h[i].cnt = s->cnt; h[i].queue = s->queue;
      for (int k = 0; k < 2; ++k) h[i].F[k] = Fields<float>{(float *)s->Er[k], (float *)s->Ez[k], (float *)s->H[k]};
      cm[i] = s->cnt;
    }
    BatchCell32 *d;
    SIM_TRY(batch_alloc(b, &d, (size_t)n));
    GASATT_CUDA(ctx, cudaMemcpy(d, h.data(), sizeof(BatchCell32) * n, cudaMemcpyHostToDevice));
    G.cells = d;
    SIM_TRY(batch_alloc(b, &G.commit, (size_t)n));
    GASATT_CUDA(ctx, cudaMemcpy(G.commit, cm.data(), sizeof(SimCounters *) * n, cudaMemcpyHostToDevice));
  } else {
    std::vector<BatchCell64> h(n);
    for (int i = 0; i < n; ++i) {
      gasatt_sim *s = G.sims[i];
      for (int jb = 0; jb < 2; ++jb) {
        h[i].P[jb] = s->P;
        h[i].P[jb].Jr = s->Jr[jb]; h[i].P[jb].Jz = s->Jz[jb];
      }
      h[i].S[0] = s->s64[0]; h[i].S[1] = s->s64[1];
      h[i].cnt = s->cnt; h[i].queue = s->queue;
      for (int k = 0; k < 2; ++k) h[i].F[k] = Fields<double>{(double *)s->Er[k], (double *)s->Ez[k], (double *)s->H[k]};
    }
    BatchCell64 *d;
    SIM_TRY(batch_alloc(b, &d, (size_t)n));
    GASATT_CUDA(ctx, cudaMemcpy(d, h.data(), sizeof(BatchCell64) * n, cudaMemcpyHostToDevice));
    G.cells = d;
  }
  const int nsm = ctx->sms;
  // one patch shape for the group: its cells' own knob value, or by all their tiles
  if (!G.ph) {
    long long t12 = 0, t16 = 0;
    for (const gasatt_sim *s : G.sims) {
      t12 += tma_tiles(12, s->cfg.n_r, s->cfg.n_z);
      t16 += tma_tiles(16, s->cfg.n_r, s->cfg.n_z);
    }
    G.ph = tma_auto(t12, t16, nsm);
  }
  std::vector<int2> table;
  for (int i = 0; i < n; ++i)
    for (int t = 0; t < tma_tiles(G.ph, G.sims[i]->cfg.n_r, G.sims[i]->cfg.n_z); ++t) table.push_back(make_int2(i, t));
  G.nitems = (int)table.size();
  SIM_TRY(batch_alloc(b, &G.table, table.size()));
  GASATT_CUDA(ctx, cudaMemcpy(G.table, table.data(), sizeof(int2) * table.size(), cudaMemcpyHostToDevice));
  for (int q = 0; q < 2; ++q) {
    std::vector<FdtdInst> hi(n);
    for (int i = 0; i < n; ++i)
      SIM_TRY(G.form == 1 ? fdtd_inst_of<float>(G.sims[i], G.ph, q, hi[i])
                          : fdtd_inst_of<double>(G.sims[i], G.ph, q, hi[i]));
    SIM_TRY(batch_alloc(b, &G.insts[q], (size_t)n));
    GASATT_CUDA(ctx, cudaMemcpy(G.insts[q], hi.data(), sizeof(FdtdInst) * n, cudaMemcpyHostToDevice));
  }
  SIM_TRY(batch_alloc(b, &G.chunk_next, 1));
  int occ = 1;
  G.fdtd_smem = G.form == 1 ? tma_block_bytes<float>(G.ph) : tma_block_bytes<double>(G.ph);
  const BatchFdtdTmaFn fk = G.form == 1 ? batch_fdtd_tma_fn<float>(G.ph) : batch_fdtd_tma_fn<double>(G.ph);
  GASATT_CUDA(ctx, cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G.fdtd_smem));
  GASATT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fk, 32 * tma_warps(G.ph), G.fdtd_smem));
  const long long fslots = (long long)nsm * (occ > 0 ? occ : 1);
  const long long fblocks = G.nitems;
  G.fdtd_grid = (unsigned)(fslots < fblocks ? fslots : (fblocks > 0 ? fblocks : 1));
  occ = 1;
  for (const gasatt_sim *s : G.sims) G.wide = G.wide || win_cols(s->cfg.n_r) < s->cfg.n_r;
  if (G.form == 1) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_pass32<true>, kBlock, 0);
  else {
    GASATT_CUDA(ctx, cudaFuncSetAttribute(k_batch_pass64, cudaFuncAttributeMaxDynamicSharedMemorySize, kWin64Bytes));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_pass64, kBlock, kWin64Bytes);
  }
  G.pass_grid = (unsigned)(nsm * (occ > 0 ? occ : 1));
  occ = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_mcc64, kMccBlock, 0);
  G.mcc_grid = (unsigned)(nsm * (occ > 0 ? occ : 1));
  return GASATT_OK;
}

// one step of group G (state buffer cur, step parity q) onto the capturing
// stream cs (side: a second stream for the FP64 collision branch).  FP32: both
// kernels start early (but for a graph's first); FP64: neither, since the
// collisions start with the field update and would find its blocks in their
// slots (6 cells 115.7 -> 123 us a step, with the spills that the signal costs
// the pass)
int batch_group_launch(gasatt_batch *b, BatchGroup &G, cudaStream_t cs, cudaStream_t side, int cur,
                       int q, bool first) {
  gasatt_ctx *ctx = b->ctx;
  const int n = (int)G.sims.size();
  const dim3 fb(32 * tma_warps(G.ph));
  if (G.form == 1) {
    GASATT_CUDA(ctx, launch_early(!first, batch_fdtd_tma_fn<float>(G.ph), dim3(G.fdtd_grid), fb, G.fdtd_smem, cs,
                                  G.insts[q], G.table, G.nitems, G.commit, n, G.chunk_next));
    GASATT_CUDA(ctx, launch_early(true, G.wide ? k_batch_pass32<true> : k_batch_pass32<false>, dim3(G.pass_grid),
                                  dim3(kBlock), 0, cs, (const BatchCell32 *)G.cells, n, cur, 1 - q, G.chunk_next));
    return GASATT_OK;
  }
  GASATT_CUDA(ctx, cudaEventRecord(b->fork_ev, cs));
  GASATT_CUDA(ctx, cudaStreamWaitEvent(side, b->fork_ev, 0));
  k_batch_clear_next64<<<1, 256, 0, side>>>((const BatchCell64 *)G.cells, n, 1 - q);
  k_batch_mcc64<<<G.mcc_grid, kMccBlock, 0, side>>>((const BatchCell64 *)G.cells, n, cur, 1 - q);
  GASATT_CUDA(ctx, cudaGetLastError());
  GASATT_CUDA(ctx, cudaEventRecord(b->join_ev, side));
  batch_fdtd_tma_fn<double>(G.ph)<<<G.fdtd_grid, fb, G.fdtd_smem, cs>>>(G.insts[q], G.table, G.nitems, nullptr, n,
                                                                       G.chunk_next);
  GASATT_CUDA(ctx, cudaGetLastError());
  GASATT_CUDA(ctx, cudaStreamWaitEvent(cs, b->join_ev, 0));
  k_batch_pass64<<<G.pass_grid, kBlock, kWin64Bytes, cs>>>((const BatchCell64 *)G.cells, n, cur, 1 - q, q,
                                                           G.chunk_next);
  GASATT_CUDA(ctx, cudaGetLastError());
  return GASATT_OK;
}

// `count` steps of the batch (state buffer bi, the first of parity q) as one
// graph: a branch per group and per cell of its own, each its steps in turn
int batch_capture_steps(gasatt_batch *b, cudaStream_t cs, cudaStream_t side, int bi, int q, int count,
                        cudaGraphExec_t *exec) {
  gasatt_ctx *ctx = b->ctx;
  int rc = GASATT_OK;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaGraphCreate(&g, 0);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "batch graph");
  for (BatchGroup &G : b->groups) {
    cudaGraph_t child = nullptr;
    e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) { rc = cuda_fail(ctx, e, "batch capture"); break; }
    for (int k = 0; k < count && !rc; ++k) rc = batch_group_launch(b, G, cs, side, bi, (q + k) & 1, k == 0);
    const cudaError_t e2 = cudaStreamEndCapture(cs, &child);
    if (!rc && e2 != cudaSuccess) rc = cuda_fail(ctx, e2, "batch capture");
    if (!rc) {
      cudaGraphNode_t node;
      e = cudaGraphAddChildGraphNode(&node, g, nullptr, 0, child);
      if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch graph");
    }
    if (child) cudaGraphDestroy(child);
    if (rc) break;
  }
  for (size_t i = 0; i < b->singles.size() && !rc; ++i) {
    cudaGraphNode_t last, node;
    for (int k = 0; k < count && !rc; ++k, last = node) {
      e = cudaGraphAddChildGraphNode(&node, g, k > 0 ? &last : nullptr, k > 0 ? 1 : 0,
                                     b->singles[i]->gr_step[bi][(q + k) & 1]);
      if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch graph");
    }
  }
  if (!rc) {
    e = cudaGraphInstantiate(exec, g, 0);
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch graph");
  }
  cudaGraphDestroy(g);
  return rc;
}

// This thread's calls are not bound, for the time of this object, by a capture that another
// thread of the program has under way: building a graph would fail, and spoil that capture.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// two capturing streams for the time of `build`
template <typename F>
int with_capture_streams(gasatt_ctx *ctx, F build) {
  const RelaxedCapture relaxed;
  cudaStream_t cs, side;
  GASATT_CUDA(ctx, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  const cudaError_t e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    cudaStreamDestroy(cs);
    return cuda_fail(ctx, e, "batch: stream");
  }
  const int rc = build(cs, side);
  cudaStreamDestroy(side);
  cudaStreamDestroy(cs);
  return rc;
}

int batch_build_graphs(gasatt_batch *b, cudaStream_t cs, cudaStream_t side) {
  gasatt_ctx *ctx = b->ctx;
  int rc = GASATT_OK;
  for (int bi = 0; bi < 2 && !rc; ++bi) {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) { rc = cuda_fail(ctx, e, "batch sort graph"); break; }
    for (size_t i = 0; i < b->sims.size() && !rc; ++i) {
      cudaGraphNode_t node;
      e = cudaGraphAddChildGraphNode(&node, g, nullptr, 0, b->sims[i]->gr_sort[bi]);
      if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch sort graph");
    }
    if (!rc) {
      e = cudaGraphInstantiate(&b->g_sort[bi], g, 0);
      if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch sort graph");
    }
    cudaGraphDestroy(g);
  }
  for (int bi = 0; bi < 2 && !rc; ++bi)
    for (int q = 0; q < 2 && !rc; ++q) rc = batch_capture_steps(b, cs, side, bi, q, 1, &b->g[bi][q]);
  // A graph of ten steps gives 4 to 6 us a step and costs, to build and to
  // destroy, 0.2 ms for chains of kernels and 1.2 ms more for each branch with the
  // FP64 form's forks (0.12 ms a fork): it is built once as many steps were taken without
  // it.  Both built at once, the creation of a batch took 4.2 ms (FP64) and 2.0 ms
  // (FP32); now 2.2 ms and 1.8 ms.
  b->worth = 40;
  for (const BatchGroup &G : b->groups) b->worth += G.form == 0 ? 320 : 0;
  for (const gasatt_sim *s : b->singles) b->worth += s->form == 0 ? 320 : 0;
  return rc;
}

// Whether the graph of ten steps is there, or worth building now (and built).  A batch that
// cannot build it, for want of memory say, goes on without.
bool batch_steps_ready(gasatt_batch *b, int cur) {
  if (!b->g_steps[cur] && b->lone[cur] >= b->worth) {
    const std::string err = b->ctx->err;
    const int rc = with_capture_streams(b->ctx, [&](cudaStream_t cs, cudaStream_t side) {
      return batch_capture_steps(b, cs, side, cur, 0, kGraphSteps, &b->g_steps[cur]);
    });
    if (rc) {
      cudaGetLastError();                  // (the capture's end may have left one)
      b->g_steps[cur] = nullptr;
      b->worth = INT64_MAX;
      b->ctx->err = err;
    }
  }
  if (b->g_steps[cur]) return true;
  b->lone[cur] += 2;                       // (asked at every other step)
  return false;
}

// flush_collisions for every cell of the batch (before its sort): a group
// whose cells are at the same step parity and state buffer does it in two
// launches (FP32: k_batch_collide32) or three (FP64: k_batch_clear_next64, then
// k_batch_mcc64) for all of its cells, then empties their queues; any other
// cell flushes on its own.  A cell with nothing pending finds an empty queue
// (its own flush emptied it).
int batch_flush_collisions(gasatt_batch *b) {
  gasatt_ctx *ctx = b->ctx;
  cudaStream_t st = ctx->stream;
  for (BatchGroup &G : b->groups) {
    const gasatt_sim *s0 = G.sims[0];
    bool same = true, any = false;
    for (const gasatt_sim *s : G.sims) {
      same = same && s->cur == s0->cur && (s->host_step & 1) == (s0->host_step & 1);
      any = any || s->mcc_pending;
    }
    if (!any) continue;
    if (!same) {
      for (gasatt_sim *s : G.sims) SIM_TRY(flush_collisions(s));
      continue;
    }
    const int n = (int)G.sims.size(), cur = s0->cur, q = (int)((s0->host_step - 1) & 1);
    if (G.form == 1) {
      k_batch_collide32<<<G.pass_grid, kMccBlock, 0, st>>>((const BatchCell32 *)G.cells, n, cur);
      k_batch_clear_cand<<<1, 256, 0, st>>>((const BatchCell32 *)G.cells, n, -1);   // see flush_collisions
      ctx->launches += 2;
    } else {
      k_batch_clear_next64<<<1, 256, 0, st>>>((const BatchCell64 *)G.cells, n, q);
      k_batch_mcc64<<<G.mcc_grid, kMccBlock, 0, st>>>((const BatchCell64 *)G.cells, n, cur, q);
      k_batch_clear_cand<<<1, 256, 0, st>>>((const BatchCell64 *)G.cells, n, q);
      ctx->launches += 3;
    }
    GASATT_CUDA(ctx, cudaGetLastError());
    for (gasatt_sim *s : G.sims) s->mcc_pending = false;
  }
  for (gasatt_sim *s : b->singles) SIM_TRY(flush_collisions(s));
  return GASATT_OK;
}

}  // namespace
}  // extern "C++"

int gasatt_batch_create(gasatt_ctx *ctx, gasatt_sim *const *sims, int n, int sort_period,
                        gasatt_batch **out) {
  if (!ctx || !sims || n < 1 || !out || sort_period < 0)
    return fail(ctx, GASATT_E_ARG, "batch: bad arguments");
  *out = nullptr;
  for (int i = 0; i < n; ++i) {
    if (!sims[i] || sims[i]->ctx != ctx)
      return fail(ctx, GASATT_E_ARG, "batch: every instance must belong to this context");
    if (sims[i]->timing) return fail(ctx, GASATT_E_STATE, "batch: disable phase timing first");
    for (int j = 0; j < i; ++j)
      if (sims[j] == sims[i]) return fail(ctx, GASATT_E_ARG, "batch: an instance appears twice");
  }
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  gasatt_batch *b = new gasatt_batch();
  b->ctx = ctx;
  b->sims.assign(sims, sims + n);
  b->sort_period = sort_period;
  for (gasatt_sim *s : b->sims) s->cfg.sort_period = sort_period;
  // groups of cells with the same form and field patch; up to kMaxBatch each
  for (gasatt_sim *s : b->sims) {
    if (s->cfg.fdtd_ratio != 1) { b->singles.push_back(s); continue; }
    BatchGroup *G = nullptr;
    for (BatchGroup &g : b->groups)
      if (g.form == s->form && g.ph == s->cfg.fdtd_tile_rows && (int)g.sims.size() < kMaxBatch) G = &g;
    if (!G) {
      b->groups.emplace_back();
      G = &b->groups.back();
      G->form = s->form;
      G->ph = s->cfg.fdtd_tile_rows;
    }
    G->sims.push_back(s);
  }
  int rc = GASATT_OK;
  if (cudaEventCreateWithFlags(&b->fork_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->join_ev, cudaEventDisableTiming) != cudaSuccess)
    rc = fail(ctx, GASATT_E_CUDA, "batch: event");
  for (size_t i = 0; i < b->groups.size() && !rc; ++i) rc = batch_group_setup(b, b->groups[i]);
  if (!rc) rc = with_capture_streams(ctx, [&](cudaStream_t cs, cudaStream_t side) { return batch_build_graphs(b, cs, side); });
  if (rc) {
    gasatt_batch_destroy(b);
    return rc;
  }
  *out = b;
  return GASATT_OK;
}

int gasatt_batch_step(gasatt_batch *b, int nsteps) {
  if (!b || nsteps < 0) return GASATT_E_ARG;
  gasatt_ctx *ctx = b->ctx;
  GASATT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  for (int k = 0; k < nsteps; ++k) {
    for (gasatt_sim *s : b->sims) SIM_TRY(sim_prime(s));
    if (b->sort_period > 0) {
      // every cell due at once (the batch keeps them in lockstep): one graph
      // sorts them all side by side
      bool all_due = true;
      for (const gasatt_sim *s : b->sims)
        all_due = all_due && s->since_sort >= b->sort_period && s->cur == b->sims[0]->cur;
      if (all_due) {
        SIM_TRY(batch_flush_collisions(b));
        GASATT_CUDA(ctx, cudaGraphLaunch(b->g_sort[b->sims[0]->cur], st));
        for (gasatt_sim *s : b->sims) {
          ctx->launches += 4;
          s->cur = 1 - s->cur;
          s->since_sort = 0;
        }
      } else {
        for (gasatt_sim *s : b->sims)
          if (s->since_sort >= b->sort_period) SIM_TRY(gasatt_sim_sort(s));
      }
    }
    const gasatt_sim *s0 = b->sims[0];
    bool lockstep = true;
    // several steps by one launch: from an even step, up to every cell's next sort and ion push
    int many = !(s0->host_step & 1) && nsteps - k >= kGraphSteps ? kGraphSteps : 1;
    for (const gasatt_sim *s : b->sims) {
      lockstep = lockstep && s->cur == s0->cur && (s->host_step & 1) == (s0->host_step & 1) &&
                 !s->timing;
      if (!steps_fit(s, b->sort_period)) many = 1;
    }
    if (!lockstep) many = 1;
    if (many > 1 && !batch_steps_ready(b, s0->cur)) many = 1;
    if (lockstep) {
      GASATT_CUDA(ctx, cudaGraphLaunch(many > 1 ? b->g_steps[s0->cur] : b->g[s0->cur][s0->host_step & 1], st));
      for (const BatchGroup &G : b->groups) ctx->launches += many * (G.form == 0 ? 4 : 2);
      for (const gasatt_sim *s : b->singles) ctx->launches += many * (s->form == 0 ? 3 : 2);
      for (const BatchGroup &G : b->groups)
        for (gasatt_sim *s : G.sims) s->batch_pass = true;
    } else {
      for (gasatt_sim *s : b->sims) {
        SIM_TRY(clear_after_batch(s, st, (int)((s->host_step - 1) & 1)));
        GASATT_CUDA(ctx, cudaGraphLaunch(s->g_step[s->cur][s->host_step & 1], st));
        ctx->launches += s->form == 0 ? 3 : 2;
      }
    }
    for (gasatt_sim *s : b->sims) {
      s->host_step += many;
      s->since_sort += many;
      s->mcc_pending = true;
      if (ion_push_due(s)) SIM_TRY(launch_ion_push(s, st));
    }
    k += many - 1;
  }
  return GASATT_OK;
}

}  // extern "C"
