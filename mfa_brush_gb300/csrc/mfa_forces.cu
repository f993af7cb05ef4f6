// mfa_forces.cu -- force kernels of the MD-DPD step.
//
// k_pair   : fluid_fluid.f90:97-261 with dpd_forces.f90:45-115 and ewald_real.f90:15-33 fused.
//            One thread per particle walks its full Verlet list (no atomics, no Newton-3 scatter);
//            each unordered pair is therefore evaluated from both sides, and the DPD noise is a
//            Philox draw keyed on (seed, step, min tag, max tag) so both sides see the same g and
//            momentum is conserved exactly in exact arithmetic.  Energies are halved per visit
//            (a fixed wall bead has no list: its pairs count in full).
//            k_pair is the mixed mode's: positions are fixed-point int4 (the int32 difference is the x,y minimum image),
//            all pair arithmetic is FP32.  In the fused mixed step the FP32 partial sums over each
//            batch of kept pairs go into an FP64 per-particle total, with the particle's bonded
//            terms (evaluated by the same thread), its 9-3 wall force and the body force; in the
//            drop-in the FP32 sum is added to the FP64 force.  With a single cut-off for every
//            type pair the screening compares against one constant (UNI).  With energies, the
//            pair, bond, angle and wall virial is summed as well.
// k_pair_lanes : the same for systems too small to fill the GPU with a thread per particle: eight
//            lanes per particle, the same bits.
// k_pair64 : the same in FP64 mode: FP32 screening, kept pairs of a warp put together.
// k_bonded : intra_molec.f90:16-188 (FENE), bending.f90:19-121 / bending_melt.f90:22-108 and
//            orientation.f90:24-88.  Owner computes: the thread of bead m evaluates every bond,
//            angle and orientation term that acts on m (terms centred on m-1, m, m+1) and adds
//            its own share, so no two threads write one particle.  The body (bonded_of) is
//            shared with the fused pair kernel.
// k_wall   : fluid_wall.f90:77-125 (implicit 9-3 walls), FP64.
// k_cforce : constant_force.f90:17-21 (Poiseuille body force m*g on every non-head bead).
#include <type_traits>

#include "mfa_integ.cuh"

namespace mfa {

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <bool MIXED>
using real_t = typename std::conditional<MIXED, float, double>::type;

// A constant in the kernel's precision: the FP32 copy for MIXED, the double otherwise.
template <bool MIXED>
__device__ __forceinline__ real_t<MIXED> cst(double d, float f) {
  if constexpr (MIXED) return f; else return d;
}

__device__ __forceinline__ double r2min_of(const SimConst& C, long long step) {
  if (!C.force_switch_on) return 0.;
  double r_time = (double)step * C.dt;
  return (r_time < C.r2min_time) ? (1. - r_time / C.r2min_time) * C.r2min_init : 0.;
}

// ---------------------------------------------------------------------------------------------
// Bonded terms
// ---------------------------------------------------------------------------------------------
template <bool MIXED>
struct BeadPos;
template <>
struct BeadPos<true> {
  int4 q;
  __device__ void load(const DevState& s, int slot) { q = __ldg(&s.pfx[slot]); }
};
template <>
struct BeadPos<false> {
  double x, y, z;
  __device__ void load(const DevState& s, int slot) { x = s.rx[slot]; y = s.ry[slot]; z = s.rz[slot]; }
};

// a - b with the x,y minimum image
template <bool MIXED>
__device__ __forceinline__ void bead_delta(const BeadPos<MIXED>& a, const BeadPos<MIXED>& b, const RepDesc& R,
                                           real_t<MIXED>* d) {
  if constexpr (MIXED) {
    d[0] = i2f_fast(fx_diff(a.q.x, b.q.x)) * R.ufx_f[0];
    d[1] = i2f_fast(fx_diff(a.q.y, b.q.y)) * R.ufx_f[1];
    d[2] = i2f_fast(fx_diff(a.q.z, b.q.z)) * R.ufx_f[2];
  } else {
    d[0] = mic_fast(a.x - b.x, R.L[0], R.invL[0]);
    d[1] = mic_fast(a.y - b.y, R.L[1], R.invL[1]);
    d[2] = a.z - b.z;
  }
}

// a * b rounded on its own, never merged into a multiply-add: a force term that the virial of an
// energy kernel also reads is rounded alike in the kernels with and without energies (whether the
// compiler merges a product into an add depends on the product's other uses)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// One angle term of bending.f90:47-109 with r_prev = r_c - r_{c-1}, r_next = r_{c+1} - r_c.
// fa acts on c-1, fc on c+1 (c gets -fa-fc).  MIXED takes the angle's sine and cosine from
// |p x n| and p.n (the harmonic form its angle as atan2(|p x n|, p.n)), which keeps FP32
// accurate for the nearly straight chains that stiff brushes produce.
template <bool MIXED>
__device__ void bend_term(const real_t<MIXED>* rp, const real_t<MIXED>* rn, const SimConst& C, real_t<MIXED> kb,
                          real_t<MIXED> aeq, real_t<MIXED>* fa, real_t<MIXED>* fc, real_t<MIXED>& e) {
  using real = real_t<MIXED>;
  real dot = 0, rp2 = 0, rn2 = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dot += rn[j] * rp[j];
    rp2 += rp[j] * rp[j];
    rn2 += rn[j] * rn[j];
  }
  real dn[3], dp[3], dn2 = 0, dp2 = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dn[j] = rp[j] * rn2 - rn[j] * dot;
    dp[j] = -rn[j] * rp2 + rp[j] * dot;
    dn2 += dn[j] * dn[j];
    dp2 += dp[j] * dp[j];
  }
  const real small = cst<MIXED>(C.bend_small, C.bend_small_f);
  const real srp = sqrt(rp2), srn = sqrt(rn2);
  if (dn2 < small) {
    real u[3], nu = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) { u[j] = rp[j] / srp - rn[j] / srn; nu += u[j] * u[j]; }
    nu = sqrt(nu);
#pragma unroll
    for (int j = 0; j < 3; ++j) dn[j] = (nu != 0) ? u[j] / nu / srn : (real)0;
  } else {
    const real sc = (real)1 / sqrt(dn2 * rn2);
#pragma unroll
    for (int j = 0; j < 3; ++j) dn[j] *= sc;
  }
  if (dp2 < small) {
    real u[3], nu = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) { u[j] = rp[j] / srp - rn[j] / srn; nu += u[j] * u[j]; }
    nu = sqrt(nu);
#pragma unroll
    for (int j = 0; j < 3; ++j) dp[j] = (nu != 0) ? u[j] / nu / srp : (real)0;
  } else {
    const real sc = (real)1 / sqrt(dp2 * rp2);
#pragma unroll
    for (int j = 0; j < 3; ++j) dp[j] *= sc;
  }
  real fm;
  if constexpr (MIXED) {
    real cx = rp[1] * rn[2] - rp[2] * rn[1];
    real cy = rp[2] * rn[0] - rp[0] * rn[2];
    real cz = rp[0] * rn[1] - rp[1] * rn[0];
    const real cr = sqrtf(cx * cx + cy * cy + cz * cz);
    if (C.bend_form == 1) {
      // the cosine form needs sin(alpha) and cos(alpha) only: |p x n| / (|p| |n|) and
      // p.n / (|p| |n|), with no angle and no library sine (the force then takes the same
      // operations whether or not the energy is formed)
      const real inv = (real)1 / (srp * srn);
      fm = kb * (cr * inv);
      e = kb * ((real)1 - dot * inv);
    } else {
      const real da = atan2f(cr, dot) - aeq;
      fm = kb * da;
      e = (real)0.5 * fm * da;
    }
  } else {
    real ca = dot / sqrt(rp2 * rn2);
    const real alpha = (ca >= 1.0) ? aeq : acos(ca);  // bending.f90:93-98 guard: delta_alpha = 0
    if (C.bend_form == 1) {
      fm = kb * sin(alpha);
      e = kb * ((real)1 - cos(alpha));
    } else {
      real da = alpha - aeq;
      fm = kb * da;
      e = (real)0.5 * fm * da;
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fa[j] = mul_rn(fm, dp[j]);
    fc[j] = mul_rn(fm, dn[j]);
  }
}

// Virial partials of the bonded terms of one particle (EFLAG kernels): FENE, brush and melt
// bending as symmetric tensors (xx yy zz xy xz yz), orientation as a full one (row-major).
template <typename T>
struct BondVir {
  T fene[6], bend[6], bendm[6], orient[9];
  __device__ void zero() {
#pragma unroll
    for (int c = 0; c < 6; ++c) fene[c] = bend[c] = bendm[c] = 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) orient[c] = 0;
  }
};

// Bonded force on the mobile particle i (owner computes, see k_bonded); adds to F[3] and, for the
// terms that i owns, to e4[4] = {FENE, brush bending, melt bending, orientation}.  With EFLAG the
// virial goes to bv: half of each of i's bonds (-fac d (x) d, the other half comes from the
// partner), the whole of the angle centred on i (-f_a (x) r_prev + f_c (x) r_next) and of the
// orientation term of a head (F_1 (x) (r_1 - r_head)).  FENE_ONLY: mask is 1.  Returns false when i is in no chain of two
// or more beads.
template <bool MIXED, bool EFLAG, bool FENE_ONLY = false>
__device__ __forceinline__ bool bonded_of(const DevState& s, const SimConst& C, int mask, int i, int w,
                                          real_t<MIXED>* F, real_t<MIXED>* e4, BondVir<real_t<MIXED>>* bv,
                                          int tag = -1) {
  using real = real_t<MIXED>;
  const RepDesc& R = s.reps[info_rep(w)];
  int kind = -1, m = 0, n = 0;
  const int t = tag >= 0 ? tag : __ldg(&s.tag[i]);
  const int lt = t - R.p0;
  if (lt < R.part_init_d) {
    kind = 0; n = R.n_mon; m = lt % n;
  } else if (lt < R.part_init_e) {
    kind = 1; n = R.n_mon_d; m = (lt - R.part_init_d) % n;
  } else if (lt < R.n_mon_tot) {
    kind = 2; n = R.n_mon_e; m = (lt - R.part_init_e) % n;
  }
  if (kind < 0 || n < 2) return false;
  const int t0 = t - m;
  {
    const bool do_fene = FENE_ONLY || (mask & 1);
    const bool do_bend = !FENE_ONLY && ((kind == 0 && (mask & 2)) || (kind == 1 && (mask & 4)));
    const bool do_or = !FENE_ONLY && kind == 0 && (mask & 8) && m <= 1;
    const int lo = max(0, m - ((do_bend) ? 2 : 1)), hi = min(n - 1, m + ((do_bend) ? 2 : 1));
    BeadPos<MIXED> P[5];  // beads m-2 .. m+2 (fixed slots, so the array stays in registers)
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int b = m - 2 + u;
      if (b >= lo && b <= hi) P[u].load(s, __ldg(&s.slot_of_tag[t0 + b]));
    }
    if (do_fene) {
      const real kc = cst<MIXED>(C.k_chain, C.k_chain_f), ir2 = cst<MIXED>(C.inv_r_chain_2, C.inv_r_chain_2_f),
                 xm = cst<MIXED>(C.fene_xmax, C.fene_xmax_f);
      if (m > 0) {  // bond (m-1, m): this bead is the second partner
        real d[3];
        bead_delta<MIXED>(P[1], P[2], R, d);
        real x = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) * ir2;
        x = x < xm ? x : xm;
        real fac = kc / ((real)1 - x) * ir2;
        F[0] += fac * d[0]; F[1] += fac * d[1]; F[2] += fac * d[2];
        if (EFLAG) sym_add(bv->fene, (real)-0.5 * fac, d[0], d[1], d[2]);
      }
      if (m < n - 1) {  // bond (m, m+1): first partner; energy counted here
        real d[3];
        bead_delta<MIXED>(P[2], P[3], R, d);
        real x = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) * ir2;
        x = x < xm ? x : xm;
        real fac = kc / ((real)1 - x) * ir2;
        F[0] -= fac * d[0]; F[1] -= fac * d[1]; F[2] -= fac * d[2];
        if (EFLAG) {
          e4[0] += kc * ((real)-0.5 * log((real)1 - x));
          sym_add(bv->fene, (real)-0.5 * fac, d[0], d[1], d[2]);
        }
      }
    }
    if (do_bend) {
      const real kb = cst<MIXED>(C.k_bend, C.k_bend_f), aeq = cst<MIXED>(C.alpha_eq, C.alpha_eq_f);
#pragma unroll
      for (int u = 1; u <= 3; ++u) {  // the angle centred on bead c = m - 2 + u
        const int c = m - 2 + u;
        if (c < 1 || c > n - 2) continue;
        real rp[3], rn[3], fa[3], fc[3], e;
        bead_delta<MIXED>(P[u], P[u - 1], R, rp);
        bead_delta<MIXED>(P[u + 1], P[u], R, rn);
        bend_term<MIXED>(rp, rn, C, kb, aeq, fa, fc, e);
        if (u == 3) { F[0] += fa[0]; F[1] += fa[1]; F[2] += fa[2]; }
        else if (u == 2) {
          F[0] -= fa[0] + fc[0]; F[1] -= fa[1] + fc[1]; F[2] -= fa[2] + fc[2];
          if (EFLAG) {
            if (kind == 0) e4[1] += e; else e4[2] += e;
            real* wb = (kind == 0) ? bv->bend : bv->bendm;
            const int ia[6] = {0, 1, 2, 0, 0, 1}, ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
            for (int c = 0; c < 6; ++c) wb[c] += fc[ia[c]] * rn[ib[c]] - fa[ia[c]] * rp[ib[c]];
          }
        } else { F[0] += fc[0]; F[1] += fc[1]; F[2] += fc[2]; }
      }
    }
    if (do_or) {
      // orientation.f90:35-88: ghost bond head -> head -/+ z, against bond 1
      const BeadPos<MIXED> H = (m == 0) ? P[2] : P[1];   // the head
      const BeadPos<MIXED> B1 = (m == 0) ? P[3] : P[2];  // bead 1 of the chain
      real rp[3], rn[3];
      bead_delta<MIXED>(B1, H, R, rn);
      double hz;
      if constexpr (MIXED) hz = (double)H.q.z * R.ufx[2]; else hz = H.z;
      if constexpr (MIXED) {
        rp[0] = 0; rp[1] = 0; rp[2] = (hz > R.L[2] / 2) ? -1.f : 1.f;
      } else {
        double g = (hz > R.L[2] / 2) ? hz + 1.0 : hz - 1.0;
        rp[0] = 0; rp[1] = 0; rp[2] = hz - g;
      }
      real dot = 0, rp2 = 0, rn2 = 0, dn[3], dn2 = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j) { dot += rn[j] * rp[j]; rp2 += rp[j] * rp[j]; rn2 += rn[j] * rn[j]; }
#pragma unroll
      for (int j = 0; j < 3; ++j) { dn[j] = rp[j] * rn2 - rn[j] * dot; dn2 += dn[j] * dn[j]; }
      const real srp = sqrt(rp2), srn = sqrt(rn2);
      if (dn2 < cst<MIXED>(C.bend_small, C.bend_small_f)) {
        real u[3], nu = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) { u[j] = rp[j] / srp - rn[j] / srn; nu += u[j] * u[j]; }
        nu = sqrt(nu);
#pragma unroll
        for (int j = 0; j < 3; ++j) dn[j] = (nu != 0) ? u[j] / nu / srn : (real)0;
      } else {
        const real sc = (real)1 / sqrt(dn2 * rn2);
#pragma unroll
        for (int j = 0; j < 3; ++j) dn[j] *= sc;
      }
      real alpha;
      if constexpr (MIXED) {
        real cx = rp[1] * rn[2] - rp[2] * rn[1];
        real cy = rp[2] * rn[0] - rp[0] * rn[2];
        real cz = rp[0] * rn[1] - rp[1] * rn[0];
        alpha = atan2f(sqrtf(cx * cx + cy * cy + cz * cz), dot);
      } else {
        real ca = dot / sqrt(rp2 * rn2);
        alpha = (ca >= 1.0) ? 0. : acos(ca);
      }
      const real da = alpha - cst<MIXED>(C.alpha_or, C.alpha_or_f);
      const real fm = cst<MIXED>(C.k_or, C.k_or_f) * da;
      const real sgn = (m == 0) ? (real)-1 : (real)1;
      const real sf = sgn * fm;
      F[0] += mul_rn(sf, dn[0]); F[1] += mul_rn(sf, dn[1]); F[2] += mul_rn(sf, dn[2]);
      if (EFLAG && m == 0) {
        e4[3] += (real)0.5 * fm * da;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) bv->orient[3 * a + b] += fm * dn[a] * rn[b];
      }
    }
  }
  return true;
}

// Slots and values of a symmetric tensor (6 components) for obs_push.
template <typename T>
__device__ __forceinline__ void sym_slots(int* sl, T* v, int base, const T* w6) {
  const int idx[6] = {0, 4, 8, 1, 2, 5};
#pragma unroll
  for (int c = 0; c < 6; ++c) { sl[c] = base + idx[c]; v[c] = w6[c]; }
}

// Slots and values of the bonded energies and virial tensors for obs_push (31 of them; terms
// that are off contribute zeros, which add nothing).
template <typename T>
__device__ __forceinline__ void bonded_slots(int* sl, T* v, const T* e4, const BondVir<T>& bv) {
  sl[0] = O_VINTRA; v[0] = e4[0];
  sym_slots(sl + 1, v + 1, O_VIR + 9 * V_FENE, bv.fene);
  sl[7] = O_VBEND; v[7] = e4[1];
  sym_slots(sl + 8, v + 8, O_VIR + 9 * V_BEND, bv.bend);
  sl[14] = O_VBENDM; v[14] = e4[2];
  sym_slots(sl + 15, v + 15, O_VIR + 9 * V_BENDM, bv.bendm);
  sl[21] = O_VOR; v[21] = e4[3];
#pragma unroll
  for (int c = 0; c < 9; ++c) { sl[22 + c] = O_VIR + 9 * V_OR + c; v[22 + c] = bv.orient[c]; }
}

// the FENE ones alone (7 of them)
template <typename T>
__device__ __forceinline__ void fene_slots(int* sl, T* v, const T* e4, const BondVir<T>& bv) {
  sl[0] = O_VINTRA; v[0] = e4[0];
  sym_slots(sl + 1, v + 1, O_VIR + 9 * V_FENE, bv.fene);
}
// bonded terms of the fused mixed kernels: none, FENE alone, all (by the mask)
constexpr int BOND_NONE = 0, BOND_FENE = 1, BOND_ALL = 2;
inline int bond_kind(int mask) { return mask == 0 ? BOND_NONE : (mask == 1 ? BOND_FENE : BOND_ALL); }
constexpr int bond_values(int bonded) { return bonded == BOND_ALL ? 31 : (bonded == BOND_FENE ? 7 : 0); }

// A thread per tag (by_tag) in larger systems: the beads of a chain are consecutive tags, so the warps
// that work are full and those of the solvent leave (by slot nearly every warp holds a few chain beads,
// and an FP64 instruction takes the same time for them).  16 brush replicas in FP64, 243 k particles, by
// slot / by tag: 42 / 30 us; charged brush, 33.6 k: 12.7 / 11.2.  A small system waits for the longer chain
// of loads instead (its slot comes first): 7200 particles 45.5 / 47.5 us a step.
template <bool MIXED, bool EFLAG>
__global__ void __launch_bounds__(128) k_bonded(DevState s, SimConst C, int mask, Acc acc, bool to_f4,
                                                   bool by_tag) {
  using real = real_t<MIXED>;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool inside = g < s.N;
  const int i = inside ? (by_tag ? __ldg(&s.slot_of_tag[g]) : g) : 0, w = inside ? __ldg(&s.info[i]) : 0;
  const int rep = info_rep(w);
  real F[3] = {0, 0, 0};
  real e4[4] = {0, 0, 0, 0};
  BondVir<real> bv;
  if (EFLAG) bv.zero();
  const bool has = inside && info_mobile(w) && bonded_of<MIXED, EFLAG>(s, C, mask, i, w, F, e4, &bv, by_tag ? g : -1);
  if (has) {
    if (MIXED && to_f4) {  // fused step: FP32 force array
      float4 f = s.f4[i];
      f.x += (float)F[0];
      f.y += (float)F[1];
      f.z += (float)F[2];
      s.f4[i] = f;
    } else {
      s.fx[i] += (double)F[0];
      s.fy[i] += (double)F[1];
      s.fz[i] += (double)F[2];
    }
  }
  if (EFLAG) {
    int sl[31];
    real v[31];
    bonded_slots(sl, v, e4, bv);
    obs_push<real, 31>(acc, sl, v, rep, has);
  }
}

// kept pairs per batch (a thread screens its list until it has this many, then they are evaluated),
// and list entries screened per group (their loads are all in flight at once).  Measured on 256
// brush replicas (4.66 M particles, skin 0.5): groups of 2 / 3 / 4 / 8 entries gave a pair kernel
// of 0.574 / 0.582 / 0.583 / 0.648 ms with the evaluation loop not unrolled; unrolling it by 2 or
// 4 cost 4 % or 20 %.  With the batch in shared memory, the kernel with the integration in its
// tail took 0.598 / 0.586 / 0.586 / 0.588 / 0.597 / 0.607 ms at batches of 8 / 10 / 12 / 16 /
// 24 / 32 (groups of 2; 12 with groups of 4: 0.585).
constexpr int PAIR_BATCH = 12;
constexpr int PAIR_G = 2;
// Every block prefetches into L2 what the block one per SM later reads from memory: the own-particle
// arrays and the first list rows (a lane per row; most WCA lists end there).  The kernel is bound by
// the latency of its loads (7.7 of 15 stall cycles per issue), and these would come from HBM: pair
// kernel 500 -> 456 us on 256 brush replicas (own-particle streams of the tail alone 490, own block's
// rows and streams 462, 2 / 4 / 10 blocks per SM ahead 458 / 463 / 490; 16, 20 or 32 rows: alike,
// alike, 1 us more).
constexpr int PAIR_ROWS_AHEAD = 18;

// Force factor fs of the pair (i, j) along d = r_i - r_j (LJ with the switch-on clamp, DPD with the
// pair's Philox noise, real-space Coulomb), fluid_fluid.f90:97-261, dpd_forces.f90:45-115,
// ewald_real.f90:15-33; with EFLAG the pair's share `half` of its energies.  FP32 (pair_fs) and
// FP64 (pair_fs64) forms.
template <bool EFLAG>
__device__ __forceinline__ float pair_fs(const DevState& s, const SimConst& C, const PairEntry<float>& e, float dx,
                                         float dy, float dz, float4 vj, float vix, float viy, float viz, int tag_i,
                                         int p0, uint32_t nkey, float r2min, float half, float& e_lj, float& e_c) {
  const float r2raw = dx * dx + dy * dy + dz * dz;
  const int fl = e.flags;
  float r2 = r2raw;
  const bool in_lj = r2raw < e.range2;
  float fs = 0;  // force factor along d = r_i - r_j
  if (in_lj) {
    r2 = r2raw < r2min ? r2min : r2raw;
    // the hardware reciprocal (2 ulp) instead of the IEEE division sequence
    const float inv_r2 = rcp_ftz(r2);
    const float s2 = e.sig2 * inv_r2;
    const float s6 = s2 * s2 * s2;
    const float s12 = s6 * s6;
    fs = e.eps4 * (12.f * s12 - 6.f * s6) * inv_r2;
    if (EFLAG) e_lj += half * e.eps4 * ((s12 - s6) - e.shift);
  }
  const bool dpd = (in_lj && (fl & PF_DPD_LJ)) || ((fl & PF_DPD_OWN) && r2 < e.dpd_rc2);
  if (dpd) {
    const int tag_j = __float_as_int(vj.w) - p0;
    const float ir = rsqrt_ftz(r2);  // one hardware reciprocal square root (2 ulp)
    const float r = r2 * ir;
    float wr, wd;
    if (C.dpd_weight1) {
      wr = wd = 1;
    } else {
      wr = 1.f - r * ((fl & PF_DPD_OWN) ? e.inv_dpd_rc : e.inv_rc);
      wd = wr * wr;
    }
    const float g = pair_gauss_f(nkey, tag_i, tag_j);
    const float rdot = ((vix - vj.x) * dx + (viy - vj.y) * dy + (viz - vj.z) * dz) * ir;
    fs += (C.sig_f * wr * g - C.gamma_f * wd * rdot) * ir;
  }
  if (fl & PF_COUL) {
    const bool in_c = (C.coul_rc2_f > 0) ? (r2raw < C.coul_rc2_f) : in_lj;
    if (in_c) {
      const float rc2 = in_lj ? r2 : r2raw;
      const float r = sqrtf(rc2), ir = 1.f / r;
      const float qq = e.qq, sqa = C.sqrt_alpha_f;
      const float ec = erfcf(sqa * r);
      if (EFLAG) e_c += half * qq * ec * ir;
      fs += (qq * sqa * C.inv_sqrt_pi_f * 2.f * expf(-C.alpha_c_f * rc2) * ir + qq * ec * ir * ir) * ir;
    }
  }
  return fs;
}

template <bool EFLAG>
__device__ __forceinline__ double pair_fs64(const DevState& s, const SimConst& C, const PairEntry<double>& e,
                                            double dx, double dy, double dz, int j, double vix, double viy,
                                            double viz, int tag_i, int p0, uint32_t nkey, double r2min, double half,
                                            double& e_lj, double& e_c) {
  const double r2raw = dx * dx + dy * dy + dz * dz;
  const int fl = e.flags;
  const bool in_lj = r2raw < e.range2;
  const double r2 = (in_lj && r2raw < r2min) ? r2min : r2raw;
  const bool dpd = (in_lj && (fl & PF_DPD_LJ)) || ((fl & PF_DPD_OWN) && r2 < e.dpd_rc2);
  const bool in_c = (fl & PF_COUL) && ((C.coul_rc2 > 0) ? (r2raw < C.coul_rc2) : in_lj);
  double fs = 0;
  if (!(in_lj || dpd || in_c)) return fs;
  const double ir = rsqrt64(r2);  // the only root and division of the pair
  if (in_lj) {
    // (rounded once: the seventh power below would enlarge the square's own error.  1 % of the step)
    double inv_r2 = ir * ir;
    inv_r2 = fma(inv_r2, fma(-inv_r2, r2, 1.), inv_r2);
    const double s2 = e.sig2 * inv_r2;
    const double s6 = s2 * s2 * s2;
    const double s12 = s6 * s6;
    fs = e.eps4 * (12. * s12 - 6. * s6) * inv_r2;
    if (EFLAG) e_lj += half * e.eps4 * ((s12 - s6) - e.shift);
  }
  if (dpd) {
    const dbl4 v4 = s.vd[j];
    const int tag_j = (int)__double_as_longlong(v4.w) - p0;
    double wr, wd;
    if (C.dpd_weight1) {
      wr = wd = 1;
    } else {
      // (r corrected as the root it stands for: r2 ir rounds twice, 0.1 % of the forces' error)
      const double q = r2 * ir, r = fma(fma(-q, q, r2), half_of(ir), q);
      wr = 1. - r * ((fl & PF_DPD_OWN) ? e.inv_dpd_rc : e.inv_rc);
      wd = wr * wr;
    }
    const double g = pair_gauss_d(s.noise, nkey, tag_i, tag_j);
    const double rdot = ((vix - v4.x) * dx + (viy - v4.y) * dy + (viz - v4.z) * dz) * ir;
    fs += (C.sig * wr * g - C.gamma * wd * rdot) * ir;
  }
  if (in_c) {
    const CoulTab* T = s.coul;
    if (T && r2 >= T->lo && r2 < T->hi) {
      const double x = (r2 - T->lo) * T->inv_h, z = x + 4503599627370496.0;  // 2^52: rounds to an integer
      int k = __double2loint(z);
      double t = x - (z - 4503599627370496.0);  // [-1/2, 1/2] from the nearest edge
      // (the last doubles below hi may round onto the table's end, edge n: the interval left of it as well)
      const bool left = t < 0. || k >= T->n;
      if (left) --k;
      t = fma(2., t, left ? 1. : -1.);  // [-1, 1] inside the interval
      fs += e.qq * coul_poly(T->f + 8 * (size_t)k, t);
      if (EFLAG) e_c += half * e.qq * coul_poly(T->e + 8 * (size_t)k, t);
    } else {
      const double r = r2 * ir, qq = e.qq, ec = erfc(C.sqrt_alpha * r);
      if (EFLAG) e_c += half * qq * ec * ir;
      fs += (qq * C.sqrt_alpha * C.inv_sqrt_pi * 2. * exp(-C.alpha_c * r2) * ir + qq * ec * ir * ir) * ir;
    }
  }
  return fs;
}

// The pair kernel of the mixed mode: FP32 pair arithmetic on the fixed-point views.  Template
// switches:
//   EFLAG   energies and the virial into the accumulators;
//   FUSED   the fused mixed-precision step: FP32 partial sums over each batch of kept
//           pairs are added to an FP64 per-particle total, together with the bonded, wall and body
//           forces of the particle, and the total is stored (rounded to FP32) in the force array
//           that the integrator reads;
//   BONDED  (FUSED only) the particle's bonded terms (bonded_of; FENE alone or all) in the same thread, which saves
//           the bonded kernel's launch and its read-modify-write of the force;
//   UNI     one screening cut-off for every type pair (SimConst::scr2_uni_f).
// Without FUSED the forces are added to (accumulate) or stored in the FP64 force arrays.
// Virial (EFLAG): each visit of a pair adds half of F_ij (x) (r_i - r_j) (the other visit adds the
// other half); a pair with a fixed wall bead, which has no list of its own, counts in full.
//   INTEG   (FUSED) the step's integration in the tail (with EFLAG also its kinetic energy and
//           tensor and the head forces, into the same warp reduction): each thread takes its
//           particle's force and runs the integrator's update (int_mixed_particle, MODE 2) on it,
//           writing the next step's views to the other view buffers (pfx_alt, vf_alt) while the
//           neighbours still read pfx and vf; wall beads copy their views across, and the step
//           counter of the other set is this one's plus one.  No force array is written.
//   PERSIST (FUSED only) a grid of the blocks that fit on the GPU at once; each block takes tiles
//           of blockDim.x particles from a queue (s.pair_q[0], one atomic ticket per tile, no
//           waiting) and the last block to finish resets the queue for the next launch.  Compiled
//           for 8 resident blocks per SM (64 registers): at 9 the tile loop spills.
template <bool EFLAG, bool FUSED = false, int BONDED = BOND_NONE, bool UNI = false, bool PERSIST = false,
          bool INTEG = false>
// Resident blocks per SM: 10 for the kernel with the integration in its tail (48 registers, no spill
// with FENE bonds alone, 52 bytes with every bonded term; 0.456 ms per step on 256 brush replicas;
// before the loads were moved ahead of their use 0.537, and 0.553 at 11 or 12 blocks), 9 for the other fused forms (an energy step of these replicas costs 125 us
// more than a plain one; 166 at 8 blocks, 210 at 7), 8 for the persistent schedule (its tile loop
// spills at 9).  FENE bonds alone have a variant of their own: compiled for every bonded term the
// energy variant spilled 200 bytes and reduced 54 values per warp instead of 30 (235 us more than a
// plain step), and the plain one took 0.559 ms.
__global__ void __launch_bounds__(128, PERSIST ? 8 : ((INTEG && !EFLAG) ? 10 : 9)) k_pair(DevState s, SimConst C,
                                                                                          bool accumulate, Acc acc,
                                                                                          int bmask = 0) {
  using real = float;
  static_assert(!BONDED || FUSED, "bonded terms are fused only into the fused form");
  static_assert(!INTEG || (FUSED && !PERSIST), "the integration is fused into the fused form");
  __shared__ PairEntry<real> tab[NPAIR];
  // FUSED: the particle's FP64 total, in shared memory while the pair loop runs (registers are
  // scarce there; it is touched once per batch)
  __shared__ double ftot[FUSED ? 3 : 1][FUSED ? 128 : 1];
  for (int k = threadIdx.x; k < NPAIR; k += blockDim.x) tab[k] = s.tabf[k];
  __shared__ int tile_sh;
  const int ntile = (s.N + blockDim.x - 1) / blockDim.x;
  for (int pass = 0;; ++pass) {
  int tile;
  if constexpr (PERSIST) {
    __syncthreads();  // every thread is done with the previous tile's ticket
    if (threadIdx.x == 0) tile_sh = atomicAdd(s.pair_q, 1);
    __syncthreads();
    tile = tile_sh;
    if (tile >= ntile) break;
  } else {
    if (pass) break;
    tile = blockIdx.x;
  }
  const int i = tile * blockDim.x + threadIdx.x;
  const bool inside = i < s.N;
  const int w = inside ? __ldg(&s.info[i]) : 0;
  const bool active = inside && info_mobile(w);
  const int rep = info_rep(w);
  float e_w = 0.f, w_wall = 0.f;  // FUSED: wall energy and virial
  {  // the streams of the block that starts about when this one ends, on their way into L2
    const int ip = i + s.nsm * (int)blockDim.x, i0 = ip & ~31, row = threadIdx.x & 31;
    if (i0 < s.N && row < min(PAIR_ROWS_AHEAD, s.nbr_cap)) prefetch_l2(s.nbr + (size_t)row * s.Np + i0);
    if (ip < s.N) {
      prefetch_l2(s.info + ip);
      prefetch_l2(s.nn + ip);
      prefetch_l2(s.pfx + ip);
      prefetch_l2(s.vf + ip);
      if (FUSED) prefetch_l2(s.rz + ip);
      if (INTEG) {
        prefetch_l2(s.rx + ip);
        prefetch_l2(s.ry + ip);
        prefetch_l2(s.vx + ip);
        prefetch_l2(s.vy + ip);
        prefetch_l2(s.vz + ip);
        prefetch_l2(s.ref + ip);
        prefetch_l2(s.tag + ip);
      }
    }
  }
  if constexpr (FUSED) {
    // the particle's external forces first: its FP64 total starts from them
    double ez = 0., ex = 0., ey = 0.;
    if (active) {
      const int ti = info_type(w);
      if (C.wall == 2) {  // fluid_wall.f90:96-121 from the FP64 position: distances to both walls
        const double zd = s.rz[i];
        const float zl = d2f_fast(zd), zh = d2f_fast(s.reps[rep].L[2] - zd);
        float fwb, fwt;
        wall93f_split(C, ti, zl, zh, fwb, fwt, e_w);
        ez = f2d_fast(fwb) + f2d_fast(fwt);
        if (EFLAG) w_wall = fwb * zl - fwt * zh;  // each wall's force times z - z_wall
      }
      if (C.poiseuille && ti != 0) {  // constant_force.f90:17-21: m g on every non-head bead
        ex = f2d_fast(C.mass_f[ti] * C.cforce_f[0]);
        ey = f2d_fast(C.mass_f[ti] * C.cforce_f[1]);
        ez += f2d_fast(C.mass_f[ti] * C.cforce_f[2]);
      }
    }
    ftot[0][threadIdx.x] = ex;
    ftot[1][threadIdx.x] = ey;
    ftot[2][threadIdx.x] = ez;
  }
  __syncthreads();
  // Shared memory of the batch of kept list entries (a column per thread) and, in the energy
  // variant with bonded terms, of the bonded virial partials after it: the batch is dead once
  // the pair loop ends, and a barrier separates the two uses, so the variant keeps room for L1.
  constexpr int JL_WORDS = PAIR_BATCH * 128;
  constexpr int BV_WORDS = (EFLAG && BONDED == BOND_ALL) ? 128 * (int)(sizeof(BondVir<real>) / 4) : 0;
  __shared__ __align__(16) int pair_pool[JL_WORDS > BV_WORDS ? JL_WORDS : BV_WORDS];
  real fx = 0, fy = 0, fz = 0;        // the current batch (FUSED), else the whole sum
  real e_lj = 0, e_c = 0;
  real wv[6] = {0, 0, 0, 0, 0, 0};   // EFLAG: pair virial, xx yy zz xy xz yz
  if (active) {
    const RepDesc& R = s.reps[rep];
    const long long step = R.s_time + *s.steps_done;
    const real r2min = C.force_switch_on ? (real)r2min_of(C, step) : (real)0;
    const int ti = info_type(w);
    const int n = __ldg(&s.nn[i]);
    const int p0 = R.p0;
    // own position / velocity
    const int4 qi = __ldg(&s.pfx[i]);
    const float4 vi = __ldg(&s.vf[i]);
    const int tag_i = __float_as_int(vi.w) - p0;
    const float ux = R.ufx_f[0], uy = R.ufx_f[1], uz = R.ufx_f[2];
    const uint32_t nkey = pair_key(R.seed, step);  // the replica's noise key of this step
    const int* __restrict__ nb = s.nbr + i;
    auto delta = [&](int j, real& dx, real& dy, real& dz) -> int {
      const int4 qj = __ldg(&s.pfx[j]);
      dx = i2f_fast(fx_diff(qi.x, qj.x)) * ux;
      dy = i2f_fast(fx_diff(qi.y, qj.y)) * uy;
      dz = i2f_fast(fx_diff(qi.z, qj.z)) * uz;
      return qj.w;
    };
    // Two phases per batch: (1) screen list entries with the cheap distance test and keep the
    // ones inside any interaction range, (2) evaluate LJ + DPD + Coulomb on the kept pairs only.
    // Without the split a warp runs the Philox/DPD body whenever any lane has an interacting
    // pair, i.e. on almost every list entry.
    constexpr int BATCH = PAIR_BATCH;
    constexpr int G = PAIR_G;  // list entries screened per group: their loads are all in flight at once
    // the batch's kept entries in shared memory, a column per thread (conflict-free): a
    // dynamically indexed local array lives in local memory, whose loads missed L1 behind the
    // gathers
    int* const jl = pair_pool + threadIdx.x;
    int k = 0;
    // screening against the largest cut-off of the type pair, with the coarse conversion (512
    // fixed-point units of resolution, inside the margin of screen2)
    const float cx = ux * 512.f, cy = uy * 512.f, cz = uz * 512.f;
    auto screen = [&](int j) -> bool {
      const int4 qj = __ldg(&s.pfx[j]);
      const float dx = i2f_coarse(fx_diff(qi.x, qj.x), 9) * cx;
      const float dy = i2f_coarse(fx_diff(qi.y, qj.y), 9) * cy;
      const float dz = i2f_coarse(fx_diff(qi.z, qj.z), 9) * cz;
      return dx * dx + dy * dy + dz * dz < (UNI ? C.scr2_uni_f : tab[ti * MAXT + info_type(qj.w)].screen2);
    };
    while (k < n) {
      int m = 0;
      // groups of G independent entries (index loads first, then the position gathers)
      // (the next group's list indices are loaded one group ahead, hiding their DRAM latency)
      int jg[G];
      if (k + G <= n) {
#pragma unroll
        for (int u = 0; u < G; ++u) jg[u] = __ldg(nb + (size_t)(k + u) * s.Np);
      }
      while (k + G <= n && m <= BATCH - G) {
        int jn[G];
        const bool more = k + 2 * G <= n;
#pragma unroll
        for (int u = 0; u < G; ++u) jn[u] = more ? __ldg(nb + (size_t)(k + G + u) * s.Np) : 0;
        bool hg[G];
#pragma unroll
        for (int u = 0; u < G; ++u) hg[u] = screen(jg[u]);
#pragma unroll
        for (int u = 0; u < G; ++u)
          if (hg[u]) jl[128 * m++] = jg[u];
        k += G;
#pragma unroll
        for (int u = 0; u < G; ++u) jg[u] = jn[u];
      }
      while (k < n && m < BATCH) {
        const int j = __ldg(nb + (size_t)k * s.Np);
        ++k;
        if (screen(j)) jl[128 * m++] = j;
      }
#pragma unroll 1
      for (int t = 0; t < m; ++t) {
        const int j = jl[128 * t];
        real dx, dy, dz;
        const float4 vj = __ldg(&s.vf[j]);  // with the position: behind the cut-off test it would wait again
        const int wj = delta(j, dx, dy, dz);
        const PairEntry<real>& e = tab[ti * MAXT + info_type(wj)];
        // half of each mobile pair (both ends sum it); a fixed wall bead has no list of its own
        const real half = info_mobile(wj) ? (real)0.5 : (real)1;
        const real fs = pair_fs<EFLAG>(s, C, e, dx, dy, dz, vj, vi.x, vi.y, vi.z, tag_i, p0, nkey, r2min, half,
                                       e_lj, e_c);
        // unmerged products and sums: alike with and without energies
        fx = __fadd_rn(fx, __fmul_rn(fs, dx));
        fy = __fadd_rn(fy, __fmul_rn(fs, dy));
        fz = __fadd_rn(fz, __fmul_rn(fs, dz));
        if (EFLAG) sym_add(wv, half * fs, dx, dy, dz);
      }
      if constexpr (FUSED) {  // the batch's FP32 partial into the FP64 total
        ftot[0][threadIdx.x] += f2d_fast(fx);
        ftot[1][threadIdx.x] += f2d_fast(fy);
        ftot[2][threadIdx.x] += f2d_fast(fz);
        fx = fy = fz = 0;
      }
    }
  }
  real eb[4] = {0, 0, 0, 0};
  // the bonded virial partials of the thread (EFLAG): with every term in shared memory, where the
  // bonded terms' registers are scarce (27 words per thread: a stride prime to the 32 banks)
  BondVir<real> bv_own;
  BondVir<real>& bv = (EFLAG && BONDED == BOND_ALL) ? reinterpret_cast<BondVir<real>*>(pair_pool)[threadIdx.x] : bv_own;
  if (EFLAG && BONDED == BOND_ALL) __syncthreads();  // every thread is past its pair loop: the batch area is free
  if (EFLAG && BONDED) bv.zero();
  double fxd = 0., fyd = 0., fzd = 0.;
  // INTEG with EFLAG: the integrator's kinetic energy, kinetic tensor and head forces
  float ike = 0.f, ikin[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, ifh[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if constexpr (FUSED) {
    fxd = ftot[0][threadIdx.x];
    fyd = ftot[1][threadIdx.x];
    fzd = ftot[2][threadIdx.x];
    if (active) {
      if constexpr (BONDED) {
        real fb[3] = {0, 0, 0};
        bonded_of<true, EFLAG, BONDED == BOND_FENE>(s, C, bmask, i, w, fb, eb, &bv);
        fxd += f2d_fast(fb[0]);
        fyd += f2d_fast(fb[1]);
        fzd += f2d_fast(fb[2]);
      }
    }
  }
  if (inside) {
    if constexpr (INTEG) {
      if (active) {
        int_mixed_particle<2, EFLAG>(s, C, i, w, d2f_fast(fxd), d2f_fast(fyd), d2f_fast(fzd), s.pfx_alt, s.vf_alt,
                                     ike, ikin, ifh);
      } else if (C.move_walls) {  // a wall bead on a moving wall: its next site
        double x, y, z;
        s.pfx_alt[i] = move_wall_bead(s, C, i, w, x, y, z);
        s.vf_alt[i] = s.vf[i];
      } else {  // a wall bead: its views as they are
        s.pfx_alt[i] = s.pfx[i];
        s.vf_alt[i] = s.vf[i];
      }
      if (i == 0) *s.steps_alt = *s.steps_done + 1;
    } else if constexpr (FUSED) {
      s.f4[i] = make_float4(d2f_fast(fxd), d2f_fast(fyd), d2f_fast(fzd), 0.f);
    } else if (accumulate) {
      if (active) {
        s.fx[i] += (double)fx;
        s.fy[i] += (double)fy;
        s.fz[i] += (double)fz;
      }
    } else {
      s.fx[i] = fx;
      s.fy[i] = fy;
      s.fz[i] = fz;
    }
  }
  if (EFLAG) {  // one warp reduction for every energy and virial component of the kernel
    constexpr int NB = bond_values(BONDED), NW = FUSED ? 2 : 0, NI = INTEG ? 13 : 0, NV = 8 + NB + NW + NI;
    int sl[NV];
    real v[NV];
    sl[0] = O_VFF; v[0] = e_lj;
    sl[1] = O_VCOUL; v[1] = e_c;
    sym_slots(sl + 2, v + 2, O_VIR + 9 * V_PAIR, wv);
    if constexpr (BONDED == BOND_ALL) bonded_slots(sl + 8, v + 8, eb, bv);
    if constexpr (BONDED == BOND_FENE) fene_slots(sl + 8, v + 8, eb, bv);
    if constexpr (FUSED) {
      sl[8 + NB] = O_VFW; v[8 + NB] = e_w;
      sl[9 + NB] = O_VIR + 9 * V_WALL + 8; v[9 + NB] = w_wall;
    }
    if constexpr (INTEG) {  // the integrator's kinetic energy, kinetic tensor and head forces
      constexpr int b = 8 + NB + NW;
      const int idx[6] = {0, 4, 8, 1, 2, 5};
      sl[b] = O_TFLUID; v[b] = ike;
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        sl[b + 1 + c] = O_KIN + idx[c]; v[b + 1 + c] = ikin[c];
        sl[b + 7 + c] = O_FH + c; v[b + 7 + c] = ifh[c];
      }
    }
    obs_push<real, NV>(acc, sl, v, rep, active);
  }
  }
  if constexpr (PERSIST) {  // the last block out resets the queue (every block has drawn its last ticket)
    if (threadIdx.x == 0 && atomicAdd(s.pair_q + 1, 1) == (int)gridDim.x - 1) {
      s.pair_q[0] = 0;
      s.pair_q[1] = 0;
    }
  }
}

// The mixed pair kernel for few particles: a small system leaves the thread-per-particle kernel four
// warps on some SMs, and its time is the latency of one thread's walk (19 us at 6400 particles).  Here
// PL_G lanes take a particle's list side by side and place the kept entries by a ballot; they evaluate
// a batch side by side too, and one lane per component adds the products of a batch in list order, so
// the sums are those of k_pair to the bit (batches of PAIR_BATCH kept entries, products and sums
// rounded apart).  A warp of its own per block evaluates the bonded terms of the 32 particles
// meanwhile and then integrates them (FUSED, BONDED, UNI, INTEG as in k_pair).
// Measured: 17.9 -> 11.5 us at 6400 particles (WCA), 59 -> 22 at 6800 (2.24 sigma), 67 -> 35 at 33,600
// (charged brush).
constexpr int PL_G = 8, PL_P = 32, PL_T = PL_P * PL_G + 32;

template <bool EFLAG, bool FUSED, int BONDED, bool UNI, bool INTEG>
__global__ void __launch_bounds__(PL_T) k_pair_lanes(DevState s, SimConst C, Acc acc, int bmask) {
  __shared__ PairEntry<float> tab[NPAIR];
  __shared__ int jl[PL_P][PAIR_BATCH + PL_G];
  __shared__ float prod[3][PL_P][PAIR_BATCH + 1];
  __shared__ double tot[3][PL_P];
  __shared__ float wall_e[PL_P], wall_w[PL_P];
  const unsigned FULL = 0xffffffffu;
  for (int k = threadIdx.x; k < NPAIR; k += PL_T) tab[k] = s.tabf[k];
  const int lane = threadIdx.x & 31;
  const bool tail = threadIdx.x >= PL_P * PL_G;
  const int pl = tail ? lane : (int)threadIdx.x / PL_G, i = blockIdx.x * PL_P + pl;
  const bool inside = i < s.N;
  const int w = inside ? __ldg(&s.info[i]) : 0;
  const bool active = inside && info_mobile(w);
  const int rep = info_rep(w);
  float fb[3] = {0.f, 0.f, 0.f}, eb[4] = {0.f, 0.f, 0.f, 0.f};
  BondVir<float> bv;
  if (EFLAG) bv.zero();
  __syncthreads();
  if (tail) {
    if constexpr (BONDED) {
      if (active) bonded_of<true, EFLAG, BONDED == BOND_FENE>(s, C, bmask, i, w, fb, eb, &bv);
    }
  } else {
    const int q8 = lane & (PL_G - 1), grp = lane / PL_G;
    const RepDesc& R = s.reps[rep];
    const int ti = info_type(w), p0 = R.p0;
    float e_w = 0.f, w_wall = 0.f;
    double sum = 0.;  // lanes 0..2: the component's total, from the external forces on
    if (FUSED && active) {
      if (q8 < 3 && C.poiseuille && ti != 0) sum = f2d_fast(C.mass_f[ti] * C.cforce_f[q8]);
      if (q8 == 2 && C.wall == 2) {  // as k_pair
        const double zd = s.rz[i];
        const float zl = d2f_fast(zd), zh = d2f_fast(R.L[2] - zd);
        float fwb, fwt;
        wall93f_split(C, ti, zl, zh, fwb, fwt, e_w);
        const double ez = f2d_fast(fwb) + f2d_fast(fwt);
        sum = ez + sum;
        if (EFLAG) w_wall = fwb * zl - fwt * zh;
      }
    }
    if (EFLAG && FUSED && q8 == 2) {
      wall_e[pl] = e_w;
      wall_w[pl] = w_wall;
    }
    float run = 0.f;  // without FUSED: the component's FP32 sum over the whole list
    float e_lj = 0.f, e_c = 0.f, wv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const long long step = R.s_time + *s.steps_done;
    const float r2min = C.force_switch_on ? (float)r2min_of(C, step) : 0.f;
    const uint32_t nkey = pair_key(R.seed, step);
    const int n = active ? __ldg(&s.nn[i]) : 0;
    const int* __restrict__ nb = s.nbr + i;
    const int4 qi = active ? __ldg(&s.pfx[i]) : make_int4(0, 0, 0, 0);
    const float4 vi = active ? __ldg(&s.vf[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int tag_i = __float_as_int(vi.w) - p0;
    const float ux = R.ufx_f[0], uy = R.ufx_f[1], uz = R.ufx_f[2];
    const float cx = ux * 512.f, cy = uy * 512.f, cz = uz * 512.f;
    int m = 0, k = 0;  // kept entries waiting in jl, list position: alike in the lanes of a particle
    for (;;) {
      while (__any_sync(FULL, m < PAIR_BATCH && k < n)) {
        const bool go = m < PAIR_BATCH && k < n;
        int j = 0;
        bool hit = false;
        if (go && k + q8 < n) {
          j = __ldg(nb + (size_t)(k + q8) * s.Np);
          const int4 qj = __ldg(&s.pfx[j]);
          const float dx = i2f_coarse(fx_diff(qi.x, qj.x), 9) * cx;
          const float dy = i2f_coarse(fx_diff(qi.y, qj.y), 9) * cy;
          const float dz = i2f_coarse(fx_diff(qi.z, qj.z), 9) * cz;
          hit = dx * dx + dy * dy + dz * dz < (UNI ? C.scr2_uni_f : tab[ti * MAXT + info_type(qj.w)].screen2);
        }
        const unsigned bits = (__ballot_sync(FULL, hit) >> (grp * PL_G)) & ((1u << PL_G) - 1u);
        if (hit) jl[pl][m + __popc(bits & ((1u << q8) - 1u))] = j;
        m += __popc(bits);
        if (go) k += PL_G;
      }
      __syncwarp();
      const int take = min(m, PAIR_BATCH);
      if (!__any_sync(FULL, take > 0)) break;
      for (int c = q8; c < take; c += PL_G) {
        const int j = jl[pl][c];
        const float4 vj = __ldg(&s.vf[j]);
        const int4 qj = __ldg(&s.pfx[j]);
        const float dx = i2f_fast(fx_diff(qi.x, qj.x)) * ux;
        const float dy = i2f_fast(fx_diff(qi.y, qj.y)) * uy;
        const float dz = i2f_fast(fx_diff(qi.z, qj.z)) * uz;
        const PairEntry<float>& e = tab[ti * MAXT + info_type(qj.w)];
        const float half = info_mobile(qj.w) ? 0.5f : 1.f;
        const float fs = pair_fs<EFLAG>(s, C, e, dx, dy, dz, vj, vi.x, vi.y, vi.z, tag_i, p0, nkey, r2min, half, e_lj,
                                        e_c);
        prod[0][pl][c] = __fmul_rn(fs, dx);
        prod[1][pl][c] = __fmul_rn(fs, dy);
        prod[2][pl][c] = __fmul_rn(fs, dz);
        if (EFLAG) sym_add(wv, half * fs, dx, dy, dz);
      }
      __syncwarp();
      if (q8 < 3) {
        float f = FUSED ? 0.f : run;
        for (int c = 0; c < take; ++c) f = __fadd_rn(f, prod[q8][pl][c]);
        if (FUSED) sum += f2d_fast(f); else run = f;
      }
      // the entries past the batch to the front
      const int left = m - take;
      const int mv = q8 < left ? jl[pl][take + q8] : 0;
      __syncwarp();
      if (q8 < left) jl[pl][q8] = mv;
      m = left;
      __syncwarp();
    }
    if (q8 < 3) tot[q8][pl] = FUSED ? sum : (double)run;
    if (EFLAG) {
      int sl[8];
      float v[8];
      sl[0] = O_VFF; v[0] = e_lj;
      sl[1] = O_VCOUL; v[1] = e_c;
      sym_slots(sl + 2, v + 2, O_VIR + 9 * V_PAIR, wv);
      obs_push<float, 8>(acc, sl, v, rep, active);
    }
  }
  __syncthreads();
  if (!tail) return;
  float ike = 0.f, ikin[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, ifh[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (inside) {
    double fxd = tot[0][lane], fyd = tot[1][lane], fzd = tot[2][lane];
    if (BONDED && active) {
      fxd += f2d_fast(fb[0]);
      fyd += f2d_fast(fb[1]);
      fzd += f2d_fast(fb[2]);
    }
    if constexpr (INTEG) {
      if (active) {
        int_mixed_particle<2, EFLAG>(s, C, i, w, d2f_fast(fxd), d2f_fast(fyd), d2f_fast(fzd), s.pfx_alt, s.vf_alt,
                                     ike, ikin, ifh);
      } else if (C.move_walls) {  // a wall bead on a moving wall: its next site
        double x, y, z;
        s.pfx_alt[i] = move_wall_bead(s, C, i, w, x, y, z);
        s.vf_alt[i] = s.vf[i];
      } else {  // a wall bead: its views as they are
        s.pfx_alt[i] = s.pfx[i];
        s.vf_alt[i] = s.vf[i];
      }
      if (i == 0) *s.steps_alt = *s.steps_done + 1;
    } else if constexpr (FUSED) {
      s.f4[i] = make_float4(d2f_fast(fxd), d2f_fast(fyd), d2f_fast(fzd), 0.f);
    } else if (active) {
      s.fx[i] += fxd;
      s.fy[i] += fyd;
      s.fz[i] += fzd;
    }
  }
  if constexpr (EFLAG && FUSED) {
    constexpr int NB = bond_values(BONDED), NI = INTEG ? 13 : 0, NV = NB + 2 + NI;
    int sl[NV];
    float v[NV];
    if constexpr (BONDED == BOND_ALL) bonded_slots(sl, v, eb, bv);
    if constexpr (BONDED == BOND_FENE) fene_slots(sl, v, eb, bv);
    sl[NB] = O_VFW; v[NB] = wall_e[lane];
    sl[NB + 1] = O_VIR + 9 * V_WALL + 8; v[NB + 1] = wall_w[lane];
    if constexpr (INTEG) {
      constexpr int b = NB + 2;
      const int idx[6] = {0, 4, 8, 1, 2, 5};
      sl[b] = O_TFLUID; v[b] = ike;
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        sl[b + 1 + c] = O_KIN + idx[c]; v[b + 1 + c] = ikin[c];
        sl[b + 7 + c] = O_FH + c; v[b + 7 + c] = ifh[c];
      }
    }
    obs_push<float, NV>(acc, sl, v, rep, active);
  }
}

template <bool EFLAG>
static void launch_pair_lanes(const DevState& s, const SimConst& C, cudaStream_t st, bool fused, Acc acc, int mask,
                              bool uni, bool integ) {
  using KernT = void (*)(DevState, SimConst, Acc, int);
  // [integ][bonded][uni]
#define LANES(I, B) {k_pair_lanes<EFLAG, true, B, false, I>, k_pair_lanes<EFLAG, true, B, true, I>}
  const KernT kf[2][3][2] = {{LANES(false, BOND_NONE), LANES(false, BOND_FENE), LANES(false, BOND_ALL)},
                             {LANES(true, BOND_NONE), LANES(true, BOND_FENE), LANES(true, BOND_ALL)}};
#undef LANES
  const KernT kd[2] = {k_pair_lanes<EFLAG, false, BOND_NONE, false, false>, k_pair_lanes<EFLAG, false, BOND_NONE, true, false>};
  const KernT k = fused ? kf[integ ? 1 : 0][bond_kind(mask)][uni ? 1 : 0] : kd[uni ? 1 : 0];
  k<<<(s.N + PL_P - 1) / PL_P, PL_T, 0, st>>>(s, C, acc, mask);
}

// The pair kernel of the FP64 mode.  The FP64 pipe bounds it (an FP64 instruction of a warp holds it
// for 16 clocks however many lanes are active), so (1) the list is screened in FP32 on the fixed-point
// view, (2) the kept pairs of a warp's particles are put together and evaluated 32 at a time, a
// lane per pair whoever owns it (a thread per particle left half of the lanes idle: the kept counts
// of neighbours differ; 16 brush replicas 6648 -> 4146 us a call of 10 steps with (3), and 9700
// before the screening in FP32; 3830 now), and (3) the roots, divisions and noise are those of mfa_dev.cuh.  The
// factors and distances go back through shared memory and each owner adds its own in list order, so the
// sums do not depend on which lane evaluated a pair (multiply-adds: products rounded before the sums were
// 0.5 % further from 64-bit-exact forces).  A warp on a replica boundary evaluates each lane's own
// pairs instead, so that the energy sums (by lane) stay with their replica.
// With G lanes per particle (4 or 8) a warp takes 32 / G particles: their lists are screened side by
// side, and a small system has G times as many warps, whose serial chain of loads and FP64 results is
// what its time is then.  The kept pairs and the order of the sums are the same.  G = 1 fills the rounds
// best (150 pairs of 32 WCA particles instead of 38 of 8).  Pair kernel, us, G = 1 / 4 / 8: WCA, 6400
// particles 42 / 19 / 19; 2.24 sigma, 6800 213 / 77 / 73; charged, 32.5 k 247 / 138 / 132.
constexpr int P64_BATCH = 8;  // kept pairs per lane and round
struct Pair64Warp {           // shared memory of a warp
  double own[6][32];          // its particles' positions and half-step velocities
  double f[32 * P64_BATCH];     // force factor of each kept pair
  double d[3][32 * P64_BATCH];  // and its distance from the owner
  int tag[32], type[32];
  int j[32 * P64_BATCH];
  unsigned char who[32 * P64_BATCH];
};

template <bool EFLAG, bool UNI, int G>
__global__ void __launch_bounds__(128, 4) k_pair64(DevState s, SimConst C, bool accumulate, Acc acc) {
  extern __shared__ __align__(16) unsigned char sh_raw[];
  __shared__ PairEntry<double> tab[NPAIR];
  __shared__ float scr[NPAIR];
  for (int k = threadIdx.x; k < NPAIR; k += blockDim.x) {
    tab[k] = s.tabd[k];
    scr[k] = s.tabf[k].screen2;
  }
  __syncthreads();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  Pair64Warp& W = reinterpret_cast<Pair64Warp*>(sh_raw)[threadIdx.x >> 5];
  constexpr int BATCH = P64_BATCH * G;
  const int own = lane / G, sub = lane % G;  // the lane's particle of the warp's 32 / G
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const bool inside = i < s.N;
  const int w = __ldg(&s.info[min(i, s.N - 1)]);  // (the lanes past the end take the last replica)
  const bool active = inside && info_mobile(w);
  const int rep = info_rep(w);
  const bool one = __all_sync(FULL, rep == __shfl_sync(FULL, rep, 0));
  const RepDesc& R = s.reps[rep];
  const long long step = R.s_time + *s.steps_done;
  const double r2min = C.force_switch_on ? r2min_of(C, step) : 0.;
  const int p0 = R.p0, ti = info_type(w);
  const uint32_t nkey = pair_key(R.seed, step);
  const double L0 = R.L[0], L1 = R.L[1], iL0 = R.invL[0], iL1 = R.invL[1];
  const int n = active ? __ldg(&s.nn[i]) : 0;
  const int* __restrict__ nb = s.nbr + i;
  int4 qi = make_int4(0, 0, 0, 0);
  if (active) {
    qi = __ldg(&s.pfx[i]);
    if (sub == 0) {
      const dbl4 x = s.pd[i], v = s.vd[i];
      W.own[0][own] = x.x; W.own[1][own] = x.y; W.own[2][own] = x.z;
      W.own[3][own] = v.x; W.own[4][own] = v.y; W.own[5][own] = v.z;
      W.tag[own] = (int)__double_as_longlong(v.w) - p0;
      W.type[own] = ti;
    }
  }
  const float cx = R.ufx_f[0] * 512.f, cy = R.ufx_f[1] * 512.f, cz = R.ufx_f[2] * 512.f;
  auto screen = [&](int j) -> bool {  // as the mixed kernel's
    const int4 qj = __ldg(&s.pfx[j]);
    const float dx = i2f_coarse(fx_diff(qi.x, qj.x), 9) * cx;
    const float dy = i2f_coarse(fx_diff(qi.y, qj.y), 9) * cy;
    const float dz = i2f_coarse(fx_diff(qi.z, qj.z), 9) * cz;
    return dx * dx + dy * dy + dz * dz < (UNI ? C.scr2_uni_f : scr[ti * MAXT + info_type(qj.w)]);
  };
  double fx = 0., fy = 0., fz = 0., e_lj = 0., e_c = 0.;
  double wv[6] = {0., 0., 0., 0., 0., 0.};  // EFLAG: pair virial, xx yy zz xy xz yz
  int k = 0;
  while (__any_sync(FULL, k < n)) {
    // the particle's next kept pairs, at most BATCH, first in its own row of W.j
    int m = 0;
    if constexpr (G == 1) {
      while (k < n && m < BATCH) {
        constexpr int F = 4;  // entries whose loads are in flight together
        if (k + F <= n && m <= BATCH - F) {
          int jg[F];
          bool hg[F];
#pragma unroll
          for (int u = 0; u < F; ++u) jg[u] = __ldg(nb + (size_t)(k + u) * s.Np);
#pragma unroll
          for (int u = 0; u < F; ++u) hg[u] = screen(jg[u]);
#pragma unroll
          for (int u = 0; u < F; ++u)
            if (hg[u]) W.j[lane * BATCH + m++] = jg[u];
          k += F;
        } else {
          const int j = __ldg(nb + (size_t)k * s.Np);
          ++k;
          if (screen(j)) W.j[lane * BATCH + m++] = j;
        }
      }
    } else {
      constexpr int F = 2;  // G entries at a time, F of these in flight together
      while (__any_sync(FULL, k < n && m <= BATCH - F * G)) {
        const bool room = m <= BATCH - F * G;
        int jg[F];
        bool hg[F];
#pragma unroll
        for (int u = 0; u < F; ++u) {
          const int e = k + u * G + sub;
          jg[u] = room && e < n ? __ldg(nb + (size_t)e * s.Np) : -1;
        }
#pragma unroll
        for (int u = 0; u < F; ++u) hg[u] = jg[u] >= 0 && screen(jg[u]);
#pragma unroll
        for (int u = 0; u < F; ++u) {
          const unsigned bits = (__ballot_sync(FULL, hg[u]) >> (own * G)) & ((1u << G) - 1u);
          if (hg[u]) W.j[own * BATCH + m + __popc(bits & ((1u << sub) - 1u))] = jg[u];
          m += __popc(bits);
        }
        if (room) k += F * G;
      }
      __syncwarp();
    }
    // then together: owner after owner, each in list order
    int at = sub == 0 ? m : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, at, o);
      if (lane >= o) at += y;
    }
    const int total = __shfl_sync(FULL, at, 31);
    at -= m;
    int mine[P64_BATCH];
#pragma unroll
    for (int t = 0; t < P64_BATCH; ++t) mine[t] = (t * G + sub < m) ? W.j[own * BATCH + t * G + sub] : 0;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < P64_BATCH; ++t)
      if (t * G + sub < m) {
        W.j[at + t * G + sub] = mine[t];
        W.who[at + t * G + sub] = (unsigned char)own;
      }
    __syncwarp();
    const int rounds = one ? (total + 31) >> 5 : ((int)__reduce_max_sync(FULL, (unsigned)m) + G - 1) / G;
    for (int t = 0; t < rounds; ++t) {
      const int q = one ? 32 * t + lane : at + t * G + sub;
      if (one ? q < total : t * G + sub < m) {
        const int j = W.j[q], o = W.who[q];
        const dbl4 pj = s.pd[j];
        const double dx = mic_fast(W.own[0][o] - pj.x, L0, iL0);
        const double dy = mic_fast(W.own[1][o] - pj.y, L1, iL1);
        const double dz = W.own[2][o] - pj.z;
        const int wj = (int)__double_as_longlong(pj.w);
        // half of each mobile pair (both ends sum it); a fixed wall bead has no list of its own
        const double half = info_mobile(wj) ? 0.5 : 1.;
        const double fs = pair_fs64<EFLAG>(s, C, tab[W.type[o] * MAXT + info_type(wj)], dx, dy, dz, j, W.own[3][o],
                                           W.own[4][o], W.own[5][o], W.tag[o], p0, nkey, r2min, half, e_lj, e_c);
        W.f[q] = fs;
        W.d[0][q] = dx;
        W.d[1][q] = dy;
        W.d[2][q] = dz;
        if (EFLAG) sym_add(wv, half * fs, dx, dy, dz);
      }
    }
    __syncwarp();
    if constexpr (G == 1) {
      for (int t = 0; t < m; ++t) {
        const double fs = W.f[at + t];
        fx = fma(fs, W.d[0][at + t], fx);
        fy = fma(fs, W.d[1][at + t], fy);
        fz = fma(fs, W.d[2][at + t], fz);
      }
    } else if (sub < 3) {  // (a lane per component, in fx)
      for (int t = 0; t < m; ++t) fx = fma(W.f[at + t], W.d[sub][at + t], fx);
    }
    __syncwarp();
  }
  if constexpr (G == 1) {
    if (inside) {
      if (!accumulate) {
        s.fx[i] = fx;
        s.fy[i] = fy;
        s.fz[i] = fz;
      } else if (active) {
        s.fx[i] += fx;
        s.fy[i] += fy;
        s.fz[i] += fz;
      }
    }
  } else if (inside && sub < 3) {
    double* f = sub == 0 ? s.fx : (sub == 1 ? s.fy : s.fz);
    if (!accumulate) f[i] = fx;
    else if (active) f[i] += fx;
  }
  if (EFLAG) {
    int sl[8];
    double v[8];
    sl[0] = O_VFF; v[0] = e_lj;
    sl[1] = O_VCOUL; v[1] = e_c;
    sym_slots(sl + 2, v + 2, O_VIR + 9 * V_PAIR, wv);
    // (a warp of one replica: every lane has evaluated pairs, the ends' lanes too)
    obs_push<double, 8>(acc, sl, v, rep, one ? true : active);
  }
}

void launch_pair(const DevState& s, const SimConst& C, cudaStream_t st, bool accumulate, bool eflag, Acc acc,
                 int block, int bonded_mask, bool integ) {
  // 32, 64 or 128 threads per block (the kernel is compiled for at most 128); anything else
  // takes the built-in 128
  const int B = (block == 32 || block == 64) ? block : 128;
  const int g = (s.N + B - 1) / B;
  const bool uni = C.scr2_uni_f > 0.f;
  // Lanes per particle for systems too small to fill the GPU with threads (an explicit block size or
  // the persistent schedule asks for k_pair).  The line follows the lists' length, for which the capacity
  // that the library chooses stands (61 entries with the WCA cut-off, 180 with 2.24 sigma, 284 with a Coulomb
  // cut-off of 3): lanes / thread per particle took 17 / 19 us at 20 k and 24 / 19 at 40 k particles (WCA), 56 / 71
  // at 42 k and 93 / 86 at 83 k (2.24 sigma), 55 / 68 at 64 k and 94 / 91 at 130 k (charged).  (A capacity of
  // 420 given by the caller put WCA channels of up to 168 k particles on the wrong side.)
  const bool lanes = s.mixed && B == 128 && block != 128 && s.N <= 400ll * s.list_len &&
                     !(s.pair_persist && !accumulate && !eflag);
  if (lanes) {
    if (eflag) launch_pair_lanes<true>(s, C, st, !accumulate, acc, bonded_mask, uni, integ);
    else launch_pair_lanes<false>(s, C, st, !accumulate, acc, bonded_mask, uni, integ);
  } else if (s.mixed && !accumulate) {  // the fused step
    using KernT = void (*)(DevState, SimConst, bool, Acc, int);
    // [eflag][bonded][uni]: forces alone, the persistent schedule, with the step's integration in the tail
#define PAIRK(E, B, P, I) {k_pair<E, true, B, false, P, I>, k_pair<E, true, B, true, P, I>}
#define PAIRB(E, P, I) {PAIRK(E, BOND_NONE, P, I), PAIRK(E, BOND_FENE, P, I), PAIRK(E, BOND_ALL, P, I)}
    const KernT ks[2][3][2] = {PAIRB(false, false, false), PAIRB(true, false, false)};
    const KernT kp[3][2] = PAIRB(false, true, false);
    const KernT ki[2][3][2] = {PAIRB(false, false, true), PAIRB(true, false, true)};
#undef PAIRB
#undef PAIRK
    const int bi = bond_kind(bonded_mask), ui = uni ? 1 : 0;
    if (integ) {
      ki[eflag ? 1 : 0][bi][ui]<<<g, B, 0, st>>>(s, C, false, acc, bonded_mask);
    } else if (s.pair_persist && !eflag) {
      const KernT k = kp[bi][ui];
      int per_sm = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, B, 0);
      const int grid = std::min(g, std::max(per_sm, 1) * s.nsm);
      k<<<grid, B, 0, st>>>(s, C, false, acc, bonded_mask);
    } else {
      ks[eflag ? 1 : 0][bi][ui]<<<g, B, 0, st>>>(s, C, false, acc, bonded_mask);
    }
  } else if (s.mixed) {  // the drop-in: added to the FP64 force
    if (eflag) k_pair<true><<<g, B, 0, st>>>(s, C, true, acc);
    else k_pair<false><<<g, B, 0, st>>>(s, C, true, acc);
  } else {
    using KernT = void (*)(DevState, SimConst, bool, Acc);
#define PAIR64(G) {{k_pair64<false, false, G>, k_pair64<true, false, G>}, {k_pair64<false, true, G>, k_pair64<true, true, G>}}
    const KernT kd[3][2][2] = {PAIR64(1), PAIR64(4), PAIR64(8)};
#undef PAIR64
    // Lanes per particle by the particles and the lists' length (as above: 61 entries with the WCA
    // cut-off, 180 with 2.24 sigma, 284 with a Coulomb cut-off of 3; an explicit block size asks for one).
    // 4 lanes / one took, us: WCA 35 / 43 at 19.6 k, 62 / 61 at 40 k, 107 / 89 at 78 k; 2.24 sigma 202 / 244
    // at 21 k, 682 / 716 at 83 k, 2471 / 2485 at 333 k; charged 138 / 247 at 32 k, 384 / 474 at 130 k.
    // 8 lanes / 4: WCA 12 / 17 at 2.3 k, 19 / 19 at 6.4 k, 42 / 35 at 20 k; 2.24 sigma 73 / 77 at 6.8 k, 207 / 202
    // at 21 k; charged 80 / 96 at 16 k, 132 / 138 at 32 k, 223 / 216 at 64 k;
    // explicit walls 23 / 21 at 7200.
    const bool given = block == 32 || block == 64 || block == 128;
    const int lg = given || s.N > 10ll * s.list_len * s.list_len ? 0 : (s.N > 60ll * s.list_len ? 1 : 2);
    const long long threads = (long long)s.N * (lg == 0 ? 1 : (lg == 1 ? 4 : 8));
    // the warps are independent, so one per block: with four the slowest holds the others' place (16 brush
    // replicas, 128 / 64 / 32 threads: 243 / 238 / 237 us; 1 M particles 911 / 890 / 886)
    const int B64 = given ? block : 32;
    kd[lg][uni ? 1 : 0][eflag ? 1 : 0]<<<(int)((threads + B64 - 1) / B64), B64, B64 / 32 * sizeof(Pair64Warp), st>>>(
        s, C, accumulate, acc);
  }
}

void launch_bonded(const DevState& s, const SimConst& C, cudaStream_t st, int mask, bool eflag, Acc acc,
                   bool fused) {
  if (!mask) return;
  int B = 128, g = (s.N + B - 1) / B;
  const bool by_tag = s.N > B * s.nsm;  // (more than four warps per SM)
  if (s.mixed) {
    if (eflag) k_bonded<true, true><<<g, B, 0, st>>>(s, C, mask, acc, fused, by_tag);
    else k_bonded<true, false><<<g, B, 0, st>>>(s, C, mask, acc, fused, by_tag);
  } else {
    if (eflag) k_bonded<false, true><<<g, B, 0, st>>>(s, C, mask, acc, false, by_tag);
    else k_bonded<false, false><<<g, B, 0, st>>>(s, C, mask, acc, false, by_tag);
  }
}

// ---------------------------------------------------------------------------------------------
// Implicit 9-3 walls and the constant body force
// ---------------------------------------------------------------------------------------------
template <bool EFLAG>
__global__ void k_wall(DevState s, SimConst C, Acc acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool inside = i < s.N;
  const int w = inside ? s.info[i] : 0;
  const bool active = inside && info_mobile(w);
  double e = 0., wzz = 0.;
  if (active) {
    const RepDesc& R = s.reps[info_rep(w)];
    const double z = s.rz[i];
    double fb, ft;
    wall93_split(C, info_type(w), z, R.L[2], fb, ft, e);
    s.fz[i] += fb + ft;
    wzz = fb * z + ft * (z - R.L[2]);  // each wall's force times z - z_wall
  }
  if (EFLAG) {
    const int sl[2] = {O_VFW, O_VIR + 9 * V_WALL + 8};
    const double v[2] = {e, wzz};
    obs_push<double, 2>(acc, sl, v, info_rep(w), active);
  }
}

void launch_wall(const DevState& s, const SimConst& C, cudaStream_t st, bool eflag, Acc acc) {
  int B = 256, g = (s.N + B - 1) / B;
  if (eflag) k_wall<true><<<g, B, 0, st>>>(s, C, acc);
  else k_wall<false><<<g, B, 0, st>>>(s, C, acc);
}

__global__ void k_cforce(DevState s, SimConst C) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.N) return;
  const int w = s.info[i];
  if (!info_mobile(w) || info_type(w) == 0) return;
  const double m = C.mass[info_type(w)];
  s.fx[i] += m * C.const_force[0];
  s.fy[i] += m * C.const_force[1];
  s.fz[i] += m * C.const_force[2];
}

void launch_const_force(const DevState& s, const SimConst& C, cudaStream_t st) {
  int B = 256, g = (s.N + B - 1) / B;
  k_cforce<<<g, B, 0, st>>>(s, C);
}

// ---------------------------------------------------------------------------------------------
// Pair list export: every interacting pair (local tags, i<j) of replica `rep`, FP64 distances.
// ---------------------------------------------------------------------------------------------
__global__ void k_pair_list(DevState s, SimConst C, int rep, int* __restrict__ out, long long cap,
                            unsigned long long* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.N) return;
  const int w = s.info[i];
  if (info_rep(w) != rep || !info_mobile(w)) return;
  const RepDesc& R = s.reps[rep];
  const int ti = info_type(w), tgi = s.tag[i];
  const int n = s.nn[i];
  for (int k = 0; k < n; ++k) {
    int j = s.nbr[(size_t)k * s.Np + i];
    int wj = s.info[j];
    int tgj = s.tag[j];
    if (!info_mobile(wj) || tgj <= tgi) continue;
    double dx = mic_ref(s.rx[i] - s.rx[j], R.L[0], R.invL[0]);
    double dy = mic_ref(s.ry[i] - s.ry[j], R.L[1], R.invL[1]);
    double dz = s.rz[i] - s.rz[j];
    double r2 = dx * dx + dy * dy + dz * dz;
    const PairEntry<double>& e = s.tabd[ti * MAXT + info_type(wj)];
    bool hit = r2 < e.range2;
    if (!hit && (e.flags & PF_DPD_OWN)) hit = r2 < e.dpd_rc2;
    if (!hit && (e.flags & PF_COUL) && C.coul_rc2 > 0.) hit = r2 < C.coul_rc2;
    if (hit) {
      unsigned long long k2 = atomicAdd(count, 1ull);
      if ((long long)k2 < cap) {
        out[2 * k2] = tgi - R.p0;
        out[2 * k2 + 1] = tgj - R.p0;
      }
    }
  }
}

void launch_pair_list(const DevState& s, const SimConst& C, cudaStream_t st, int rep, int* pairs, long long cap,
                      unsigned long long* count) {
  int B = 128, g = (s.N + B - 1) / B;
  k_pair_list<<<g, B, 0, st>>>(s, C, rep, pairs, cap, count);
}

}  // namespace mfa
