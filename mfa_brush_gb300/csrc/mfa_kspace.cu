// mfa_kspace.cu -- reciprocal-space Ewald sum with the slab correction on the device.
//
// ewald_k.f90:128-202 evaluates rho(k) = sum_i q_i exp(i k.r_i) over N_k half-space vectors and
// then F_i = -(8 pi q_i / V) sum_k k G(k) (cos(k.r_i) Im rho - sin(k.r_i) Re rho),
// U = (4 pi / V) sum_k G(k) |rho(k)|^2, G(k) = exp(-k^2/(4 alpha_c)) / k^2, storing an N x N_k
// phase array.  Here nothing of size N x N_k is stored.  The k-vectors come kz outer, ky, kx
// inner, so a (ky, kz) "row" of k shares the factor Y(ky) Z(kz) and only X(kx) varies along it:
//   k_ks_tables:  per charged particle, X(nx) = exp(i nx dkx x), Y(ny), Z(nz) for n >= 0, each
//                 from a phase in 64-bit turns (plain FP64 form: reduced in FP64); stored column-major
//                 ([column][particle]) so that a warp reads 32 particles of one column at once;
//   k_ks_rho:     rho(row, nx) = sum_p (q Y Z)(p, row) X(p, nx) as a complex matrix product per
//                 block of up to 64 rows x 16 |nx| slots x a particle chunk, +nx and -nx from the same
//                 four real sums (X(-n) = conj X(n)): lane = slot, half-warp = 4 rows, tiles of
//                 32 particles in shared memory; plain sums over a tile and Kahan-compensated
//                 sums across tiles in FP32 (MIXED), or FP64 sums; one partial per particle
//                 chunk;
//   k_ks_rho_sum: the partials of each k summed in a fixed order; G rho per k and the dense
//                 (row, slot) table of (G rho, kx G rho) for the force; U reduced
//                 deterministically (per-block partials, the last block adds them);
//   k_ks_force_dense (mixed, nxm <= 15): thread per particle with X(0..nxm) in registers, a
//                 chunk of 32 rows per block streamed from the dense table with its +nx and -nx
//                 slots folded together: per row S = sum conj(X) G rho and
//                 S_x = sum conj(X) kx G rho, then Im(conj(Y Z) S_x) to F_x and ky, kz times
//                 Im(conj(Y Z) S) to F_y, F_z; rows added with Kahan compensation;
//   k_ks_force:   the same per row, one k at a time from shared memory (nxm > 15);
//   k_ks_rho_q, k_ks_fold_q, k_ks_force_q: rho, the folded table and the dense force of the FP64 mode
//                 for nxm <= 15, in two-limb integers;
//   k_ks_force_sum: the chunk partials in a fixed order, times -8 pi q / V, into the force array.
// dipolar_correction.f90:20-33 (Yeh-Berkowitz slab term), FP64: the moment in blocks of its own of
// k_ks_tables, the force in k_ks_force_sum.
// Every sum has a fixed order, so a charged run is reproducible bit for bit.  A batch runs each
// kernel once for all replicas (the last grid dimension; the blocks past a replica's own extent
// leave): launched replica by replica, 7 kernels each, twelve small charged channels spent 825 us a
// step in launches one behind the other.  A replica's work is divided as it is alone, so its sums
// are those of the replica run alone.
#include <algorithm>
#include <type_traits>

#include "mfa_grid.h"
#include "mfa_state.cuh"

namespace mfa {

template <bool MIXED>
using kreal = typename std::conditional<MIXED, float, double>::type;
template <bool MIXED>
using kcplx = typename std::conditional<MIXED, float2, double2>::type;

__device__ __forceinline__ void cmul(float2 a, float2 b, float2& c) {
  c = make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cmul(double2 a, double2 b, double2& c) {
  c = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// s += y: Kahan-compensated in FP32 (c carries the negated lost low part) unless `plain` (the
// precision study of mfa_options.kspace_plain_sums), plain in FP64
template <bool MIXED>
__device__ __forceinline__ void ksum(kreal<MIXED>& s, kreal<MIXED>& c, kreal<MIXED> y, bool plain = false) {
  if constexpr (MIXED) {
    if (plain) {
      s += y;
      return;
    }
    const float z = y - c;
    const float t = s + z;
    c = (t - s) - z;
    s = t;
  } else {
    s += y;
  }
}

template <bool MIXED>
__device__ __forceinline__ const kcplx<MIXED>* ktab(const KSpace& K) {
  if constexpr (MIXED) return K.tabf; else return K.tabd;
}

// Two FP32 multiply-adds in one instruction (each rounded as fmaf rounds): the sums below are bound by
// instruction issue, and a packed one takes one slot for two.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}

// (a - ca) + (b - cb) with the compensations ca, cb of sums a, b: rounded sum and remainder (Knuth)
__device__ __forceinline__ float2 two_sum(float a, float b, float ca, float cb) {
  const float h = __fadd_rn(a, b), t = __fsub_rn(h, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(h, t)), __fsub_rn(b, t));
  return make_float2(h, __fsub_rn(e, __fadd_rn(ca, cb)));
}

// a column of the tables into shared memory, asynchronously
template <typename Cx>
__device__ __forceinline__ void cp_async(Cx* to, const Cx* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
               "n"(sizeof(Cx))
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---- the FP64 mode's sums in integers -----------------------------------------------------------
// An FP64 multiply-add of a warp holds the SM's FP64 pipe for 16 clocks; three 32 x 32 + 64 bit integer
// ones do the same work in two fifths of that (charged brush, 13,760 charges and 8070 k: rho 903 -> 306
// us, force 1740 -> 597).  A number v, |v| <= 1, is held in two limbs, v = h 2^-27 +
// l 2^-57 with |l| <= 2^29 (57 bits behind the point; a double in [1/2, 1) has 53).  A product keeps
// h h' (in units of 2^-54) and h l' + l h' (2^-84), each summed exactly in 64 bits; l l', at most 2^-56
// and of either sign, is left out.  The k sets of up to 15 waves per axis (nxm) take this path.
constexpr double QL_MAGIC = 6755399441055744.0;  // 1.5 * 2^52: the low word of the sum is the integer

__device__ __forceinline__ int2 ql_of(double v) {
  const double t = fma(v, 134217728.0, QL_MAGIC);
  const double r = fma(v, 134217728.0, QL_MAGIC - t);
  return make_int2(__double2loint(t), __double2loint(fma(r, 1073741824.0, QL_MAGIC)));
}
struct QlSum {
  long long h, m;
  __device__ __forceinline__ void zero() { h = m = 0; }
  __device__ __forceinline__ void add(int2 a, int2 b) {
    h += (long long)a.x * b.x;
    m += (long long)a.x * b.y;
    m += (long long)a.y * b.x;
  }
  __device__ __forceinline__ long long q54() const { return h + ((m + (1ll << 29)) >> 30); }  // units of 2^-54
  // units of 2^-58, for sums below 16
  __device__ __forceinline__ long long q58() const { return (h << 4) + ((m + (1ll << 25)) >> 26); }
};
// The high limb of a number that is not finite: in a q Z column it marks the particle, and what its
// chunk sums (k_ks_rho_q) is then NaN, as a sum in floating point would be.
constexpr int QL_NAN = (int)0x80000000;
__device__ __forceinline__ bool nonfinite(double v) { return (__double2hiint(v) & 0x7FF00000) == 0x7FF00000; }
__device__ __forceinline__ int2 ql_neg(int2 a) { return make_int2(-a.x, -a.y); }
// the limbs of t units of 2^-58, |t| <= 2^58
__device__ __forceinline__ int2 ql_limbs(long long t) {
  const long long h = (t + (1ll << 30)) >> 31;
  return make_int2((int)h, ((int)(t - (h << 31)) + 1) >> 1);
}
__device__ __forceinline__ int2 ql_re(int4 a) { return make_int2(a.x, a.y); }
__device__ __forceinline__ int2 ql_im(int4 a) { return make_int2(a.z, a.w); }
// (a b) of complex numbers of modulus at most 1
__device__ __forceinline__ int4 ql_cmul(int4 a, int4 b) {
  QlSum re, im;
  re.zero();
  im.zero();
  re.add(ql_re(a), ql_re(b));
  re.add(ql_neg(ql_im(a)), ql_im(b));
  im.add(ql_re(a), ql_im(b));
  im.add(ql_im(a), ql_re(b));
  const int2 x = ql_limbs(re.q58()), y = ql_limbs(im.q58());
  return make_int4(x.x, x.y, y.x, y.y);
}

constexpr int KS_TILE = 32;  // particles per shared-memory tile of k_ks_rho (one per lane)

// rho(row, nx) = sum_p A(p, row) X(p, nx), A = q Y(ny) Z(nz), with X(p, -n) = conj X(p, n): the
// four real sums P1 = sum a c, P2 = sum b d, P3 = sum a d, P4 = sum b c over A = a + ib,
// X(p, n) = c + id give both rho(row, n) = (P1 - P2, P3 + P4) and rho(row, -n) = (P1 + P2,
// P4 - P3).  A block takes KS_RB rows, 16 slots n = 16 z .. 16 z + 15 and a chunk of
// particles, in tiles of 32.  Lane l owns slot n = 16 z + (l & 15); warp w owns rows 8 w .. 8 w + 7,
// four of them per half-warp (l >> 4).  Per particle a lane reads its X (the half-warps share the 16
// slots) and its four A (two 16-byte loads, one address per half-warp) for 16 multiply-adds, packed
// by two in FP32 (P1, P2 from (a, b) (c, d), P3, P4 from (a, b) (d, c)), which cover up to eight k.
// Slots outside a row's k-range are computed and not stored.  The table columns that the block's
// rows and slots use are copied a tile ahead (cp.async); the A of a tile is formed from them.  (Read
// from global memory when the tile began, their latency stood before every tile: with the packed
// sums 57 -> 39 us on the charged brush.)  The Y and Z columns are the ranges
// that the block's rows use, at most KS_BC of them (KsRowBlock): they fit however long the box is.  (A block
// of one or two tiles waits mostly for its first loads: with the ranges read one load behind K, or a list of
// columns behind a barrier, twelve small charged channels took 21.8 us, now 20.7.)
constexpr int KS_RHO_T = 256;  // threads of a k_ks_rho block (8 warps)
constexpr int KS_RW = 8;       // rows per warp (four per half-warp)
constexpr int KS_CS = KS_TILE + 1;  // column stride (odd: 16 slots of one particle are 16 banks apart)
constexpr int KS_AS = KS_RB + 2;  // A row stride (16-byte aligned rows)
static_assert(KS_TILE * KS_AS * sizeof(float2) % 16 == 0, "the columns follow the A rows 16-byte aligned");

template <bool MIXED>
__global__ void __launch_bounds__(KS_RHO_T, MIXED ? 3 : 1) k_ks_rho(const KSpace* __restrict__ Ks,
                                                                             const KsRowBlock* __restrict__ rblk, int nz) {
  const KSpace K = Ks[blockIdx.z / nz];
  const KsRowBlock Q = rblk[blockIdx.z / nz * gridDim.x + blockIdx.x];  // (beside K, not behind it)
  const int zs = blockIdx.z % nz;
  if (Q.nr == 0 || (int)blockIdx.y >= K.npchunks || zs * KS_SL > K.nxm || K.nq == 0) return;
  if (!MIXED && K.dense) return;  // (k_ks_rho_q)
  using real = kreal<MIXED>;
  using Cx = kcplx<MIXED>;
  extern __shared__ __align__(16) unsigned char shraw[];
  Cx* As = reinterpret_cast<Cx*>(shraw);              // [KS_TILE][KS_AS]
  int2* rc = reinterpret_cast<int2*>(As + KS_TILE * KS_AS);  // [KS_RB] signed Y column, Z column (of a tile)
  Cx* cols = reinterpret_cast<Cx*>(rc + KS_RB);       // two tiles of columns: 16 X, the block's Y and Z
  const Cx* tab = ktab<MIXED>(K);
  const int rbeg = Q.row, nr = Q.nr, ncols = KS_SL + Q.ny + Q.nz;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  constexpr int NW = KS_RHO_T / 32;
  constexpr int RL = KS_RW / 2;  // rows per lane
  const int slot = zs * KS_SL + (lane & (KS_SL - 1));  // |nx| of the lane
  const int r0 = warp * KS_RW + half * RL;             // the lane's first row
  const bool act = r0 < nr;
  const int p_beg = blockIdx.y * K.pchunk, p_end = min(K.nq, p_beg + K.pchunk);
  auto fetch = [&](int t0, int buf) {
    const int pq = t0 + lane;
    if (pq < p_end) {
      Cx* to = cols + buf * ncols * KS_CS + lane;
      for (int c = warp; c < ncols; c += NW) {
        const int n = zs * KS_SL + c;  // X column
        const int col = c < KS_SL ? n : (c < KS_SL + Q.ny ? K.nxm + 1 + Q.ylo + c - KS_SL
                                                          : K.nxm + K.nym + 2 + Q.zlo + c - KS_SL - Q.ny);
        if (c >= KS_SL || n <= K.nxm) cp_async(to + c * KS_CS, tab + (size_t)col * K.nq + pq);
      }
    }
    cp_async_commit();
  };
  // (X slots past nxm are never fetched: zero in both tiles)
  for (int c = K.nxm + 1 - zs * KS_SL + warp; c < KS_SL; c += NW) {
    Cx zero;
    zero.x = zero.y = 0;
    if (c >= 0) cols[c * KS_CS + lane] = cols[(ncols + c) * KS_CS + lane] = zero;
  }
  real s[4][RL], c[4][RL];  // sums P1..P4 across tiles and their compensations
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int i = 0; i < RL; ++i) s[a][i] = c[a][i] = 0;
  fetch(p_beg, 0);
  for (int r = threadIdx.x; r < nr; r += KS_RHO_T) {
    const int4 R = K.rows[rbeg + r];
    const int yc = KS_SL + abs(R.z) - Q.ylo;
    rc[r] = make_int2(R.z < 0 ? -yc : yc, KS_SL + Q.ny + R.w - Q.zlo);
  }
  int buf = 0;
  for (int t0 = p_beg; t0 < p_end; t0 += KS_TILE, buf ^= 1) {
    const int nt = min(KS_TILE, p_end - t0);
    real q = 0;
    if (lane < nt) {
      if constexpr (MIXED) q = K.qvalf[t0 + lane]; else q = K.qval[t0 + lane];
    }
    cp_async_wait<0>();
    __syncthreads();  // this tile's columns are here; the A and columns of the tile before are used up
    fetch(t0 + KS_TILE, buf ^ 1);  // (nothing past the last tile)
    const Cx* col = cols + buf * ncols * KS_CS;
    if (lane < nt) {
#pragma unroll
      for (int h = 0; h < KS_RB / NW; ++h) {
        const int r = warp + NW * h;
        if (r < nr) {
          const int2 R = rc[r];
          Cx y = col[abs(R.x) * KS_CS + lane];
          const Cx z = col[R.y * KS_CS + lane];
          if (R.x < 0) y.y = -y.y;
          Cx A;
          cmul(y, z, A);
          A.x *= q;
          A.y *= q;
          As[lane * KS_AS + r] = A;
        }
      }
    }
    __syncthreads();
    if (act) {
      // plain sums over the tile's particles, compensated sums across tiles
      const Cx* xs = col + (lane & (KS_SL - 1)) * KS_CS;
      if constexpr (MIXED) {
        float2 t01[RL], t23[RL];
#pragma unroll
        for (int i = 0; i < RL; ++i) t01[i] = t23[i] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int p = 0; p < nt; ++p) {
          const float2 x = xs[p], xr = make_float2(x.y, x.x);
          const float4* A4 = reinterpret_cast<const float4*>(As + p * KS_AS + r0);
#pragma unroll
          for (int i = 0; i < RL / 2; ++i) {
            const float4 u = A4[i];
            const float2 a = make_float2(u.x, u.y), b = make_float2(u.z, u.w);
            t01[2 * i] = ffma2(a, x, t01[2 * i]);
            t23[2 * i] = ffma2(a, xr, t23[2 * i]);
            t01[2 * i + 1] = ffma2(b, x, t01[2 * i + 1]);
            t23[2 * i + 1] = ffma2(b, xr, t23[2 * i + 1]);
          }
        }
#pragma unroll
        for (int i = 0; i < RL; ++i) {
          ksum<MIXED>(s[0][i], c[0][i], t01[i].x, K.plain);
          ksum<MIXED>(s[1][i], c[1][i], t01[i].y, K.plain);
          ksum<MIXED>(s[2][i], c[2][i], t23[i].x, K.plain);
          ksum<MIXED>(s[3][i], c[3][i], t23[i].y, K.plain);
        }
      } else {
        real t[4][RL];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int i = 0; i < RL; ++i) t[a][i] = 0;
#pragma unroll 1
        for (int p = 0; p < nt; ++p) {
          const Cx x = xs[p];
#pragma unroll
          for (int i = 0; i < RL; ++i) {
            const Cx A = As[p * KS_AS + r0 + i];
            t[0][i] = fma(A.x, x.x, t[0][i]);
            t[1][i] = fma(A.y, x.y, t[1][i]);
            t[2][i] = fma(A.x, x.y, t[2][i]);
            t[3][i] = fma(A.y, x.x, t[3][i]);
          }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int i = 0; i < RL; ++i) ksum<MIXED>(s[a][i], c[a][i], t[a][i], K.plain);
      }
    }
  }
  if (act && slot <= K.nxm) {
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      const int r = r0 + i;
      if (r < nr) {
        const int4 R = K.rows[rbeg + r];
        const int lo = K.kn[R.x].x;  // the row's first nx
        const int kp = R.x + slot - lo, km = R.x - slot - lo;
        const bool hp = kp >= R.x && kp < R.y, hm = slot > 0 && km >= R.x && km < R.y;
        if constexpr (MIXED) {
          // P +- P' as an unevaluated FP32 sum (48 bits): FP64 here, all blocks at their ends at
          // once, took a quarter of the kernel
          float4* o = reinterpret_cast<float4*>(K.rho_part) + (size_t)blockIdx.y * K.nk;
          const float2 a = two_sum(s[0][i], -s[1][i], c[0][i], -c[1][i]), b = two_sum(s[2][i], s[3][i], c[2][i], c[3][i]);
          const float2 e = two_sum(s[0][i], s[1][i], c[0][i], c[1][i]), f = two_sum(s[3][i], -s[2][i], c[3][i], -c[2][i]);
          if (hp) o[kp] = make_float4(a.x, a.y, b.x, b.y);
          if (hm) o[km] = make_float4(e.x, e.y, f.x, f.y);
        } else {
          double2* o = reinterpret_cast<double2*>(K.rho_part) + (size_t)blockIdx.y * K.nk;
          if (hp) o[kp] = make_double2(s[0][i] - s[1][i], s[2][i] + s[3][i]);
          if (hm) o[km] = make_double2(s[0][i] + s[1][i], s[3][i] - s[2][i]);
        }
      }
    }
  }
}

// The same in integer limbs (FP64 mode, K.dense): lanes, rows and tiles as k_ks_rho; the tables are
// those of X, Y and q Z / q_max.  A tile's sums go to 64-bit totals in units of 2^-51 (a chunk holds at most
// 2048 particles: a total, and the sums of two that a k takes, stay at or below 2^62).
__global__ void __launch_bounds__(KS_RHO_T, 2) k_ks_rho_q(const KSpace* __restrict__ Ks, const KsRowBlock* __restrict__ rblk,
                                                           int nz) {
  const KSpace K = Ks[blockIdx.z / nz];
  const KsRowBlock Q = rblk[blockIdx.z / nz * gridDim.x + blockIdx.x];
  const int zs = blockIdx.z % nz;
  if (!K.dense || Q.nr == 0 || (int)blockIdx.y >= K.npchunks || zs > 0 || K.nq == 0) return;
  extern __shared__ __align__(16) unsigned char shraw[];
  int4* As = reinterpret_cast<int4*>(shraw);                 // [KS_TILE][KS_RB + 1]
  int2* rc = reinterpret_cast<int2*>(As + KS_TILE * (KS_RB + 1));
  int4* cols = reinterpret_cast<int4*>(rc + KS_RB);          // two tiles of columns: 16 X, the block's Y and Z
  const int rbeg = Q.row, nr = Q.nr, ncols = KS_SL + Q.ny + Q.nz;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  constexpr int NW = KS_RHO_T / 32, RL = KS_RW / 2;
  const int slot = lane & (KS_SL - 1), r0 = warp * KS_RW + half * RL;
  const bool act = r0 < nr;
  const int p_beg = blockIdx.y * K.pchunk, p_end = min(K.nq, p_beg + K.pchunk);
  auto fetch = [&](int t0, int buf) {
    const int pq = t0 + lane;
    if (pq < p_end) {
      int4* to = cols + buf * ncols * KS_CS + lane;
      for (int c = warp; c < ncols; c += NW) {
        const int col = c < KS_SL ? c : (c < KS_SL + Q.ny ? K.nxm + 1 + Q.ylo + c - KS_SL
                                                          : K.ncol + Q.zlo + c - KS_SL - Q.ny);
        if (c >= KS_SL || c <= K.nxm) cp_async(to + c * KS_CS, K.tabq + (size_t)col * K.nq + pq);
      }
    }
    cp_async_commit();
  };
  for (int c = K.nxm + 1 + warp; c < KS_SL; c += NW)
    cols[c * KS_CS + lane] = cols[(ncols + c) * KS_CS + lane] = make_int4(0, 0, 0, 0);
  long long tot[4][RL];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int i = 0; i < RL; ++i) tot[a][i] = 0;
  int bad = 0;  // a particle that is not finite (every particle of the chunk comes by with the first row)
  fetch(p_beg, 0);
  for (int r = threadIdx.x; r < nr; r += KS_RHO_T) {
    const int4 R = K.rows[rbeg + r];
    const int yc = KS_SL + abs(R.z) - Q.ylo;
    rc[r] = make_int2(R.z < 0 ? -yc : yc, KS_SL + Q.ny + R.w - Q.zlo);
  }
  int buf = 0;
  for (int t0 = p_beg; t0 < p_end; t0 += KS_TILE, buf ^= 1) {
    const int nt = min(KS_TILE, p_end - t0);
    cp_async_wait<0>();
    __syncthreads();  // this tile's columns are here; the A and columns of the tile before are used up
    fetch(t0 + KS_TILE, buf ^ 1);
    const int4* col = cols + buf * ncols * KS_CS;
    if (lane < nt) {
#pragma unroll 2
      for (int h = 0; h < KS_RB / NW; ++h) {
        const int r = warp + NW * h;
        if (r < nr) {
          const int2 R = rc[r];
          int4 y = col[abs(R.x) * KS_CS + lane];
          if (R.x < 0) { y.z = -y.z; y.w = -y.w; }
          const int4 z = col[R.y * KS_CS + lane];
          bad |= z.x == QL_NAN;
          As[lane * (KS_RB + 1) + r] = ql_cmul(y, z);
        }
      }
    }
    __syncthreads();
    if (act) {
      const int4* xs = col + slot * KS_CS;
      QlSum t[4][RL];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int i = 0; i < RL; ++i) t[a][i].zero();
#pragma unroll 1
      for (int p = 0; p < nt; ++p) {
        const int4 x = xs[p];
#pragma unroll
        for (int i = 0; i < RL; ++i) {
          const int4 A = As[p * (KS_RB + 1) + r0 + i];
          t[0][i].add(ql_re(A), ql_re(x));
          t[1][i].add(ql_im(A), ql_im(x));
          t[2][i].add(ql_re(A), ql_im(x));
          t[3][i].add(ql_im(A), ql_re(x));
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int i = 0; i < RL; ++i) tot[a][i] += (t[a][i].q54() + 4) >> 3;
    }
  }
  bad = __syncthreads_or(bad);
  if (act && slot <= K.nxm) {
    const double sc = bad ? nan("") : K.qmax * 4.4408920985006262e-16;  // 2^-51
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      const int r = r0 + i;
      if (r < nr) {
        const int4 R = K.rows[rbeg + r];
        const int lo = K.kn[R.x].x, kp = R.x + slot - lo, km = R.x - slot - lo;
        double2* o = reinterpret_cast<double2*>(K.rho_part) + (size_t)blockIdx.y * K.nk;
        if (kp >= R.x && kp < R.y)
          o[kp] = make_double2((double)(tot[0][i] - tot[1][i]) * sc, (double)(tot[2][i] + tot[3][i]) * sc);
        if (slot > 0 && km >= R.x && km < R.y)
          o[km] = make_double2((double)(tot[0][i] + tot[1][i]) * sc, (double)(tot[3][i] - tot[2][i]) * sc);
      }
    }
  }
}

// Block sum of v (all threads, warps in order); the same value in every thread.
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double b = 0.;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b += red[w];
  return b;
}

// Block sum of v (all threads), then the last of `blocks` blocks to finish adds the per-block
// partials: each of its threads a strided subset in order, then a block sum; a fixed order for
// a given grid.  Returns true in thread 0 of that block, with the total in `total`.
__device__ __forceinline__ bool grid_sum_last(double v, double* part, unsigned* ticket, unsigned blocks,
                                              double& total) {
  __shared__ double red[32];
  __shared__ bool last;
  const double b = block_sum(v, red);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(ticket, 1u) == blocks - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double t = 0.;
  for (unsigned k = threadIdx.x; k < blocks; k += blockDim.x) t += ((volatile double*)part)[k];
  t = block_sum(t, red);
  if (threadIdx.x != 0) return false;
  total = t;
  *ticket = 0u;  // ready for the next launch
  return true;
}

// The same for NV values at once; part holds blocks x NV partials.
template <int NV>
__device__ __forceinline__ bool grid_sum_last_n(const double* v, double* part, unsigned* ticket, unsigned blocks,
                                                double* total) {
  __shared__ double red[32];
  __shared__ bool last;
  double b[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) b[c] = block_sum(v[c], red);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < NV; ++c) part[(size_t)blockIdx.x * NV + c] = b[c];
    __threadfence();
    last = atomicAdd(ticket, 1u) == blocks - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double t[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) t[c] = 0.;
  for (unsigned k = threadIdx.x; k < blocks; k += blockDim.x)
#pragma unroll
    for (int c = 0; c < NV; ++c) t[c] += ((volatile double*)part)[(size_t)k * NV + c];
#pragma unroll
  for (int c = 0; c < NV; ++c) t[c] = block_sum(t[c], red);
  if (threadIdx.x != 0) return false;
#pragma unroll
  for (int c = 0; c < NV; ++c) total[c] = t[c];
  *ticket = 0u;  // ready for the next launch
  return true;
}

// parts of the sum that a launch covers
constexpr int KS_RECIP = 1, KS_DIPOLE = 2;
__host__ __device__ inline int ks_dipole_blocks(int nq) {
  return nq > 0 ? (nq + KS_TAB_T - 1) / KS_TAB_T < KS_RED_MAX ? (nq + KS_TAB_T - 1) / KS_TAB_T : KS_RED_MAX : 0;
}

// Blocks 0 .. ks_dipole_blocks - 1 of a replica: the dipole moment; the blocks from dblk on: the tables.
template <bool MIXED>
__global__ void __launch_bounds__(KS_TAB_T) k_ks_tables(DevState s, const KSpace* __restrict__ Ks, int dblk, int what,
                                                        double pi, Acc acc, bool eflag) {
  const KSpace& K = Ks[blockIdx.y];
  if ((int)blockIdx.x < dblk) {
    const int nb = ks_dipole_blocks(K.nq);
    if (!(what & KS_DIPOLE) || (int)blockIdx.x >= nb) return;
    double m = 0.;
    for (int p = blockIdx.x * KS_TAB_T + threadIdx.x; p < K.nq; p += nb * KS_TAB_T)
      m += K.qval[p] * (s.rz[s.slot_of_tag[K.qtag[p]]] - K.lz_half);
    double tot;
    if (grid_sum_last(m, K.red_part + 7 * KS_RED_MAX, K.ticket + 1, nb, tot)) {
      K.mz[0] = tot;
      if (eflag) acc.col(O_VDIP)[K.rep] += 2. * pi * tot * tot * K.inv_V;
    }
    return;
  }
  const unsigned idx = (blockIdx.x - dblk) * KS_TAB_T + threadIdx.x, nq = K.nq;
  const int ncol = (!MIXED && K.dense) ? K.ncolq : K.ncol;
  if (!(what & KS_RECIP) || K.nk == 0 || idx >= nq * ncol) return;
  int col = idx / nq;
  const int p = idx - col * nq;
  const int i = s.slot_of_tag[K.qtag[p]];
  const bool times_q = col >= K.ncol;  // (the limb tables hold q Z / q_max as well)
  if (times_q) col -= K.nzm + 1;
  int n = col, ax = 0;
  if (col > K.nxm + 1 + K.nym) { n = col - K.nxm - K.nym - 2; ax = 2; }
  else if (col > K.nxm) { n = col - K.nxm - 1; ax = 1; }
  // the phase of n = 1 in turns as a 64-bit fixed point (2^-58), times n with wrap-around: as a signed
  // number of 2^-64 it is the phase in [-1/2, 1/2) turns.  One FP64 product; in FP64 the products, the reduction
  // and the conversions of a column bound this kernel.
  double t = (ax == 0 ? K.cx * s.rx[i] : (ax == 1 ? K.cy * s.ry[i] : K.cz * s.rz[i]));
  bool bad = nonfinite(t);  // (the integers below know no NaN)
  if ((__double2hiint(t) & 0x7FFFFFFF) >= 0x40200000) t -= rint(t);  // (8 turns away: not wrapped yet)
  if constexpr (MIXED) {
    const unsigned long long ph = (unsigned long long)round_bits<58>(t) * (unsigned)n << 6;
    float sn, cs;
    // 2 ph / 2^64 from all of its bits: the upper half in two exact parts, the lower half rounded (below the
    // rounding of the sum)
    const int hi = (int)(ph >> 32);
    const float low = fmaf(__int_as_float(0x4B000000 | (hi & 0xFFFF)) - 8388608.0f, 4294967296.0f, __uint2float_rn((unsigned)ph));
    sincospif(fmaf(__int_as_float(0x4B400000 + (hi >> 16)) - 12582912.0f, 3.0517578125e-05f,
                   low * 1.08420217248550443401e-19f), &sn, &cs);
    K.tabf[idx] = bad ? make_float2(nanf(""), nanf("")) : make_float2(cs, sn);
  } else if (K.dense) {
    // the same phase to 64 bits: the nearest of 1024 table angles and the angle from it by the series
    const unsigned long long ph = (unsigned long long)round_bits<58>(t) * (unsigned)n << 6;
    const int k = (int)((ph + (1ull << 53)) >> 54) & 1023;
    const long long lo = (long long)(ph << 10) >> 10;  // ph mod 2^54, signed
    const double d = (double)lo * (6.283185307179586476925 / 18446744073709551616.0);  // 2 pi / 2^64
    const double2 a = __ldg(&s.noise->cs[k]);
    const double d2 = d * d, c = fma(d2, fma(d2, 1.0 / 24.0, -0.5), 1.0);
    const double e = d * fma(d2, fma(d2, 1.0 / 120.0, -1.0 / 6.0), 1.0);
    double re = fma(a.x, c, -(a.y * e)), im = fma(a.y, c, a.x * e);
    if (times_q) {
      const double q = K.qval[p] * K.inv_qmax;
      re *= q;
      im *= q;
      bad = bad || nonfinite(s.rx[i]) || nonfinite(s.ry[i]);
    }
    const int2 x = ql_of(re), y = ql_of(im);
    K.tabq[idx] = make_int4(bad ? QL_NAN : x.x, x.y, y.x, y.y);
  } else {
    double u = (double)n * t;
    u -= rint(u);  // turns in [-1/2, 1/2]
    double sn, cs;
    sincospi(2. * u, &sn, &cs);
    K.tabd[idx] = make_double2(cs, sn);
  }
}

// Thread (k, g) of a block of 32 k x 8 groups sums the chunk partials c = g, g + 8, ..; the
// eight group sums are then added in group order: a fixed order for every k.  With energies, the
// reciprocal-space virial sum over k of u_k (delta_ab - 2 k_a k_b (1/k^2 + 1/(4 alpha_c))) as well
// (u_k = G |rho|^2, the k's term of the energy), the derivative of the energy under a deformation
// of the cell.
template <bool MIXED>
__global__ void __launch_bounds__(256) k_ks_rho_sum(const KSpace* __restrict__ Ks, double pi4, double fac_alpha, Acc acc,
                                                    bool eflag) {
  const KSpace K = Ks[blockIdx.y];
  const int nkb = (K.nk + 31) / 32, blocks = min(KS_RED_MAX, nkb);  // blocks of this replica
  if ((int)blockIdx.x >= blocks || K.nq == 0) return;
  __shared__ double2 part[8][32];
  const int kl = threadIdx.x & 31, g = threadIdx.x >> 5;
  double u[7] = {0., 0., 0., 0., 0., 0., 0.};  // energy, then the virial xx yy zz xy xz yz
  for (int kb = blockIdx.x; kb < nkb; kb += blocks) {
    const int k = kb * 32 + kl;
    double re = 0., im = 0.;
    if (k < K.nk) {
#pragma unroll 4
      for (int c = g; c < K.npchunks; c += 8) {
        if constexpr (MIXED) {
          const float4 v = reinterpret_cast<const float4*>(K.rho_part)[(size_t)c * K.nk + k];
          re += f2d_nan(v.x) + f2d_nan(v.y);
          im += f2d_nan(v.z) + f2d_nan(v.w);
        } else {
          const double2 v = reinterpret_cast<const double2*>(K.rho_part)[(size_t)c * K.nk + k];
          re += v.x;
          im += v.y;
        }
      }
    }
    part[g][kl] = make_double2(re, im);
    __syncthreads();
    if (g == 0 && k < K.nk) {
      re = 0.;
      im = 0.;
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        re += part[h][kl].x;
        im += part[h][kl].y;
      }
      const double G = K.kfac[k];
      const double uk = G * (re * re + im * im);
      u[0] += uk;
      if (eflag) {
        const double kx = K.kvec[3 * k], ky = K.kvec[3 * k + 1], kz = K.kvec[3 * k + 2];
        const double c = 2. * (1. / (kx * kx + ky * ky + kz * kz) + fac_alpha) * uk;
        u[1] += uk - c * kx * kx;
        u[2] += uk - c * ky * ky;
        u[3] += uk - c * kz * kz;
        u[4] -= c * kx * ky;
        u[5] -= c * kx * kz;
        u[6] -= c * ky * kz;
      }
      if constexpr (MIXED) {
        const double kx = K.kvec[3 * k], a = G * re, b = G * im;
        const int xi = K.kn[k].x + K.nxm;
        K.kdf[k] = make_float4((float)kx, (float)a, (float)b, __int_as_float(xi));
        K.wdense[(size_t)K.fpos[K.krow[k]] * 4 * K.qx + xi] =
            make_float4((float)a, (float)b, (float)(kx * a), (float)(kx * b));
      } else {
        K.kdd[k] = make_double2(G * re, G * im);
      }
    }
    __syncthreads();
  }
  if (!eflag) return;
  double tot[7];
  if (grid_sum_last_n<7>(u, K.red_part, K.ticket, blocks, tot)) {
    const double sc = pi4 * K.inv_V;
    acc.col(O_VCOULK)[K.rep] += tot[0] * sc;
    const int idx[6] = {0, 4, 8, 1, 2, 5};
    for (int c = 0; c < 6; ++c) acc.col(O_VIR + 9 * V_KSPACE + idx[c])[K.rep] += tot[1 + c] * sc;
  }
}

template <bool MIXED>
struct KD;
template <>
struct KD<true> {
  float kx, a, b;  // kx, G Re rho, G Im rho
  int xi;          // nx + nxm
};
template <>
struct KD<false> {
  double kx, a, b;
  int xi, pad;
};

template <bool MIXED>
__global__ void __launch_bounds__(KS_FB) k_ks_force(const KSpace* __restrict__ Ks) {
  const KSpace K = Ks[blockIdx.z];
  if (K.dense || (int)blockIdx.x * KS_FB >= K.nq || (int)blockIdx.y >= K.nkchunks) return;
  using real = kreal<MIXED>;
  using Cx = kcplx<MIXED>;
  using real2 = kcplx<MIXED>;
  extern __shared__ __align__(16) unsigned char shraw[];
  const int nxc = 2 * K.nxm + 1;
  Cx* Xs = reinterpret_cast<Cx*>(shraw);                              // [nxc][KS_FB]
  KD<MIXED>* kd = reinterpret_cast<KD<MIXED>*>(Xs + nxc * KS_FB);     // [fchunk_k_max]
  int4* rs = reinterpret_cast<int4*>(kd + K.fchunk_k_max);            // [fchunk_rows_max]
  real2* ryz = reinterpret_cast<real2*>(rs + K.fchunk_rows_max);      // [fchunk_rows_max] ky, kz
  const int rb = K.chunk_row[blockIdx.y], re = K.chunk_row[blockIdx.y + 1];
  const int kb = K.rows[rb].x, ke = K.rows[re - 1].y;
  for (int k = kb + threadIdx.x; k < ke; k += KS_FB) {
    KD<MIXED> d;
    if constexpr (MIXED) {
      const float4 v = K.kdf[k];
      d.kx = v.x;
      d.a = v.y;
      d.b = v.z;
      d.xi = __float_as_int(v.w);
    } else {
      const double2 v = K.kdd[k];
      d.kx = K.kvec[3 * k];
      d.a = v.x;
      d.b = v.y;
      d.xi = K.kn[k].x + K.nxm;
      d.pad = 0;
    }
    kd[k - kb] = d;
  }
  for (int r = rb + threadIdx.x; r < re; r += KS_FB) {
    const int4 R = K.rows[r];
    const int yc = K.nxm + 1 + abs(R.z);
    rs[r - rb] = make_int4(R.x - kb, R.y - kb, R.z < 0 ? -yc : yc, K.nxm + K.nym + 2 + R.w);
    real2 w;
    w.x = (real)K.kvec[3 * R.x + 1];
    w.y = (real)K.kvec[3 * R.x + 2];
    ryz[r - rb] = w;
  }
  const Cx* tab = ktab<MIXED>(K);
  const int p = blockIdx.x * KS_FB + threadIdx.x;
  const int pc = min(p, K.nq - 1);
  for (int c = 0; c < nxc; ++c) {
    Cx v = tab[(size_t)abs(c - K.nxm) * K.nq + pc];
    if (c < K.nxm) v.y = -v.y;
    Xs[c * KS_FB + threadIdx.x] = v;
  }
  __syncthreads();
  if (p >= K.nq) return;
  const Cx* T = tab + pc;
  const Cx* X = Xs + threadIdx.x;
  real fx = 0, fy = 0, fz = 0, cx = 0, cy = 0, cz = 0;
  const int nr = re - rb;
  int4 R = rs[0];
  Cx Y = T[(size_t)abs(R.z) * K.nq], Z = T[(size_t)R.w * K.nq];
  for (int r = 0; r < nr; ++r) {
    // the next row's factors are loaded while this row is summed
    int4 Rn = R;
    Cx Yn = Y, Zn = Z;
    if (r + 1 < nr) {
      Rn = rs[r + 1];
      Yn = T[(size_t)abs(Rn.z) * K.nq];
      Zn = T[(size_t)Rn.w * K.nq];
    }
    if (R.z < 0) Y.y = -Y.y;
    Cx YZ;
    cmul(Y, Z, YZ);
    // plain sums along the row (at most 2 nxm + 1 terms), compensated sums across rows
    real srow = 0, sxrow = 0;
#pragma unroll 4
    for (int k = R.x; k < R.y; ++k) {
      const KD<MIXED> d = kd[k];
      Cx E;
      cmul(X[d.xi * KS_FB], YZ, E);
      const real sg = E.x * d.b - E.y * d.a;
      sxrow = fma(d.kx, sg, sxrow);
      srow += sg;
    }
    const real2 w = ryz[r];
    ksum<MIXED>(fx, cx, sxrow, K.plain);
    ksum<MIXED>(fy, cy, w.x * srow, K.plain);
    ksum<MIXED>(fz, cz, w.y * srow, K.plain);
    R = Rn;
    Y = Yn;
    Z = Zn;
  }
  double* o = K.fpart + ((size_t)blockIdx.y * K.nq + p) * 3;
  o[0] = (double)fx - (double)cx;
  o[1] = (double)fy - (double)cy;
  o[2] = (double)fz - (double)cz;
}

// Mixed precision, nxm <= 15: the thread keeps X(p, n) for n = 0 .. nxm in registers and reads
// the slot table of a chunk of rows from shared memory.  With S = sum_nx conj(X) W and
// Sx = sum_nx conj(X) kx W over a row (W = G rho), that row adds Im(conj(Y Z) Sx) to F_x and
// ky, kz times Im(conj(Y Z) S) to F_y, F_z.  X(p, -n) = conj X(p, n) and kx(-n) = -kx(n), so the
// two signed slots +-n fold into one: with X(n) = c + id, W(n) = u + iv, W(-n) = u' + iv',
//   S  gets c (u + u') + d (v - v') + i [c (v + v') - d (u - u')],
//   Sx gets c (ku + ku') + d (kv - kv') + i [c (kv + kv') - d (ku - ku')],
// where ku = kx(n) u, ku' = kx(-n) u' (the table's kx W columns): eight FMAs per |n| from two
// broadcast 16-byte loads, where the signed slots took sixteen.  The block folds the signed slot
// table (k_ks_rho_sum's (W, kx W) per signed slot) while staging it.  The rows are taken in order
// of their slot range (frow), so that the rows of a chunk share a narrow window of slots; slots
// outside the window are skipped (a branch uniform over the block).
// A thread takes PP particles KS_FB apart: with one, the broadcast loads of the slots bound the kernel (L1
// at 83 %); two share them (68 -> 51 us on the charged brush, 13,760 charges and 509 rows; the
// multiply-adds alone, at 16 slots a row, are 23 us of the FP32 pipe).
template <int QF, int PP>
__global__ void __launch_bounds__(KS_FB) k_ks_force_dense(const KSpace* __restrict__ Ks) {
  const KSpace K = Ks[blockIdx.z];
  if (!K.dense || (int)blockIdx.x * KS_FB * PP >= K.nq || (int)blockIdx.y >= K.nkchunks) return;
  constexpr int NF = 4 * QF;  // folded slots |n| = 0 .. NF - 1
  extern __shared__ __align__(16) unsigned char shraw[];
  float4* Wd = reinterpret_cast<float4*>(shraw);              // [KS_FR][NF][2]
  int2* rc = reinterpret_cast<int2*>(Wd + KS_FR * NF * 2);    // [KS_FR] signed Y column, Z column
  float2* ryz = reinterpret_cast<float2*>(rc + KS_FR);        // [KS_FR] ky, kz
  const int rbeg = blockIdx.y * KS_FR, nr = min(KS_FR, K.nrows - rbeg);
  const int nxm = K.nxm, nsig = 4 * K.qx;
  const int2 win = K.fwin[blockIdx.y];  // signed slots win.x .. win.y (slot j is nx = j - nxm)
  // the folded window: |nx| from mlo to mhi
  const int ax = abs(win.x - nxm), ay = abs(win.y - nxm);
  const int mlo = (win.x <= nxm && nxm <= win.y) ? 0 : min(ax, ay), mhi = max(ax, ay);
  const float4* wsrc = K.wdense + (size_t)rbeg * nsig;
  for (int e = threadIdx.x; e < nr * NF; e += KS_FB) {
    const int r = e / NF, m = e - r * NF;
    float4 wp = make_float4(0.f, 0.f, 0.f, 0.f), wm = wp;
    if (m <= nxm) {
      wp = wsrc[r * nsig + nxm + m];
      if (m > 0) wm = wsrc[r * nsig + nxm - m];
    }
    // slots side by side by two, for the packed multiply-adds: of slots m, m + 1 the words 2 q, 2 q + 1
    // hold the q-th of (u + u', v - v', v + v', u' - u) and of the same of the Sx columns
    float* o = reinterpret_cast<float*>(Wd) + 16 * (e >> 1) + (e & 1);
    o[0] = wp.x + wm.x; o[2] = wp.y - wm.y; o[4] = wp.y + wm.y; o[6] = wm.x - wp.x;
    o[8] = wp.z + wm.z; o[10] = wp.w - wm.w; o[12] = wp.w + wm.w; o[14] = wm.z - wp.z;
  }
  for (int r = threadIdx.x; r < nr; r += KS_FB) {
    const int4 R = K.rows[K.frow[rbeg + r]];
    const int yc = nxm + 1 + abs(R.z);
    rc[r] = make_int2(R.z < 0 ? -yc : yc, nxm + K.nym + 2 + R.w);
    ryz[r] = make_float2((float)K.kvec[3 * R.x + 1], (float)K.kvec[3 * R.x + 2]);
  }
  const int p0 = blockIdx.x * KS_FB * PP + threadIdx.x;
  const float2* T[PP];
  float2 Xc[PP][NF / 2], Xd[PP][NF / 2];  // X = c + id of slots 2 j, 2 j + 1 as (c, c'), (d, d')
#pragma unroll
  for (int a = 0; a < PP; ++a) {
    T[a] = K.tabf + min(p0 + a * KS_FB, K.nq - 1);
#pragma unroll
    for (int j = 0; j < NF / 2; ++j) {
      float2 x = make_float2(0.f, 0.f), y = x;
      if (2 * j >= mlo && 2 * j <= mhi && 2 * j <= nxm) x = T[a][(size_t)(2 * j) * K.nq];
      if (2 * j + 1 >= mlo && 2 * j + 1 <= mhi && 2 * j + 1 <= nxm) y = T[a][(size_t)(2 * j + 1) * K.nq];
      Xc[a][j] = make_float2(x.x, y.x);
      Xd[a][j] = make_float2(x.y, y.y);
    }
  }
  __syncthreads();
  if (p0 >= K.nq) return;
  float F[PP][3], Fc[PP][3];  // sums and compensations
  float2 Y[PP], Z[PP];
  int2 R = rc[0];
#pragma unroll
  for (int a = 0; a < PP; ++a) {
#pragma unroll
    for (int d = 0; d < 3; ++d) F[a][d] = Fc[a][d] = 0.f;
    Y[a] = T[a][(size_t)abs(R.x) * K.nq];
    Z[a] = T[a][(size_t)R.y * K.nq];
  }
  for (int r = 0; r < nr; ++r) {
    int2 Rn = R;
    float2 YZ[PP];
#pragma unroll
    for (int a = 0; a < PP; ++a) {
      if (R.x < 0) Y[a].y = -Y[a].y;
      cmul(Y[a], Z[a], YZ[a]);
    }
    if (r + 1 < nr) {  // the next row's factors, while this one is summed
      Rn = rc[r + 1];
#pragma unroll
      for (int a = 0; a < PP; ++a) {
        Y[a] = T[a][(size_t)abs(Rn.x) * K.nq];
        Z[a] = T[a][(size_t)Rn.y * K.nq];
      }
    }
    const float4* w = Wd + r * NF * 2;
    float2 sr[PP], si[PP], xr[PP], xi[PP];  // S and Sx over even and odd slots
#pragma unroll
    for (int a = 0; a < PP; ++a) sr[a] = si[a] = xr[a] = xi[a] = make_float2(0.f, 0.f);
#pragma unroll
    for (int g = 0; g < QF; ++g) {  // groups of four slots; a group outside the window is skipped
      if (4 * g + 3 < mlo || 4 * g > mhi) continue;
#pragma unroll
      for (int i = 2 * g; i < 2 * g + 2; ++i) {
        const float4 u = w[4 * i], v = w[4 * i + 1], ux = w[4 * i + 2], vx = w[4 * i + 3];
#pragma unroll
        for (int a = 0; a < PP; ++a) {
          sr[a] = ffma2(Xc[a][i], make_float2(u.x, u.y), ffma2(Xd[a][i], make_float2(u.z, u.w), sr[a]));
          si[a] = ffma2(Xc[a][i], make_float2(v.x, v.y), ffma2(Xd[a][i], make_float2(v.z, v.w), si[a]));
          xr[a] = ffma2(Xc[a][i], make_float2(ux.x, ux.y), ffma2(Xd[a][i], make_float2(ux.z, ux.w), xr[a]));
          xi[a] = ffma2(Xc[a][i], make_float2(vx.x, vx.y), ffma2(Xd[a][i], make_float2(vx.z, vx.w), xi[a]));
        }
      }
    }
    const float2 kyz = ryz[r];
#pragma unroll
    for (int a = 0; a < PP; ++a) {
      const float srow = YZ[a].x * (si[a].x + si[a].y) - YZ[a].y * (sr[a].x + sr[a].y);
      const float sxrow = YZ[a].x * (xi[a].x + xi[a].y) - YZ[a].y * (xr[a].x + xr[a].y);
      ksum<true>(F[a][0], Fc[a][0], sxrow, K.plain);
      ksum<true>(F[a][1], Fc[a][1], kyz.x * srow, K.plain);
      ksum<true>(F[a][2], Fc[a][2], kyz.y * srow, K.plain);
    }
    R = Rn;
  }
#pragma unroll
  for (int a = 0; a < PP; ++a) {
    const int p = p0 + a * KS_FB;
    if (p >= K.nq) return;
    double* o = K.fpart + ((size_t)blockIdx.y * K.nq + p) * 3;
#pragma unroll
    for (int d = 0; d < 3; ++d) o[d] = f2d_nan(F[a][d]) - f2d_nan(Fc[a][d]);
  }
}

// The folded slot table of the dense force in limbs: a warp per row, lane m = |n|.  Per slot the eight
// words of k_ks_force_dense (kx as n; its unit goes into the row's factor), each row scaled by powers
// of two so that the sums over its slots stay within 1, and per row (ky, kz, dk) times its scale and the units of the integer sums.
__global__ void __launch_bounds__(128) k_ks_fold_q(const KSpace* __restrict__ Ks, int nf) {
  const KSpace K = Ks[blockIdx.y];
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), m = threadIdx.x & 31;  // (row in force order)
  if (!K.dense || K.nq == 0 || row >= K.nrows) return;
  const int4 R = K.rows[K.frow[row]];
  const int lo = K.kn[R.x].x, kp = R.x + m - lo, km = R.x - m - lo;
  double2 w = make_double2(0., 0.), v = w;
  if (m <= K.nxm && kp >= R.x && kp < R.y) w = K.kdd[kp];
  if (m > 0 && m <= K.nxm && km >= R.x && km < R.y) v = K.kdd[km];
  double a[8] = {w.x + v.x, w.y - v.y, w.y + v.y, v.x - w.x,
                 m * (w.x - v.x), m * (w.y + v.y), m * (w.y - v.y), -m * (w.x + v.x)};
  double sc[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    double br = fabs(a[4 * g]) + fabs(a[4 * g + 1]), bi = fabs(a[4 * g + 2]) + fabs(a[4 * g + 3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      br += __shfl_xor_sync(0xffffffffu, br, o);
      bi += __shfl_xor_sync(0xffffffffu, bi, o);
    }
    const double big = fmax(br, bi);
    // 2^-e with 2^e > big (1 for a row of zeros)
    const int e = big > 0. ? ((__double2hiint(big) >> 20) & 0x7FF) - 1022 : 0;
    const double down = __hiloint2double((1023 - e) << 20, 0);
    sc[g] = big == big ? __hiloint2double((1023 + e) << 20, 0) : big;  // (a NaN goes on in the row's factors)
#pragma unroll
    for (int c = 0; c < 4; ++c) a[4 * g + c] *= down;
  }
  if (m < nf) {
    int4* o = K.wq + ((size_t)row * nf + m) * 4;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int2 x = ql_of(a[2 * c]), y = ql_of(a[2 * c + 1]);
      o[c] = make_int4(x.x, x.y, y.x, y.y);
    }
  }
  if (m == 0) {
    const double unit = 3.4694469519536142e-18;  // 2^-58
    K.rowq[3 * row] = (double)(2. * M_PI) * K.cx * sc[1] * unit;
    K.rowq[3 * row + 1] = K.kvec[3 * R.x + 1] * sc[0] * unit;
    K.rowq[3 * row + 2] = K.kvec[3 * R.x + 2] * sc[0] * unit;
  }
}

// The dense force in integer limbs (FP64 mode): rows, slots, windows and partials as
// k_ks_force_dense; the sums of a row's 32 products are exact in 64 bits, and only the row's two results go to
// FP64.  Against 80-bit arithmetic the forces are 3.5e-16 off (r.m.s., of the largest), as the FP64
// kernels' were (3 to 15 waves, 40 to 4100 charges).
template <int QF>
__global__ void __launch_bounds__(KS_FB) k_ks_force_q(const KSpace* __restrict__ Ks, int nf) {
  const KSpace K = Ks[blockIdx.z];
  if (!K.dense || (int)blockIdx.x * KS_FB >= K.nq || (int)blockIdx.y >= K.nkchunks) return;
  constexpr int NF = 4 * QF;
  extern __shared__ __align__(16) unsigned char shraw[];
  int4* Wq = reinterpret_cast<int4*>(shraw);                // [KS_FR][NF][4]
  double* rw = reinterpret_cast<double*>(Wq + KS_FR * NF * 4);  // [KS_FR][3]
  int2* rc = reinterpret_cast<int2*>(rw + 3 * KS_FR);       // [KS_FR] signed Y column, Z column
  const int rbeg = blockIdx.y * KS_FR, nr = min(KS_FR, K.nrows - rbeg), nxm = K.nxm;
  const int2 win = K.fwin[blockIdx.y];
  const int ax = abs(win.x - nxm), ay = abs(win.y - nxm);
  const int mlo = (win.x <= nxm && nxm <= win.y) ? 0 : min(ax, ay), mhi = max(ax, ay);
  for (int e = threadIdx.x; e < nr * NF * 4; e += KS_FB) {
    const int r = e / (4 * NF), m = (e >> 2) - r * NF;
    Wq[e] = m < nf ? K.wq[((size_t)(rbeg + r) * nf + m) * 4 + (e & 3)] : make_int4(0, 0, 0, 0);
  }
  for (int r = threadIdx.x; r < 3 * nr; r += KS_FB) rw[r] = K.rowq[3 * rbeg + r];
  for (int r = threadIdx.x; r < nr; r += KS_FB) {
    const int4 R = K.rows[K.frow[rbeg + r]];
    const int yc = nxm + 1 + abs(R.z);
    rc[r] = make_int2(R.z < 0 ? -yc : yc, nxm + K.nym + 2 + R.w);
  }
  const int p = blockIdx.x * KS_FB + threadIdx.x;
  const int4* T = K.tabq + min(p, K.nq - 1);
  int4 X[NF];
#pragma unroll
  for (int j = 0; j < NF; ++j) {
    X[j] = make_int4(0, 0, 0, 0);
    if (j >= mlo && j <= mhi && j <= nxm) X[j] = T[(size_t)j * K.nq];
  }
  __syncthreads();
  if (p >= K.nq) return;
  double fx = 0., fy = 0., fz = 0.;
  int2 R = rc[0];
  int4 Y = T[(size_t)abs(R.x) * K.nq], Z = T[(size_t)R.y * K.nq];
#pragma unroll 1
  for (int r = 0; r < nr; ++r) {
    if (R.x < 0) { Y.z = -Y.z; Y.w = -Y.w; }
    const int4 YZ = ql_cmul(Y, Z);
    if (r + 1 < nr) {  // the next row's factors, while this one is summed
      R = rc[r + 1];
      Y = T[(size_t)abs(R.x) * K.nq];
      Z = T[(size_t)R.y * K.nq];
    }
    const int4* w = Wq + r * NF * 4;
    QlSum sr, si, xr, xi;
    sr.zero(); si.zero(); xr.zero(); xi.zero();
#pragma unroll
    for (int g = 0; g < QF; ++g) {  // (a branch per slot or two, or more blocks per SM, were 2-7 % slower)
      if (4 * g + 3 < mlo || 4 * g > mhi) continue;
#pragma unroll
      for (int j = 4 * g; j < 4 * g + 4; ++j) {
        const int4 u = w[4 * j], v = w[4 * j + 1], ux = w[4 * j + 2], vx = w[4 * j + 3];
        const int2 c = ql_re(X[j]), d = ql_im(X[j]);
        sr.add(c, ql_re(u)); sr.add(d, ql_im(u));
        si.add(c, ql_re(v)); si.add(d, ql_im(v));
        xr.add(c, ql_re(ux)); xr.add(d, ql_im(ux));
        xi.add(c, ql_re(vx)); xi.add(d, ql_im(vx));
      }
    }
    // Im(conj(Y Z) S) and Im(conj(Y Z) Sx) of the row
    QlSum a, b;
    a.zero();
    b.zero();
    const int2 yr = ql_re(YZ), yi = ql_neg(ql_im(YZ));
    a.add(yr, ql_limbs(si.q58())); a.add(yi, ql_limbs(sr.q58()));
    b.add(yr, ql_limbs(xi.q58())); b.add(yi, ql_limbs(xr.q58()));
    const double srow = (double)a.q58(), sxrow = (double)b.q58();
    fx = fma(sxrow, rw[3 * r], fx);
    fy = fma(srow, rw[3 * r + 1], fy);
    fz = fma(srow, rw[3 * r + 2], fz);
  }
  double* o = K.fpart + ((size_t)blockIdx.y * K.nq + p) * 3;
  o[0] = fx;
  o[1] = fy;
  o[2] = fz;
}

// F_i = -(8 pi q_i / V) * sum over k-chunks in a fixed order, and the slab term's -4 pi q_i M_z / V
// along z, added to the FP64 force array or, in the fused mixed-precision step, to the FP32 one.  A
// thread per component: the partials of a chunk are read in order.
__global__ void __launch_bounds__(128) k_ks_force_sum(DevState s, const KSpace* __restrict__ Ks, double pi, int what,
                                                      bool to_f4) {
  const KSpace K = Ks[blockIdx.y];
  const int idx = blockIdx.x * 128 + threadIdx.x;
  if (idx >= 3 * K.nq) return;
  const int p = idx / 3, d = idx - 3 * p;
  const int i = s.slot_of_tag[K.qtag[p]];
  const double q = K.qval[p];
  double* fd = d == 0 ? s.fx : (d == 1 ? s.fy : s.fz);
  float* f4 = reinterpret_cast<float*>(s.f4 + i) + d;
  if ((what & KS_RECIP) && K.nk > 0) {
    double f = 0.;
#pragma unroll 8
    for (int c = 0; c < K.nkchunks; ++c) f += K.fpart[(size_t)c * K.nq * 3 + idx];
    const double qf = -(8. * pi) * q * K.inv_V;
    if (to_f4) *f4 += (float)(qf * f);
    else fd[i] += qf * f;
  }
  if ((what & KS_DIPOLE) && d == 2) {
    const double f = -4. * pi * q * K.mz[0] * K.inv_V;
    if (to_f4) *f4 += (float)f;
    else fd[i] += f;
  }
}

namespace {
// (yz: the most Y and Z columns that the rows of a block use)
size_t rho_smem(int yz, bool mixed) {
  return ((size_t)KS_TILE * KS_AS + 2 * (size_t)(KS_SL + yz) * KS_CS) *
             (mixed ? sizeof(float2) : sizeof(double2)) +
         (size_t)KS_RB * sizeof(int2);
}
size_t force_smem(const KSpace& K, bool mixed) {
  const size_t cx = mixed ? sizeof(float2) : sizeof(double2);
  return (size_t)(2 * K.nxm + 1) * KS_FB * cx + (size_t)K.fchunk_k_max * (mixed ? sizeof(KD<true>) : sizeof(KD<false>)) +
         (size_t)K.fchunk_rows_max * (sizeof(int4) + cx);
}
// groups of four folded slots |nx| = 0 .. nxm of k_ks_force_dense
int dense_qf(const KSpace& K) { return (K.nxm + 4) / 4; }
// (the limb forms of the FP64 mode)
size_t rho_q_smem(int yz) {
  return ((size_t)KS_TILE * (KS_RB + 1) + 2 * (size_t)(KS_SL + yz) * KS_CS) * sizeof(int4) +
         (size_t)KS_RB * sizeof(int2);
}
size_t force_q_smem(int qf) {
  return (size_t)KS_FR * (4 * qf * 4 * sizeof(int4) + 3 * sizeof(double) + sizeof(int2));
}
size_t dense_smem(int qf) {
  return (size_t)KS_FR * (4 * qf * 2 * sizeof(float4) + sizeof(int2) + sizeof(float2));
}
constexpr int KS_DENSE_QX_MAX = 8;  // the register-resident X of k_ks_force_dense: nxm <= 15

template <int QF>
void launch_dense(const KSpace* Ks, size_t shm, dim3 g, int pp, cudaStream_t st) {
  if (pp == 2) k_ks_force_dense<QF, 2><<<g, KS_FB, shm, st>>>(Ks);
  else k_ks_force_dense<QF, 1><<<g, KS_FB, shm, st>>>(Ks);
}
template <int QF>
void launch_force_q(const KSpace* Ks, dim3 g, cudaStream_t st) {
  k_ks_force_q<QF><<<g, KS_FB, force_q_smem(QF), st>>>(Ks, 4 * QF);
}
typedef void (*force_q_launcher)(const KSpace*, dim3, cudaStream_t);
const force_q_launcher kForceQ[5] = {nullptr, launch_force_q<1>, launch_force_q<2>, launch_force_q<3>, launch_force_q<4>};
typedef void (*dense_launcher)(const KSpace*, size_t, dim3, int, cudaStream_t);
const dense_launcher kDense[5] = {nullptr, launch_dense<1>, launch_dense<2>, launch_dense<3>, launch_dense<4>};
}  // namespace

bool kspace_dense(const KSpace& K) { return K.qx <= KS_DENSE_QX_MAX; }
size_t kspace_force_smem(const KSpace& K, bool mixed) { return force_smem(K, mixed); }

int kspace_prepare(const KSpace& K, bool mixed) {
  const bool q = kspace_dense(K) && !mixed;
  const size_t a = q ? rho_q_smem(K.yz_max) : rho_smem(K.yz_max, mixed);
  const size_t b = q ? force_q_smem(dense_qf(K)) : (kspace_dense(K) ? dense_smem(dense_qf(K)) : force_smem(K, mixed));
  if (a > KS_SMEM_MAX || b > KS_SMEM_MAX) return (int)cudaErrorInvalidConfiguration;
  // The opt-in is a property of the kernel for the whole process, not of a context: set it to the
  // largest allowed size once, so that no context lowers it below another's needs (occupancy
  // follows the size of each launch, not this limit).
  const int mx = (int)KS_SMEM_MAX;
  cudaError_t e = cudaFuncSetAttribute(k_ks_rho<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ks_rho<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ks_force<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ks_force<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ks_rho_q, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  return (int)e;  // force_q_smem and dense_smem stay below 48 KB: 32 rows x 16 folded slots x 64 or 32 B + 1 KB
}

KSpaceBatch kspace_batch(const std::vector<KSpace>& Ks, bool mixed, int nsm) {
  KSpaceBatch B = {};
  // two particles per thread of the dense force kernel when that leaves every SM two blocks
  long long two = 0;
  for (const KSpace& K : Ks)
    if (kspace_dense(K)) two += (long long)((K.nq + 2 * KS_FB - 1) / (2 * KS_FB)) * K.nkchunks;
  B.pp = mixed && two >= 2 * nsm ? 2 : 1;
  B.n = (int)Ks.size();
  for (const KSpace& K : Ks) {
    if (K.nq == 0) continue;  // no charges: every block of this replica leaves
    B.dip = std::max(B.dip, ks_dipole_blocks(K.nq));
    const int ncol = (!mixed && kspace_dense(K)) ? K.ncolq : K.ncol;
    B.tab = std::max(B.tab, K.nk ? table_blocks(K.nq, ncol) : 0);
    B.nq = std::max(B.nq, K.nq);
    if (K.nk == 0) continue;
    if (!mixed && kspace_dense(K)) B.rho_q_shm = std::max(B.rho_q_shm, rho_q_smem(K.yz_max));
    else B.rho_shm = std::max(B.rho_shm, rho_smem(K.yz_max, mixed));
    B.nrows = std::max(B.nrows, K.nrows);
    B.rows = std::max(B.rows, K.nrblk);
    B.pchunks = std::max(B.pchunks, K.npchunks);
    B.nz = std::max(B.nz, (K.nxm + KS_SL) / KS_SL);
    B.sum = std::max(B.sum, std::min(KS_RED_MAX, (K.nk + 31) / 32));
    const int fb = (K.nq + KS_FB - 1) / KS_FB;
    if (kspace_dense(K)) {
      B.dense_p = std::max(B.dense_p, (fb + B.pp - 1) / B.pp);
      B.dense_k = std::max(B.dense_k, K.nkchunks);
      B.qf = std::max(B.qf, dense_qf(K));
    } else {
      B.force_p = std::max(B.force_p, fb);
      B.force_k = std::max(B.force_k, K.nkchunks);
      B.force_shm = std::max(B.force_shm, force_smem(K, mixed));
    }
  }
  return B;
}

static int launch_ks(const DevState& s, const SimConst& C, KSpaceBatch B, cudaStream_t st, int what, bool eflag,
                     Acc acc, bool to_f4) {
  if (B.nq == 0) return 0;
  const int most = 65535 / std::max(B.nz, 1);  // the last grid dimension holds nz per replica
  if (B.n > most) {
    KSpaceBatch A = B;
    A.n = most;
    B.d += most;
    B.rblk += (size_t)most * B.rows;
    B.n -= most;
    return launch_ks(s, C, A, st, what, eflag, acc, to_f4) + launch_ks(s, C, B, st, what, eflag, acc, to_f4);
  }
  const double pi = (double)3.1415926536f;  // mfa_common.f90:315 (single-precision literal)
  const bool recip = (what & KS_RECIP) && B.rows > 0;
  const int dblk = (what & KS_DIPOLE) ? B.dip : 0, tblk = recip ? B.tab : 0;
  int launches = 0;
  if (dblk + tblk > 0) {
    const dim3 g(dblk + tblk, B.n);
    if (s.mixed) k_ks_tables<true><<<g, KS_TAB_T, 0, st>>>(s, B.d, dblk, what, pi, acc, eflag);
    else k_ks_tables<false><<<g, KS_TAB_T, 0, st>>>(s, B.d, dblk, what, pi, acc, eflag);
    ++launches;
  }
  if (recip) {
    const dim3 g1(B.rows, B.pchunks, B.nz * B.n), g2(B.sum, B.n);
    const double fac_alpha = 1. / (4. * C.alpha_c);
    if (s.mixed) {
      k_ks_rho<true><<<g1, KS_RHO_T, B.rho_shm, st>>>(B.d, B.rblk, B.nz);
      k_ks_rho_sum<true><<<g2, 256, 0, st>>>(B.d, 4. * pi, fac_alpha, acc, eflag);
    } else {
      if (B.rho_shm) k_ks_rho<false><<<g1, KS_RHO_T, B.rho_shm, st>>>(B.d, B.rblk, B.nz);
      if (B.rho_q_shm) k_ks_rho_q<<<g1, KS_RHO_T, B.rho_q_shm, st>>>(B.d, B.rblk, B.nz);
      k_ks_rho_sum<false><<<g2, 256, 0, st>>>(B.d, 4. * pi, fac_alpha, acc, eflag);
    }
    launches += 2;
    if (B.dense_p && !s.mixed) {
      k_ks_fold_q<<<dim3((B.nrows + 3) / 4, B.n), 128, 0, st>>>(B.d, 4 * B.qf);
      kForceQ[B.qf](B.d, dim3(B.dense_p, B.dense_k, B.n), st);
      launches += 2;
    } else if (B.dense_p) {
      kDense[B.qf](B.d, dense_smem(B.qf), dim3(B.dense_p, B.dense_k, B.n), B.pp, st);
      ++launches;
    }
    if (B.force_p) {
      const dim3 g3(B.force_p, B.force_k, B.n);
      if (s.mixed) k_ks_force<true><<<g3, KS_FB, B.force_shm, st>>>(B.d);
      else k_ks_force<false><<<g3, KS_FB, B.force_shm, st>>>(B.d);
      ++launches;
    }
  }
  k_ks_force_sum<<<dim3((3 * B.nq + 127) / 128, B.n), 128, 0, st>>>(s, B.d, pi, what, to_f4);
  return launches + 1;
}

int launch_kspace(const DevState& s, const SimConst& C, const KSpaceBatch& B, cudaStream_t st, bool eflag, Acc acc) {
  return launch_ks(s, C, B, st, KS_RECIP, eflag, acc, false);
}

int launch_dipolar(const DevState& s, const SimConst& C, const KSpaceBatch& B, cudaStream_t st, bool eflag, Acc acc) {
  return launch_ks(s, C, B, st, KS_DIPOLE, eflag, acc, false);
}

int launch_kspace_step(const DevState& s, const SimConst& C, const KSpaceBatch& B, cudaStream_t st, bool eflag,
                       Acc acc) {
  return launch_ks(s, C, B, st, KS_RECIP | KS_DIPOLE, eflag, acc, s.mixed);
}

}  // namespace mfa
