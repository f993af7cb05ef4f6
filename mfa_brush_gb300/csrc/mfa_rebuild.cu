// mfa_rebuild.cu -- cell sort and Verlet-list rebuild on the device.
//
// Replaces the reference's neighbour bookkeeping: the linked cells of cell_list.f90:56-268
// (BIN_TYPE 2, rebuilt incrementally every step) and the skin-based Verlet lists of
// binning.f90 / check_skin.f90 (BIN_TYPE 0, rebuilt when a particle moved > skin/2).  Here the
// list is rebuilt when the position kernel has raised `rebuild_flag` (displacement > skin/2), by
// two kernels.  k_sort, a cooperative launch whose phases a grid barrier separates:
//   1. bin:      cell of every particle on the replica's list grid (cell edge >= r_cut_max+skin),
//                counts per cell, cell row and cell plane, the particle's tag into its cell's bucket;
//   2. starts:   a warp per row of cells: the planes and rows before it, then a scan along the row;
//   3. permute:  a particle's slot is its cell's start plus the number of smaller tags in the bucket:
//                the FP64 state goes there (the final order (replica, cell, tag) and every later
//                FP sum order are deterministic);
//   4. back:     the state in the new order, views and rebuild references rewritten.
// and k_nlist, the full neighbour list over the surrounding cells (x,y periodic, z bounded).
// The decision is per replica, as the reference decides per system: the position kernel raises the
// flag of the replica whose particle moved.  Every block lists the flagged replicas with prefix sums
// of their particles and cells, and the phases stride over that work; the other replicas' slots,
// cells and lists stay as they are (a replica's slots are one fixed range, its cells one fixed range,
// and its lists name only its own slots).
// In a captured CUDA graph the sequence sits in the body of a conditional node that runs only on
// steps where some replica is flagged.
#include "mfa_grid.h"
#include "mfa_state.cuh"

namespace mfa {

// Cell of a fixed-point position on the replica's list grid: one integer multiply per axis (x, y
// wrap with the fixed point; z is clamped to the grid).  Shared by the binning and the list build
// of both precisions, so they agree to the bit.
__device__ __forceinline__ void cell_coords(const RepDesc& R, const int4& q, int& ix, int& iy, int& iz) {
  ix = (int)(((unsigned long long)(unsigned)q.x * (unsigned)R.nc[0]) >> 32);
  iy = (int)(((unsigned long long)(unsigned)q.y * (unsigned)R.nc[1]) >> 32);
  iz = (int)(((long long)q.z * R.nc[2]) >> 30);
  iz = min(max(iz, 0), R.nc[2] - 1);
}

// ---- work list ------------------------------------------------------------------------------
// particles per chunk of the list builder (a warp's, consecutive slots of one replica)
constexpr int NL_CHUNK = 32;
constexpr int WL_SHARED = 1024;  // replicas whose work list fits in shared memory

// The replicas to rebuild (n of them) in ascending order and the prefix sums over them of their
// particles, cells, rows of cells and list chunks.
struct WorkList {
  int *rep, *p, *c, *y, *k;
  int n;
};

// Work item g of a prefix array pre (n listed replicas): the last k with pre[k] <= g.
__device__ __forceinline__ int wl_find(const int* pre, int n, int g) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}
// Particle i of a rebuilt replica into its cell: the cell's count and the particle's rank in it.
__device__ __forceinline__ void bin_particle(const DevState& s, int i) {
  int w = s.info[i];
  const RepDesc& R = s.reps[info_rep(w)];
  if (s.mixed) {
    // (x, y need no check: the fixed-point view wraps them; the integrator flags NaN); the z
    // check in FP32, as FP64 compares and the cell-height division issue on the FP64 pipe
    const double zd = s.rz[i];
    const float z = d2f_fast(zd);
    const int ez = (__double2hiint(zd) >> 20) & 0x7FF;  // (the conversion is right below 2^127)
    if (ez >= 1023 + 127 || !(z >= R.zlim_f[0] && z <= R.zlim_f[1]))
      atomicOr(s.status, ez == 0x7FF ? ST_NAN : ST_OUT_OF_BOX);
  } else {
    const double lz = 1. / R.inv_lc[2];
    const double x = s.rx[i], y = s.ry[i], z = s.rz[i];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(s.status, ST_NAN);
    else if (z < -lz || z > R.L[2] + lz) atomicOr(s.status, ST_OUT_OF_BOX);
  }
  int ix, iy, iz;
  cell_coords(R, s.pfx[i], ix, iy, iz);
  const int row = iz * R.nc[1] + iy, c = R.cell_off + row * R.nc[0] + ix;
  s.cell_of[i] = c;
  // Particles are still nearly sorted by cell, so neighbouring lanes share cells, rows and planes:
  // the lanes of one cell take consecutive ranks from a single atomicAdd (the buckets are ordered by
  // tag afterwards, so the order of the ranks does not matter), those of a row or plane one sum.
  const unsigned here = __activemask();
  const int lane = threadIdx.x & 31;
  const unsigned gc = __match_any_sync(here, c), gr = __match_any_sync(here, R.row_off + row),
                 gz = __match_any_sync(here, R.plane_off + iz);
  const int leader = __ffs(gc) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&s.cell_count[c], __popc(gc));
  if (lane == __ffs(gr) - 1) atomicAdd(&s.row_count[R.row_off + row], __popc(gr));
  if (lane == __ffs(gz) - 1) atomicAdd(&s.plane_count[R.plane_off + iz], __popc(gz));
  base = __shfl_sync(gc, base, leader);
  const int rank = base + __popc(gc & ((1u << lane) - 1u));
  s.rank[i] = rank;
  if (rank < s.bucket_cap) s.bucket[(size_t)c * s.bucket_cap + rank] = s.tag[i];
  else s.wl_n[3] = 1;  // a cell denser than its bucket: this rebuild orders the cells the long way
}

// The starts of the cells of one row (a warp): the particles of the planes and rows before it in
// its replica, then a scan along the row.
__device__ __forceinline__ void row_starts(const DevState& s, const RepDesc& R, int row) {
  const int lane = threadIdx.x & 31, iz = row / R.nc[1];
  int v = 0;
  for (int z = lane; z < iz; z += 32) v += s.plane_count[R.plane_off + z];
  for (int y = iz * R.nc[1] + lane; y < row; y += 32) v += s.row_count[R.row_off + y];
  int at = R.p0 + (int)__reduce_add_sync(0xffffffffu, (unsigned)v);
  const int c0 = R.cell_off + row * R.nc[0];
  for (int b = 0; b < R.nc[0]; b += 32) {
    const int n = b + lane < R.nc[0] ? s.cell_count[c0 + b + lane] : 0;
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += u;
    }
    if (b + lane < R.nc[0]) s.cell_start[c0 + b + lane] = at + x - n;
    at += __shfl_sync(0xffffffffu, x, 31);
  }
}

// The slot of particle i (tag t) in the new order, from its cell's bucket of tags.
__device__ __forceinline__ int bucket_slot(const DevState& s, int i, int t) {
  const int c = s.cell_of[i], n = s.cell_count[c];
  const int4* b = reinterpret_cast<const int4*>(s.bucket + (size_t)c * s.bucket_cap);  // (a multiple of 4)
  int less = 0;
  for (int k = 0; k < n; k += 4) {
    const int4 q = b[k >> 2];
    less += (q.x < t) + (k + 1 < n && q.y < t) + (k + 2 < n && q.z < t) + (k + 3 < n && q.w < t);
  }
  return s.cell_start[c] + less;
}

// The slots of cell c ordered by tag (a rebuild with a cell denser than its bucket).
__device__ __forceinline__ void sort_cell(const DevState& s, int c) {
  const int b = s.cell_start[c], n = s.cell_count[c];
  for (int k = 1; k < n; ++k) {
    int p = s.perm[b + k];
    int t = s.tag[p];
    int m = k - 1;
    while (m >= 0 && s.tag[s.perm[b + m]] > t) {
      s.perm[b + m + 1] = s.perm[b + m];
      --m;
    }
    s.perm[b + m + 1] = p;
  }
}

// The state of slot o to slot to(o) of the new order; the loads are issued before the slot is known.
template <typename F>
__device__ __forceinline__ void permute_slot(const DevState& s, int o, F to) {
  const double x = s.rx[o], y = s.ry[o], z = s.rz[o], vx = s.vx[o], vy = s.vy[o], vz = s.vz[o];
  const int wo = s.info[o], t = s.tag[o];
  const int i = to(t);
  s.tmp[0][i] = x;
  s.tmp[1][i] = y;
  s.tmp[2][i] = z;
  s.tmp[3][i] = vx;
  s.tmp[4][i] = vy;
  s.tmp[5][i] = vz;
  if (s.permute_accel || !info_mobile(wo)) {
    s.tmp[6][i] = s.ax[o];
    s.tmp[7][i] = s.ay[o];
    s.tmp[8][i] = s.az[o];
  }
  s.tmp_tag[i] = t;
  s.tmp_info[i] = wo;
}

// Writes the pair-kernel views of slot i and returns the fixed-point position (w in q.w).
__device__ __forceinline__ int4 write_views(const DevState& s, int i, const RepDesc& R, double x, double y, double z,
                                            double vx, double vy, double vz, int w, int t) {
  int4 q;
  q.x = to_fx_periodic(x, R.sfx[0]);
  q.y = to_fx_periodic(y, R.sfx[1]);
  q.z = to_fx_z(z, R.sfx[2]);
  q.w = w;
  s.pfx[i] = q;
  if (s.mixed) {
    s.vf[i] = make_float4(d2f_fast(vx), d2f_fast(vy), d2f_fast(vz), __int_as_float(t));
  } else {
    s.pd[i] = mk_dbl4(x, y, z, __longlong_as_double((long long)w));
    s.vd[i] = mk_dbl4(vx, vy, vz, __longlong_as_double((long long)t));
  }
  return q;
}

// Slot i of the new order back into the state, with its views and its position of this rebuild.
__device__ __forceinline__ void copyback_slot(const DevState& s, int i) {
  double x = s.tmp[0][i], y = s.tmp[1][i], z = s.tmp[2][i];
  double vx = s.tmp[3][i], vy = s.tmp[4][i], vz = s.tmp[5][i];
  s.rx[i] = x; s.ry[i] = y; s.rz[i] = z;
  s.vx[i] = vx; s.vy[i] = vy; s.vz[i] = vz;
  int t = s.tmp_tag[i], w = s.tmp_info[i];
  if (s.permute_accel || !info_mobile(w)) {
    s.ax[i] = s.tmp[6][i]; s.ay[i] = s.tmp[7][i]; s.az[i] = s.tmp[8][i];
  }
  s.tag[i] = t;
  s.info[i] = w;
  s.slot_of_tag[t] = i;
  const RepDesc& R = s.reps[info_rep(w)];
  int4 q = write_views(s, i, R, x, y, z, vx, vy, vz, w, t);
  // the list builder's view: sigma from the fixed point (so that it wraps alike), to 512 units
  s.lp[i] = make_float4((__int_as_float(0x4B000000 | ((unsigned)q.x >> 9)) - 8388608.0f) * (512.f * R.ufx_f[0]),
                        (__int_as_float(0x4B000000 | ((unsigned)q.y >> 9)) - 8388608.0f) * (512.f * R.ufx_f[1]),
                        i2f_coarse(q.z, 9) * (512.f * R.ufx_f[2]), __int_as_float(w));
  q.w = 0;
  s.ref[i] = q;
}

// Grid barrier of a cooperative launch: every block arrives at the k-th barrier (k = 1, 2, ..) on a
// counter that the list builder's end sets back to zero.  The wait is bounded (about a second): then
// the status word gets ST_BARRIER and the block leaves.  A block goes on only when all have arrived, so
// whatever a block does rests on finished phases.  The counts and the slots may then be half-way, so
// from that on every sort leaves at once (sort_failed) and the list builder finds no work: the lists stay
// those of the last complete rebuild, whose slots are in range, and the host refuses further steps.
__device__ __forceinline__ bool grid_barrier(const DevState& s, int k) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned* cnt = reinterpret_cast<unsigned*>(s.wl_n + 4);
    const unsigned target = (unsigned)k * gridDim.x;
    unsigned seen, old;
    __threadfence();
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(cnt) : "memory");
    seen = old + 1;
    for (int t = 0; t < s.barrier_spins && seen < target; ++t)
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(cnt) : "memory");
    ok = seen >= target;
    if (!ok) {
      atomicOr(s.status, ST_BARRIER);
      s.wl_n[0] = s.wl_k[0] = 0;  // (block 0 wrote its own before it arrived here, or gives up later)
    }
    __threadfence();
  }
  __syncthreads();
  return ok;
}

__device__ __forceinline__ unsigned sort_failed(const DevState& s) {
  return s.status[0] & ST_BARRIER;
}

// block-wide exclusive scan of v; the block's total in `total`
__device__ __forceinline__ int block_scan_excl(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();  // sh may still be read from the call before
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  int off = 0, t = 0;
  for (int q = 0; q < nw; ++q) {
    const int y = sh[q];
    off += q < wid ? y : 0;
    t += y;
  }
  total = t;
  return off + x - v;
}

// The work list of the flagged replicas (all when forced), by one block into L.
__device__ __forceinline__ void make_worklist(const DevState& s, bool force, WorkList& L, int* sh) {
  int n = 0, at[4] = {0, 0, 0, 0};
  for (int base = 0; base < s.nrep; base += SORT_T) {
    const int r = base + threadIdx.x;
    const bool sel = r < s.nrep && (force || s.rebuild_flag[1 + r] != 0);
    int v[4] = {0, 0, 0, 0};
    if (sel) {
      const RepDesc& R = s.reps[r];
      v[0] = R.n_part; v[1] = R.ncell; v[2] = R.nc[1] * R.nc[2]; v[3] = (R.n_part + NL_CHUNK - 1) / NL_CHUNK;
    }
    int tn, t[4], e[4];
    const int en = block_scan_excl(sel ? 1 : 0, sh, tn);
    if (tn == 0) continue;  // (uniform)
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = at[q] + block_scan_excl(v[q], sh, t[q]);
    if (sel) {
      L.rep[n + en] = r;
      L.p[n + en] = e[0]; L.c[n + en] = e[1]; L.y[n + en] = e[2]; L.k[n + en] = e[3];
    }
    n += tn;
#pragma unroll
    for (int q = 0; q < 4; ++q) at[q] += t[q];
  }
  if (threadIdx.x == 0) { L.p[n] = at[0]; L.c[n] = at[1]; L.y[n] = at[2]; L.k[n] = at[3]; }
  L.n = n;
  __syncthreads();
}

// The sort of the flagged replicas, see the top of the file.  Its passes over memory are short: with
// a kernel each (ten of them) their launches and ramps took most of the time of a rebuild of a few
// replicas; with a cluster of eight blocks per replica instead of the whole grid the phases of one
// large replica took 100 us.  With the list builder below, a rebuild of a 6400-particle channel went
// from 79 to 36 us, of 32 brush replicas (447 k particles) from 188 to 159, of 256 (4.66 M) from 1451
// to 1336, and a step's rebuild of the flagged ones of these 256 from 229 to 197 us.
__global__ void __launch_bounds__(SORT_T, SORT_PER_SM) k_sort(DevState s, bool force) {
  const unsigned failed = sort_failed(s);
  if (!force && s.rebuild_flag[0] == 0) {  // (the same for every block: the list builder's end clears it)
    if (blockIdx.x == 0 && threadIdx.x == 0) s.wl_n[0] = s.wl_k[0] = 0;
    return;
  }
  if (__syncthreads_or(failed)) return;  // (another block of this launch may set it meanwhile)
  __shared__ int wl[5][WL_SHARED + 1];
  __shared__ int sh[SORT_T / 32];
  WorkList L;
  int bar = 0;
  if (s.nrep <= WL_SHARED) {  // every block makes its own
    L.rep = wl[0]; L.p = wl[1]; L.c = wl[2]; L.y = wl[3]; L.k = wl[4];
    make_worklist(s, force, L, sh);
    if (blockIdx.x == 0)  // the list builder's copy
      for (int q = threadIdx.x; q <= L.n; q += SORT_T) {
        s.wl_k[q] = L.k[q];
        if (q < L.n) s.wl_rep[q] = L.rep[q];
      }
  } else {
    L.rep = s.wl_rep; L.p = s.wl_p; L.c = s.wl_c; L.y = s.wl_y; L.k = s.wl_k;
    if (blockIdx.x == 0) {
      make_worklist(s, force, L, sh);
      if (threadIdx.x == 0) s.wl_n[0] = L.n;
    }
    if (!grid_barrier(s, ++bar)) return;
    L.n = s.wl_n[0];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s.wl_n[0] = L.n;
    s.wl_n[1] = 0;  // the list builder's chunk queue
  }
  // every block takes one contiguous share of the particles, cells and rows in each phase
  auto share = [&](int total, int unit, int& lo, int& hi) {
    const int per = ((total + unit - 1) / unit + gridDim.x - 1) / gridDim.x * unit;
    lo = min(total, (int)blockIdx.x * per);
    hi = min(total, lo + per);
  };
  // f(list position k, item g) for the thread's items of a share, k found once and then stepped on
  auto each = [&](const int* pre, int lo, int hi, auto f) {
    int g = lo + threadIdx.x;
    if (g >= hi) return;
    int k = wl_find(pre, L.n, g);
    for (; g < hi; g += SORT_T) {
      while (k + 1 < L.n && pre[k + 1] <= g) ++k;
      f(k, g - pre[k]);
    }
  };
  int plo, phi, clo, chi, ylo, yhi;
  share(L.p[L.n], 32, plo, phi);
  share(L.c[L.n], 32, clo, chi);
  share(L.y[L.n], 1, ylo, yhi);
  each(L.p, plo, phi, [&](int k, int g) { bin_particle(s, s.reps[L.rep[k]].p0 + g); });
  if (!grid_barrier(s, ++bar)) return;
  const bool dense = *(volatile int*)(s.wl_n + 3) != 0;
  for (int g = ylo + (threadIdx.x >> 5); g < yhi; g += SORT_T / 32) {
    const int k = wl_find(L.y, L.n, g);
    row_starts(s, s.reps[L.rep[k]], g - L.y[k]);
  }
  if (!grid_barrier(s, ++bar)) return;
  if (!dense) {
    each(L.p, plo, phi, [&](int k, int g) {
      const int i = s.reps[L.rep[k]].p0 + g;
      permute_slot(s, i, [&](int t) { return bucket_slot(s, i, t); });
    });
  } else {
    each(L.p, plo, phi, [&](int k, int g) {
      const int i = s.reps[L.rep[k]].p0 + g;
      s.perm[s.cell_start[s.cell_of[i]] + s.rank[i]] = i;
    });
    if (!grid_barrier(s, ++bar)) return;
    each(L.c, clo, chi, [&](int k, int g) { sort_cell(s, s.reps[L.rep[k]].cell_off + g); });
    if (!grid_barrier(s, ++bar)) return;
    each(L.p, plo, phi, [&](int k, int g) {
      const int i = s.reps[L.rep[k]].p0 + g;
      permute_slot(s, s.perm[i], [&](int) { return i; });
    });
  }
  if (!grid_barrier(s, ++bar)) return;
  each(L.p, plo, phi, [&](int k, int g) { copyback_slot(s, s.reps[L.rep[k]].p0 + g); });
  // the counts back to zero for the next binning
  each(L.c, clo, chi, [&](int k, int g) { s.cell_count[s.reps[L.rep[k]].cell_off + g] = 0; });
  each(L.y, ylo, yhi, [&](int k, int g) {
    const RepDesc& R = s.reps[L.rep[k]];
    s.row_count[R.row_off + g] = 0;
    if (g % R.nc[1] == 0) s.plane_count[R.plane_off + g / R.nc[1]] = 0;
  });
}

// The end of a rebuild, in the list builder's last block to finish: counts it (when some replica was
// flagged) and the flagged replicas' rebuilds, and clears the flags.
__device__ __forceinline__ void rebuild_done(const DevState& s) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(s.wl_n + 2, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  int* flag = s.rebuild_flag;
  const bool failed = sort_failed(s), any = flag[0] != 0 && !failed;
  __syncthreads();
  for (int r = threadIdx.x; r < s.nrep && any; r += blockDim.x) {
    if (flag[1 + r]) {
      s.rep_rebuilds[r] += 1;
      flag[1 + r] = 0;
    }
  }
  if (threadIdx.x == 0) {
    s.wl_n[2] = 0;
    if (!failed) s.wl_n[3] = s.wl_n[4] = 0;
    if (any) {
      *s.rebuilds += 1;
      flag[0] = 0;
    }
  }
}

// Full Verlet list: every mobile particle lists all j (mobile or wall) with r^2 < (rc_ij+skin)^2,
// decided in FP32 with a margin (fx_margin in mfa_api.cu) on an FP32 view of the positions, in both
// precisions.  Cells are at least 1/H of the list cut-off wide (1/HX along x), and the cells around a
// particle are walked as (2H+1)^2 x-rows: the cells of a row are consecutive in the sorted order
// unless the row wraps in x, so a row is one contiguous slot range (two when it wraps).  Rows whose
// y/z distance from the particle exceeds the largest list cut-off of its type are skipped, and each
// kept row is trimmed in x to the cells within that cut-off, which removes about half of the
// candidates.  A range lies in one periodic image, so its shift goes into the particle's
// coordinates once and a candidate costs three subtractions, three products and a compare (with
// integer minimum images and conversions per candidate it took twice the instructions).
//
// The list's order is by row, then by slot, whichever way it is built:
//   a thread per particle, when there are particles enough to fill the GPU with NL_G lanes each (2048
//     threads per SM; the least work, as the lanes of a warp walk nearly the same rows);
//   NL_G lanes per particle, when there are not: one or a few replicas flagged, where a thread's walk
//     of ~80 candidates one after the other is 36 us of latency, and this is 14.  The lanes set up a
//     row each, take the candidates of a row side by side and place the hits by a ballot.  (With
//     four or sixteen times as many particles built this way the steps of 64 and 256 brush replicas
//     took 4 and 10 % longer.)
// Bound by the latency of the candidates' loads and by issue (60 % active, 19 of 32 lanes).  Short
// lists gain nothing from unrolled candidate loops, long ones 2 %.
// Each lane (group) stages its first NL_STAGE entries in shared memory and the warp writes them out
// row by row: the k-th neighbours of 32 consecutive particles are 32 consecutive ints of nbr
// (scattered 4-byte stores into the column-major list cost read-modify-writes in HBM).
constexpr int NL_STAGE = 32;  // staged entries per particle (later ones go straight to the list)

struct NlRow {  // slot ranges of a row, the second when it wraps in x
  int b0, e0, b1, e1;
  float x0, x1, y;  // the particle's coordinates in the image of each range
};

// exact for small integers, without a conversion instruction
__device__ __forceinline__ float nl_float(int v) { return i2f_coarse(v, 0); }
// squared gap to a cell edge, d the distance before it (0 when the particle is past it)
__device__ __forceinline__ float nl_gap2(float d) {
  d = fmaxf(d, 0.f);
  return d * d;
}

template <int H, int HX>
__device__ __forceinline__ NlRow nl_row(const DevState& s, const RepDesc& R, int row, float4 q, int ix, int iy, int iz,
                                        float rl2max) {
  NlRow r = {0, 0, 0, 0, q.x, q.x, q.y};
  const int dz = row / (2 * H + 1) - H, dy = row - (dz + H) * (2 * H + 1) - H;
  const int cz = iz + dz;
  int cy = iy + dy;
  if (cz < 0 || cz >= R.nc[2]) return r;
  const float lx = R.lc_f[0], ly = R.lc_f[1], lz = R.lc_f[2];
  const float rem2 = rl2max - (dz > 0 ? nl_gap2(nl_float(cz) * lz - q.z) : (dz < 0 ? nl_gap2(q.z - nl_float(cz + 1) * lz) : 0.f)) -
                     (dy > 0 ? nl_gap2(nl_float(cy) * ly - q.y) : (dy < 0 ? nl_gap2(q.y - nl_float(cy + 1) * ly) : 0.f));
  if (rem2 <= 0.f) return r;  // the whole row is beyond the list cut-off
  const int nx = R.nc[0];
  int xa = ix, xb = ix;
#pragma unroll
  for (int k = 1; k <= HX; ++k) {
    xa -= nl_gap2(q.x - nl_float(ix - k + 1) * lx) < rem2;
    xb += nl_gap2(nl_float(ix + k) * lx - q.x) < rem2;
  }
  if (cy < 0) { cy += R.nc[1]; r.y += R.L_f[1]; }
  else if (cy >= R.nc[1]) { cy -= R.nc[1]; r.y -= R.L_f[1]; }
  const int* __restrict__ st = s.cell_start + R.cell_off + (cz * R.nc[1] + cy) * nx;
  // (cell_start[c + 1] ends cell c; there is one entry past the last cell)
  if (xa < 0) {
    r.b0 = st[0]; r.e0 = st[xb + 1];
    r.b1 = st[nx + xa]; r.e1 = st[nx];
    r.x1 += R.L_f[0];
  } else if (xb >= nx) {
    r.b0 = st[xa]; r.e0 = st[nx];
    r.b1 = st[0]; r.e1 = st[xb - nx + 1];
    r.x1 -= R.L_f[0];
  } else {
    r.b0 = st[xa]; r.e0 = st[xb + 1];
  }
  return r;
}

template <bool UNI, int H, int HX = H>
__global__ void __launch_bounds__(NL_T, NL_PER_SM) k_nlist(DevState s) {
  constexpr int NR = (2 * H + 1) * (2 * H + 1);
  const int nwl = s.wl_n[0], nchunks = s.wl_k[nwl];
  const int lane = threadIdx.x & 31, warp = (blockIdx.x * NL_T + threadIdx.x) >> 5, nwarps = gridDim.x * (NL_T / 32);
  __shared__ int nl_sh[NL_T * (NL_STAGE | 1)];
  __shared__ float rl2f[NPAIR];
  __shared__ float rlmax[MAXT];
  if (nchunks > 0) {
    for (int k = threadIdx.x; k < NPAIR; k += NL_T) rl2f[k] = s.tabf[k].rlist2;
    if (threadIdx.x < MAXT) {  // largest list cut-off of each type, with the culling margin
      float m = 0.f;
      for (int t = 0; t < MAXT; ++t) m = fmaxf(m, s.tabf[threadIdx.x * MAXT + t].rlist2);
      m = sqrtf(m) + s.fx_err;
      rlmax[threadIdx.x] = m * m * 1.0002f;
    }
    __syncthreads();
    const unsigned FULL = 0xffffffffu;
    const int cap = s.nbr_cap;
    const float rl_uni = s.rl2_uni;  // UNI: one list cut-off for every pair
    int most = 0;  // neighbours found (more than the capacity when the list overflows)
    auto hit_of = [&](float x, float y, float z, float4 c, int ti) {
      const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
      return dx * dx + dy * dy + dz * dz < (UNI ? rl_uni : rl2f[ti * MAXT + info_type(__float_as_int(c.w))]);
    };
    if ((long long)nchunks * NL_CHUNK * NL_G > (long long)s.nsm * 2048) {
      // ---- a thread per particle, chunks from a queue (they differ in cost)
      int* mine = nl_sh + threadIdx.x * (NL_STAGE | 1);  // odd stride: distinct banks
      for (;;) {
        int ch = 0;
        if (lane == 0) ch = atomicAdd(s.wl_n + 1, 1);
        ch = __shfl_sync(FULL, ch, 0);
        if (ch >= nchunks) break;
        const int lk = wl_find(s.wl_k, nwl, ch);
        const RepDesc& R = s.reps[s.wl_rep[lk]];
        const int loc = (ch - s.wl_k[lk]) * NL_CHUNK + lane, i = R.p0 + loc;
        const bool doit = loc < R.n_part;
        int cnt = 0;
        if (doit) {
          const float4 q = s.lp[i];
          const int w = __float_as_int(q.w);
          if (info_mobile(w)) {
            const int ti = info_type(w);
            int ix, iy, iz;
            cell_coords(R, s.pfx[i], ix, iy, iz);
            const float rl2max = rlmax[ti];
            const float lx = R.lc_f[0], ly = R.lc_f[1], lz = R.lc_f[2];
            const int nx = R.nc[0], ny = R.nc[1];
            float gxm[HX], gxp[HX];  // squared gaps to the cells ix - k and ix + k
#pragma unroll
            for (int k = 1; k <= HX; ++k) {
              gxm[k - 1] = nl_gap2(q.x - nl_float(ix - k + 1) * lx);
              gxp[k - 1] = nl_gap2(nl_float(ix + k) * lx - q.x);
            }
            for (int cz = max(iz - H, 0); cz <= min(iz + H, R.nc[2] - 1); ++cz) {
              const float rz2 = rl2max - (cz > iz ? nl_gap2(nl_float(cz) * lz - q.z)
                                                  : (cz < iz ? nl_gap2(q.z - nl_float(cz + 1) * lz) : 0.f));
              for (int dy = -H; dy <= H; ++dy) {
                int cy = iy + dy;
                const float rem2 = rz2 - (dy > 0 ? nl_gap2(nl_float(cy) * ly - q.y)
                                                 : (dy < 0 ? nl_gap2(q.y - nl_float(cy + 1) * ly) : 0.f));
                if (rem2 <= 0.f) continue;  // the whole row is beyond the list cut-off
                int xa = ix, xb = ix;
#pragma unroll
                for (int k = 0; k < HX; ++k) {
                  xa -= gxm[k] < rem2;
                  xb += gxp[k] < rem2;
                }
                float y = q.y;
                if (cy < 0) { cy += ny; y += R.L_f[1]; }
                else if (cy >= ny) { cy -= ny; y -= R.L_f[1]; }
                const int* __restrict__ st = s.cell_start + R.cell_off + (cz * ny + cy) * nx;
                // (cell_start[c + 1] ends cell c; there is one entry past the last cell)
                int b = st[max(xa, 0)], e = st[min(xb, nx - 1) + 1], b1 = 0, e1 = 0;
                float x = q.x, x1 = q.x;
                if (xa < 0) { b1 = st[nx + xa]; e1 = st[nx]; x1 += R.L_f[0]; }
                else if (xb >= nx) { b1 = st[0]; e1 = st[xb - nx + 1]; x1 -= R.L_f[0]; }
                // (one loop for both ranges and every lane: with a loop per kind of row the lanes of a
                // warp that walk different kinds take turns, 17 % slower on 256 brush replicas)
                for (int g = 0; g < 2; ++g) {
#pragma unroll(UNI ? 1 : 2)
                  for (int j = b; j < e; ++j) {
                    const bool hit = hit_of(x, y, q.z, s.lp[j], ti) && j != i;
                    mine[min(cnt, NL_STAGE)] = j;  // kept when it hits; the last word takes the rest
                    if (hit && cnt >= NL_STAGE && cnt < cap) s.nbr[(size_t)cnt * s.Np + i] = j;
                    cnt += hit;
                  }
                  b = b1; e = e1; x = x1;
                }
              }
            }
          }
        }
        most = max(most, cnt);
        const int kept = min(cnt, cap), rows = min((int)__reduce_max_sync(FULL, (unsigned)kept), NL_STAGE);
        for (int k = 0; k < rows; ++k)
          if (k < kept) s.nbr[(size_t)k * s.Np + i] = mine[k];
        if (doit) s.nn[i] = kept;
      }
    } else {
      // ---- NL_G lanes per particle
      constexpr int PW = 32 / NL_G;  // particles of a warp at a time
      const int q8 = lane & (NL_G - 1), grp = lane / NL_G;
      int* mine = nl_sh + (threadIdx.x / NL_G) * (NL_STAGE | 1);
      const int units = nchunks * (NL_CHUNK / PW);
      for (int u = warp; u < units; u += nwarps) {
        const int ch = u / (NL_CHUNK / PW);
        const int lk = wl_find(s.wl_k, nwl, ch);
        const RepDesc& R = s.reps[s.wl_rep[lk]];
        const int loc = (ch - s.wl_k[lk]) * NL_CHUNK + (u % (NL_CHUNK / PW)) * PW + grp, i = R.p0 + loc;
        const bool doit = loc < R.n_part;
        const float4 q = s.lp[doit ? i : R.p0];
        const int w = __float_as_int(q.w), ti = info_type(w);
        const bool walk = doit && info_mobile(w);
        int ix = 0, iy = 0, iz = 0;
        if (walk) cell_coords(R, s.pfx[i], ix, iy, iz);
        const float rl2max = rlmax[ti];
        int cnt = 0;
        for (int rb = 0; rb < NR; rb += NL_G) {  // each lane sets up a row
          NlRow r = {0, 0, 0, 0, 0.f, 0.f, 0.f};
          if (walk && rb + q8 < NR) r = nl_row<H, HX>(s, R, rb + q8, q, ix, iy, iz, rl2max);
          const bool any1 = __any_sync(FULL, r.e1 > r.b1);
          for (int o = 0; o < NL_G && rb + o < NR; ++o) {
            for (int g = 0; g < (any1 ? 2 : 1); ++g) {
              const int b = __shfl_sync(FULL, g ? r.b1 : r.b0, o, NL_G), e = __shfl_sync(FULL, g ? r.e1 : r.e0, o, NL_G);
              const float x = __shfl_sync(FULL, g ? r.x1 : r.x0, o, NL_G), y = __shfl_sync(FULL, r.y, o, NL_G);
              const int it = ((int)__reduce_max_sync(FULL, (unsigned)(e - b)) + NL_G - 1) / NL_G;
              for (int t = 0; t < it; ++t) {
                const int j = b + t * NL_G + q8;
                bool hit = false;
                if (j < e) hit = hit_of(x, y, q.z, s.lp[j], ti) && j != i;
                const unsigned bits = (__ballot_sync(FULL, hit) >> (grp * NL_G)) & ((1u << NL_G) - 1u);
                if (hit) {
                  const int k = cnt + __popc(bits & ((1u << q8) - 1u));
                  if (k < NL_STAGE) mine[k] = j;
                  else if (k < cap) s.nbr[(size_t)k * s.Np + i] = j;
                }
                cnt += __popc(bits);
              }
            }
          }
        }
        most = max(most, cnt);
        const int kept = min(cnt, cap);
        __syncwarp();
        // (consecutive lanes take consecutive particles of one list row)
        const int pi = lane % PW;
        const int kp = __shfl_sync(FULL, kept, pi * NL_G), ip = __shfl_sync(FULL, i, pi * NL_G);
        const int* from = nl_sh + ((threadIdx.x & ~31) / NL_G + pi) * (NL_STAGE | 1);
        for (int k = lane / PW; k < min(kp, NL_STAGE); k += NL_G) s.nbr[(size_t)k * s.Np + ip] = from[k];
        if (doit && q8 == 0) s.nn[i] = kept;
        __syncwarp();  // the staging area is the next particles'
      }
    }
    // the true count, so that the host grows the capacity past it
    most = (int)__reduce_max_sync(FULL, (unsigned)most);
    if (lane == 0 && (unsigned)most > *(volatile unsigned*)(s.status + 1)) {
      atomicMax(s.status + 1, (unsigned)most);
      if (most > cap) atomicOr(s.status, ST_NLIST_OVERFLOW);
    }
  }
  rebuild_done(s);
}

int rebuild_launches() { return 2; }

cudaError_t launch_rebuild(const DevState& s, cudaStream_t st, bool force) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sort_blocks(s.N, s.nsm));
  cfg.blockDim = dim3(SORT_T);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  // (the launches' own results: the thread's last error may be the caller's)
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_sort, s, force);
  if (e != cudaSuccess) return e;
  const int uni = s.rl2_uni > 0.f ? 1 : 0;
  using KernT = void (*)(DevState);
  const KernT kerns[3][2] = {{k_nlist<false, 1>, k_nlist<true, 1>},
                             {k_nlist<false, 2>, k_nlist<true, 2>},
                             {k_nlist<false, 3>, k_nlist<true, 3>}};
  // cells finer along x alone (with 3x3 rows in y, z)
  const KernT kx[2][2] = {{k_nlist<false, 1, 2>, k_nlist<true, 1, 2>}, {k_nlist<false, 1, 3>, k_nlist<true, 1, 3>}};
  const KernT kern = (s.nl_hx != s.nl_h) ? kx[s.nl_hx - 2][uni] : kerns[s.nl_h - 1][uni];
  cfg.gridDim = dim3(list_blocks(s.N, s.nsm));
  cfg.blockDim = dim3(NL_T);
  cfg.numAttrs = 0;
  return cudaLaunchKernelEx(&cfg, kern, s);
}

// ---------------------------------------------------------------------------------------------
// Parity exports with the reference's own grid (cell_list.f90:129-213, 285-433)
// ---------------------------------------------------------------------------------------------
__global__ void k_ref_cells(DevState s, int rep, double il0, double il1, double il2, int n0, int n1, int n2,
                            int* __restrict__ cell_of_tag, int* __restrict__ counts) {
  const RepDesc& R = s.reps[rep];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= R.n_mon_tot) return;
  int i = s.slot_of_tag[R.p0 + t];
  double r[3] = {s.rx[i], s.ry[i], s.rz[i]};
  double il[3] = {il0, il1, il2};
  int nc[3] = {n0, n1, n2};
  int pc = 1, pf = 1;
  for (int d = 0; d < 3; ++d) {
    int c = (int)(r[d] * il[d]);
    c = min(max(c, 0), nc[d] - 1);
    pc += pf * c;
    pf *= nc[d];
  }
  cell_of_tag[t] = pc;
  atomicAdd(&counts[pc], 1);
}

void launch_ref_cells(const DevState& s, cudaStream_t st, int rep, const double* il, const int* nc, int* cell_of_tag,
                      int* counts) {
  int n = s.N;  // upper bound; the kernel checks the replica's own count
  k_ref_cells<<<(n + 255) / 256, 256, 0, st>>>(s, rep, il[0], il[1], il[2], nc[0], nc[1], nc[2], cell_of_tag, counts);
}

__global__ void k_cell_neigh(int n0, int n1, int n2, int n_nei, int* __restrict__ out) {
  int in_cell = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int nct = n0 * n1 * n2;
  if (in_cell > nct) return;
  int z_cell = (in_cell - 1) / (n0 * n1) + 1;
  int y_cell = (in_cell - n0 * n1 * (z_cell - 1) - 1) / n0 + 1;
  int x_cell = in_cell - n0 * n1 * (z_cell - 1) - n0 * (y_cell - 1);
  int* o = out + (size_t)(in_cell - 1) * n_nei;
  int il = 0;
  int lo = (n_nei == 13) ? 1 : 0, hi = (n_nei == 13) ? 3 : 4, ilo = 2, ihi = (n_nei == 13) ? 3 : 4;
  for (int i = ilo; i <= ihi; ++i)
    for (int j = lo; j <= hi; ++j) {
      if (i == 2 && j <= 1) continue;
      for (int k = lo; k <= hi; ++k) {
        if (i == 2 && j == 2 && k >= 3) continue;
        int jc = in_cell + i - 2 + (j - 2) * n0 + (k - 2) * n1 * n0;
        if (jc == in_cell) continue;
        if (n_nei == 13) {
          if (x_cell == 1 && i == 1) jc += n0;
          if (x_cell == n0 && i == 3) jc -= n0;
          if (y_cell == 1 && j == 1) jc += n0 * n1;
          if (y_cell == n1 && j == 3) jc -= n0 * n1;
        } else {
          if (x_cell + i - 2 > n0) jc -= n0;
          if (y_cell + j - 2 < 1) jc += n0 * n1;
          if (y_cell + j - 2 > n1) jc -= n0 * n1;
        }
        if (z_cell + k - 2 < 1) jc = 0;
        if (z_cell + k - 2 > n2) jc = 0;
        o[il++] = jc;
      }
    }
}

void launch_cell_neigh(const int* nc, int n_nei, int* out, cudaStream_t st) {
  int nct = nc[0] * nc[1] * nc[2];
  k_cell_neigh<<<(nct + 127) / 128, 128, 0, st>>>(nc[0], nc[1], nc[2], n_nei, out);
}

}  // namespace mfa
