// clmd_cycle.cu -- the MD step as ONE persistent cooperative kernel.
//
// A launch runs `nsteps` consecutive integrator(i) calls (int-verlet-mav.f
// or int-verlet-nh-mav.f, with scalev velocity scaling before each step when
// ethst == 'X', main.f:207) for one system, or one neighbor() call.  Phases
// are separated by a grid barrier instead of kernel boundaries:
//
//   velocity Verlet, per step:  [force_n + kick_n + drift_n+1] -> barrier
//                               -> skin decision -> (rebuild: 5 barriers)
//   Nose-Hoover, per step:      [velocities_n + drift_n+1] -> barrier ->
//                               (rebuild) -> force_n+1 -> barrier
//
// Forces of step n read the positions of step n while the fused drift writes
// step n+1's, so positions are double-buffered (pos0/pos1); v and a are only
// ever touched by their own atom.  Every block keeps a replica of the scalar
// state (clmd_scalars, grid geometry) in shared memory and updates it from
// the same reduced values in the same order, so all blocks take the same
// branches; block 0 writes the replica back at the end.  Grid-wide sums are
// per-block partials reduced by every block in a fixed order: deterministic.
//
// Per-atom arithmetic is the same code as the standalone kernels (built with
// -fmad=false): positions, velocities, accelerations and lists stay
// bit-identical to the serial FP64 reference.
#include <cuda_runtime.h>
#include <stdio.h>

#include "clmd_cycle.cuh"

namespace clmd {

#ifndef CLMD_PB
#define CLMD_PB 512
#endif
constexpr int kPB = CLMD_PB;      // threads per block
#ifndef CLMD_CYCLE_MINB
#define CLMD_CYCLE_MINB (1024 / CLMD_PB)         // resident blocks per SM the registers must allow
#endif
constexpr int kRedSlots = 16;     // partial-sum slots per buffer

// ---------------------------------------------------------------------------
// grid barrier (co-residency guaranteed by the cooperative launch); every
// wait is bounded and reports CLMD_ERR_TIMEOUT instead of hanging
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool gbar(DevState* st) {
  __shared__ int fail;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int* gen = &st->bar_gen;
    unsigned int g = *gen;
    __threadfence();
    unsigned int arrived = atomicAdd(&st->bar_count, 1u);
    fail = 0;
    if (arrived == gridDim.x - 1 + st->bar_extra) {
      atomicExch(&st->bar_count, 0u);
      __threadfence();
      atomicAdd(&st->bar_gen, 1u);
    } else {
      const long long limit = st->bar_limit > 0 ? st->bar_limit : (1ll << 25);
      long long spins = 0;
      while (*gen == g) {
        __nanosleep(32);
        if (++spins > limit) {
          fail = 1;
          // recorded here as well: a rebuild cut short by a timeout leaves
          // the launch through its normal end, which latches err_new
          atomicCAS(&st->err_new, 0, CLMD_ERR_TIMEOUT);
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return fail == 0;
}

// partials: buf[slot * nb + block]
__device__ __forceinline__ void put_sum(double* buf, int slot, double v, double* sh) {
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) buf[slot * gridDim.x + blockIdx.x] = t;
}
__device__ __forceinline__ void put_max(double* buf, int slot, double v, double* sh) {
  double t = block_max(v, sh);
  if (threadIdx.x == 0) buf[slot * gridDim.x + blockIdx.x] = t;
}
// every thread of every block gets the same total
__device__ __forceinline__ double get_sum(const double* buf, int slot, double* sh,
                                          double* bc) {
  double v = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x)
    v += __ldcg(buf + slot * gridDim.x + k);
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) *bc = t;
  __syncthreads();
  double r = *bc;
  __syncthreads();
  return r;
}
__device__ __forceinline__ double get_max(const double* buf, int slot, double* sh,
                                          double* bc) {
  double v = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x)
    v = fmax(v, __ldcg(buf + slot * gridDim.x + k));
  double t = block_max(v, sh);
  if (threadIdx.x == 0) *bc = t;
  __syncthreads();
  double r = *bc;
  __syncthreads();
  return r;
}

constexpr int kTileLog = 11, kMaxTiles = 2048;

// exclusive scan over the block (sh: a warp's sum each); total: the block's
__device__ __forceinline__ int block_scan(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();
  if (lane == 31) sh[w] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < kPB / 32; k++) {
    const int t = sh[k];
    before += k < w ? t : 0;
    total += t;
  }
  return before + incl - v;
}

// The list rebuild, in place: positions wrapped and, with the velocities and
// perm, put in cell order (gathered into pos_s, vx_s.., perm_s; the search
// reads the new order there and copies each slot back as it takes it).
// Returns false if the grid must stop (error).  acc: carry the accelerations
// into the new order too; a rebuild inside the step loop runs between the
// drift (the last reader of a step's accelerations) and the force pass that
// overwrites them, so there they are not moved
static __device__ bool rebuild(const Params& P, DevState* st, Blk& B, const CycleArgs& A,
                               double4* pos, WarpStage* stage, bool acc) {
  const int N = P.N;
  const int G = gridDim.x * blockDim.x;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const Geo& g = B.g;
  __shared__ int ssh[kPB / 32];
  int* toff = (int*)stage;  // [kMaxTiles], until the search
  static_assert(sizeof(WarpStage) * (kPB / 32) >= sizeof(int) * kMaxTiles, "tile offsets");
  // R1: histogram of the wrapped positions (neighbor-pbc-mav.f:67-71; R4
  // stores them wrapped); the count before an atom's own is its arrival
  // number in the cell (kept in row_lo, dead until the search writes it)
  if (t0 == 0) st->list_used = 0ull;
  for (int p = t0; p < N; p += G) {
    const double4 v = wrap_box(P, pos[p]);
    const int cx = clmd_cell(v.x, g.cfx, g.ncx);
    const int cy = clmd_cell(v.y, g.cfy, g.ncy);
    const int cz = clmd_cell(v.z, g.cfz, g.ncz);
    int c = (cz * g.ncy + cy) * g.ncx + cx;
    A.atom_cell[p] = c;
    A.row_lo[p] = atomicAdd(&A.cell_count[c], 1);
  }
  if (!gbar(st)) return false;
  // R2: per tile of cells an exclusive scan (into cell_fill) and its sum;
  // the counts go back to zero.  At most kMaxTiles tiles, so that every
  // block can hold the tiles' offsets in shared memory
  const int ncell = g.ncell;
  int tlog = kTileLog;
  while (((ncell - 1) >> tlog) >= kMaxTiles) tlog++;
  const int ntiles = ((ncell - 1) >> tlog) + 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int b = blockIdx.x; b < ntiles; b += gridDim.x) {
    constexpr int per = (1 << kTileLog) / kPB;
    int carry = 0;
    for (int sub = 0; sub < 1 << (tlog - kTileLog); sub++) {
      const int c0 = (b << tlog) + (sub << kTileLog) + threadIdx.x * per;
      int n[per], s = 0;
#pragma unroll
      for (int k = 0; k < per; k++) {
        n[k] = c0 + k < ncell ? __ldcg(A.cell_count + c0 + k) : 0;
        s += n[k];
      }
      int total;
      int ex = carry + block_scan(s, ssh, total);
#pragma unroll
      for (int k = 0; k < per; k++) {
        if (c0 + k < ncell) {
          A.cell_fill[c0 + k] = ex;
          A.cell_count[c0 + k] = 0;
        }
        ex += n[k];
      }
      carry += total;
    }
    if (threadIdx.x == 0) A.scan_aux[b] = carry;
  }
  if (!gbar(st)) return false;
  // R3: every block scans the tiles' sums; the atoms' reference numbers go
  // to their cells in arrival order, and the cells get their final starts
  {
    constexpr int kT = kMaxTiles / kPB;
    int s = 0, loc[kT];
#pragma unroll
    for (int k = 0; k < kT; k++) {
      const int t = threadIdx.x * kT + k;
      loc[k] = t < ntiles ? __ldcg(A.scan_aux + t) : 0;
      s += loc[k];
    }
    int total;
    int ex = block_scan(s, ssh, total);
#pragma unroll
    for (int k = 0; k < kT; k++) {
      toff[threadIdx.x * kT + k] = ex;
      ex += loc[k];
    }
    __syncthreads();
  }
  for (int p = t0; p < N; p += G) {
    const int c = A.atom_cell[p];
    A.cell_atoms[__ldcg(A.cell_fill + c) + toff[c >> tlog] + A.row_lo[p]] = A.perm[p];
  }
  for (int c = t0; c < ncell; c += G) A.cell_start[c] = __ldcg(A.cell_fill + c) + toff[c >> tlog];
  if (t0 == 0) A.cell_start[ncell] = N;
  if (!gbar(st)) return false;
  // R4: each atom's place is its cell's start plus the number of smaller
  // reference indices in the cell; its state goes there in the scratch arrays
  for (int p = t0; p < N; p += G) {
    const int c = A.atom_cell[p], ref = A.perm[p];
    const int c0 = __ldcg(A.cell_start + c), c1 = __ldcg(A.cell_start + c + 1);
    const double4 v = wrap_box(P, pos[p]);
    int q = c0;
    for (int k = c0; k < c1; k++) q += __ldcg(A.cell_atoms + k) < ref;
    A.pos_s[q] = v;
    A.posf[q] = make_float4((float)v.x, (float)v.y, (float)v.z, __int_as_float(ref));
    A.vx_s[q] = A.vx[p];
    A.vy_s[q] = A.vy[p];
    A.vz_s[q] = A.vz[p];
    if (acc) {
      A.ax_s[q] = A.ax[p];
      A.ay_s[q] = A.ay[p];
      A.az_s[q] = A.az[p];
    }
    A.perm_s[q] = ref;
  }
  if (!gbar(st)) return false;
  // R5: rows (neighbor-pbc-mav.f:73-99), warp-aligned grid-stride, over the
  // new order in the scratch arrays; each slot is committed (copied back)
  // by the thread that takes it
  const double4* npos = A.pos_s;
  const int* perm = A.perm_s;
  for (int base0 = t0 - lane; base0 < N; base0 += G) {
    int p = base0 + lane;
    bool active = p < N;
    int cnt = 0, refi = 0;
    double4 pi = make_double4(0, 0, 0, 0);
    int2* buf = (int2*)&stage[w] + lane;
    if (active) {
      pi = npos[p];
      refi = perm[p];
      pos[p] = pi;
      A.vx[p] = A.vx_s[p];
      A.vy[p] = A.vy_s[p];
      A.vz[p] = A.vz_s[p];
      if (acc) {
        A.ax[p] = A.ax_s[p];
        A.ay[p] = A.ay_s[p];
        A.az[p] = A.az_s[p];
      }
      A.perm[p] = refi;
      A.iperm[refi] = p;
      cnt = row_search(P, g, p, refi, pi, npos, A.posf, A.cell_start, buf, nullptr);
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    unsigned long long start = 0;
    if (lane == 31) start = atomicAdd(&st->list_used, (unsigned long long)incl);
    start = __shfl_sync(0xffffffffu, start, 31) + (unsigned long long)(incl - cnt);
    int lo = 0, longer = 0;
    if (start + (unsigned long long)cnt > (unsigned long long)P.list_cap) {
      raise_err(st, CLMD_ERR_LIST_OVERFLOW);
      start = 0;
      cnt = 0;
    } else if (cnt > kRowCap) {
      longer = cnt;
      row_search(P, g, p, refi, pi, npos, A.posf, A.cell_start, nullptr, A.list + start);
    } else {
      lo = row_store(buf, cnt, refi, A.list + start);
    }
    sort_long_rows(A.list, perm, start, longer, refi, lo);
    if (!active) continue;
    A.row_start[p] = (int)start;
    A.row_len[p] = cnt;
    A.row_lo[p] = lo;
  }
  if (!gbar(st)) return false;
  // neighbor-pbc-mav.f:95-97: the half list's write cursor after the last
  // row (1 + natom headers + half pairs) plus natom must stay within mxnlist
  const bool full = P.half_cap > 0 &&
                    (long long)(__ldcg(&st->list_used) / 2ull) + 2LL * P.N + 1 > P.half_cap;
  if (__ldcg(&st->err_new) != 0 || full) {
    if (threadIdx.x == 0 && B.q.status == 0) {
      B.q.status = CLMD_ERR_LIST_OVERFLOW;
      B.q.fail_step = st->cur_step;
    }
    return false;
  }
  return true;
}

enum { SLOT_MAX = 0, SLOT_SUMV2 = 1, SLOT_EPOT = 2, SLOT_VIR = 3, SLOT_EKIN = 4,
       SLOT_WV = 5, SLOT_VV = 4, SLOT_EK0 = 6 /* ek per species: 6..15 */ };

// Nose-Hoover by the reference's own sweeps where the closed form does not
// stand for them (clmd_nh_closed): the two further sums, then the number of
// sweeps.  red0, red1: the partial buffers, the next one first.
struct Swept {
  int n;     // sweeps; kNhSweeps + 1: no convergence; 0: a barrier timed out
  double p;  // the new PSI
};
static __device__ __noinline__ Swept nh_sweep(DevState* st, int N, const double* vx,
                                              const double* vy, const double* vz,
                                              const double* ax, const double* ay,
                                              const double* az, double dt, double m, double nkt3,
                                              double Q, double sww, double psi, double* red0,
                                              double* red1, double* sh, double* bc) {
  const int G = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const double dth = dt / 2;
  double wv = 0.0, vv = 0.0, swv = 0.0, svv = 0.0;
  int need = 1;
  for (int pass = 0; pass < 2; pass++) {
    for (int p = t0; p < N; p += G) {
      const double V[3] = {vx[p], vy[p], vz[p]};
      const double W[3] = {V[0] + dth * ax[p], V[1] + dth * ay[p], V[2] + dth * az[p]};
      if (pass == 0) {
        wv = wv + W[0] * V[0] + W[1] * V[1] + W[2] * V[2];
        vv = vv + V[0] * V[0] + V[1] * V[1] + V[2] * V[2];
      } else {
        need = max(need, clmd_nh_sweeps(W, V, sww, swv, svv, psi, m, nkt3, dt, Q));
      }
    }
    if (pass == 0) {
      put_sum(red0, SLOT_WV, wv, sh);
      put_sum(red0, SLOT_VV, vv, sh);
      if (!gbar(st)) return {0, 0.0};
      swv = get_sum(red0, SLOT_WV, sh, bc);
      svv = get_sum(red0, SLOT_VV, sh, bc);
    } else {
      put_max(red1, SLOT_MAX, (double)need, sh);
      if (!gbar(st)) return {0, 0.0};
      need = (int)get_max(red1, SLOT_MAX, sh, bc);
    }
  }
  return {need, clmd_nh_swept(need, sww, swv, svv, psi, m, nkt3, dt, Q)};
}

template <bool NH, bool THERMO, bool MIXED>
__global__ void __launch_bounds__(kPB, CLMD_CYCLE_MINB) k_cycle(Params P, DevState* st,
                                                                CycleArgs A, int nsteps,
                                                                int mode, int first,
                                                                int set) {
  // set: the first step's number (main.f's loop counter) comes with the call
  if (set && blockIdx.x == 0 && threadIdx.x == 0) st->cur_step = first;
  if (gated(st)) return;
  __shared__ Blk B;
  __shared__ double sh[kPB / 32];
  extern __shared__ __align__(16) WarpStage stage[];  // [kPB / 32]
  const int N = P.N;
  const int G = gridDim.x * blockDim.x;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr bool nh = NH;
  constexpr bool thermo = THERMO;
  const double dt = P.dt;
  if (threadIdx.x == 0) {
    B.q = st->s;
    B.g.rs2 = st->rs2;
    B.g.cfx = st->cfx; B.g.cfy = st->cfy; B.g.cfz = st->cfz;
    B.g.ncx = st->ncx; B.g.ncy = st->ncy; B.g.ncz = st->ncz; B.g.ncell = st->ncell;
    B.g.nox = st->nox; B.g.noy = st->noy; B.g.noz = st->noz;
    B.stop = 0;
    B.rebuild = 0;
  }
  __syncthreads();
  int step = set ? first : st->cur_step;
  int cur = 0;  // positions of the current step live in pos0 / pos1
  auto posb = [&](int k) { return k ? A.pos1 : A.pos0; };
  int rb = 0;  // partial-buffer toggle
  auto red = [&]() { return A.red + (size_t)rb * kRedSlots * gridDim.x; };

  if (mode == 1) {
    // neighbor(step) called directly: a forced rebuild
    if (threadIdx.x == 0) {
      B.rebuild = 1;
      prologue(P, B, step);
    }
    __syncthreads();
    if (!B.stop) rebuild(P, st, B, A, posb(0), stage, true);
    goto done;
  }

  {
    bool drift_done = false;  // the current step's drift already ran (fused)
    const double psi0 = B.q.psi;
    (void)psi0;
    for (int s = 0; s < nsteps; s++, step++) {
      const bool last = (s == nsteps - 1);
      if (!drift_done) {
        // ---- velocity scaling (scalev-nh-m.f), main.f:207, before the step
        if (thermo) {
          for (int sp = 0; sp < P.atsorts; sp++) {
            double e = 0.0;
            for (int p = t0; p < N; p += G) {
              int b = sp_block(P, A.perm[p]);
              if (b == sp)
                e = e + 0.5 * P.apmas[sp] * (A.vx[p] * A.vx[p] + A.vy[p] * A.vy[p] +
                                             A.vz[p] * A.vz[p]);
            }
            put_sum(red(), SLOT_EK0 + sp, e, sh);
          }
          if (!gbar(st)) goto timeout;
          for (int sp = 0; sp < P.atsorts; sp++) {
            double ek = get_sum(red(), SLOT_EK0 + sp, sh, B.bcast);
            if (threadIdx.x == 0) {
              B.kf[sp] = sqrt(P.ekinT[sp] / ek);
              B.scale[sp] = (P.apth[sp] == 'X');
            }
          }
          __syncthreads();
          rb ^= 1;
        }
        // ---- drift (int-verlet-mav.f:44-56 / int-verlet-nh-mav.f:49-61)
        double d2 = 0.0, sv = 0.0;
        const double psi = B.q.psi;
        const double dt2 = dt * dt / 2, dth = dt / 2;
        double4* pos = posb(cur);
        for (int p = t0; p < N; p += G) {
          double vxi = A.vx[p], vyi = A.vy[p], vzi = A.vz[p];
          if (thermo) {
            int b = sp_block(P, A.perm[p]);
            if (b >= 0 && B.scale[b]) {
              double kf = B.kf[b];
              vxi = vxi * kf;
              vyi = vyi * kf;
              vzi = vzi * kf;
            }
          }
          double4 q = pos[p];
          double axi = A.ax[p], ayi = A.ay[p], azi = A.az[p];
          double dx, dy, dz;
          if (!nh) {
            double hx = 0.5 * axi * dt, hy = 0.5 * ayi * dt, hz = 0.5 * azi * dt;
            dx = (vxi + hx) * dt;
            dy = (vyi + hy) * dt;
            dz = (vzi + hz) * dt;
            vxi = vxi + hx;
            vyi = vyi + hy;
            vzi = vzi + hz;
          } else {
            dx = dt * vxi + dt2 * (axi - psi * vxi);
            dy = dt * vyi + dt2 * (ayi - psi * vyi);
            dz = dt * vzi + dt2 * (azi - psi * vzi);
            sv = sv + vxi * vxi + vyi * vyi + vzi * vzi;
            vxi = vxi + dth * (axi - psi * vxi);
            vyi = vyi + dth * (ayi - psi * vyi);
            vzi = vzi + dth * (azi - psi * vzi);
          }
          q.x = q.x + dx;
          q.y = q.y + dy;
          q.z = q.z + dz;
          pos[p] = q;
          A.vx[p] = vxi;
          A.vy[p] = vyi;
          A.vz[p] = vzi;
          d2 = fmax(d2, dx * dx + dy * dy + dz * dz);
        }
        put_max(red(), SLOT_MAX, d2, sh);
        if (nh) put_sum(red(), SLOT_SUMV2, sv, sh);
        if (!gbar(st)) goto timeout;
      }
      // ---- scalars after the drift: NH s/PSI half step, skin decision
      {
        double dmmr = get_max(red(), SLOT_MAX, sh, B.bcast);
        double sumv2 = nh ? get_sum(red(), SLOT_SUMV2, sh, B.bcast) : 0.0;
        if (threadIdx.x == 0) {
          if (nh) {
            clmd_scalars& q = B.q;
            const double dt2 = dt * dt / 2, dth = dt / 2;
            q.sumv2 = sumv2;
            if (P.ethst == 'N') {  // int-verlet-nh-mav.f:64-67
              q.s = q.s + q.psi * dt + (P.apmas[0] * q.sumv2 - P.nkt3_d) * dt2 / P.Q;
              q.psi = q.psi + (P.apmas[0] * q.sumv2 - P.nkt3_d) * dth / P.Q;
            }
          }
          skin(P, B, dmmr, step);
        }
        __syncthreads();
        rb ^= 1;
        if (B.stop) goto done;
        if (B.rebuild) {
          if (!rebuild(P, st, B, A, posb(cur), stage, false)) goto stop_or_timeout;
        }
      }
      // ---- forces (+ kick, + next drift)
      {
        double4* pos = posb(cur);
        double4* nxt = posb(cur ^ 1);
        const double bf1 = 2.0 + (double)(int)(B.q.atrskin / P.sig1);
        const double bf2 = bf1 + 0.5;
        const bool fuse = !nh && !thermo && !last;
        // mixed Nose-Hoover: the velocity pass fuses the next drift unless
        // this is the launch's last step or velocities are rescaled first
        const bool keep64 = last || thermo;
        (void)keep64;
        double esum = 0.0, vir = 0.0, ek = 0.0, d2 = 0.0, sv = 0.0, wv = 0.0, vv = 0.0;
        const double dth = dt / 2;
        WarpStage& W = stage[threadIdx.x >> 5];
        const int lane = threadIdx.x & 31;
        bool bad = false;  // (raised in st->err_new too)
        for (int base0 = t0 - lane; base0 < N; base0 += G) {
          const int p = base0 + lane;
          const bool act = p < N;
          double4 pa = act ? pos[p] : make_double4(0.0, 0.0, 0.0, 1.0);
          Pair f;
          f.esum = 0.0;
          f.vir = 0.0;
          // lane 0 is active whenever the warp is; only its row start is used
          warp_forces<MIXED>(P, st, pos, A.list, lane == 0 ? A.row_start[p] : 0,
                      act ? A.row_len[p] : 0,
                      act ? A.row_lo[p] : 0, pa, bf1, bf2, f.fx, f.fy, f.fz, f.esum, f.vir,
                      last, W, bad);
          // lanes past N still evaluated pair terms of their warp's atoms
          esum = esum + f.esum;
          vir = vir + f.vir;
          if (!act) continue;
          int sa = (int)pa.w;
          double iatm = 1.0 / P.apmas[sa - 1];
          // int-verlet-mav.f:76-84: a = 0, AccAtom adds fsum/m
          double axi = 0.0 + f.fx * iatm, ayi = 0.0 + f.fy * iatm, azi = 0.0 + f.fz * iatm;
          if (MIXED && nh) {
            // FP32 accelerations (the pair terms' precision); FP64 in the
            // state only where the next reader is an unfused drift
            const float fx32 = (float)axi, fy32 = (float)ayi, fz32 = (float)azi;
            axi = fx32;
            ayi = fy32;
            azi = fz32;
            if (!keep64) {
              A.afx[p] = fx32;
              A.afy[p] = fy32;
              A.afz[p] = fz32;
            }
          }
          if (!(MIXED && nh) || keep64) {
            A.ax[p] = axi;
            A.ay[p] = ayi;
            A.az[p] = azi;
          }
          if (!nh) {
            // :86-92
            double vxi = A.vx[p] + 0.5 * axi * dt;
            double vyi = A.vy[p] + 0.5 * ayi * dt;
            double vzi = A.vz[p] + 0.5 * azi * dt;
            if (last || thermo)
              ek = ek + 0.5 * P.apmas[sa - 1] * (vxi * vxi + vyi * vyi + vzi * vzi);
            if (fuse) {
              // next step's drift (:44-56)
              double hx = 0.5 * axi * dt, hy = 0.5 * ayi * dt, hz = 0.5 * azi * dt;
              double dx = (vxi + hx) * dt, dy = (vyi + hy) * dt, dz = (vzi + hz) * dt;
              double4 q = pa;
              q.x = q.x + dx;
              q.y = q.y + dy;
              q.z = q.z + dz;
              nxt[p] = q;
              vxi = vxi + hx;
              vyi = vyi + hy;
              vzi = vzi + hz;
              d2 = fmax(d2, dx * dx + dy * dy + dz * dz);
            }
            A.vx[p] = vxi;
            A.vy[p] = vyi;
            A.vz[p] = vzi;
          } else {
            // closed-form solve (clmd_nh_root): sv = sum W^2, W = V + dth a
            // (the velocity pass forms W again from V and a)
            const double vxi = A.vx[p], vyi = A.vy[p], vzi = A.vz[p];
            const double wx = vxi + dth * axi, wy = vyi + dth * ayi, wz = vzi + dth * azi;
            sv = sv + wx * wx + wy * wy + wz * wz;
            if (!MIXED && last) {  // for the count of the reference's sweeps
              wv = wv + wx * vxi + wy * vyi + wz * vzi;
              vv = vv + vxi * vxi + vyi * vyi + vzi * vzi;
            }
          }
        }
        if (last) {
          put_sum(red(), SLOT_EPOT, esum, sh);
          put_sum(red(), SLOT_VIR, vir, sh);
          if (!nh) put_sum(red(), SLOT_EKIN, ek, sh);
        }
        if (fuse) put_max(red(), SLOT_MAX, d2, sh);
        if (nh) {
          put_sum(red(), SLOT_SUMV2, sv, sh);
          if (!MIXED && last) {
            put_sum(red(), SLOT_WV, wv, sh);
            put_sum(red(), SLOT_VV, vv, sh);
          }
        }
        if (!gbar(st)) goto timeout;
        if (__ldcg(&st->err_new) != 0) {
          if (threadIdx.x == 0 && B.q.status == 0) {
            B.q.status = __ldcg(&st->err_new);
            B.q.fail_step = step;
          }
          goto done;
        }
        if (last) {
          double e = get_sum(red(), SLOT_EPOT, sh, B.bcast);
          double w = get_sum(red(), SLOT_VIR, sh, B.bcast);
          double k = nh ? 0.0 : get_sum(red(), SLOT_EKIN, sh, B.bcast);
          if (threadIdx.x == 0) {
            B.q.epot = e;
            B.q.virial = w;
            if (!nh) B.q.ekin = k;
          }
        }
        if (fuse) {
          cur ^= 1;
          drift_done = true;
        } else {
          drift_done = false;
        }
        if (!nh) {
          // the fused drift's reduction stays in this buffer for the
          // decision of the next step
          if (!fuse) rb ^= 1;
          continue;
        }
      }
      // ---- Nose-Hoover implicit solve (int-verlet-nh-mav.f:105-180)
      {
        const double dt2 = dt * dt / 2, dth = dt / 2, m = P.apmas[0], Q = P.Q;
        const double psi = B.q.psi;
        double sumv2 = get_sum(red(), SLOT_SUMV2, sh, B.bcast);
        const double swv = !MIXED && last ? get_sum(red(), SLOT_WV, sh, B.bcast) : 0.0;
        const double svv = !MIXED && last ? get_sum(red(), SLOT_VV, sh, B.bcast) : 0.0;
        rb ^= 1;
        // every block solves the same scalar equation from the same sums
        double pn;
        bool ok = clmd_nh_root(m * sumv2, psi, P.nkt3_i, dth, Q, pn);
        int iters = 1;
        if (!MIXED && !clmd_nh_closed(ok, psi, dth)) {
          double* const r0 = red();
          rb ^= 1;
          const Swept w = nh_sweep(st, N, A.vx, A.vy, A.vz, A.ax, A.ay, A.az, dt, m, P.nkt3_i, Q,
                                   sumv2, psi, r0, red(), sh, B.bcast);
          rb ^= 1;
          if (w.n == 0) goto timeout;
          iters = w.n;
          pn = w.p;
          ok = iters <= kNhSweeps;
        }
        if (!ok) {
          if (threadIdx.x == 0 && B.q.status == 0) {
            B.q.status = CLMD_ERR_NH_NOCONVERGE;
            B.q.fail_step = step;
            if (!MIXED) B.q.nh_iters = min(iters, kNhSweeps);
          }
          __syncthreads();
          goto done;
        }
        // v = W c, fused with the next step's drift (the same expressions
        // as the drift at the top of the step, PSI = pn) unless this is the
        // launch's last step or velocities are rescaled before each step
        const double c = 1.0 / (1.0 + dth * pn);
        const bool fuse = !thermo && !last;
        double d2 = 0.0, sv = 0.0;
        int sweeps = 1;
        double4* pos = posb(cur);
        for (int p = t0; p < N; p += G) {
          double axi, ayi, azi;
          if (MIXED && fuse) {
            axi = A.afx[p];
            ayi = A.afy[p];
            azi = A.afz[p];
          } else {
            axi = A.ax[p];
            ayi = A.ay[p];
            azi = A.az[p];
          }
          const double V[3] = {A.vx[p], A.vy[p], A.vz[p]};
          const double W[3] = {V[0] + dth * axi, V[1] + dth * ayi, V[2] + dth * azi};
          double vxi = W[0] * c, vyi = W[1] * c, vzi = W[2] * c;
          if (!MIXED && last)
            sweeps = max(sweeps, clmd_nh_sweeps(W, V, sumv2, swv, svv, psi, m, P.nkt3_i, dt, Q));
          if (fuse) {
            double dx = dt * vxi + dt2 * (axi - pn * vxi);
            double dy = dt * vyi + dt2 * (ayi - pn * vyi);
            double dz = dt * vzi + dt2 * (azi - pn * vzi);
            sv = sv + vxi * vxi + vyi * vyi + vzi * vzi;
            vxi = vxi + dth * (axi - pn * vxi);
            vyi = vyi + dth * (ayi - pn * vyi);
            vzi = vzi + dth * (azi - pn * vzi);
            double4 q = pos[p];
            q.x = q.x + dx;
            q.y = q.y + dy;
            q.z = q.z + dz;
            pos[p] = q;
            d2 = fmax(d2, dx * dx + dy * dy + dz * dz);
          }
          A.vx[p] = vxi;
          A.vy[p] = vyi;
          A.vz[p] = vzi;
        }
        if (threadIdx.x == 0) {
          B.q.nh_iters = iters;
          B.q.sumv2 = sumv2 * c * c;
          B.q.psi = pn;
          B.q.ekin = 0.5 * m * B.q.sumv2;
        }
        if (fuse) {
          // the forces' reads of pos ended at the barrier before the root
          put_max(red(), SLOT_MAX, d2, sh);
          put_sum(red(), SLOT_SUMV2, sv, sh);
          if (!gbar(st)) goto timeout;
          drift_done = true;
        } else {
          __syncthreads();
          drift_done = false;
        }
        if (!MIXED && last) {  // the sweeps the reference takes for this step
          put_max(red(), SLOT_MAX, (double)sweeps, sh);
          if (!gbar(st)) goto timeout;
          const double n = get_max(red(), SLOT_MAX, sh, B.bcast);
          if (threadIdx.x == 0) B.q.nh_iters = min((int)n, kNhSweeps);
          rb ^= 1;
        }
      }
    }
  }
  goto done;
stop_or_timeout:
  goto done;
timeout:
  if (threadIdx.x == 0) atomicCAS(&st->s.status, 0, CLMD_ERR_TIMEOUT);
  return;
done:
  // positions back in pos0, then block 0 publishes its replica
  if (cur == 1)
    for (int p = t0; p < N; p += G) A.pos0[p] = A.pos1[p];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    clmd_scalars q = B.q;
    q.npairs_half = (long long)(st->list_used / 2ull);
    // err_new stays set (other blocks may still read it); the status latches it
    int err = __ldcg(&st->err_new);
    if (err && q.status == 0) {
      q.status = err;
      q.fail_step = step;
    }
    st->s = q;
    st->cur_step = (mode == 1) ? st->cur_step : step;
    st->rs2 = B.g.rs2;
    st->cfx = B.g.cfx; st->cfy = B.g.cfy; st->cfz = B.g.cfz;
    st->ncx = B.g.ncx; st->ncy = B.g.ncy; st->ncz = B.g.ncz; st->ncell = B.g.ncell;
    st->nox = B.g.nox; st->noy = B.g.noy; st->noz = B.g.noz;
  }
}

// This file is compiled twice: as is (the FP64 kernels and the host side)
// and with CLMD_CYCLE_MIXED (the mixed-precision kernels only).  In one
// translation unit the two sets got larger local frames and ran ~4% slower.
typedef void (*CycleKernel)(Params, DevState*, CycleArgs, int, int, int, int);

#ifdef CLMD_CYCLE_MIXED
CycleKernel cycle_kernel_mixed(bool nh, bool th) {
  if (nh) return th ? k_cycle<true, true, true> : k_cycle<true, false, true>;
  return th ? k_cycle<false, true, true> : k_cycle<false, false, true>;
}
#else
CycleKernel cycle_kernel_mixed(bool nh, bool th);

static CycleArgs cycle_args(clmd_system* S) {
  CycleArgs A;
  A.pos0 = S->pos;
  A.pos1 = S->pos_alt;
  A.vx = S->vx; A.vy = S->vy; A.vz = S->vz;
  A.ax = S->ax; A.ay = S->ay; A.az = S->az;
  A.afx = S->afx; A.afy = S->afy; A.afz = S->afz;
  A.perm = S->perm; A.iperm = S->iperm;
  A.pos_s = S->pos_s;
  A.vx_s = S->vx_s; A.vy_s = S->vy_s; A.vz_s = S->vz_s;
  A.ax_s = S->ax_s; A.ay_s = S->ay_s; A.az_s = S->az_s;
  A.perm_s = S->perm_s;
  A.posf = S->posf;
  A.cell_count = S->cell_count; A.cell_start = S->cell_start; A.cell_fill = S->cell_fill;
  A.cell_atoms = S->cell_atoms; A.atom_cell = S->atom_cell; A.scan_aux = S->scan_aux;
  A.list = S->list; A.row_start = S->row_start; A.row_len = S->row_len; A.row_lo = S->row_lo;
  A.red = S->red;
  return A;
}

static CycleKernel cycle_kernel(const clmd_system* S) {
  bool nh = S->P.integrator == CLMD_INT_NOSE, th = S->P.ethst == 'X';
  if (S->P.precision == CLMD_PREC_MIXED) return cycle_kernel_mixed(nh, th);
  if (nh) return th ? k_cycle<true, true, false> : k_cycle<true, false, false>;
  return th ? k_cycle<false, true, false> : k_cycle<false, false, false>;
}

constexpr int kStageBytes = (kPB / 32) * (int)sizeof(WarpStage);

int cycle_blocks_for(clmd_system* S) {
  small_setup(S);
  int per_sm = 0;
  cudaFuncSetAttribute(cycle_kernel(S), cudaFuncAttributeMaxDynamicSharedMemorySize, kStageBytes);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cycle_kernel(S), kPB, kStageBytes);
  if (per_sm < 1) per_sm = 1;
  int nb = S->num_sms * per_sm;
  int need = (S->P.N + kPB - 1) / kPB;
  need = need < 1 ? 1 : need;
  return nb < need ? nb : need;
}

void cycle_launch(clmd_system* S, int nsteps, int mode, const int* step) {
  // small systems on one cluster, unless a failure-path test has changed the
  // grid barrier, which that kernel does not use
  if (S->small_ctas && !S->debug_barrier) {
    small_launch(S, cycle_args(S), nsteps, mode, step);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S->cyc_blocks);
  cfg.blockDim = dim3(kPB);
  cfg.dynamicSmemBytes = kStageBytes;
  cfg.stream = S->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, cycle_kernel(S), S->P, S->st, cycle_args(S), nsteps, mode,
                     step ? *step : 0, step != nullptr);
  S->launches++;
}
#endif  // CLMD_CYCLE_MIXED

}  // namespace clmd
