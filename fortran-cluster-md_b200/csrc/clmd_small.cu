// clmd_small.cu -- the persistent step kernel for small systems: one
// thread-block cluster, one atom per thread.
//
// The same work as k_cycle (clmd_cycle.cu): a launch runs `nsteps`
// consecutive integrator(i) calls, or one neighbor() call.  With a few
// thousand atoms a step is a chain of latencies, not work: on the grid
// kernel a step of 1,000 atoms (velocity Verlet) took 13.6 us and one of
// 5,921 (Nose-Hoover, FP64 sweeps) 49 us, nearly all of it grid barriers,
// partial sums fetched through L2 and per-atom state read back from memory.
// Here
//   - a barrier is the hardware cluster barrier (up to 16 CTAs, one per SM);
//   - a thread keeps its atom's position, velocity, acceleration and row in
//     registers between rebuilds; only positions go through memory, where
//     the neighbours' threads gather them;
//   - each warp writes its partial sums into every CTA's shared memory
//     (distributed shared memory) before the barrier, and after it every
//     warp adds them in one fixed order: all threads hold the same totals
//     without a further exchange;
//   - the atoms are spread over as many CTAs as possible (at least a few
//     warps each): the fewer warps share an SM, the shorter a step.
// Now 5.9 us a step at 1,000 atoms and 17 us at 5,921 (Nose-Hoover solved in
// closed form).  What is left is instruction latency: force pass ~2.5k cycles
// a chunk of 32 pair terms, cluster barrier ~1-2k, skin decision ~1.3k, a tenth
// of a ~40k-cycle rebuild; one CTA of 128 atoms is not much faster (6.5 us).
//
// Per-atom arithmetic, list order and the rows' chunks are those of k_cycle
// (same functions, same flags): positions, velocities, accelerations and
// lists are bit-identical to it.  Every CTA applies the same scalar logic to
// the same totals, errors included (they travel with the partial sums), so
// all CTAs take the same branches and leave together.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "clmd_cycle.cuh"

namespace clmd {

namespace cg = cooperative_groups;

constexpr int kSC = 16;              // CTAs of a cluster at most
constexpr int kSNT = kSmallThreads;  // threads of a CTA at most
constexpr int kSW = kSNT / 32;
constexpr int kSSlots = 10;

struct SmallShared {
  Blk B;
  double part[2][kSSlots][kSC * kSW];  // partial sums: phase parity, slot, warp of the cluster
  int err[2];                          // an error of this phase, from any CTA
  int csum[kSC];
  int wsum[kSW + 1];
  WarpStage stage[kSW];
};

struct Grp {
  int C, nw, rank, lane;
  int mine;  // this warp's number in the cluster
  SmallShared* s;
  int rb;  // parity of the phase whose partial sums are being written

  __device__ __forceinline__ void barrier() const {
    if (C == 1)
      __syncthreads();
    else
      cg::this_cluster().sync();
  }
  template <class T>
  __device__ __forceinline__ T* at(T* p, int r) const {
    return C == 1 ? p : cg::this_cluster().map_shared_rank(p, r);
  }
  __device__ __forceinline__ void put(int slot, double warp_total) const {
    if (lane < C) *at(&s->part[rb][slot][mine], lane) = warp_total;
  }
  __device__ __forceinline__ void put_sum(int slot, double v) const { put(slot, warp_sum(v)); }
  __device__ __forceinline__ void put_max(int slot, double v) const { put(slot, warp_max(v)); }
  __device__ __forceinline__ void put_err(int code) const {
    for (int r = 0; r < C; r++) *at(&s->err[rb], r) = code;
  }
  // after the barrier, the same value in every thread of the cluster
  __device__ __forceinline__ double get_sum(int slot) const {
    double v = 0.0;
    for (int k = lane; k < C * nw; k += 32) v += s->part[rb][slot][k];
    return warp_sum(v);
  }
  __device__ __forceinline__ double get_max(int slot) const {
    double v = 0.0;
    for (int k = lane; k < C * nw; k += 32) v = fmax(v, s->part[rb][slot][k]);
    return warp_max(v);
  }
};

// one atom's state, in its thread's registers
struct Atom {
  double4 q;
  double vx, vy, vz, ax, ay, az;
  int ref;                // reference index (perm)
  int start, len, lo;     // its list row
  bool act;
};

template <class T>
__device__ __forceinline__ T s_pre(T v, int lane) {  // inclusive scan over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// neighbor-pbc-mav.f:67-99: positions wrapped, atoms put in cell order (ties
// by reference index, as k_cycle), rows searched and sorted.  acc: the
// accelerations move with their atoms (a rebuild inside a step runs before
// the force pass that overwrites them).  False: the cluster must stop.
static __device__ bool s_rebuild(const Params& P, DevState* st, SmallShared& S, Grp& G,
                                 const CycleArgs& A, double4* pos, Atom& a, int p, bool acc) {
  const Geo& g = S.B.g;
  const int tid = threadIdx.x, NT = blockDim.x, lane = G.lane, w = tid >> 5;
  if (p == 0) st->list_used = 0ull;
  int cell = 0, arrival = 0;
  if (a.act) {
    a.q = wrap_box(P, a.q);
    const int cx = clmd_cell(a.q.x, g.cfx, g.ncx);
    const int cy = clmd_cell(a.q.y, g.cfy, g.ncy);
    const int cz = clmd_cell(a.q.z, g.cfz, g.ncz);
    cell = (cz * g.ncy + cy) * g.ncx + cx;
    arrival = atomicAdd(&A.cell_count[cell], 1);
  }
  G.barrier();
  // cell starts: each CTA scans its share of the cells, then adds the sums
  // of the CTAs before it; the counts go back to zero
  const int share = (g.ncell + G.C - 1) / G.C;
  const int per = (share + NT - 1) / NT;
  const int c0 = G.rank * share + tid * per;
  const int c1 = min(min(c0 + per, (G.rank + 1) * share), g.ncell);
  int sum = 0;
  for (int c = c0; c < c1; c++) sum += __ldcg(A.cell_count + c);
  const int incl = s_pre(sum, lane);
  if (lane == 31) S.wsum[w] = incl;
  __syncthreads();
  int before = 0, total = 0;
  for (int k = 0; k < G.nw; k++) {
    const int t = S.wsum[k];
    before += k < w ? t : 0;
    total += t;
  }
  if (tid < G.C) *G.at(&S.csum[G.rank], tid) = total;
  G.barrier();
  int ex = before + incl - sum;
  for (int r = 0; r < G.rank; r++) ex += S.csum[r];
  for (int c = c0; c < c1; c++) {
    const int n = __ldcg(A.cell_count + c);
    A.cell_start[c] = ex;
    A.cell_count[c] = 0;
    ex += n;
  }
  if (p == 0) A.cell_start[g.ncell] = P.N;
  G.barrier();
  // reference numbers by cell in arrival order; then every atom's place is
  // its cell's start plus the number of smaller reference indices in it
  int s0 = 0;
  if (a.act) {
    s0 = A.cell_start[cell];
    A.cell_atoms[s0 + arrival] = a.ref;
  }
  G.barrier();
  if (a.act) {
    const int s1 = A.cell_start[cell + 1];
    int dst = s0;
    for (int k = s0; k < s1; k++) dst += A.cell_atoms[k] < a.ref;
    A.pos_s[dst] = a.q;
    A.vx_s[dst] = a.vx;
    A.vy_s[dst] = a.vy;
    A.vz_s[dst] = a.vz;
    if (acc) {
      A.ax_s[dst] = a.ax;
      A.ay_s[dst] = a.ay;
      A.az_s[dst] = a.az;
    }
    A.perm_s[dst] = a.ref;
    A.posf[dst] = make_float4((float)a.q.x, (float)a.q.y, (float)a.q.z, __int_as_float(a.ref));
    A.iperm[a.ref] = dst;
  }
  G.barrier();
  int2* buf = (int2*)&S.stage[w] + lane;
  int cnt = 0;
  if (a.act) {
    a.q = A.pos_s[p];
    a.vx = A.vx_s[p];
    a.vy = A.vy_s[p];
    a.vz = A.vz_s[p];
    if (acc) {
      a.ax = A.ax_s[p];
      a.ay = A.ay_s[p];
      a.az = A.az_s[p];
    }
    a.ref = A.perm_s[p];
    A.perm[p] = a.ref;
    pos[p] = a.q;
    cnt = row_search(P, g, p, a.ref, a.q, A.pos_s, A.posf, A.cell_start, buf, nullptr);
  }
  // one warp-wide cursor step: a warp's 32 rows are contiguous
  const int inc = s_pre(cnt, lane);
  unsigned long long base = 0;
  if (lane == 31 && inc) base = atomicAdd(&st->list_used, (unsigned long long)inc);
  base = __shfl_sync(0xffffffffu, base, 31) + (unsigned long long)(inc - cnt);
  a.start = (int)base;
  a.len = cnt;
  a.lo = 0;
  const bool over = base + (unsigned long long)cnt > (unsigned long long)P.list_cap;
  int longer = 0;
  if (over) {
    raise_err(st, CLMD_ERR_LIST_OVERFLOW);
    G.put_err(CLMD_ERR_LIST_OVERFLOW);
    a.start = a.len = 0;
  } else if (cnt > kRowCap) {
    longer = cnt;
    row_search(P, g, p, a.ref, a.q, A.pos_s, A.posf, A.cell_start, nullptr, A.list + base);
  } else {
    a.lo = row_store(buf, cnt, a.ref, A.list + base);
  }
  sort_long_rows(A.list, A.perm_s, base, longer, a.ref, a.lo);
  if (a.act) {
    A.row_start[p] = a.start;
    A.row_len[p] = a.len;
    A.row_lo[p] = a.lo;
  }
  G.barrier();
  const int err = S.err[G.rb];
  G.rb ^= 1;
  // neighbor-pbc-mav.f:95-97: the half list's write cursor after the last
  // row (1 + natom headers + half pairs) plus natom must stay within mxnlist
  const bool full = P.half_cap > 0 &&
                    (long long)(__ldcg(&st->list_used) / 2ull) + 2LL * P.N + 1 > P.half_cap;
  if (err || full) {
    if (tid == 0 && S.B.q.status == 0) {
      S.B.q.status = CLMD_ERR_LIST_OVERFLOW;
      S.B.q.fail_step = st->cur_step;
    }
    return false;
  }
  return true;
}

enum { SS_MAX = 0, SS_SUMV2, SS_EPOT, SS_VIR, SS_EKIN, SS_WV, SS_VV };

// Nose-Hoover by the reference's own sweeps where the closed form does not
// stand for them (clmd_nh_closed).  Two phases: G's parity stays as it is.
struct Swept {
  int n;     // sweeps; kNhSweeps + 1: no convergence
  double p;  // the new PSI
};
static __device__ __noinline__ Swept s_sweep(Grp G, bool act, double wx, double wy, double wz,
                                             double vx, double vy, double vz, double sww,
                                             double psi, double m, double nkt3, double dt,
                                             double Q) {
  G.put_sum(SS_WV, wx * vx + wy * vy + wz * vz);
  G.put_sum(SS_VV, vx * vx + vy * vy + vz * vz);
  G.barrier();
  const double swv = G.get_sum(SS_WV), svv = G.get_sum(SS_VV);
  G.rb ^= 1;
  int n = 1;
  if (act) {
    const double W[3] = {wx, wy, wz}, V[3] = {vx, vy, vz};
    n = clmd_nh_sweeps(W, V, sww, swv, svv, psi, m, nkt3, dt, Q);
  }
  G.put_max(SS_MAX, (double)n);
  G.barrier();
  n = (int)G.get_max(SS_MAX);
  return {n, clmd_nh_swept(n, sww, swv, svv, psi, m, nkt3, dt, Q)};
}

template <bool NH, bool THERMO, bool MIXED>
__global__ void __launch_bounds__(kSNT, 1) k_small(Params P, DevState* st, CycleArgs A, int nsteps,
                                                   int mode, int first, int set, int per) {
  // set: the first step's number (main.f's loop counter) comes with the call
  if (set && blockIdx.x == 0 && threadIdx.x == 0) st->cur_step = first;
  if (gated(st)) return;  // uniform: CTA 0 writes it back after the last barrier
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmallShared& S = *reinterpret_cast<SmallShared*>(smem_raw);
  Blk& B = S.B;
  const int tid = threadIdx.x, NT = blockDim.x, N = P.N;
  Grp G;
  G.C = gridDim.x;
  G.nw = NT >> 5;
  G.rank = blockIdx.x;
  G.lane = tid & 31;
  G.mine = G.rank * G.nw + (tid >> 5);
  G.s = &S;
  G.rb = 0;
  {
    const int* src = (const int*)&st->s;
    int* dst = (int*)&B.q;
    for (int k = tid; k < (int)(sizeof(clmd_scalars) / 4); k += NT) dst[k] = __ldcg(src + k);
  }
  if (tid == 0) {
    B.g.rs2 = st->rs2;
    B.g.cfx = st->cfx; B.g.cfy = st->cfy; B.g.cfz = st->cfz;
    B.g.ncx = st->ncx; B.g.ncy = st->ncy; B.g.ncz = st->ncz; B.g.ncell = st->ncell;
    B.g.nox = st->nox; B.g.noy = st->noy; B.g.noz = st->noz;
    B.stop = 0;
    B.rebuild = 0;
    S.err[0] = S.err[1] = 0;
  }
  int step = set ? first : st->cur_step;
  // `per` atoms per warp, in its first lanes
  const int p = G.lane < per ? G.mine * per + G.lane : N;
  Atom a;
  a.act = p < N;
  a.q = make_double4(0.0, 0.0, 0.0, 1.0);
  a.vx = a.vy = a.vz = a.ax = a.ay = a.az = 0.0;
  a.ref = a.start = a.len = a.lo = 0;
  if (a.act) {
    a.q = A.pos0[p];
    a.vx = A.vx[p]; a.vy = A.vy[p]; a.vz = A.vz[p];
    a.ax = A.ax[p]; a.ay = A.ay[p]; a.az = A.az[p];
    a.ref = A.perm[p];
    a.start = A.row_start[p]; a.len = A.row_len[p]; a.lo = A.row_lo[p];
  }
  G.barrier();  // every CTA has started (its shared memory may be written)
  WarpStage& W = S.stage[tid >> 5];
  const double dt = P.dt, dt2 = dt * dt / 2, dth = dt / 2;
  int cur = 0;  // the current positions: pos0 / pos1

  if (mode == 1) {
    if (tid == 0) {
      B.rebuild = 1;
      prologue(P, B, step);
    }
    __syncthreads();
    if (!B.stop) s_rebuild(P, st, S, G, A, A.pos0, a, p, true);
    goto done;
  }
  {
    bool drift_done = false;
    for (int s = 0; s < nsteps; s++, step++) {
      const bool last = (s == nsteps - 1);
      if (!drift_done) {
        if (THERMO) {  // scalev-nh-m.f, main.f:207
          const int b = a.act ? sp_block(P, a.ref) : -1;
          for (int sp = 0; sp < P.atsorts; sp++)
            G.put_sum(sp, b == sp ? 0.5 * P.apmas[sp] * (a.vx * a.vx + a.vy * a.vy + a.vz * a.vz)
                                  : 0.0);
          G.barrier();
          for (int sp = 0; sp < P.atsorts; sp++) {
            const double ek = G.get_sum(sp);
            const double kf = sqrt(P.ekinT[sp] / ek);
            if (b == sp && P.apth[sp] == 'X') {
              a.vx = a.vx * kf;
              a.vy = a.vy * kf;
              a.vz = a.vz * kf;
            }
          }
          G.rb ^= 1;
        }
        // drift (int-verlet-mav.f:44-56 / int-verlet-nh-mav.f:49-61)
        double d2 = 0.0, sv = 0.0;
        if (a.act) {
          double dx, dy, dz;
          if (!NH) {
            const double hx = 0.5 * a.ax * dt, hy = 0.5 * a.ay * dt, hz = 0.5 * a.az * dt;
            dx = (a.vx + hx) * dt;
            dy = (a.vy + hy) * dt;
            dz = (a.vz + hz) * dt;
            a.vx = a.vx + hx;
            a.vy = a.vy + hy;
            a.vz = a.vz + hz;
          } else {
            const double psi = B.q.psi;
            dx = dt * a.vx + dt2 * (a.ax - psi * a.vx);
            dy = dt * a.vy + dt2 * (a.ay - psi * a.vy);
            dz = dt * a.vz + dt2 * (a.az - psi * a.vz);
            sv = a.vx * a.vx + a.vy * a.vy + a.vz * a.vz;
            a.vx = a.vx + dth * (a.ax - psi * a.vx);
            a.vy = a.vy + dth * (a.ay - psi * a.vy);
            a.vz = a.vz + dth * (a.az - psi * a.vz);
          }
          a.q.x = a.q.x + dx;
          a.q.y = a.q.y + dy;
          a.q.z = a.q.z + dz;
          (cur ? A.pos1 : A.pos0)[p] = a.q;
          d2 = dx * dx + dy * dy + dz * dz;
        }
        G.put_max(SS_MAX, d2);
        if (NH) G.put_sum(SS_SUMV2, sv);
        G.barrier();
      }
      // scalars after the drift: NH s/PSI half step, skin decision
      {
        const double dmmr = G.get_max(SS_MAX);
        const double sumv2 = NH ? G.get_sum(SS_SUMV2) : 0.0;
        __syncthreads();  // the replica's readers of the step before are done
        if (tid == 0) {
          if (NH) {
            clmd_scalars& q = B.q;
            q.sumv2 = sumv2;
            if (P.ethst == 'N') {  // int-verlet-nh-mav.f:64-67
              q.s = q.s + q.psi * dt + (P.apmas[0] * q.sumv2 - P.nkt3_d) * dt2 / P.Q;
              q.psi = q.psi + (P.apmas[0] * q.sumv2 - P.nkt3_d) * dth / P.Q;
            }
          }
          skin(P, B, dmmr, step);
        }
        __syncthreads();
        G.rb ^= 1;
        if (B.stop) goto done;
        if (B.rebuild && !s_rebuild(P, st, S, G, A, cur ? A.pos1 : A.pos0, a, p, false))
          goto done;
      }
      // forces, kick, next drift
      const double psi = B.q.psi, m = P.apmas[0], Q = P.Q;
      const bool fuse = !NH && !THERMO && !last;
      double wx = 0.0, wy = 0.0, wz = 0.0;
      {
        const double bf1 = 2.0 + (double)(int)(B.q.atrskin / P.sig1), bf2 = bf1 + 0.5;
        double fx, fy, fz, esum = 0.0, vir = 0.0, ek = 0.0, d2 = 0.0, sv = 0.0;
        bool bad = false;
        warp_forces<MIXED>(P, st, cur ? A.pos1 : A.pos0, A.list, a.start, a.len, a.lo, a.q, bf1,
                           bf2, fx, fy, fz, esum, vir, last, W, bad);
        if (bad) G.put_err(CLMD_ERR_BAD_SPECIES);
        if (a.act) {
          const double mass = P.apmas[(int)a.q.w - 1], iatm = 1.0 / mass;
          // int-verlet-mav.f:76-84: a = 0, AccAtom adds fsum/m
          a.ax = 0.0 + fx * iatm;
          a.ay = 0.0 + fy * iatm;
          a.az = 0.0 + fz * iatm;
          if (MIXED && NH) {  // FP32 accelerations, the pair terms' precision
            a.ax = (float)a.ax;
            a.ay = (float)a.ay;
            a.az = (float)a.az;
          }
          if (!NH) {  // :86-92
            a.vx = a.vx + 0.5 * a.ax * dt;
            a.vy = a.vy + 0.5 * a.ay * dt;
            a.vz = a.vz + 0.5 * a.az * dt;
            if (last || THERMO) ek = 0.5 * mass * (a.vx * a.vx + a.vy * a.vy + a.vz * a.vz);
            if (fuse) {  // the next step's drift (:44-56)
              const double hx = 0.5 * a.ax * dt, hy = 0.5 * a.ay * dt, hz = 0.5 * a.az * dt;
              const double dx = (a.vx + hx) * dt, dy = (a.vy + hy) * dt, dz = (a.vz + hz) * dt;
              a.q.x = a.q.x + dx;
              a.q.y = a.q.y + dy;
              a.q.z = a.q.z + dz;
              (cur ? A.pos0 : A.pos1)[p] = a.q;
              a.vx = a.vx + hx;
              a.vy = a.vy + hy;
              a.vz = a.vz + hz;
              d2 = dx * dx + dy * dy + dz * dz;
            }
          } else {
            // closed-form solve (clmd_nh_root): W = V + dth a
            wx = a.vx + dth * a.ax;
            wy = a.vy + dth * a.ay;
            wz = a.vz + dth * a.az;
            sv = wx * wx + wy * wy + wz * wz;
          }
        }
        if (last) {
          G.put_sum(SS_EPOT, esum);
          G.put_sum(SS_VIR, vir);
          if (!NH) G.put_sum(SS_EKIN, ek);
        }
        if (fuse) G.put_max(SS_MAX, d2);
        if (NH) {
          G.put_sum(SS_SUMV2, sv);
          if (!MIXED && last) {  // for the count of the reference's sweeps
            G.put_sum(SS_WV, wx * a.vx + wy * a.vy + wz * a.vz);
            G.put_sum(SS_VV, a.vx * a.vx + a.vy * a.vy + a.vz * a.vz);
          }
        }
        G.barrier();
        if (const int err = S.err[G.rb]) {
          // the positions of this step, not the fused drift's
          if (fuse && a.act) a.q = (cur ? A.pos1 : A.pos0)[p];
          if (tid == 0 && B.q.status == 0) {
            B.q.status = err;
            B.q.fail_step = step;
          }
          goto done;
        }
        if (last) {
          const double e = G.get_sum(SS_EPOT), v = G.get_sum(SS_VIR);
          const double k = NH ? 0.0 : G.get_sum(SS_EKIN);
          if (tid == 0) {
            B.q.epot = e;
            B.q.virial = v;
            if (!NH) B.q.ekin = k;
          }
        }
        if (fuse) cur ^= 1;
        drift_done = fuse;
        if (!NH) {
          // a fused drift's maximum stays in this buffer for the next step
          if (!fuse) G.rb ^= 1;
          continue;
        }
      }
      // Nose-Hoover implicit solve (int-verlet-nh-mav.f:105-180)
      const double sumv2 = G.get_sum(SS_SUMV2);
      const double swv = !MIXED && last ? G.get_sum(SS_WV) : 0.0;
      const double svv = !MIXED && last ? G.get_sum(SS_VV) : 0.0;
      G.rb ^= 1;
      double pn;  // every thread takes the same root of the same sum
      int sweeps = 1;
      bool ok = clmd_nh_root(m * sumv2, psi, P.nkt3_i, dth, Q, pn);
      if (!MIXED && !clmd_nh_closed(ok, psi, dth)) {
        const Swept w = s_sweep(G, a.act, wx, wy, wz, a.vx, a.vy, a.vz, sumv2, psi, m, P.nkt3_i,
                                dt, Q);
        pn = w.p;
        sweeps = min(w.n, kNhSweeps);
        ok = w.n <= kNhSweeps;
      } else if (!MIXED && last) {
        if (a.act) {
          const double W3[3] = {wx, wy, wz}, V3[3] = {a.vx, a.vy, a.vz};
          sweeps = clmd_nh_sweeps(W3, V3, sumv2, swv, svv, psi, m, P.nkt3_i, dt, Q);
        }
        G.put_max(SS_MAX, (double)sweeps);
        G.barrier();
        sweeps = min((int)G.get_max(SS_MAX), kNhSweeps);
        G.rb ^= 1;
      }
      if (!ok) {
        if (tid == 0 && B.q.status == 0) {
          B.q.status = CLMD_ERR_NH_NOCONVERGE;
          B.q.fail_step = step;
          if (!MIXED) B.q.nh_iters = sweeps;
        }
        goto done;
      }
      const double c = 1.0 / (1.0 + dth * pn);
      a.vx = wx * c;
      a.vy = wy * c;
      a.vz = wz * c;
      __syncthreads();  // every thread has read this step's PSI
      if (tid == 0) {
        B.q.nh_iters = sweeps;
        B.q.sumv2 = sumv2 * c * c;
        B.q.psi = pn;
        B.q.ekin = 0.5 * m * B.q.sumv2;
      }
      __syncthreads();
    }
  }
done:
  G.barrier();  // no CTA reads st, err_new or another's shared memory any more
  if (a.act) {
    A.pos0[p] = a.q;
    A.vx[p] = a.vx; A.vy[p] = a.vy; A.vz[p] = a.vz;
    A.ax[p] = a.ax; A.ay[p] = a.ay; A.az[p] = a.az;
  }
  if (G.rank != 0) return;
  if (tid == 0) {
    clmd_scalars& q = B.q;
    q.npairs_half = (long long)(__ldcg(&st->list_used) / 2ull);
    const int err = __ldcg(&st->err_new);  // stays set; the status latches it
    if (err && q.status == 0) {
      q.status = err;
      q.fail_step = step;
    }
    if (mode != 1) st->cur_step = step;
    st->rs2 = B.g.rs2;
    st->cfx = B.g.cfx; st->cfy = B.g.cfy; st->cfz = B.g.cfz;
    st->ncx = B.g.ncx; st->ncy = B.g.ncy; st->ncz = B.g.ncz; st->ncell = B.g.ncell;
    st->nox = B.g.nox; st->noy = B.g.noy; st->noz = B.g.noz;
  }
  __syncthreads();
  {
    const int* src = (const int*)&B.q;
    int* dst = (int*)&st->s;
    for (int k = tid; k < (int)(sizeof(clmd_scalars) / 4); k += NT) dst[k] = src[k];
  }
}

// compiled twice, like clmd_cycle.cu: FP64 kernels with the host side, and
// the mixed-precision kernels alone
typedef void (*SmallKernel)(Params, DevState*, CycleArgs, int, int, int, int, int);

#ifdef CLMD_CYCLE_MIXED
SmallKernel small_kernel_mixed(bool nh, bool th) {
  if (nh) return th ? k_small<true, true, true> : k_small<true, false, true>;
  return th ? k_small<false, true, true> : k_small<false, false, true>;
}
#else
SmallKernel small_kernel_mixed(bool nh, bool th);

static SmallKernel small_kernel(const clmd_system* S) {
  const bool nh = S->P.integrator == CLMD_INT_NOSE, th = S->P.ethst == 'X';
  if (S->P.precision == CLMD_PREC_MIXED) return small_kernel_mixed(nh, th);
  if (nh) return th ? k_small<true, true, false> : k_small<true, false, false>;
  return th ? k_small<false, true, false> : k_small<false, false, false>;
}

static void small_config(const clmd_system* S, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
  cfg.gridDim = dim3(S->small_ctas);
  cfg.blockDim = dim3(S->small_threads);
  cfg.dynamicSmemBytes = sizeof(SmallShared);
  cfg.stream = S->stream;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S->small_ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

// Whether the system runs on one cluster, and its shape.  The shortest step
// has the fewest pair terms per warp: 8 or 16 atoms in a warp's first lanes
// while 16 CTAs of 16 warps hold the system at that, else 32.  (Mixed
// precision sums a row's terms by chunks of the warp's entries: always 32, the
// grid kernel's grouping.)  4 warps a CTA until that takes 16 CTAs, then more.
void small_setup(clmd_system* S) {
  S->small_ctas = 0;
  const int N = S->P.N;
  if (N > kSC * kSmallThreads) return;
  int per = 32;
  if (S->P.precision != CLMD_PREC_MIXED)
    while (per > 8 && (N + per / 2 - 1) / (per / 2) <= kSC * kSW) per /= 2;
  const int warps = (N + per - 1) / per;
  int c = (warps + 3) / 4, nt = 128;
  if (c > kSC) {
    c = kSC;
    nt = (warps + c - 1) / c * 32;
  }
  S->small_per = per;
  SmallKernel k = small_kernel(S);
  S->small_ctas = c;
  S->small_threads = nt;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  small_config(S, cfg, at);
  int n = 0;
  if ((c > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                    cudaSuccess) ||
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(SmallShared)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, (void*)k, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    S->small_ctas = 0;  // no such cluster here: the grid kernel
  }
}

void small_launch(clmd_system* S, const CycleArgs& A, int nsteps, int mode, const int* step) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  small_config(S, cfg, at);
  cudaLaunchKernelEx(&cfg, small_kernel(S), S->P, S->st, A, nsteps, mode, step ? *step : 0,
                     step != nullptr, S->small_per);
  S->launches++;
}
#endif  // CLMD_CYCLE_MIXED

}  // namespace clmd
