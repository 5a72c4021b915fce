// clmd_cycle.cuh -- what the persistent step kernels share (clmd_cycle.cu: any
// size, the whole GPU, grid barriers; clmd_small.cu: small systems, one
// thread-block cluster): the replicated scalar logic (skin, rebuild
// decision), the list search of one atom, and the warp-cooperative pair
// forces.
#pragma once

#include "clmd_mixed.cuh"
#include "clmd_system.hpp"

namespace clmd {

constexpr int kSmallThreads = 512; // threads per CTA of the small-system kernel at most
struct Geo {
  double rs2, cfx, cfy, cfz;
  int ncx, ncy, ncz, ncell;
  int nox, noy, noz, pad;  // cells searched per dimension: 1, 2 or 3
  // the FP32 list test: r^2 below flo is a neighbour, above fhi is none; in
  // between the FP64 test decides
  float flo, fhi;
  int sel;  // a dimension has fewer than three cells: images per pair
};

struct Blk {
  clmd_scalars q;
  Geo g;
  double kf[CLMD_MXSORTS];
  double bcast[4];
  int scale[CLMD_MXSORTS];
  int rebuild;
  int stop;
};

// ---------------------------------------------------------------------------
// scalar logic (thread 0 of each block on its replica)
// ---------------------------------------------------------------------------

// neighbor-pbc-mav.f:48-60, 101-105 and the cell grid
static __device__ void prologue(const Params& P, Blk& B, int step) {
  clmd_scalars& q = B.q;
  if (q.dmms > (q.atrskin - P.atrcut)) {  // :48-51
    if (q.status == 0) {
      q.status = CLMD_ERR_SKIN;
      q.fail_step = step;
    }
    B.stop = 1;
    B.rebuild = 0;
    return;
  }
  q.dmmav = (double)(float)q.dmmst * q.dmmsu / 256.0;  // :53
  if (step != P.btim && step > 0) {                      // :55-60
    q.atrskin = P.atrcut + (q.atrskin - P.atrcut) * (double)P.nbtim / (double)q.dmmst;
    q.atrskin = fmin(P.boxx / 2.0, q.atrskin);
    q.atrskin = fmin(P.boxy / 2.0, q.atrskin);
    q.atrskin = fmin(P.boxz / 2.0, q.atrskin);
  }
  Geo& g = B.g;
  g.rs2 = q.atrskin * q.atrskin;
  double side = q.atrskin * (1.0 + 1e-9);
  int n3[3] = {(int)floor(P.boxx / side), (int)floor(P.boxy / side), (int)floor(P.boxz / side)};
  int mx[3] = {P.ncx_max, P.ncy_max, P.ncz_max};
  int* nos[3] = {&g.nox, &g.noy, &g.noz};
  for (int d = 0; d < 3; d++) {
    n3[d] = max(1, min(n3[d], mx[d]));
    *nos[d] = min(n3[d], 3);
  }
  g.ncx = n3[0];
  g.ncy = n3[1];
  g.ncz = n3[2];
  g.ncell = n3[0] * n3[1] * n3[2];
  g.cfx = (double)g.ncx / P.boxx;
  g.cfy = (double)g.ncy / P.boxy;
  g.cfz = (double)g.ncz / P.boxz;
  g.sel = g.ncx < 3 || g.ncy < 3 || g.ncz < 3;
  {
    // FP32 coordinates in [0, L] and shifted by L are off by at most
    // e = 4 L 2^-24 together; r^2 by 2 e (|dx| + |dy| + |dz|) + 3 e^2 and its
    // own few roundings
    const double e = fmax(fmax(P.boxx, P.boxy), P.boxz) * 2.4e-7;
    const double band = 4.0 * e * q.atrskin + 3.0 * e * e + 1e-6 * g.rs2;
    g.flo = (float)(g.rs2 - band);
    g.fhi = (float)(g.rs2 + band);
  }
  q.dmmax = fmax(q.dmms, q.dmmax);  // :101-105
  q.dmms = 0.0;
  q.dmmst = 0;
  q.nrebuild = q.nrebuild + 1;
  q.last_rebuild_step = step;
}

// int-verlet-mav.f:64-74 / int-verlet-nh-mav.f:70-78
static __device__ void skin(const Params& P, Blk& B, double dmmr, int step) {
  clmd_scalars& q = B.q;
  dmmr = 2.2 * sqrt(dmmr);
  q.dmms = q.dmms + dmmr;
  q.dmmsu = q.dmmsu + dmmr - q.dmmh[q.dmmi];
  q.dmmh[q.dmmi] = dmmr;
  q.dmmi = (q.dmmi + 1) & 255;
  q.dmmst = q.dmmst + 1;
  B.rebuild = q.dmms > (q.atrskin - P.atrcut - 2.0 * q.dmms / (double)(float)q.dmmst);
  if (B.rebuild) prologue(P, B, step);
}

// ---------------------------------------------------------------------------
// the list rebuild (neighbor-pbc-mav.f:67-99) as barrier-separated phases
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool nbt(const Params& P, double rs2, const double4& a,
                                    const double4& b) {
  double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
  dx = mimage_nb(dx, P.boxx, P.ibx);
  dy = mimage_nb(dy, P.boxy, P.iby);
  dz = mimage_nb(dz, P.boxz, P.ibz);
  double r2 = dx * dx + dy * dy + dz * dz;
  return r2 <= rs2;
}

// One row of m <= 32 T entries (slots, in any order), by the whole warp: T
// entries per lane in registers, and every entry's place is the count of
// smaller reference indices (distinct, so the places are a permutation).
// Returns the number of entries below `ref`.
template <int T>
__device__ __forceinline__ int sort_row(int* row, const int* perm, int m, int ref) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int q[T], key[T], rank[T], below = 0;
#pragma unroll
  for (int t = 0; t < T; t++) {
    const int k = lane + 32 * t;
    q[t] = k < m ? row[k] : 0;
    key[t] = k < m ? perm[q[t]] : 0x7fffffff;
    rank[t] = 0;
  }
#pragma unroll
  for (int t = 0; t < T; t++)
    below += __popc(__ballot_sync(FULL, lane + 32 * t < m && key[t] < ref));
#pragma unroll
  for (int u = 0; u < T; u++) {
    if (32 * u >= m) break;
#pragma unroll 8
    for (int l = 0; l < 32; l++) {
      const int other = __shfl_sync(FULL, key[u], l);
#pragma unroll
      for (int t = 0; t < T; t++) rank[t] += other < key[t];
    }
  }
  __syncwarp();  // every lane has read the row
#pragma unroll
  for (int t = 0; t < T; t++)
    if (lane + 32 * t < m) row[rank[t]] = q[t];
  __syncwarp();
  return below;
}

// Rows longer than the search's buffer, one after the other by the whole
// warp: lanes with n > 0 name a row of n entries that starts at list[start];
// each is put in ascending reference order, *lo gets the number of entries
// below the owner's reference index.  A row of more than 256 entries is left
// to its lane's insertion sort (in memory: ~130 us for a droplet's row of 130).
static __device__ __noinline__ void sort_long_rows(int* list, const int* perm,
                                                   unsigned long long start, int n, int refi,
                                                   int& lo) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned todo = __ballot_sync(FULL, n > 0);
  __syncwarp();  // the owners' entries are visible to every lane
  while (todo) {
    const int ow = __ffs(todo) - 1;
    todo &= todo - 1;
    const int m = __shfl_sync(FULL, n, ow), ref = __shfl_sync(FULL, refi, ow);
    int* row = list + __shfl_sync(FULL, start, ow);
    int below = 0;
    if (m <= 64) {
      below = sort_row<2>(row, perm, m, ref);
    } else if (m <= 128) {
      below = sort_row<4>(row, perm, m, ref);
    } else if (m <= 256) {
      below = sort_row<8>(row, perm, m, ref);
    } else {
      if (lane == ow) {
        for (int a = 1; a < m; a++) {
          int kq = row[a], kr = perm[kq];
          int b = a - 1;
          while (b >= 0 && perm[row[b]] > kr) {
            row[b + 1] = row[b];
            b--;
          }
          row[b + 1] = kq;
        }
        for (int a = 0; a < m; a++) below += perm[row[a]] < refi;
      }
      __syncwarp();
    }
    if (lane == ow) lo = below;
  }
}

struct CycleArgs {
  double4* pos0;
  double4* pos1;
  double *vx, *vy, *vz, *ax, *ay, *az;
  // mixed Nose-Hoover: the accelerations between a step's force pass and its
  // velocity pass
  float *afx, *afy, *afz;
  int *perm, *iperm;
  double4* pos_s;
  double *vx_s, *vy_s, *vz_s, *ax_s, *ay_s, *az_s;
  int* perm_s;
  float4* posf;  // positions in FP32, reference index in .w, in cell order
  int *cell_count, *cell_start, *cell_fill, *cell_atoms, *atom_cell, *scan_aux;
  int *list, *row_start, *row_len, *row_lo;
  double* red;  // 2 x kRedSlots x gridDim partials
};

// neighbor-pbc-mav.f:67-71, dmod(dmod(x, L) + L, L).  Within one box length
// of the box both dmods are a subtraction or nothing, exact either way (of
// neighbouring binades at most), so the result is the same bits without the
// two library calls
__device__ __forceinline__ double wrap_1(double x, double L) {
  if (x > -L && x < L + L) {
    const double u = (x >= L ? x - L : x) + L;
    return u >= L + L ? u - (L + L) : u >= L ? u - L : u;
  }
  return fmod(fmod(x, L) + L, L);
}
__device__ __forceinline__ double4 wrap_box(const Params& P, double4 v) {
  v.x = wrap_1(v.x, P.boxx);
  v.y = wrap_1(v.y, P.boxy);
  v.z = wrap_1(v.z, P.boxz);
  return v;
}

// for-a-lj-n-pbc-m.f:92-142 for one atom: fsum in the reference's order
// (accumulated by warp_forces below)
struct Pair {
  double fx, fy, fz, esum, vir;
};

// Pair forces, warp-cooperative, for the 32 consecutive slots of a warp, whose
// rows are contiguous in the list (the search allocates them with one
// warp-wide cursor step).  Lanes evaluate the pair terms of 32 consecutive
// list entries at a time (balanced work whatever the row lengths), stage them
// in shared memory, and each owner lane then adds its own terms in list
// order, i.e. in the reference's order, with the same +/- as the serial code.
// FP64: the terms of kGroup chunks are staged before the owner lanes add
// theirs, so that more owners work at once (a row's terms still go in
// list order)
#ifndef CLMD_FORCE_GROUP
#define CLMD_FORCE_GROUP 4
#endif
constexpr int kGroup = CLMD_FORCE_GROUP;
// (the term an owner adds: negated where the reference subtracts it, zero
// beyond the cut-off; adding a zero leaves a sum as it is)
struct WarpStage {
  double tx[32 * kGroup], ty[32 * kGroup], tz[32 * kGroup];
  int more[32 * kGroup];  // (the search's buffer is a little larger)
};

template <bool MIXED>
__device__ __forceinline__ void warp_forces(const Params& P, DevState* st, const double4* pos,
                                            const int* list, int st0, int len, int lo,
                                            const double4& pa, double bf1, double bf2,
                                            double& fx, double& fy, double& fz, double& esum,
                                            double& vir, bool energies, WarpStage& W,
                                            bool& bad) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int e = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(FULL, e, o);
    if (lane >= o) e += t;
  }
  const int tot = __shfl_sync(FULL, e, 31);
  e -= len;  // exclusive prefix: this lane's row starts at wbase + e
  const int wbase = __shfl_sync(FULL, st0, 0);
  const int sa = (int)pa.w;
  constexpr bool mixed = MIXED;
  float sx = 0.f, sy = 0.f, sz = 0.f, kx = 0.f, ky = 0.f, kz = 0.f;  // mixed: Kahan sums
  fx = 0.0;
  fy = 0.0;
  fz = 0.0;
  // this chunk's entry and neighbour position are fetched first, and the
  // next chunk's entry with them, so that the loads overlap the owner search
  int jnext = lane < tot ? list[wbase + lane] : 0;
  for (int c = 0; c < tot; c += 32) {
    const int k = c + lane;
    const int kk = k < tot ? k : tot - 1;
    const int jc = jnext;
    double4 pb = make_double4(0.0, 0.0, 0.0, 0.0);
    if (k < tot) pb = pos[jc];
    if (k + 32 < tot) jnext = list[wbase + k + 32];
    int ow = 0;
#pragma unroll
    for (int sft = 16; sft >= 1; sft >>= 1) {
      int cand = ow + sft;
      int ec = __shfl_sync(FULL, e, cand & 31);
      if (cand <= 31 && ec <= kk) ow = cand;
    }
    const double ox = __shfl_sync(FULL, pa.x, ow);
    const double oy = __shfl_sync(FULL, pa.y, ow);
    const double oz = __shfl_sync(FULL, pa.z, ow);
    const int osp = __shfl_sync(FULL, sa, ow);
    const int oe = __shfl_sync(FULL, e, ow);
    const int olo = __shfl_sync(FULL, lo, ow);
    int flag = 0;
    double tx = 0.0, ty = 0.0, tz = 0.0;
    if (k < tot) {
      bool own = (k - oe) >= olo;  // neighbour has the larger reference index
      double dx, dy, dz;
      if (own) {
        dx = ox - pb.x; dy = oy - pb.y; dz = oz - pb.z;
      } else {
        dx = pb.x - ox; dy = pb.y - oy; dz = pb.z - oz;
      }
      mimage_bf3(P, dx, dy, dz, bf1, bf2);
      double rij2 = dx * dx + dy * dy + dz * dz;
      if (rij2 <= P.atr2) {
        double r2 = rij2;
        double rij6 = 0.0;
        if (!mixed) {
          rij2 = 1.0 / rij2;
          rij6 = rij2 * rij2 * rij2;
        }
        int ij = osp + (int)pb.w;
        if (ij < 2 || ij > 4) {
          raise_err(st, CLMD_ERR_BAD_SPECIES);
          bad = true;
        } else if (mixed) {
          double e, w;
          pair_term_f32(P, ij, r2, dx, dy, dz, tx, ty, tz, e, w);
          if (own && energies) {
            esum = esum + e;
            vir = vir + w;
          }
          flag = own ? 1 : 2;
        } else {
          double fij = pair_fij(P, ij, rij2, rij6);
          tx = fij * dx;
          ty = fij * dy;
          tz = fij * dz;
          if (own && energies) {
            esum = esum + pair_e(P, ij, rij6);
            vir = vir + fij * r2;
          }
          flag = own ? 1 : 2;
        }
      }
    }
    const int a0 = e > c ? e : c;
    const int a1 = (e + len) < (c + 32) ? (e + len) : (c + 32);
    if (mixed) {
      // each row's terms in this chunk summed by a segmented scan across the
      // lanes (a fixed tree: deterministic), then added to the owner's
      // Kahan sums chunk by chunk: every lane works, where the ordered
      // FP64 sum below has only the owners working
      const float sg = flag == 1 ? 1.0f : (flag == 2 ? -1.0f : 0.0f);
      float v0 = sg * (float)tx, v1 = sg * (float)ty, v2 = sg * (float)tz;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int ou = __shfl_up_sync(FULL, ow, off);
        const float u0 = __shfl_up_sync(FULL, v0, off);
        const float u1 = __shfl_up_sync(FULL, v1, off);
        const float u2 = __shfl_up_sync(FULL, v2, off);
        if (lane >= off && ou == ow) {
          v0 = __fadd_rn(v0, u0);
          v1 = __fadd_rn(v1, u1);
          v2 = __fadd_rn(v2, u2);
        }
      }
      const int last = a1 > a0 ? a1 - 1 - c : 0;  // my row's last entry in the chunk
      const float p0 = __shfl_sync(FULL, v0, last);
      const float p1 = __shfl_sync(FULL, v1, last);
      const float p2 = __shfl_sync(FULL, v2, last);
      if (a1 > a0) {
        kahan_add(sx, kx, p0);
        kahan_add(sy, ky, p1);
        kahan_add(sz, kz, p2);
      }
      continue;
    }
    const int g = (c >> 5) % kGroup;
    W.tx[32 * g + lane] = flag == 2 ? -tx : tx;
    W.ty[32 * g + lane] = flag == 2 ? -ty : ty;
    W.tz[32 * g + lane] = flag == 2 ? -tz : tz;
    if (g != kGroup - 1 && c + 32 < tot) continue;  // the group is not full yet
    __syncwarp();
    const int cg = c - 32 * g;  // the group's first entry
    const int b0 = e > cg ? e : cg;
    const int b1 = (e + len) < (c + 32) ? (e + len) : (c + 32);
#pragma unroll 2
    for (int q = b0 - cg; q < b1 - cg; q++) {
      fx = fx + W.tx[q];
      fy = fy + W.ty[q];
      fz = fz + W.tz[q];
    }
    __syncwarp();
  }
  if (mixed) {
    fx = (double)sx;
    fy = (double)sy;
    fz = (double)sz;
  }
}

__device__ __forceinline__ int sp_block(const Params& P, int ref) {
  for (int s = 0; s < P.atsorts; s++)
    if (ref >= P.sp_start[s] && ref < P.sp_start[s + 1]) return s;
  return -1;
}

// the search's hits of one thread, until its row is written: in the
// pair-force stage's memory, not in use then (entry k of lane l at
// [32 k + l]; arrays of a thread's own would live in local memory)
constexpr int kRowCap = (int)(sizeof(WarpStage) / 32 / 8);

// neighbor-pbc-mav.f:73-99: the neighbours of one atom (slot p, wrapped
// position pa) among the cells around it, into buf (the first kRowCap) or all
// of them into out; returns their number.  cf: the atoms' positions in FP32
// with the reference index in .w, in cell order.
// The test is FP32 (with three or more cells per dimension the image is the
// cell range's shift) and FP64, the reference's expression, only within the
// FP32 rounding of the list radius: the same list, a quarter of the FP64
// instructions, and 16 bytes a candidate instead of 36.  Two candidates are
// loaded at a time and the next cell row's range ahead of this one's tests:
// a thread's chain of loads, not their number, bounds the search.  With the
// rank sort of long rows neighbor() took 553 -> 380 us (N = 1,000,003) and
// 440 -> 150 us (30,011 atoms, 30 liquid droplets).
__device__ __forceinline__ int row_search(const Params& P, const Geo& g, int p, int ref,
                                          const double4& pa, const double4* pos,
                                          const float4* cf, const int* cs, int2* buf, int* out) {
  const int ncx = g.ncx, ncy = g.ncy, ncz = g.ncz, noy = g.noy, noz = g.noz;
  const int cx = clmd_cell(pa.x, g.cfx, ncx);
  const int cy = clmd_cell(pa.y, g.cfy, ncy);
  const int cz = clmd_cell(pa.z, g.cfz, ncz);
  const float lx = (float)P.boxx, ly = (float)P.boxy, lz = (float)P.boxz;
  const float px = (float)pa.x, py = (float)pa.y, pz = (float)pa.z;
  const float flo = g.flo, fhi = g.fhi;
  const bool sel = g.sel != 0;
  // the cells of a row: [xa, xb), and the one the row wraps to (edge), at a
  // box length's shift
  const int xa = ncx < 3 ? 0 : max(cx - 1, 0), xb = ncx < 3 ? ncx : min(cx + 2, ncx);
  const bool edge = ncx >= 3 && (cx == 0 || cx == ncx - 1);
  const int xw = cx == 0 ? ncx - 1 : 0;
  const float wx = sel ? 0.f : (cx == 0 ? lx : -lx);
  int n = 0, ka = 0, kb = 0;
  float ny, nz;  // the next row's image shifts
  int a0, b0, a1 = 0, b1 = 0;
  auto next = [&]() {  // cell ranges and shifts of row (ka, kb), then on to the next
    int zz = cz + ka - (noz == 3), yy = cy + kb - (noy == 3);
    nz = sel ? 0.f : (zz < 0 ? lz : (zz >= ncz ? -lz : 0.f));
    ny = sel ? 0.f : (yy < 0 ? ly : (yy >= ncy ? -ly : 0.f));
    zz += zz < 0 ? ncz : (zz >= ncz ? -ncz : 0);
    yy += yy < 0 ? ncy : (yy >= ncy ? -ncy : 0);
    const int* row = cs + (zz * ncy + yy) * ncx;
    a0 = row[xa];
    b0 = row[xb];
    if (edge) {
      a1 = row[xw];
      b1 = row[xw + 1];
    }
    if (++kb == noy) {
      kb = 0;
      ka++;
    }
  };
  auto test = [&](const float4& c, int q, float x, float y, float z) {
    float dx = x - c.x, dy = y - c.y, dz = z - c.z;
    if (sel) {
      dx -= fabsf(dx) > 0.5f * lx ? copysignf(lx, dx) : 0.f;
      dy -= fabsf(dy) > 0.5f * ly ? copysignf(ly, dy) : 0.f;
      dz -= fabsf(dz) > 0.5f * lz ? copysignf(lz, dz) : 0.f;
    }
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (!(r2 <= fhi) || q == p) return;  // (a NaN is no neighbour)
    const int refq = __float_as_int(c.w);
    if (!(r2 < flo)) {
      const double4 pq = pos[q];
      if (!((ref < refq) ? nbt(P, g.rs2, pa, pq) : nbt(P, g.rs2, pq, pa))) return;
    }
    if (out)
      out[n] = q;
    else if (n < kRowCap)
      buf[n * 32] = make_int2(q, refq);
    n++;
  };
  next();
  for (bool more = true; more;) {
    int q = a0, e = b0;
    const int q1 = a1, e1 = edge ? b1 : a1;
    const float y = py + ny, z = pz + nz;
    float x = px;
    more = ka < noz;
    if (more) next();
    for (int part = 0;; part++) {
#pragma unroll 1
      for (; q < e; q += 2) {
        const float4 c0 = cf[q], c1 = cf[min(q + 1, e - 1)];
        test(c0, q, x, y, z);
        if (q + 1 < e) test(c1, q + 1, x, y, z);
      }
      if (part || !edge) break;
      q = q1;
      e = e1;
      x = px + wx;
    }
  }
  return n;
}

// a row's hits in the buffer (n <= kRowCap) put in ascending reference order
// and written out; returns how many lie below the owner's reference index
__device__ __forceinline__ int row_store(int2* buf, int n, int ref, int* row) {
  for (int k = 1; k < n; k++) {
    const int2 e = buf[k * 32];
    int b = k - 1;
    while (b >= 0 && buf[b * 32].y > e.y) {
      buf[(b + 1) * 32] = buf[b * 32];
      b--;
    }
    buf[(b + 1) * 32] = e;
  }
  int lo = 0;
  for (int k = 0; k < n; k++) {
    const int2 e = buf[k * 32];
    row[k] = e.x;
    lo += e.y < ref;
  }
  return lo;
}

// clmd_small.cu: systems of up to 16 * kSmallThreads atoms
void small_setup(clmd_system* S);
void small_launch(clmd_system* S, const CycleArgs& A, int nsteps, int mode, const int* step);

}  // namespace clmd
