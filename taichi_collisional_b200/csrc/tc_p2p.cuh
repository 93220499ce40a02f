// Near field: P2P over the (target cell, source cell) list, target-stationary.
// Restates P2P_simple (kernel_fast_lean.h:268-459; a = sum m d / r^3, p = sum m / r, r = 0
// skipped, no softening) and the jerk P2P (taichi_with_jerks/kernel_fast_lean.h:499-699;
// J = sum m [dv / r^3 - 3 (d.dv) d / r^5]).
//
// A warp per work item, a target per lane.  A row of r <= 16 targets uses floor(32 / r) groups of r
// lanes, each group taking every ng-th source body, so small leaves still fill the warp; the groups are
// combined with a fixed shuffle tree (deterministic sums).
#pragma once
#include "tc_down.cuh"

namespace tc {

template <bool JERK>
struct TcAcc {
  double pot, ax, ay, az, jx, jy, jz;
  __device__ __forceinline__ void zero() { pot = ax = ay = az = jx = jy = jz = 0.0; }
  __device__ __forceinline__ void add_xor(int o) {
    pot += __shfl_xor_sync(0xffffffffu, pot, o);
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
    az += __shfl_xor_sync(0xffffffffu, az, o);
    if (JERK) {
      jx += __shfl_xor_sync(0xffffffffu, jx, o);
      jy += __shfl_xor_sync(0xffffffffu, jy, o);
      jz += __shfl_xor_sync(0xffffffffu, jz, o);
    }
  }
  // sum of the ng lane groups (group g = lanes [g gsz, (g + 1) gsz)) into group 0 by a fixed
  // tree: at step s, group g (a multiple of 2 s) adds group g + s
  __device__ __forceinline__ void add_groups(int gsz, int ng, int grp) {
    for (int st = 1; st < ng; st <<= 1) {
      const int off = st * gsz;
      const bool take = (grp % (2 * st)) == 0 && grp + st < ng;
      double v;
      v = __shfl_down_sync(0xffffffffu, pot, off); if (take) pot += v;
      v = __shfl_down_sync(0xffffffffu, ax, off); if (take) ax += v;
      v = __shfl_down_sync(0xffffffffu, ay, off); if (take) ay += v;
      v = __shfl_down_sync(0xffffffffu, az, off); if (take) az += v;
      if (JERK) {
        v = __shfl_down_sync(0xffffffffu, jx, off); if (take) jx += v;
        v = __shfl_down_sync(0xffffffffu, jy, off); if (take) jy += v;
        v = __shfl_down_sync(0xffffffffu, jz, off); if (take) jz += v;
      }
    }
  }
};

template <bool JERK>
__device__ __forceinline__ void tc_p2p_one(double xi, double yi, double zi, double vxi, double vyi, double vzi,
                                           const TcBodies& b, int j, TcAcc<JERK>& a) {
  if (!(b.flags[j] & 2)) return;
  double dx = b.x[j] - xi, dy = b.y[j] - yi, dz = b.z[j] - zi;
  double r2 = dx * dx + dy * dy + dz * dz;
  if (!(r2 > 0.0)) return;
  double invr = rsqrt(r2 + b.eps2), invr2 = invr * invr;
  double f = b.m[j] * invr;
  a.pot += f;
  f *= invr2;
  a.ax += dx * f;
  a.ay += dy * f;
  a.az += dz * f;
  if (JERK) {
    double dvx = b.vx[j] - vxi, dvy = b.vy[j] - vyi, dvz = b.vz[j] - vzi;
    double vr = 3.0 * (dx * dvx + dy * dvy + dz * dvz);
    a.jx += dvx * f;
    a.jy += dvy * f;
    a.jz += dvz * f;
    f *= -invr2 * vr;
    a.jx += dx * f;
    a.jy += dy * f;
    a.jz += dz * f;
  }
}

constexpr int kP2PWarps = 4;

// ---------------------------------------------------------------------------------------
// Work items of the near field.
//
// A row is up to 32 consecutive bodies of one target leaf; its work is the bodies of the leaf's
// source cells.  That work varies by orders of magnitude: a few wide leaves of the outer halo
// have nearly the whole system in their list, and a warp that walks such a list alone holds the
// launch for tens of milliseconds (N = 131,072, p = 12: 56 ms for 0.85e9 pairs, whose FP64
// arithmetic takes 2 ms).  So a row whose cost exceeds C is split into chunks of about C:
// C = total cost / K, K a few times the warps the GPU holds, but at least kP2PMinCost, so that
// small systems fill the GPU as well (this replaces a fixed number of chunks per leaf chosen by
// n).  Chunk boundaries are multiples of 32 bodies of the row's source sequence: the tiles of a
// split row hold the same bodies as those of an unsplit one.  Chunks store their sums in a slot
// each, folded in chunk order by k_p2p_join, so the sums depend on the lists alone and not on the
// order in which warps take items.
//
// Split items are handed out before the unsplit rows, so the long ones start first.
// ---------------------------------------------------------------------------------------
struct __align__(8) TcP2PItem {
  int t, t0;   // target leaf, first body of the row in it
  int q, off;  // first source cell (index into the list) and first body in it
  int cnt;     // source bodies of the chunk
  int pad;
};
struct TcP2PRow {
  int t, t0, base, nch;  // a split row: its first slot and its number of chunks
};
struct TcP2PWork {
  const TcP2PItem* items;  // split rows' chunks; item k owns slot k
  const int2* singles;     // unsplit rows (t, t0)
  const unsigned* cnt;     // [0] items, [1] singles, [2] split rows
  unsigned* next;          // work counter, zero before the launch
  double* slots;           // [item][component][32]
  bool shared;             // a body may be in several target cells (see tc_p2p_add)
};
constexpr int kP2PMinCost = 64;

// source bodies a warp steps through for a row of r targets (floor(32 / r) lane groups share them)
__device__ __forceinline__ int tc_p2p_cost(int S, int r) {
  const int ng = r > 16 ? 1 : 32 / r;
  return (S + ng - 1) / ng;
}

// S[k] = source bodies of target k (0 when it has no sink); the total cost and pair count.  A warp per
// target, four list entries a lane in flight (an outlier's list holds thousands of cells).
__global__ void __launch_bounds__(256) k_p2p_work(const int* __restrict__ tlist, int ntl,
                                                  const int* __restrict__ tstart, const int* __restrict__ src,
                                                  const TcCells c, int* __restrict__ S, unsigned long long* inter,
                                                  unsigned long long* cost, const unsigned* ntldev = nullptr) {
  if (ntldev) ntl = (int)*ntldev;  // device-sized launch (graph)
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (blockDim.x >> 5);
  unsigned long long wi = 0, wc = 0;
  for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < ntl; k += nw) {
    const int t = tlist[k];
    unsigned s = 0;
    if (c.has_sink[t]) {
      const int sb = tstart[t], se = tstart[t + 1];
      for (int q = sb + lane; q < se; q += 128) {
        int id[4];
#pragma unroll
        for (int u = 0; u < 4; u++) id[u] = q + 32 * u < se ? src[q + 32 * u] : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) s += id[u] >= 0 ? (unsigned)c.nbody[id[u]] : 0u;
      }
      s = __reduce_add_sync(0xffffffffu, s);
    }
    if (lane == 0) {
      S[k] = (int)s;
      const int nt = c.nbody[t];
      wi += (unsigned long long)nt * s;
      wc += (unsigned long long)(nt >> 5) * s;
      if (nt & 31) wc += (unsigned long long)tc_p2p_cost((int)s, nt & 31);
    }
  }
  if (lane == 0 && wi) {
    atomicAdd(inter, wi);
    atomicAdd(cost, wc);
  }
}

// rows -> singles and chunk items, a warp per target
__global__ void __launch_bounds__(256) k_p2p_plan(const int* __restrict__ tlist, int ntl,
                                                  const int* __restrict__ tstart, const int* __restrict__ src,
                                                  const TcCells c, const int* __restrict__ S,
                                                  const unsigned long long* cost, int K, int cap,
                                                  int2* __restrict__ singles, TcP2PItem* __restrict__ items,
                                                  TcP2PRow* __restrict__ rows, unsigned* __restrict__ cnt,
                                                  const unsigned* ntldev = nullptr) {
  if (ntldev) ntl = (int)*ntldev;  // device-sized launch (graph)
  const int lane = threadIdx.x & 31;
  const unsigned long long C64 = (*cost + K - 1) / K;
  const int C = (int)(C64 < kP2PMinCost ? kP2PMinCost : C64 > 0x7fffffffull ? 0x7fffffff : C64);
  const int nw = gridDim.x * (blockDim.x >> 5);
  for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < ntl; k += nw) {
    const int s = S[k];
    if (s == 0) continue;
    const int t = tlist[k], nt = c.nbody[t], nrow = (nt + 31) >> 5;
    const int sb = tstart[t], se = tstart[t + 1];
    // the rows of the target, 32 at a time (one per lane): unsplit rows first
    for (int r0 = 0; r0 < nrow; r0 += 32) {
      const int t0 = 32 * (r0 + lane);
      const bool row = t0 < nt, split = row && tc_p2p_cost(s, min(32, nt - t0)) > C;
      const unsigned one = __ballot_sync(0xffffffffu, row && !split);
      unsigned m = __ballot_sync(0xffffffffu, split);
      if (one) {
        int base = 0;
        if (lane == 0) base = (int)atomicAdd(&cnt[1], (unsigned)__popc(one));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (row && !split) singles[base + __popc(one & ((1u << lane) - 1u))] = make_int2(t, t0);
      }
      for (; m; m &= m - 1) {
        const int ts = 32 * (r0 + __ffs(m) - 1);
        const int want = (int)(((unsigned)tc_p2p_cost(s, min(32, nt - ts)) + (unsigned)C - 1u) / (unsigned)C);
        const int B = ((s + want - 1) / want + 31) & ~31;
        const int nch = (s + B - 1) / B;
        int ib = 0;
        if (lane == 0) ib = (int)atomicAdd(&cnt[0], (unsigned)nch);
        ib = __shfl_sync(0xffffffffu, ib, 0);
        if (ib + nch > cap) continue;  // cannot happen: a split row costs more than C, so it has less than 2 cost / C
                                       // items, and C is at least cost / K (or as large as any row's cost)
        if (lane == 0) rows[atomicAdd(&cnt[2], 1u)] = TcP2PRow{t, ts, ib, nch};
        int p = 0;  // bodies before the window of 128 cells, four consecutive ones a lane
        for (int q0 = sb; q0 < se; q0 += 128) {
          int nb[4], sum = 0;
#pragma unroll
          for (int u = 0; u < 4; u++) nb[u] = q0 + 4 * lane + u < se ? src[q0 + 4 * lane + u] : -1;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            nb[u] = nb[u] >= 0 ? c.nbody[nb[u]] : 0;
            sum += nb[u];
          }
          int pi = sum;
          for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pi, d);
            if (lane >= d) pi += v;
          }
          int pb = p + pi - sum;  // bodies before this lane's cell
#pragma unroll
          for (int u = 0; u < 4; u++) {
            for (int h = (pb + B - 1) / B; nb[u] > 0 && h < nch && h * B < pb + nb[u]; h++)
              items[ib + h] = TcP2PItem{t, ts, q0 + 4 * lane + u, h * B - pb, min(B, s - h * B), 0};
            pb += nb[u];
          }
          p += __shfl_sync(0xffffffffu, pi, 31);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// FP64 near field of small systems (below kP2PSmallN bodies): every leaf's source list is cut into
// kP2PChunks pieces of as many cells, without a plan.  The block-time-step integrator's compensation terms
// are rounding residues of these sums, so the order of its small kicks' sums is part of what it reproduces,
// and this is that order.  Pieces of as many cells are as even as the leaves are: near field with the pieces /
// with work items (ms), top tree N = 1,000 and ncrit 16 0.057 / 0.069, 64 0.111 / 0.071; N = 2,000 0.064 / 0.083 and
// 0.165 / 0.087.
// ---------------------------------------------------------------------------------------
constexpr int kP2PSmallN = 2048, kP2PChunks = 16;

template <bool JERK>
__global__ void __launch_bounds__(kP2PWarps * 32) k_p2p_chunks(const int* __restrict__ tlist, int ntl,
                                                        const int* __restrict__ tstart, const int* __restrict__ src,
                                                        const TcBodies b, const TcCells c, TcOut out,
                                                        const unsigned* ntldev, int nsplit,
                                                        double* __restrict__ part, int pstride,
                                                        unsigned long long* inter) {
  // Work item k: target leaf k / nsplit, chunk k % nsplit of its source-cell list; its partial sums
  // go to part[(chunk * NC + component) * pstride + body] for k_p2p_chunks_join.
  if (ntldev) ntl = (int)*ntldev;  // device-sized launch (graph)
  constexpr int NC = JERK ? 7 : 4;
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long nitem = (long long)ntl * nsplit;
  for (long long k = (long long)blockIdx.x * kP2PWarps + w; k < nitem; k += (long long)gridDim.x * kP2PWarps) {
    const int kk = (int)(k / nsplit), chunk = (int)(k % nsplit);
    int t = tlist[kk];
    if (!c.has_sink[t]) continue;
    int tb = c.begin[t], nt = c.nbody[t];
    const int sb0 = tstart[t], len = tstart[t + 1] - sb0;
    const int sb = sb0 + (int)((long long)len * chunk / nsplit);
    const int se = sb0 + (int)((long long)len * (chunk + 1) / nsplit);
    unsigned ns = 0;  // pair count of the item
    for (int q = sb + lane; q < se; q += 32) ns += (unsigned)c.nbody[src[q]];
    ns = __reduce_add_sync(0xffffffffu, ns);
    if (lane == 0 && ns) atomicAdd(inter, (unsigned long long)nt * ns);
    for (int t0 = 0; t0 < nt; t0 += 32) {
      // up to 32 targets per pass; a last pass of r <= 16 targets runs floor(32 / r) lane
      // groups of r lanes, each over every ng-th source
      const int r = min(32, nt - t0);
      const int gsz = r > 16 ? 32 : r, ng = 32 / gsz;
      const int grp = lane / gsz, ti = lane % gsz;
      int i = tb + t0 + ti;
      bool vi = grp < ng && (t0 + ti) < nt;
      double xi = 0, yi = 0, zi = 0, vxi = 0, vyi = 0, vzi = 0;
      if (vi) {
        xi = b.x[i]; yi = b.y[i]; zi = b.z[i];
        if (JERK) { vxi = b.vx[i]; vyi = b.vy[i]; vzi = b.vz[i]; }
      }
      TcAcc<JERK> a;
      a.zero();
      if (vi) {
        for (int q = sb; q < se; q++) {
          int s = src[q];
          int jb = c.begin[s], je = jb + c.nbody[s];
          for (int j = jb + grp; j < je; j += ng) tc_p2p_one<JERK>(xi, yi, zi, vxi, vyi, vzi, b, j, a);
        }
      }
      a.add_groups(gsz, ng, grp);
      if (vi && grp == 0) {
        double* pp = part + (size_t)chunk * NC * pstride + i;
        pp[0] = a.pot;
        pp[(size_t)pstride] = a.ax;
        pp[2 * (size_t)pstride] = a.ay;
        pp[3 * (size_t)pstride] = a.az;
        if (JERK) {
          pp[4 * (size_t)pstride] = a.jx;
          pp[5 * (size_t)pstride] = a.jy;
          pp[6 * (size_t)pstride] = a.jz;
        }
      }
    }
  }
}

// Folds the nsplit chunk partials of k_p2p_chunks (chunk 0 first) into the sink bodies of each target
// leaf: one warp per leaf, one lane per body.
template <bool JERK>
__global__ void __launch_bounds__(kP2PWarps * 32) k_p2p_chunks_join(const int* __restrict__ tlist, int ntl,
                                                             const TcBodies b, const TcCells c, TcOut out,
                                                             int nsplit, const double* __restrict__ part,
                                                             int pstride, const unsigned* ntldev = nullptr) {
  if (ntldev) ntl = (int)*ntldev;  // device-sized launch (graph)
  constexpr int NC = JERK ? 7 : 4;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = blockIdx.x * kP2PWarps + w; k < ntl; k += gridDim.x * kP2PWarps) {
    const int t = tlist[k];
    if (!c.has_sink[t]) continue;
    const int tb = c.begin[t], nt = c.nbody[t];
    for (int u = lane; u < nt; u += 32) {
      const int i = tb + u;
      if (!(b.flags[i] & 1)) continue;
      double v[NC];
#pragma unroll
      for (int q = 0; q < NC; q++) v[q] = 0.0;
      for (int ch = 0; ch < nsplit; ch++) {
        const double* pp = part + (size_t)ch * NC * pstride + i;
#pragma unroll
        for (int q = 0; q < NC; q++) v[q] += pp[(size_t)q * pstride];
      }
      out.pot[i] += v[0];
      out.ax[i] += v[1];
      out.ay[i] += v[2];
      out.az[i] += v[3];
      if (JERK) {
        out.jx[i] += v[4];
        out.jy[i] += v[5];
        out.jz[i] += v[6];
      }
    }
  }
}

// The next item of a warp: an item of a split row (slot >= 0) or an unsplit row; false at the end
__device__ __forceinline__ bool tc_p2p_take(const TcP2PWork& W, unsigned ni, unsigned ns, const int* tstart, int lane,
                                            TcP2PItem& it, int& slot) {
  unsigned k = 0;
  if (lane == 0) k = atomicAdd(W.next, 1u);
  k = __shfl_sync(0xffffffffu, k, 0);
  if (k >= ni + ns) return false;
  if (k < ni) {
    it = W.items[k];
    slot = (int)k;
  } else {
    const int2 r = W.singles[k - ni];
    it.t = r.x;
    it.t0 = r.y;
    it.q = tstart[r.x];
    it.off = 0;
    it.cnt = 0x7fffffff;
    slot = -1;
  }
  return true;
}

// The top tree sums accepted pairs of at most 2 and 8 bodies directly (traverse_eager.h:160), and with
// ncrit < 8 such a cell can be an inner one: its bodies are then in the rows of several targets, whose
// sums meet in the same output.
__device__ __forceinline__ void tc_p2p_add(bool shared, double* p, double v) {
  if (shared)
    atomicAdd(p, v);
  else
    *p += v;
}

// a row's sums: into its slot, or added to the sinks of an unsplit row
template <bool JERK>
__device__ __forceinline__ void tc_p2p_put(const TcP2PWork& W, int slot, int lane, int i, const TcBodies& b,
                                           const TcOut& out, const TcAcc<JERK>& a) {
  if (slot >= 0) {
    double* pp = W.slots + (size_t)slot * (JERK ? 7 : 4) * 32 + lane;
    pp[0] = a.pot; pp[32] = a.ax; pp[64] = a.ay; pp[96] = a.az;
    if (JERK) { pp[128] = a.jx; pp[160] = a.jy; pp[192] = a.jz; }
  } else if (b.flags[i] & 1) {
    tc_p2p_add(W.shared, &out.pot[i], a.pot);
    tc_p2p_add(W.shared, &out.ax[i], a.ax);
    tc_p2p_add(W.shared, &out.ay[i], a.ay);
    tc_p2p_add(W.shared, &out.az[i], a.az);
    if (JERK) {
      tc_p2p_add(W.shared, &out.jx[i], a.jx);
      tc_p2p_add(W.shared, &out.jy[i], a.jy);
      tc_p2p_add(W.shared, &out.jz[i], a.jz);
    }
  }
}

// The next tile of a target's sources, taken as one sequence of bodies (its source cells'
// bodies one after the other), so a tile holds 32 sources even where the source leaves are
// small.  (q, off) is the warp-uniform cursor: the next source cell and the next body in it.
// The first body and body count of cells q0 + l are held by lane l (cjb, cjn), reloaded 32 cells
// at a time.  Returns the tile's count; lane l gets the body index of slot l (-1 past the count).
__device__ __forceinline__ void tc_src_cells(const int* __restrict__ src, const TcCells& c, int q0, int se, int lane,
                                             int& cjb, int& cjn) {
  cjb = 0;
  cjn = 0;
  if (q0 + lane < se) {
    const int s = src[q0 + lane];
    cjb = c.begin[s];
    cjn = c.nbody[s];
  }
}
__device__ __forceinline__ int tc_next_tile(const int* __restrict__ src, const TcCells& c, int se, int& q, int& off,
                                            int& q0, int& cjb, int& cjn, int lane, int& myj) {
  int fill = 0;
  myj = -1;
  while (fill < 32 && q < se) {
    if (q >= q0 + 32) {
      q0 = q;
      tc_src_cells(src, c, q0, se, lane, cjb, cjn);
    }
    const int jb = __shfl_sync(0xffffffffu, cjb, q - q0), jn = __shfl_sync(0xffffffffu, cjn, q - q0);
    const int take = min(32 - fill, jn - off);
    if (lane >= fill && lane < fill + take) myj = jb + off + lane - fill;
    fill += take;
    off += take;
    if (off >= jn) {
      q++;
      off = 0;
    }
  }
  return fill;
}

// A tile of FP64 sources in shared memory: one 16-byte broadcast load per two fields.  A body that
// is no source gets x = NaN, so its r^2 fails the r^2 > 0 test that drops coincident bodies.
template <bool JERK>
struct TcTile64 {
  double2 xy[32], zm[32];
  double2 uv[JERK ? 32 : 1];
  double w[JERK ? 32 : 1];
};
template <bool JERK>
struct TcSrc64 {
  double x, y, z, m, u, v, w;
  __device__ __forceinline__ void load(const TcBodies& b, int j) {
    x = y = z = m = u = v = w = 0.0;
    if (j < 0) return;
    x = (b.flags[j] & 2) ? b.x[j] : __longlong_as_double(0x7ff8000000000000ll);
    y = b.y[j]; z = b.z[j]; m = b.m[j];
    if (JERK) { u = b.vx[j]; v = b.vy[j]; w = b.vz[j]; }
  }
  __device__ __forceinline__ void put(TcTile64<JERK>& T, int l) const {
    T.xy[l] = make_double2(x, y);
    T.zm[l] = make_double2(z, m);
    if (JERK) {
      T.uv[l] = make_double2(u, v);
      T.w[l] = w;
    }
  }
};

// one staged source on one target
template <bool JERK>
__device__ __forceinline__ void tc_p2p_staged(const TcTile64<JERK>& T, int s, double xi, double yi, double zi,
                                              double vxi, double vyi, double vzi, double eps2, TcAcc<JERK>& a) {
  const double2 xy = T.xy[s], zm = T.zm[s];
  const double dx = xy.x - xi, dy = xy.y - yi, dz = zm.x - zi;
  const double r2 = dx * dx + dy * dy + dz * dz;
  if (r2 > 0.0) {
    const double invr = rsqrt(r2 + eps2), invr2 = invr * invr;
    double f = zm.y * invr;
    a.pot += f;
    f *= invr2;
    a.ax += dx * f;
    a.ay += dy * f;
    a.az += dz * f;
    if (JERK) {
      const double2 uv = T.uv[s];
      const double dvx = uv.x - vxi, dvy = uv.y - vyi, dvz = T.w[s] - vzi;
      const double vr = 3.0 * (dx * dvx + dy * dvy + dz * dvz);
      a.jx += dvx * f;
      a.jy += dvy * f;
      a.jz += dvz * f;
      f *= -invr2 * vr;
      a.jx += dx * f;
      a.jy += dy * f;
      a.jz += dz * f;
    }
  }
}

// 1 / sqrt(x) of a positive normal x well inside the exponent range (2^-900 ... 2^900): the hardware
// estimate (its relative error e0 is about 2^-20) corrected by the binomial series of (1 - e)^(-1/2)
// to second order, e = 1 - x y^2, Householder's third-order iteration: y (1 + e / 2 + 3 e^2 / 8)
// leaves 5/16 e^3 < 2^-58 before rounding.
__device__ __forceinline__ double tc_rsqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ bool tc_rsqrt_in_range(double x) {
  return (unsigned)(__double2hiint(x) - (123 << 20)) < (unsigned)(1800 << 20);
}

// A velocity whose difference from another such one is finite, so that 0 times it is 0
__device__ __forceinline__ bool tc_vel_bounded(double v) { return fabs(v) < 0x1p1023; }

// Two staged sources on one target without a branch between them, so their dependent chains overlap
// (every source of the tile is one and every velocity is bounded, see k_p2p).  A pair at r = 0 adds
// zero; an r^2 outside tc_rsqrt_normal's range takes the library's root.
template <bool JERK>
__device__ __forceinline__ void tc_p2p_staged2(const TcTile64<JERK>& T, int s0, int s1, double xi, double yi,
                                               double zi, double vxi, double vyi, double vzi, double eps2,
                                               TcAcc<JERK>& a) {
  double dx[2], dy[2], dz[2], r2[2], invr[2], f[2], mj[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double2 xy = T.xy[k ? s1 : s0], zm = T.zm[k ? s1 : s0];
    dx[k] = xy.x - xi; dy[k] = xy.y - yi; dz[k] = zm.x - zi;
    mj[k] = zm.y;
    r2[k] = dx[k] * dx[k] + dy[k] * dy[k] + dz[k] * dz[k];
  }
  const double e0 = r2[0] + eps2, e1 = r2[1] + eps2;
  invr[0] = tc_rsqrt_normal(e0);
  invr[1] = tc_rsqrt_normal(e1);
  if (!(tc_rsqrt_in_range(r2[0]) && tc_rsqrt_in_range(r2[1]) && tc_rsqrt_in_range(e0) && tc_rsqrt_in_range(e1))) {
    invr[0] = r2[0] > 0.0 ? rsqrt(e0) : 0.0;
    invr[1] = r2[1] > 0.0 ? rsqrt(e1) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double invr2 = invr[k] * invr[k];
    f[k] = mj[k] * invr[k];
    a.pot += f[k];
    f[k] *= invr2;
    a.ax += dx[k] * f[k];
    a.ay += dy[k] * f[k];
    a.az += dz[k] * f[k];
    if (JERK) {
      const double2 uv = T.uv[k ? s1 : s0];
      const double dvx = uv.x - vxi, dvy = uv.y - vyi, dvz = T.w[k ? s1 : s0] - vzi;
      const double g = -3.0 * (dx[k] * dvx + dy[k] * dvy + dz[k] * dvz) * invr2 * f[k];
      a.jx += dvx * f[k] + dx[k] * g;
      a.jy += dvy * f[k] + dy[k] * g;
      a.jz += dvz * f[k] + dz[k] * g;
    }
  }
}

// FP64 near field over the work items: a warp per item, a target per lane (rows of r <= 16 targets:
// floor(32 / r) lane groups, each over every ng-th source of a tile).  The next tile's bodies are
// loaded into registers while the current one is summed.  Bound by the FP64 pipe: 69 % busy, 3.1 ms for
// 0.85e9 pairs at N = 131,072 (p = 12, jerks); one source at a time behind the r^2 test 3.2 ms at 63 %;
// reading every field of every source from global memory, one warp per leaf, 55 ms at 17 %.
template <bool JERK>
__global__ void __launch_bounds__(kP2PWarps * 32, JERK ? 4 : 5) k_p2p(const int* __restrict__ tstart,
                                                                      const int* __restrict__ src, const TcBodies b,
                                                                      const TcCells c, TcOut out,
                                                                      const TcP2PWork W) {
  __shared__ TcTile64<JERK> tile[kP2PWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TcTile64<JERK>& T = tile[w];
  const unsigned ni = W.cnt[0], ns = W.cnt[1];
  TcP2PItem it;
  int slot;
  while (tc_p2p_take(W, ni, ns, tstart, lane, it, slot)) {
    const int tb = c.begin[it.t], r = min(32, c.nbody[it.t] - it.t0), se = tstart[it.t + 1];
    const int gsz = r > 16 ? 32 : r, ng = 32 / gsz;
    const int grp = lane / gsz, ti = lane % gsz;
    const int i = tb + it.t0 + ti;
    const bool vi = grp < ng && ti < r;
    double xi = 0, yi = 0, zi = 0, vxi = 0, vyi = 0, vzi = 0;
    if (vi) {
      xi = b.x[i]; yi = b.y[i]; zi = b.z[i];
      if (JERK) { vxi = b.vx[i]; vyi = b.vy[i]; vzi = b.vz[i]; }
    }
    const bool bounded_i =
        !JERK || __all_sync(0xffffffffu, tc_vel_bounded(vxi) && tc_vel_bounded(vyi) && tc_vel_bounded(vzi));
    TcAcc<JERK> a;
    a.zero();
    int q = it.q, off = it.off, left = it.cnt, q0 = q, cjb, cjn, myj;
    tc_src_cells(src, c, q0, se, lane, cjb, cjn);
    int cnt = min(left, tc_next_tile(src, c, se, q, off, q0, cjb, cjn, lane, myj));
    TcSrc64<JERK> sb;
    sb.load(b, myj);
    while (cnt > 0) {
      __syncwarp();
      sb.put(T, lane);
      // every source of the tile is one (x is not NaN) and has a bounded velocity
      const bool plain = bounded_i && __all_sync(0xffffffffu, isfinite(sb.x) && (!JERK || (tc_vel_bounded(sb.u) &&
                                                                                           tc_vel_bounded(sb.v) &&
                                                                                           tc_vel_bounded(sb.w))));
      __syncwarp();
      const int now = cnt;
      left -= now;
      cnt = left > 0 ? min(left, tc_next_tile(src, c, se, q, off, q0, cjb, cjn, lane, myj)) : 0;
      if (cnt > 0) sb.load(b, myj);
      if (vi) {
        int s = grp;
        if (plain)
          for (; s + ng < now; s += 2 * ng)
            tc_p2p_staged2<JERK>(T, s, s + ng, xi, yi, zi, vxi, vyi, vzi, b.eps2, a);
        for (; s < now; s += ng) tc_p2p_staged<JERK>(T, s, xi, yi, zi, vxi, vyi, vzi, b.eps2, a);
      }
    }
    a.add_groups(gsz, ng, grp);
    if (vi && grp == 0) tc_p2p_put<JERK>(W, slot, lane, i, b, out, a);
  }
}

// Folds the chunks of the split rows (first chunk first) into their sink bodies: a warp per row, a
// lane per body.  NC components per slot: the TcOut arrays in order, with STEPS the time-step sum.
template <int NC, bool STEPS>
__global__ void __launch_bounds__(kP2PWarps * 32) k_p2p_join(const TcP2PRow* __restrict__ rows,
                                                             const unsigned* __restrict__ cnt, const TcBodies b,
                                                             const TcCells c, TcOut out, double* __restrict__ tsum,
                                                             const double* __restrict__ slots, bool shared) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = (int)cnt[2];
  for (int k = blockIdx.x * kP2PWarps + w; k < nr; k += gridDim.x * kP2PWarps) {
    const TcP2PRow R = rows[k];
    if (lane >= min(32, c.nbody[R.t] - R.t0)) continue;
    const int i = c.begin[R.t] + R.t0 + lane;
    if (!(b.flags[i] & 1)) continue;
    double v[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) v[q] = 0.0;
    const double* pp = slots + (size_t)R.base * NC * 32 + lane;
    for (int ch = 0; ch < R.nch; ch++, pp += NC * 32) {
#pragma unroll
      for (int q = 0; q < NC; q++) v[q] += pp[32 * q];
    }
    tc_p2p_add(shared, &out.pot[i], v[0]);
    tc_p2p_add(shared, &out.ax[i], v[1]);
    tc_p2p_add(shared, &out.ay[i], v[2]);
    tc_p2p_add(shared, &out.az[i], v[3]);
    if (STEPS) {
      tc_p2p_add(shared, &tsum[i], v[4]);
    } else if (NC == 7) {
      tc_p2p_add(shared, &out.jx[i], v[4]);
      tc_p2p_add(shared, &out.jy[i], v[5]);
      tc_p2p_add(shared, &out.jz[i], v[6]);
    }
  }
}

// Direct summation (N below the direct threshold).  One CTA per 16 targets; its 32 half-warps take
// every 32nd source of each 512-body tile staged in shared memory, and their sums are folded in a
// fixed order.  Bound by the FP64 pipe: 0.15 ms at N = 7,001, 0.11 of it pipe time (a thread per target with
// all sources in series, 219 warps for 592 schedulers, takes 3.07 ms).  Reads the caller's arrays and
// writes the caller's outputs.
constexpr int kDirT = 16, kDirThreads = 512;
template <bool JERK>
__global__ void __launch_bounds__(kDirThreads) k_direct(int n, const double* __restrict__ x,
                                                        const double* __restrict__ y, const double* __restrict__ z,
                                                        const double* __restrict__ vx, const double* __restrict__ vy,
                                                        const double* __restrict__ vz, const double* __restrict__ m,
                                                        const uint8_t* __restrict__ flags, double eps2, TcOut out,
                                                        unsigned* err) {
  __shared__ TcTile64<JERK> tile[kDirThreads / 32];
  __shared__ double red[kDirThreads / 32][JERK ? 7 : 4][kDirT];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kDirT + (lane & (kDirT - 1));
  const bool vi = i < n;
  TcBodies b;
  b.x = const_cast<double*>(x); b.y = const_cast<double*>(y); b.z = const_cast<double*>(z);
  b.m = const_cast<double*>(m);
  b.vx = const_cast<double*>(vx); b.vy = const_cast<double*>(vy); b.vz = const_cast<double*>(vz);
  const double xi = vi ? x[i] : 0, yi = vi ? y[i] : 0, zi = vi ? z[i] : 0;
  const double vxi = JERK && vi ? vx[i] : 0, vyi = JERK && vi ? vy[i] : 0, vzi = JERK && vi ? vz[i] : 0;
  const bool sink = vi && (!flags || (flags[i] & 1));
  if (err && threadIdx.x < kDirT && vi && !(isfinite(xi) && isfinite(yi) && isfinite(zi) && isfinite(m[i])))
    tc_set_err(err, TC_EBIT_NAN);
  TcAcc<JERK> a;
  a.zero();
  for (int t0 = 0; t0 < n; t0 += kDirThreads) {
    const int j = t0 + threadIdx.x;
    TcSrc64<JERK> s;
    s.x = s.y = s.z = s.m = s.u = s.v = s.w = 0.0;
    if (j < n) {
      s.x = !flags || (flags[j] & 2) ? x[j] : __longlong_as_double(0x7ff8000000000000ll);
      s.y = y[j]; s.z = z[j]; s.m = m[j];
      if (JERK) { s.u = vx[j]; s.v = vy[j]; s.w = vz[j]; }
    }
    __syncthreads();
    s.put(tile[w], lane);
    __syncthreads();
    // half-warp h of warp w: sources h, h + 2, ... of the warp's own 32
    const int cnt = min(32, n - t0 - 32 * w);
    if (sink)
      for (int q = lane >> 4; q < cnt; q += 2)
        tc_p2p_staged<JERK>(tile[w], q, xi, yi, zi, vxi, vyi, vzi, eps2, a);
  }
  a.add_xor(16);
  if (lane < kDirT) {
    red[w][0][lane] = a.pot; red[w][1][lane] = a.ax; red[w][2][lane] = a.ay; red[w][3][lane] = a.az;
    if (JERK) { red[w][4][lane] = a.jx; red[w][5][lane] = a.jy; red[w][6][lane] = a.jz; }
  }
  __syncthreads();
  const int k = threadIdx.x >> 4, o = blockIdx.x * kDirT + (threadIdx.x & (kDirT - 1));
  if (k < (JERK ? 7 : 4) && o < n) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kDirThreads / 32; q++) v += red[q][k][threadIdx.x & (kDirT - 1)];
    double* const dst[7] = {out.pot, out.ax, out.ay, out.az, out.jx, out.jy, out.jz};
    if (dst[k]) dst[k][o] = v;
  }
}

// Direct sums of at most kChainN bodies (the integrator's smallest systems) in the sources' order.
// A CTA takes 8 targets: its threads form all pair terms in shared memory, then a lane per target
// and component adds its terms one after the other -- the rounding of the plain loop over the
// sources, at the latency of one dependent FMA per source instead of a whole pair.
constexpr int kChainN = 128, kChainT = 8;
__global__ void __launch_bounds__(256) k_direct_chain(int n, const double* __restrict__ x,
                                                      const double* __restrict__ y, const double* __restrict__ z,
                                                      const double* __restrict__ m,
                                                      const uint8_t* __restrict__ flags, double eps2, TcOut out) {
  __shared__ double d[3][kChainT][kChainN + 1], f[2][kChainT][kChainN + 1];  // padded: no bank conflicts
  for (int k = threadIdx.x; k < kChainT * n; k += blockDim.x) {
    const int t = k / n, j = k % n, i = blockIdx.x * kChainT + t;
    double dx = 0, dy = 0, dz = 0, f0 = 0, f3 = 0;
    if (i < n && (!flags || (flags[j] & 2))) {
      dx = x[j] - x[i]; dy = y[j] - y[i]; dz = z[j] - z[i];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > 0.0) {
        const double invr = rsqrt(r2 + eps2), invr2 = invr * invr;
        f0 = m[j] * invr;
        f3 = f0 * invr2;
      } else {
        dx = dy = dz = 0;
      }
    }
    d[0][t][j] = dx; d[1][t][j] = dy; d[2][t][j] = dz;
    f[0][t][j] = f0; f[1][t][j] = f3;
  }
  __syncthreads();
  const int t = threadIdx.x & (kChainT - 1), q = threadIdx.x / kChainT, i = blockIdx.x * kChainT + t;
  if (q > 3 || i >= n) return;
  double a = 0.0;
  if (!flags || (flags[i] & 1)) {
    if (q == 3) {
#pragma unroll 8
      for (int j = 0; j < n; j++) a += f[0][t][j];
    } else {
#pragma unroll 8
      for (int j = 0; j < n; j++) a = __fma_rn(d[q][t][j], f[1][t][j], a);
    }
  }
  double* const dst[4] = {out.ax, out.ay, out.az, out.pot};
  dst[q][i] = a;
}

// FP64 direct sums at selected bodies: the judge of the selector, and tc_direct_sums.  Block
// (c, g) takes the source chunk c and up to 256 targets (one per thread, group g); sources pass
// through shared memory in tiles, so every body is read once per block.
// part[(k * nchunk + c) * 8 + q] = chunk c's (pot, ax, ay, az, jx, jy, jz) of target k.
constexpr int kJudgeTile = 256;
template <bool JERK>
__global__ void __launch_bounds__(kJudgeTile) k_direct_targets(int n, int nt, int nchunk, const int* __restrict__ tgt,
                                                               const TcBodies b, double* __restrict__ part) {
  __shared__ double sx[kJudgeTile], sy[kJudgeTile], sz[kJudgeTile], sm[kJudgeTile];
  __shared__ double su[JERK ? kJudgeTile : 1], sv[JERK ? kJudgeTile : 1], sw[JERK ? kJudgeTile : 1];
  const int c = blockIdx.x, k = blockIdx.y * kJudgeTile + threadIdx.x;
  const int chunk = (n + nchunk - 1) / nchunk;
  const int j0 = c * chunk, j1 = min(n, j0 + chunk);
  const int i = k < nt ? tgt[k] : 0;
  const double xi = b.x[i], yi = b.y[i], zi = b.z[i];
  const double ui = JERK ? b.vx[i] : 0.0, vi = JERK ? b.vy[i] : 0.0, wi = JERK ? b.vz[i] : 0.0;
  double pot = 0.0, ax = 0.0, ay = 0.0, az = 0.0, jx = 0.0, jy = 0.0, jz = 0.0;
  for (int t0 = j0; t0 < j1; t0 += kJudgeTile) {
    const int j = t0 + threadIdx.x;
    __syncthreads();
    if (j < j1) {
      sx[threadIdx.x] = b.x[j];
      sy[threadIdx.x] = b.y[j];
      sz[threadIdx.x] = b.z[j];
      sm[threadIdx.x] = (b.flags[j] & 2) ? b.m[j] : 0.0;
      if (JERK) {
        su[threadIdx.x] = b.vx[j];
        sv[threadIdx.x] = b.vy[j];
        sw[threadIdx.x] = b.vz[j];
      }
    }
    __syncthreads();
    const int cnt = min(kJudgeTile, j1 - t0);
    for (int q = 0; q < cnt; q++) {
      const double dx = sx[q] - xi, dy = sy[q] - yi, dz = sz[q] - zi;
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > 0.0) {
        const double invr = rsqrt(r2 + b.eps2), invr2 = invr * invr;
        const double f = sm[q] * invr;
        pot += f;
        const double f3 = f * invr2;
        ax += dx * f3;
        ay += dy * f3;
        az += dz * f3;
        if (JERK) {
          const double du = su[q] - ui, dv = sv[q] - vi, dw = sw[q] - wi;
          const double g = -3.0 * f3 * invr2 * (dx * du + dy * dv + dz * dw);
          jx += du * f3 + dx * g;
          jy += dv * f3 + dy * g;
          jz += dw * f3 + dz * g;
        }
      }
    }
  }
  if (k < nt) {
    double* o = part + ((size_t)k * nchunk + c) * 8;
    o[0] = pot; o[1] = ax; o[2] = ay; o[3] = az; o[4] = jx; o[5] = jy; o[6] = jz;
  }
}

// judge: out[k] = {direct pot, ax, ay, az (chunks summed in order), evaluated ax, ay, az}
__global__ void k_direct_targets_sum(int nt, int nchunk, const int* __restrict__ tgt, const double* __restrict__ part,
                                     TcOut ev, double* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nt) return;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < nchunk; c++)
    for (int q = 0; q < 4; q++) v[q] += part[((size_t)k * nchunk + c) * 8 + q];
  const int i = tgt[k];
  double* o = out + 7 * (size_t)k;
  o[0] = v[0]; o[1] = v[1]; o[2] = v[2]; o[3] = v[3];
  o[4] = ev.ax[i]; o[5] = ev.ay[i]; o[6] = ev.az[i];
}

// tc_direct_sums: out[k] = direct (pot, ax, ay, az, jx, jy, jz), chunks summed in order
__global__ void k_direct_targets_out(int nt, int nchunk, const double* __restrict__ part, double* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nt) return;
  double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < nchunk; c++)
    for (int q = 0; q < 7; q++) v[q] += part[((size_t)k * nchunk + c) * 8 + q];
  for (int q = 0; q < 7; q++) out[7 * (size_t)k + q] = v[q];
}

// Time-step pass of the top-level tree (get_force_and_potential(bodies, true) on the theta
// path): P2P of kernel_fast_lean.h:462-548 (the SIMD / DOUBLE_P2P branch), in FP64.  For a
// target body and one source cell: pot and acc from the cell's sources as in P2P_simple, and
// the pairwise step
//   tau1 = dt/sqrt2 r sqrt(r/mi) / (1 - dtau1/2),  dtau1 = min(1, 3/2 tau1 (d.dv)/r^2)
//   tau2 = dt r/|dv|       / (1 - dtau2/2),  dtau2 = min(1, tau2 (d.dv)/r^2 (1 + mi/(v^2 r)))
// minimised over the cell's bodies; the target's step sum gains 1/min^4.  As in the
// reference, mi starts at the target's mass and accumulates every body of the cell met so far
// (sources or not, self excluded) in the cell's body order, so each lane (one target) walks
// each source cell's bodies in order.
//
// The two steps enter as 1 / tau, of which the largest is kept: with q = 1 / sqrt(r mi) and the
// reciprocal roots of r^2 and v^2,
//   1 / tau1 = (r mi) q / (dt/sqrt2 r^2),  1 / tau2 = |dv| / (dt r),  1/min^4 = max^4,
// three reciprocal square roots and no division or square root per pair.  That order of
// comparison needs dt > 0 (and finite); POS = false is the direct form for any other dt_param.
//
// A warp per work item (whole source cells: a chunk takes the cells that begin in it); rows of
// r <= 16 targets run floor(32 / r) lane groups, each over every ng-th cell.
template <bool POS>
__global__ void __launch_bounds__(kP2PWarps * 32) k_p2p_steps(const int* __restrict__ tstart,
                                                              const int* __restrict__ src, const TcBodies b,
                                                              const TcCells c, TcOut out, double dtp,
                                                              double* __restrict__ tsum, const TcP2PWork W) {
  const int lane = threadIdx.x & 31;
  const double dts = dtp / 1.41421356237309504880;  // dt_param / M_SQRT2
  const double idts = 1.0 / dts, idtp = 1.0 / dtp;
  const unsigned ni = W.cnt[0], ns = W.cnt[1];
  TcP2PItem it;
  int slot;
  while (tc_p2p_take(W, ni, ns, tstart, lane, it, slot)) {
    const int tb = c.begin[it.t], r = min(32, c.nbody[it.t] - it.t0), se = tstart[it.t + 1];
    const int gsz = r > 16 ? 32 : r, ng = 32 / gsz;
    const int grp = lane / gsz, ti = lane % gsz;
    const bool vi = grp < ng && ti < r;
    const int i = tb + it.t0 + (vi ? ti : 0);
    const double xi = b.x[i], yi = b.y[i], zi = b.z[i], ui = b.vx[i], vvi = b.vy[i], wi = b.vz[i];
    const double m0 = b.m[i];
    double pot = 0.0, ax = 0.0, ay = 0.0, az = 0.0, ts = 0.0;
    // the cells that begin inside the chunk: bodies before the first of them, then `left` more
    const int q1 = it.off > 0 ? it.q + 1 : it.q;
    int left = it.cnt;
    if (it.off > 0) left -= c.nbody[src[it.q]] - it.off;
    for (int q0 = q1; q0 < se && left > 0; q0 += 32) {
      int cjb, cjn;
      tc_src_cells(src, c, q0, se, lane, cjb, cjn);
      int pi = cjn;
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pi, d);
        if (lane >= d) pi += v;
      }
      // cells of this window that begin before the chunk's end (bodies before a cell: pi - cjn)
      const int ncw = __popc(__ballot_sync(0xffffffffu, q0 + lane < se && pi - cjn < left));
      left -= __shfl_sync(0xffffffffu, pi, 31);
      for (int l0 = 0; l0 < ncw; l0 += ng) {
        const int l = l0 + (vi ? grp : 0);
        const int jb = __shfl_sync(0xffffffffu, cjb, l & 31);
        const int jn = __shfl_sync(0xffffffffu, cjn, l & 31);
        if (!vi || l >= ncw) continue;
        double mi = m0, tmin = 1e38, gmax = 1e-38;
        for (int j = jb; j < jb + jn; j++) {
          double mj = b.m[j];
          const double dx = b.x[j] - xi, dy = b.y[j] - yi, dz = b.z[j] - zi;
          const double du = b.vx[j] - ui, dv = b.vy[j] - vvi, dw = b.vz[j] - wi;
          const bool source = (b.flags[j] & 2) != 0;
          double r2 = dx * dx + dy * dy + dz * dz;
          const double v2 = du * du + dv * dv + dw * dw + 1e-20;
          if (!(r2 > 0.0)) {
            mj = 0.0;
            r2 = 1e38;
          }
          mi += mj;
          double invr, invr2;
          if (POS) {
            invr = rsqrt(r2);
            invr2 = invr * invr;
            // 1 / |dv|, at least 2^-520: where v2 overflowed, |dv| = v2 iv is then infinite and not inf * 0 = NaN,
            // which no comparison keeps (a finite v2 has a root of 2^-512 or more)
            double iv = rsqrt(v2);
            iv = __hiloint2double(max(__double2hiint(iv), 503 << 20), __double2loint(iv));
            const double rr = r2 * invr, rm = rr * mi, qm = rsqrt(rm);
            const double vdotdr2 = (dx * du + dy * dv + dz * dw) * invr2;
            double dtau = 1.5 * (dts * r2 * qm) * vdotdr2;
            if (!(dtau < 1.0)) dtau = 1.0;
            const double g1 = rm * qm * invr2 * idts * (1.0 - 0.5 * dtau);
            gmax = g1 > gmax ? g1 : gmax;
            dtau = dtp * rr * iv * vdotdr2 * (1.0 + mi * (iv * iv) * invr);
            if (!(dtau < 1.0)) dtau = 1.0;
            const double g2 = v2 * iv * invr * idtp * (1.0 - 0.5 * dtau);
            gmax = g2 > gmax ? g2 : gmax;
          } else {
            const double vdotdr2 = (dx * du + dy * dv + dz * dw) / r2;
            const double rr = sqrt(r2);
            invr = 1.0 / rr;
            invr2 = invr * invr;
            double tau = dts * rr * sqrt(rr / mi);
            double dtau = 3.0 * tau * vdotdr2 / 2.0;
            if (!(dtau < 1.0)) dtau = 1.0;
            tau /= (1.0 - dtau / 2.0);
            tmin = tau < tmin ? tau : tmin;
            tau = dtp * rr / sqrt(v2);
            dtau = tau * vdotdr2 * (1.0 + mi / (v2 * rr));
            if (!(dtau < 1.0)) dtau = 1.0;
            tau /= (1.0 - dtau / 2.0);
            tmin = tau < tmin ? tau : tmin;
          }
          mj = source ? mj * invr : 0.0;
          pot += mj;
          const double f = mj * invr2;
          ax += dx * f;
          ay += dy * f;
          az += dz * f;
        }
        if (POS) {
          gmax *= gmax;
          ts += gmax * gmax;
        } else {
          tmin *= tmin;
          tmin *= tmin;
          ts += 1.0 / tmin;
        }
      }
    }
    for (int st = 1; st < ng; st <<= 1) {  // the lane groups' sums, a fixed tree
      const bool take = (grp % (2 * st)) == 0 && grp + st < ng;
      double v;
      v = __shfl_down_sync(0xffffffffu, pot, st * gsz); if (take) pot += v;
      v = __shfl_down_sync(0xffffffffu, ax, st * gsz); if (take) ax += v;
      v = __shfl_down_sync(0xffffffffu, ay, st * gsz); if (take) ay += v;
      v = __shfl_down_sync(0xffffffffu, az, st * gsz); if (take) az += v;
      v = __shfl_down_sync(0xffffffffu, ts, st * gsz); if (take) ts += v;
    }
    if (!vi || grp != 0) continue;
    if (slot >= 0) {
      double* pp = W.slots + (size_t)slot * 5 * 32 + lane;
      pp[0] = pot; pp[32] = ax; pp[64] = ay; pp[96] = az; pp[128] = ts;
    } else if (b.flags[i] & 1) {
      tc_p2p_add(W.shared, &out.pot[i], pot);
      tc_p2p_add(W.shared, &out.ax[i], ax);
      tc_p2p_add(W.shared, &out.ay[i], ay);
      tc_p2p_add(W.shared, &out.az[i], az);
      tc_p2p_add(W.shared, &tsum[i], ts);
    }
  }
}

// one array, Morton order -> caller order
__global__ void k_scatter_one(int n, const int* __restrict__ perm, const double* __restrict__ s,
                              double* __restrict__ d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[perm[i]] = s[i];
}

// Morton order -> caller order
__global__ void k_scatter_out(int n, const int* __restrict__ perm, TcOut s, double* pot, double* ax, double* ay,
                              double* az, double* jx, double* jy, double* jz) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int j = perm[i];
  pot[j] = s.pot[i]; ax[j] = s.ax[i]; ay[j] = s.ay[i]; az[j] = s.az[i];
  if (jx) { jx[j] = s.jx ? s.jx[i] : 0.0; jy[j] = s.jy ? s.jy[i] : 0.0; jz[j] = s.jz ? s.jz[i] : 0.0; }
}

}  // namespace tc

namespace tc {

// ---------------------------------------------------------------------------------------
// k_p2p_mixed: the mixed-precision near field.
//
// One warp per work item (a row of up to 32 targets and all or a chunk of its sources), one target per
// lane; a row of r <= 16 targets runs floor(32 / r) lane groups, each over every ng-th source pair of
// each tile (so small leaves still fill the warp).  A tile takes the next 32 bodies of the target's source cells read as
// one sequence, so small source leaves still fill it.
//
// Arithmetic.  Sources are staged per 32-source tile as FP32 (hi, lo) pairs of positions and of
// masses, formed in FP64 once per evaluation (k_body_f32), so dx = (xj_hi - xi_hi) + (xj_lo -
// xi_lo) carries one rounding even for close pairs (the hi parts of neighbours subtract exactly).  Each lane evaluates two
// sources at once with the packed FP32x2 instructions of sm_100 (FADD2/FMUL2/FFMA2: one issue
// for two pairs); the tile stores the two sources' fields side by side so one 16-byte
// broadcast load feeds both halves.  1/r is the hardware estimate refined by one Newton
// step; each tile's FP32 sums are folded into (hi, lo) accumulators by a two-sum; the final
// sums are FP64.
//
// Accuracy.  The FP32 pair terms carry a few units of 2^-24 each, and so does their per-tile
// FP32 sum -- relative to the largest term in the sum.  A term far larger than the target's
// acceleration would leave an error far larger than the FMM's own.  So every pair whose
// strength m / r^2 exceeds tau = excl_frac |a_far| (the target's far-field acceleration,
// which the downward pass has already written into out) is left out of the FP32 sums and
// recorded; after the loop the recorded pairs are added in FP64.  A lane with more than kP2PRec
// strong pairs (a zero far field makes every pair strong) goes over its sources a second time,
// in the same tiles and lane groups, and adds every strong pair in FP64 (the same FP32 test
// decides).
// ---------------------------------------------------------------------------------------
constexpr int kP2PRec = 16;
// strong-pair threshold: pairs with m / r^2 above this fraction of the far-field acceleration
// are summed in FP64
constexpr float kP2PExclFrac = 1e-2f;

struct TcF2 {
  float hi, lo;
  __device__ __forceinline__ void add(float t) {  // two-sum
    float s = hi + t;
    float bp = s - hi;
    float e = (hi - (s - bp)) + (t - bp);
    hi = s;
    lo += e;
  }
  __device__ __forceinline__ double val() const { return (double)hi + (double)lo; }
};

// FP32 (hi, lo) split of x - c
__device__ __forceinline__ void tc_split(double x, double c, float& h, float& l) {
  double d = x - c;
  h = (float)d;
  l = (float)(d - (double)h);
}

__device__ __forceinline__ float2 tc_f2(float a) { return make_float2(a, a); }

// the hardware 1/sqrt estimate (inputs here are never subnormal: r2 + eps2 of a pair that is
// kept, or 0 for a pair that is dropped)
__device__ __forceinline__ float tc_rsqrt_est(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A tile: 32 sources as 16 pairs (2p, 2p + 1); field group g of pair p is one float4 holding
// both sources' values of two fields: g0 (xh, yh), g1 (zh, xl), g2 (yl, zl), g3 (mh, ml),
// g4 (vx, vy), g5 (vz, -), each as (source 2p, source 2p + 1).
constexpr int kP2PGroups = 6;
struct TcTile {
  float4 g[kP2PGroups][16];
};

// one target's FP32 state; the target's fields are negated and duplicated into both halves
template <bool JERK>
struct TcMixP {
  float2 nxh, nyh, nzh, nxl, nyl, nzl, nvx, nvy, nvz, eps2;
  float tau;
  float2 sp, sx, sy, sz, qx, qy, qz;  // this tile's sums, one per half
  TcF2 pot, ax, ay, az, jx, jy, jz;   // compensated totals
};

// The FP32 splits of every body, once per evaluation: positions as (hi, lo) pairs of the
// coordinates themselves (the difference (xj_hi - xi_hi) + (xj_lo - xi_lo) of two bodies keeps
// one rounding, the hi parts of neighbours subtracting exactly), the source mass likewise (0 for
// a non-source), velocities rounded.  Each tile then reads three 16-byte words per source.
template <bool JERK>
__global__ void k_body_f32(int n, const TcBodies b) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  float xh, yh, zh, xl, yl, zl, mh, ml;
  tc_split(b.x[j], 0.0, xh, xl);
  tc_split(b.y[j], 0.0, yh, yl);
  tc_split(b.z[j], 0.0, zh, zl);
  tc_split((b.flags[j] & 2) ? b.m[j] : 0.0, 0.0, mh, ml);
  b.f32[3 * (size_t)j] = make_float4(xh, yh, zh, mh);
  b.f32[3 * (size_t)j + 1] = make_float4(xl, yl, zl, ml);
  b.f32[3 * (size_t)j + 2] =
      JERK ? make_float4((float)b.vx[j], (float)b.vy[j], (float)b.vz[j], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// stage source j (or a zero-mass source at the origin when j < 0) at tile slot l
template <bool JERK>
__device__ __forceinline__ void tc_tile_put(TcTile& T, int l, const TcBodies& b, int j) {
  float xh = 0.f, yh = 0.f, zh = 0.f, xl = 0.f, yl = 0.f, zl = 0.f, mh = 0.f, ml = 0.f, vx = 0.f, vy = 0.f, vz = 0.f;
  if (j >= 0) {
    const float4 h = b.f32[3 * (size_t)j], lo = b.f32[3 * (size_t)j + 1];
    xh = h.x; yh = h.y; zh = h.z; mh = h.w;
    xl = lo.x; yl = lo.y; zl = lo.z; ml = lo.w;
    if (JERK) {
      const float4 v = b.f32[3 * (size_t)j + 2];
      vx = v.x; vy = v.y; vz = v.z;
    }
  }
  const int p = l >> 1, h = l & 1;
  float* g0 = reinterpret_cast<float*>(&T.g[0][p]);
  float* g1 = reinterpret_cast<float*>(&T.g[1][p]);
  float* g2 = reinterpret_cast<float*>(&T.g[2][p]);
  float* g3 = reinterpret_cast<float*>(&T.g[3][p]);
  g0[h] = xh; g0[2 + h] = yh;
  g1[h] = zh; g1[2 + h] = xl;
  g2[h] = yl; g2[2 + h] = zl;
  g3[h] = mh; g3[2 + h] = ml;
  if (JERK) {
    float* g4 = reinterpret_cast<float*>(&T.g[4][p]);
    float* g5 = reinterpret_cast<float*>(&T.g[5][p]);
    g4[h] = vx; g4[2 + h] = vy;
    g5[h] = vz;
  }
}

// The FP32 geometry of source pair p: differences, 1/r, m/r, and whether each half's m/r^2
// exceeds the target's threshold.  The only definition of "strong": the main loop and the
// overflow pass both call it.
template <bool JERK>
__device__ __forceinline__ void tc_mixp_geom(const TcMixP<JERK>& T, const TcTile& S, int p, float2& dx, float2& dy,
                                             float2& dz, float2& ri, float2& f0, bool& sa, bool& sb) {
  const float4 g0 = S.g[0][p], g1 = S.g[1][p], g2 = S.g[2][p], g3 = S.g[3][p];
  dx = __fadd2_rn(__fadd2_rn(make_float2(g0.x, g0.y), T.nxh), __fadd2_rn(make_float2(g1.z, g1.w), T.nxl));
  dy = __fadd2_rn(__fadd2_rn(make_float2(g0.z, g0.w), T.nyh), __fadd2_rn(make_float2(g2.x, g2.y), T.nyl));
  dz = __fadd2_rn(__fadd2_rn(make_float2(g1.x, g1.y), T.nzh), __fadd2_rn(make_float2(g2.z, g2.w), T.nzl));
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
  const float2 rs = __fadd2_rn(r2, T.eps2);  // softened (eps2 = 0: unchanged)
  const float2 y = make_float2(tc_rsqrt_est(rs.x), tc_rsqrt_est(rs.y));
  // one Newton step: ri = y + (y / 2) (1 - rs y^2), written as y - (y / 2) (rs y^2 - 1)
  const float2 e = __ffma2_rn(__fmul2_rn(rs, y), y, tc_f2(-1.f));
  ri = __ffma2_rn(__fmul2_rn(y, tc_f2(-0.5f)), e, y);
  ri.x = r2.x > 0.f ? ri.x : 0.f;  // coincident bodies (and the target itself) add nothing
  ri.y = r2.y > 0.f ? ri.y : 0.f;
  f0 = __ffma2_rn(make_float2(g3.z, g3.w), ri, __fmul2_rn(make_float2(g3.x, g3.y), ri));
  const float2 st = __fmul2_rn(f0, ri);
  sa = st.x > T.tau;
  sb = st.y > T.tau;
}

template <bool JERK>
__device__ __forceinline__ void tc_mixp_pair(TcMixP<JERK>& T, const TcTile& S, int p, bool& sa, bool& sb) {
  float2 dx, dy, dz, ri, f0;
  tc_mixp_geom<JERK>(T, S, p, dx, dy, dz, ri, f0, sa, sb);
  if (sa) f0.x = 0.f;  // strong: summed in FP64 instead
  if (sb) f0.y = 0.f;
  const float2 ri2 = __fmul2_rn(ri, ri);
  const float2 f = __fmul2_rn(f0, ri2);
  T.sp = __fadd2_rn(T.sp, f0);
  T.sx = __ffma2_rn(dx, f, T.sx);
  T.sy = __ffma2_rn(dy, f, T.sy);
  T.sz = __ffma2_rn(dz, f, T.sz);
  if (JERK) {
    const float4 g4 = S.g[4][p];
    const float2 g5 = *reinterpret_cast<const float2*>(&S.g[5][p]);
    const float2 dvx = __fadd2_rn(make_float2(g4.x, g4.y), T.nvx);
    const float2 dvy = __fadd2_rn(make_float2(g4.z, g4.w), T.nvy);
    const float2 dvz = __fadd2_rn(g5, T.nvz);
    // g = -f / r^2 * 3 (d . dv)
    const float2 vrn = __fmul2_rn(tc_f2(-3.f), __ffma2_rn(dx, dvx, __ffma2_rn(dy, dvy, __fmul2_rn(dz, dvz))));
    const float2 g = __fmul2_rn(__fmul2_rn(f, ri2), vrn);
    T.qx = __ffma2_rn(dx, g, __ffma2_rn(dvx, f, T.qx));
    T.qy = __ffma2_rn(dy, g, __ffma2_rn(dvy, f, T.qy));
    T.qz = __ffma2_rn(dz, g, __ffma2_rn(dvz, f, T.qz));
  }
}

template <bool JERK>
__device__ __forceinline__ void tc_mixp_fold(TcMixP<JERK>& T) {
  T.pot.add(__fadd_rn(T.sp.x, T.sp.y));
  T.ax.add(__fadd_rn(T.sx.x, T.sx.y));
  T.ay.add(__fadd_rn(T.sy.x, T.sy.y));
  T.az.add(__fadd_rn(T.sz.x, T.sz.y));
  if (JERK) {
    T.jx.add(__fadd_rn(T.qx.x, T.qx.y));
    T.jy.add(__fadd_rn(T.qy.x, T.qy.y));
    T.jz.add(__fadd_rn(T.qz.x, T.qz.y));
  }
  T.sp = T.sx = T.sy = T.sz = T.qx = T.qy = T.qz = tc_f2(0.f);
}

template <bool JERK>
__device__ __forceinline__ void tc_mixp_init(TcMixP<JERK>& T, const TcBodies& b, const TcOut& out, int i, bool v,
                                             float excl_frac) {
  float xh = 0.f, yh = 0.f, zh = 0.f, xl = 0.f, yl = 0.f, zl = 0.f, vx = 0.f, vy = 0.f, vz = 0.f;
  T.tau = 0.f;
  if (v) {
    const float4 h = b.f32[3 * (size_t)i], lo = b.f32[3 * (size_t)i + 1];
    xh = h.x; yh = h.y; zh = h.z;
    xl = lo.x; yl = lo.y; zl = lo.z;
    if (JERK) {
      const float4 w = b.f32[3 * (size_t)i + 2];
      vx = w.x; vy = w.y; vz = w.z;
    }
    const double a = sqrt(out.ax[i] * out.ax[i] + out.ay[i] * out.ay[i] + out.az[i] * out.az[i]);
    T.tau = (float)(excl_frac * a);
  }
  T.nxh = tc_f2(-xh); T.nyh = tc_f2(-yh); T.nzh = tc_f2(-zh);
  T.nxl = tc_f2(-xl); T.nyl = tc_f2(-yl); T.nzl = tc_f2(-zl);
  T.nvx = tc_f2(-vx); T.nvy = tc_f2(-vy); T.nvz = tc_f2(-vz);
  T.eps2 = tc_f2((float)b.eps2);
  T.sp = T.sx = T.sy = T.sz = T.qx = T.qy = T.qz = tc_f2(0.f);
  T.pot = T.ax = T.ay = T.az = T.jx = T.jy = T.jz = TcF2{0.f, 0.f};
}

template <bool JERK>
__device__ __forceinline__ TcAcc<JERK> tc_mixp_total(const TcMixP<JERK>& T) {
  TcAcc<JERK> a;
  a.pot = T.pot.val(); a.ax = T.ax.val(); a.ay = T.ay.val(); a.az = T.az.val();
  a.jx = T.jx.val(); a.jy = T.jy.val(); a.jz = T.jz.val();
  return a;
}

// Seven CTAs (28 warps) per SM: the register cap (73) spills a few words per thread, and the
// occupancy still wins at N = 4M (79.6 ms against 84.2 ms at five CTAs, 81.2 at six; the compensated
// totals kept in shared memory instead of registers measured no better).
template <bool JERK>
__global__ void __launch_bounds__(kP2PWarps * 32, 7) k_p2p_mixed(const int* __restrict__ tstart,
                                                                 const int* __restrict__ src, const TcBodies b,
                                                                 const TcCells c, TcOut out, float excl_frac,
                                                                 const TcP2PWork W) {
  // per warp: the source tile and each lane's recorded strong pairs
  __shared__ TcTile tile[kP2PWarps];
  __shared__ int tj[kP2PWarps][32];  // body index of each tile slot
  __shared__ int rec[kP2PWarps][kP2PRec][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TcTile& TL = tile[w];
  TcP2PItem it;
  int slot;
  while (tc_p2p_take(W, W.cnt[0], W.cnt[1], tstart, lane, it, slot)) {
      // up to 32 targets; a row of r <= 16 targets runs floor(32 / r) lane groups of r lanes, each
      // over every ng-th source pair
      const int se = tstart[it.t + 1];
      const int r = min(32, c.nbody[it.t] - it.t0);
      const int gsz = r > 16 ? 32 : r, ng = 32 / gsz;
      const int grp = lane / gsz, ti = lane % gsz;
      const bool act = grp < ng && ti < r;
      const int i = c.begin[it.t] + it.t0 + ti;
      int nrl = 0;  // strong pairs this lane met
      TcMixP<JERK> A;
      tc_mixp_init<JERK>(A, b, out, i, act, excl_frac);
      int q0 = it.q, cjb, cjn;
      tc_src_cells(src, c, q0, se, lane, cjb, cjn);
      for (int q = it.q, off = it.off, left = it.cnt; q < se && left > 0;) {
        int myj;
        const int cnt = min(left, tc_next_tile(src, c, se, q, off, q0, cjb, cjn, lane, myj)), np = (cnt + 1) >> 1;
        left -= cnt;
        __syncwarp();
        if (lane < 2 * np) tc_tile_put<JERK>(TL, lane, b, myj);
        tj[w][lane] = myj;
        __syncwarp();
        if (act) {
          for (int p = grp; p < np; p += ng) {
            bool sa, sbb;
            tc_mixp_pair<JERK>(A, TL, p, sa, sbb);
            if (sa | sbb) {
              if (sa) {
                if (nrl < kP2PRec) rec[w][nrl][lane] = tj[w][2 * p];
                nrl++;
              }
              if (sbb) {
                if (nrl < kP2PRec) rec[w][nrl][lane] = tj[w][2 * p + 1];
                nrl++;
              }
            }
          }
        }
        tc_mixp_fold<JERK>(A);
      }
      TcAcc<JERK> a = tc_mixp_total<JERK>(A);
      const bool ovf = act && nrl > kP2PRec;
      if (__any_sync(0xffffffffu, ovf)) {
        // a lane whose list overflowed goes over its own sources again (the same tiles, the same
        // lane groups) and adds every strong pair in FP64; the other lanes only stage the tiles
        const double xi = ovf ? b.x[i] : 0.0, yi = ovf ? b.y[i] : 0.0, zi = ovf ? b.z[i] : 0.0;
        const double vxi = (JERK && ovf) ? b.vx[i] : 0.0, vyi = (JERK && ovf) ? b.vy[i] : 0.0,
                     vzi = (JERK && ovf) ? b.vz[i] : 0.0;
        q0 = it.q;
        tc_src_cells(src, c, q0, se, lane, cjb, cjn);
        for (int q = it.q, off = it.off, left = it.cnt; q < se && left > 0;) {
          int myj;
          const int cnt = min(left, tc_next_tile(src, c, se, q, off, q0, cjb, cjn, lane, myj)), np = (cnt + 1) >> 1;
          left -= cnt;
          __syncwarp();
          if (lane < 2 * np) tc_tile_put<JERK>(TL, lane, b, myj);
          tj[w][lane] = myj;
          __syncwarp();
          if (ovf) {
            for (int p = grp; p < np; p += ng) {
              float2 dx, dy, dz, ri, f0;
              bool sa, sbb;
              tc_mixp_geom<JERK>(A, TL, p, dx, dy, dz, ri, f0, sa, sbb);
              if (sa) tc_p2p_one<JERK>(xi, yi, zi, vxi, vyi, vzi, b, tj[w][2 * p], a);
              if (sbb) tc_p2p_one<JERK>(xi, yi, zi, vxi, vyi, vzi, b, tj[w][2 * p + 1], a);
            }
          }
        }
      }
      // each lane adds its own recorded strong pairs in FP64
      if (act && !ovf && nrl > 0) {
        const double xi = b.x[i], yi = b.y[i], zi = b.z[i];
        const double vxi = JERK ? b.vx[i] : 0.0, vyi = JERK ? b.vy[i] : 0.0, vzi = JERK ? b.vz[i] : 0.0;
        for (int e = 0; e < nrl; e++) tc_p2p_one<JERK>(xi, yi, zi, vxi, vyi, vzi, b, rec[w][e][lane], a);
      }
      a.add_groups(gsz, ng, grp);
      if (act && grp == 0) tc_p2p_put<JERK>(W, slot, lane, i, b, out, a);
  }
}

}  // namespace tc
