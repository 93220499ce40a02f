// Dual-tree traversal on the device: breadth-first expansion of (target, source) cell pairs.
// Each pair takes exactly the decision of the reference recursion (traverse_eager.h:151-203;
// taichi_with_jerks/traverse_eager.h:125-155):
//   |Xi - Xj|^2 theta^2 > (Ri + Rj)^2  -> M2L (top tree: P2P when one cell holds <= 2 and
//                                          the other <= 8 bodies, :160)
//   both leaves                        -> P2P
//   Cj leaf, or Ri >= Rj and Ci inner  -> (child of Ci, Cj) for every child
//   otherwise                          -> (Ci, child of Cj) for every child
// so the set of emitted pairs equals the set the recursion visits.  The emission order is
// not deterministic; the lists are put in (target, source) order afterwards (k_list_*).
#pragma once
#include "tc_common.cuh"

namespace tc {

// acceptance test of a traversal (mode 0: theta, traverse_eager.h:151-203; 1: the low-order
// pre-pass, |d|^2 > 3 (Ri + Rj)^2 on geometric cells, :220-245; 2: the top tree's error-
// controlled MAC of horizontalPassHigh, :61-148, with the reference's binomials comb[k] =
// combinator_coef[P][k]; 3: the jerks tree's one-sided horizontalPassHigh,
// taichi_with_jerks/traverse_eager.h:59-122)
struct TcMac {
  int mode = 0;
  int p = 0;
  double fa = 0.0;
  const double* pn = nullptr;       // (p + 1) per cell
  const double* min_acc = nullptr;  // per cell
  double comb[TC_PMAX_DEV + 1];
  // > 0: an accepted pair whose target is a leaf and whose body counts multiply to at most this
  // becomes a P2P pair (exact, and cheaper than its M2L); the order selectors' form only
  long long p2p_max = 0;
};

// x^-k correctly rounded (k >= 1): x^k in double-double by repeated products, then the
// reciprocal's leading term refined by one Newton step on the pair
__device__ __forceinline__ double tc_pow_neg_int(double x, int k) {
  double h = x, l = 0.0;
  for (int i = 1; i < k; i++) {
    const double p = h * x;
    const double e = __fma_rn(h, x, -p);
    h = p;
    l = __fma_rn(l, x, e);
    const double s = h + l;
    l = l - (s - h);
    h = s;
  }
  const double y = 1.0 / h;
  // residual of y (h + l) - 1 in extended precision
  const double r = __fma_rn(-y, h, 1.0) - y * l;
  return __fma_rn(y, r, y);
}

struct TcTravCounters {
  unsigned long long frontier[3];  // rotating frontier sizes
  unsigned long long n_m2l, n_p2p;
};

__device__ __forceinline__ unsigned long long tc_warp_append(unsigned long long* counter, bool want) {
  unsigned mask = __ballot_sync(0xffffffffu, want);
  if (!mask) return 0;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(mask & ((1u << lane) - 1u));
}

__global__ void k_trav_init(int2* frontier, TcTravCounters* cnt) {
  if (threadIdx.x || blockIdx.x) return;
  frontier[0] = make_int2(0, 0);
  cnt->frontier[0] = 1;
  cnt->frontier[1] = 0;
  cnt->frontier[2] = 0;
  cnt->n_m2l = 0;
  cnt->n_p2p = 0;
}

// step s reads frontier slot s%3, writes slot (s+1)%3 and clears slot (s+2)%3
__global__ void k_trav_step(int s, const int2* __restrict__ fin, int2* __restrict__ fout, unsigned long long fcap,
                            TcTravCounters* cnt, const TcCells c, double theta2, int top_variant, int sbits,
                            unsigned long long* __restrict__ m2l, unsigned long long m2l_cap,
                            unsigned long long* __restrict__ p2p, unsigned long long p2p_cap, unsigned int* err,
                            int* __restrict__ m2l_cnt, int* __restrict__ p2p_cnt, bool ranked,
                            const TcMac mac = TcMac()) {
  unsigned long long nin = cnt->frontier[s % 3];
  if (nin > fcap) nin = fcap;  // an overflowed step was flagged; never read past the buffer
  if (blockIdx.x == 0 && threadIdx.x == 0) cnt->frontier[(s + 2) % 3] = 0;
  unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long nround = (nin + stride - 1) / stride * stride;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < nround; k += stride) {
    bool valid = k < nin;
    int i = 0, j = 0;
    int act = -1;  // 0 m2l, 1 p2p, 2 split i, 3 split j
    if (valid) {
      int2 pr = fin[k];
      i = pr.x;
      j = pr.y;
      double dx = c.X[i] - c.X[j], dy = c.Y[i] - c.Y[j], dz = c.Z[i] - c.Z[j];
      double rs = c.R[i] + c.R[j];
      int nci = c.nchild[i], ncj = c.nchild[j];
      bool accept;
      if (mac.mode == 0) {
        double R2 = (dx * dx + dy * dy + dz * dz) * theta2;
        accept = R2 > rs * rs;
      } else if (mac.mode == 1) {
        accept = dx * dx + dy * dy + dz * dz > rs * rs * 3;
      } else if (mac.mode == 3) {
        // f2 only, pre-test |d|^2 0.4 > (Ra + Rb)^2; operation order and contractions of the
        // reference's x86-64 build (norm(): fma(dz, dz, fma(dx, dx, dy dy)); Eba += (Pn pa) comb
        // as one fma; R^-(P+1) correctly rounded)
        const double R2 = __fma_rn(dz, dz, __fma_rn(dx, dx, __dmul_rn(dy, dy)));
        double f2 = 10;
        const double Ra = c.R[i], Rb = c.R[j];
        if (__dmul_rn(R2, 0.4) > __dmul_rn(rs, rs)) {
          const int P = mac.p;
          const double Rp = tc_pow_neg_int(__dsqrt_rn(R2), P + 1);
          double pa = 1, Eba = 0;
          for (int k = 0; k <= P; k++) {
            Eba = __fma_rn(__dmul_rn(mac.pn[(size_t)j * (P + 1) + P - k], pa), mac.comb[k], Eba);
            pa = __dmul_rn(pa, Ra);
          }
          const double fac = __dmul_rn(__dmul_rn(8.0, fmax(Ra, Rb)), Rp);
          f2 = __ddiv_rn(__dmul_rn(fac, Eba), __dmul_rn(mac.min_acc[i], mac.fa));
        }
        accept = f2 < 1;
      } else {
        const double R2 = dx * dx + dy * dy + dz * dz;
        double f1 = 10, f2 = 10;
        const double Ra = c.R[i], Rb = c.R[j];
        if (R2 > rs * rs) {
          const double R = sqrt(R2);
          double Rp = R2, pa = 1, pb = 1, Eba = 0, Eab = 0;
          const int P = mac.p;
          for (int k = 0; k <= P; k++) {
            const double fac = mac.comb[k];
            Eab += mac.pn[(size_t)i * (P + 1) + P - k] * pb * fac;
            Eba += mac.pn[(size_t)j * (P + 1) + P - k] * pa * fac;
            pa *= Ra;
            pb *= Rb;
            Rp *= R;
          }
          const double fac = 8 * fmax(Ra, Rb) / rs / Rp;
          Eab *= fac;
          f1 = Eab / (mac.fa * mac.min_acc[j]);
          Eba *= fac;
          f2 = Eba / (mac.fa * mac.min_acc[i]);
        }
        accept = f2 < 1 && f1 < 1;
      }
      if (accept) {
        int ni = c.nbody[i], nj = c.nbody[j];
        act = (mac.mode != 1 && top_variant && ((ni <= 2 && nj <= 8) || (nj <= 2 && ni <= 8))) ? 1 : 0;
        if (mac.p2p_max > 0 && nci == 0 && (long long)ni * nj <= mac.p2p_max) act = 1;
      } else if (nci == 0 && ncj == 0) {
        act = 1;
      } else if (ncj == 0 || (c.R[i] >= c.R[j] && nci != 0)) {
        act = 2;
      } else {
        act = 3;
      }
    }
    // a pair's key: its rank among its target's pairs so far, target, source.  Keys that a radix sort orders
    // (trees of more than kListMaxCells cells) carry no rank: its passes are whole bytes, and the last one
    // would reach past bit 2 sbits into the rank.
    unsigned long long key = ((unsigned long long)(unsigned)i << sbits) | (unsigned)j;
    if (ranked) {
      // one atomic for all lanes of the warp with the same target and list (neighbours in the frontier
      // are children of one pair)
      const bool emit = act == 0 || act == 1;
      const unsigned lane = threadIdx.x & 31;
      const unsigned peers = __match_any_sync(0xffffffffu, emit ? 2u * (unsigned)i + (unsigned)act : 0xffffffffu);
      const int lead = __ffs(peers) - 1;
      int rank = 0;
      if (emit && (int)lane == lead) rank = atomicAdd(act == 0 ? m2l_cnt + i : p2p_cnt + i, __popc(peers));
      rank = __shfl_sync(0xffffffffu, rank, lead) + __popc(peers & ((1u << lane) - 1u));
      if (emit) key |= (unsigned long long)rank << (2 * sbits);
    }
    unsigned long long o = tc_warp_append(&cnt->n_m2l, act == 0);
    if (act == 0) {
      if (o < m2l_cap) m2l[o] = key; else tc_set_err(err, TC_EBIT_M2L_CAP);
    }
    o = tc_warp_append(&cnt->n_p2p, act == 1);
    if (act == 1) {
      if (o < p2p_cap) p2p[o] = key; else tc_set_err(err, TC_EBIT_P2P_CAP);
    }
    // children pairs: reserve per thread with one atomic per warp
    int nadd = act == 2 ? c.nchild[i] : act == 3 ? c.nchild[j] : 0;
    int incl = nadd;
    int lane = threadIdx.x & 31;
    for (int d = 1; d < 32; d <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total) base = atomicAdd(&cnt->frontier[(s + 1) % 3], (unsigned long long)total);
    base = __shfl_sync(0xffffffffu, base, 31) + (incl - nadd);
    if (nadd) {
      // what fits is written, so that the next step reads no slot below fcap that was never written
      if (base + nadd > fcap) tc_set_err(err, TC_EBIT_FRONTIER_CAP);
      const int nw = base >= fcap ? 0 : (int)min((unsigned long long)nadd, fcap - base);
      const int c0 = c.child[act == 2 ? i : j];
      for (int q = 0; q < nw; q++) fout[base + q] = act == 2 ? make_int2(c0 + q, j) : make_int2(i, c0 + q);
    }
  }
}

// ---------------------------------------------------------------------------------------
// Per-target source lists in source order.  The traversal counts each target's pairs and gives every
// pair its rank, so after a scan of the counts (excl_scan) one pass moves each source to its target's
// segment (k_list_scatter); a segment is then put in order through a bitmap of the cells (a target
// meets a source once): set its sources' bits, read the bits out.  Bound by the L2 and by the latency of a
// CTA's few loads (N = 4M: 5.8 of the traversal's 14.2 ms); radix-sorting the 8-byte (target, source) keys takes
// three to five passes over each list (11.5 of 20 ms there, 0.45 of 1.1 ms at N = 12,345).
// (ndev, ncdev optional: counts on the device for device-sized launches; n is then the capacity.)
// ---------------------------------------------------------------------------------------
// Larger trees are radix-sorted.  A CTA of k_list_order holds a bit per cell, so their CTAs get few (16 an SM
// up to 96,000 cells, 4 at 400,000, one from 840,000 on) while the sort's time follows the pairs alone.
// Traversal with the lists in order, bitmaps against sort (ms; p = 4, theta = 0.5): 106,000 cells 2.0 / 2.6,
// 237,000 5.4 / 6.7, 319,000 11.5 / 14.5, 412,000 9.0 / 9.1, 452,000 13.2 / 12.9, 593,000 7.7 / 5.1,
// 849,000 38.9 / 18.4, 1,481,000 33.7 / 12.7.
constexpr int kListMaxCells = 416 << 10;
// shared memory of k_list_order for `cells` cells: the bits, and two counters per block of 1,024
__host__ __device__ constexpr int tc_list_blocks(int cells) { return (cells + 1023) >> 10; }
constexpr size_t tc_list_bytes(int cells) { return (size_t)tc_list_blocks(cells) * (128 + 8); }

// cells: cells that the bitmap of k_list_order covers.  Where a replay's list or tree has outgrown what it
// was planned for (flagged; the host redoes it), every list is made empty, so that what follows in the
// graph reads no entry that was never written.
__global__ void k_list_scatter(const unsigned long long* __restrict__ keys, unsigned long long n, int ncell, int cells,
                               int sbits, int* __restrict__ tgt_start, int* __restrict__ src, unsigned int* err,
                               const unsigned long long* ndev = nullptr, const int* ncdev = nullptr) {
  if (ncdev) ncell = *ncdev;
  if (ncell > cells || (ndev && *ndev > n)) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= ncell; i += gridDim.x * blockDim.x) tgt_start[i] = 0;
    if (ncell > cells && blockIdx.x == 0 && threadIdx.x == 0) tc_set_err(err, TC_EBIT_CELL_CAP);
    return;
  }
  if (ndev) n = *ndev;
  const unsigned long long mask = (1ull << sbits) - 1ull;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long key = keys[k];
    src[tgt_start[(key >> sbits) & mask] + (int)(key >> (2 * sbits))] = (int)(key & mask);
  }
}

constexpr int kListThreads = 128;
// One CTA per target: its segment of src put in ascending order.  A source's place is the number of set
// bits below it: the counts of the blocks of 1,024 cells before its own, the words of its block before its
// own, and the bits of its word (reading out the whole bitmap instead took 5 ms a list at N = 4M).  Lists
// longer than kListHeld entries a thread read it out.
constexpr int kListHeld = 8;
__global__ void __launch_bounds__(kListThreads) k_list_order(int ncell, int cells, const int* __restrict__ tgt_start,
                                                             int* __restrict__ src, const int* ncdev = nullptr) {
  extern __shared__ uint32_t tc_list_bits[];  // a bit for each of `cells` cells, then the block counts and sums
  __shared__ int wsum[kListThreads / 32];
  if (ncdev) ncell = *ncdev;
  if (ncell > cells) return;  // the lists are empty
  const int nblk = tc_list_blocks(ncell), words = 32 * nblk, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* cnt = reinterpret_cast<int*>(tc_list_bits + 32 * tc_list_blocks(cells));
  int* pre = cnt + tc_list_blocks(cells);
  for (int i = threadIdx.x; i < words; i += kListThreads) tc_list_bits[i] = 0u;
  for (int i = threadIdx.x; i < nblk; i += kListThreads) cnt[i] = 0;
  // exclusive sum over the threads of n (every thread takes part)
  auto before = [&](int n) {
    int incl = n;
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int at = incl - n;
    for (int i = 0; i < w; i++) at += wsum[i];
    return at;
  };
  for (int t = blockIdx.x; t < ncell; t += gridDim.x) {
    const int b = tgt_start[t], e = tgt_start[t + 1];
    if (e - b < 2) continue;
    __syncthreads();  // bits and counts are clear, wsum is free
    if (e - b <= kListHeld * kListThreads) {
      int v[kListHeld];
#pragma unroll
      for (int h = 0; h < kListHeld; h++) {
        const int k = b + h * kListThreads + threadIdx.x;
        v[h] = k < e ? src[k] : -1;
        if (v[h] >= 0) {
          atomicOr(&tc_list_bits[v[h] >> 5], 1u << (v[h] & 31));
          atomicAdd(&cnt[v[h] >> 10], 1);
        }
      }
      __syncthreads();
      const int per = (nblk + kListThreads - 1) / kListThreads, i0 = threadIdx.x * per, i1 = min(nblk, i0 + per);
      int n = 0;
      for (int i = i0; i < i1; i++) n += cnt[i];
      int at = before(n);
      for (int i = i0; i < i1; i++) {
        pre[i] = at;
        at += cnt[i];
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < kListHeld; h++) {
        if (v[h] < 0) continue;
        int rank = pre[v[h] >> 10];
        for (int i = v[h] >> 10 << 5; i < v[h] >> 5; i++) rank += __popc(tc_list_bits[i]);
        rank += __popc(tc_list_bits[v[h] >> 5] & ((1u << (v[h] & 31)) - 1u));
        src[b + rank] = v[h];
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < kListHeld; h++)
        if (v[h] >= 0) {
          tc_list_bits[v[h] >> 5] = 0u;
          cnt[v[h] >> 10] = 0;
        }
    } else {
      const int per = words / kListThreads + 1;  // consecutive words a thread reads out
      for (int k = b + threadIdx.x; k < e; k += kListThreads) {
        const int s = src[k];
        atomicOr(&tc_list_bits[s >> 5], 1u << (s & 31));
      }
      __syncthreads();
      const int w0 = min(words, (int)threadIdx.x * per), w1 = min(words, w0 + per);
      int n = 0;
      for (int i = w0; i < w1; i++) n += __popc(tc_list_bits[i]);
      int at = b + before(n);
      for (int i = w0; i < w1; i++) {
        uint32_t m = tc_list_bits[i];
        if (!m) continue;
        tc_list_bits[i] = 0u;
        for (; m; m &= m - 1) src[at++] = 32 * i + __ffs(m) - 1;
      }
    }
  }
}

// (target << sbits | source) keys, sorted (trees of more than kListMaxCells cells): per-target offsets
__global__ void k_list_csr(const unsigned long long* __restrict__ keys, unsigned long long n, int ncell, int sbits,
                           int* __restrict__ tgt_start, int* __restrict__ src,
                           const unsigned long long* ndev = nullptr, const int* ncdev = nullptr) {
  if (ndev && *ndev < n) n = *ndev;
  if (ncdev) ncell = *ncdev;
  const unsigned long long smask = (1ull << sbits) - 1ull;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long key = keys[k];
    int t = (int)(key >> sbits);
    src[k] = (int)(key & smask);
    int tp = k == 0 ? -1 : (int)(keys[k - 1] >> sbits);
    for (int q = tp + 1; q <= t; q++) tgt_start[q] = (int)k;
    if (k == n - 1)
      for (int q = t + 1; q <= ncell; q++) tgt_start[q] = (int)n;
  }
  if (n == 0 && blockIdx.x == 0)
    for (int q = threadIdx.x; q <= ncell; q += blockDim.x) tgt_start[q] = 0;
}

// compact list of targets that have at least one entry
__global__ void k_list_targets(const int* __restrict__ tgt_start, int ncell, int* __restrict__ tlist,
                               unsigned int* __restrict__ ntl, const int* ncdev = nullptr) {
  if (ncdev) ncell = *ncdev;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool has = i < ncell && tgt_start[i + 1] > tgt_start[i];
  unsigned mask = __ballot_sync(0xffffffffu, has);
  int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (lane == 0 && mask) base = atomicAdd(ntl, (unsigned)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (has) tlist[base + __popc(mask & ((1u << lane) - 1u))] = i;
}

}  // namespace tc
