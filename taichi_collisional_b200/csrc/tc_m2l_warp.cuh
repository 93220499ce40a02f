// Rotation M2L in FP64, one warp per target: the form of systems with many targets (tc_m2l_by_warp).
//
// The operator of tc_m2l.cuh (rotate about z, swap, rotate about x, swap, translate along z and
// back), arranged around what bounds it on this GPU, the instruction supply.  Unrolled in registers,
// the code of all degrees is some 130 KB at order 12; schedulers whose warps run different degrees
// fetch all of it for every batch of pairs (a kernel of 49 KB of such code waits for instructions
// 0.2 cycles per issue, one of 74 KB 3.8, one of 185 KB 12).  So:
//   - every warp runs all degrees of its own 32 pairs (a lane per pair), and the warps of the CTA go
//     through the code together, meeting once per half: one fetch serves 4 to 16 batches (waiting for
//     instructions vanishes; meeting after every second degree costs 6 % more in barriers);
//   - a pair's translation then stays in its lane: the exchange rows are private to the lane, and no
//     barrier protects them;
//   - the z-translation of an order-Q M2L joins the orders m <= min(n, Q - n) of degree n only, so the
//     second forward swap produces, and the first backward swap reads, just those (285 instead of 737
//     coefficients each at Q = 12), and 85 instead of 169 rows are exchanged;
//   - r^-k enters the exchanged values and r^-(n+1) the translated ones, which leaves one FMA with a
//     literal per term of the translation;
//   - the source expansions are read from a copy made once per evaluation (k_m2l_pack), already scaled
//     by (n+|m|)!(n-|m|)! and with every degree on a 32-byte boundary: a lane reads whole sectors with
//     32-byte loads, a degree ahead of their use (the natural layout took one 8-byte load per
//     coefficient, each touching 32 cache lines);
//   - the lanes' sums accumulate in tensor memory, folded once across the half-warps so that two
//     to four warps share a lane quarter; the next target is looked up a load at a time behind the work.
// Per pair and expansion 5,050 FP64 lane-operations at Q = 12 against 7,100; nothing is spilled.
// Measured (M2L of both expansions, ms, tc_m2l.cuh's form -> this one; N = 131,072 unless stated):
// p = 4 1.01 -> 0.78, 6 1.82 -> 1.47, 8 2.84 -> 2.27, 10 4.27 -> 3.69, 12 6.45 -> 4.70, 16 27.1 -> 19.5;
// N = 4M with per-pair orders 153 -> 105.  FP64 pipe 46 % at p = 12: two warps a scheduler (shared
// memory holds no more exchange rows) leave dependent-issue latency uncovered.
#pragma once
#include "tc_m2l.cuh"

namespace tc {

// When a target gets a warp.  A work item is one expansion of one target, about n / ncrit targets; with few
// items the warps end unevenly, and k_m2l's four warps per batch of pairs finish sooner, the more so at low
// orders, where an item is short.  M2L time of this form over that of k_m2l (98,304 to 2M bodies, ncrit 32 to
// 256):
//   theta criterion    items      768          1,536        3,072        12,500
//                      p =  8     1.12 - 1.30  0.86 - 0.95  0.71 - 0.82  0.62 - 0.74
//                      p = 10     1.04 - 1.18  0.92 - 0.98  0.82 - 0.89  0.73 - 0.83
//                      p = 12     0.90 - 1.02  0.81 - 0.88  0.69 - 0.75  0.62 - 0.71
//                      p = 16     0.85         0.79 - 0.80  0.70 - 0.77  0.66 - 0.73   (384: 0.91)
// The error-controlled criterion gives a few outlying targets lists many times the others', which one warp
// walks alone; in the top tree that costs more items,
//                      items      1,536        3,072        4,096        12,500
//                      p =  8     1.10         1.06 - 1.18  0.85         0.79
//                      p = 10     1.58         1.02 - 1.24  0.91         0.81
//                      p = 12     1.21         0.73 - 0.90  0.71         0.67
// and in the jerks tree this form is no faster at any size measured up to p = 10 (0.94 to 1.39 up to 31,000
// items) but from p = 12 on (0.62 to 1.08).  Below 98,304 bodies k_m2l stays; there the items would decide
// alike (65,537 bodies with jerks, ncrit 64: p = 8 0.85, p = 12 0.79; ncrit 256: p = 10 1.37).
constexpr int kM2LWarpN = 98304;
inline bool tc_m2l_by_warp(int n, int ncrit, int p, bool jerk, bool emac) {
  if (n < kM2LWarpN) return false;
  const long long items = (long long)n * (jerk ? 2 : 1) / ncrit;
  if (emac) return p >= 12 ? jerk || items >= 3072 : !jerk && items >= 4096;
  return items >= (p >= 16 ? 384 : p >= 12 ? 768 : 1536);
}

// ---- packed source expansions: degree d at tc_pk_off(d), (2 d + 1) rounded up to 4 doubles
__host__ __device__ constexpr int tc_pk_width(int d) { return (2 * d + 1 + 3) / 4 * 4; }
__host__ __device__ constexpr int tc_pk_off(int d) {
  int o = 0;
  for (int k = 0; k < d; k++) o += tc_pk_width(k);
  return o;
}

// M (and Mdot) -> the packed, scaled copy, NA expansions per cell.  The reference's factorial table
// stops at (2P - 1)! (kernel_fast_lean.h:127), so the scaled (P, +-P) entries are zero.
template <int P, int NA>
__global__ void __launch_bounds__(256) k_m2l_pack(int ncell, const double* __restrict__ M,
                                                  const double* __restrict__ Md, double* __restrict__ out,
                                                  const int* ncdev = nullptr) {
  constexpr int NT = (P + 1) * (P + 1), NP = tc_pk_off(P + 1);
  __shared__ int nat[NP];
  for (int i = threadIdx.x; i < NP; i += blockDim.x) {
    int d = 0;
    while (tc_pk_off(d + 1) <= i) d++;
    const int k = i - tc_pk_off(d);
    nat[i] = k < 2 * d + 1 && !(d == P && (k == 0 || k == 2 * P)) ? d * d + k : -1;
  }
  __syncthreads();
  if (ncdev) ncell = *ncdev;  // device-sized launch (graph)
  const int lane = threadIdx.x & 31, nw = gridDim.x * 8;
  for (int c = blockIdx.x * 8 + (threadIdx.x >> 5); c < ncell; c += nw) {
    double* o = out + (size_t)c * NA * NP;
    for (int i = lane; i < NP; i += 32) {
      const int k = nat[i];
      const double f = k >= 0 ? c_fc[k] : 0.0;
      o[i] = k >= 0 ? M[(size_t)c * NT + k] * f : 0.0;
      if (NA == 2) o[NP + i] = k >= 0 ? Md[(size_t)c * NT + k] * f : 0.0;
    }
  }
}

// 4 consecutive doubles (32-byte aligned), read-only
__device__ __forceinline__ void tc_ld4(const double* p, double* v) {
  asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// warps per CTA: as many as the exchange rows in shared memory, the accumulators in tensor memory and
// the registers of the largest degree leave room for
template <int Q> struct TcWarps { static constexpr int N = Q <= 8 ? 16 : Q <= 10 ? 12 : Q <= 12 ? 8 : 4; };

template <int Q>
struct TcM2LW {
  static constexpr int NW = TcWarps<Q>::N, THREADS = 32 * NW;
  // exchange rows: orders |m| <= min(k, Q - k) of degree k
  __host__ __device__ static constexpr int R(int k) { return k < Q - k ? k : Q - k; }
  __host__ __device__ static constexpr int row(int k) {
    int r = 0;
    for (int j = 0; j < k; j++) r += 2 * R(j) + 1;
    return r;
  }
  static constexpr int ROWS = row(Q + 1);
  // per warp: the exchange rows, and for the current and the next item the target's centre (3 of 32) and
  // the pairs' source centres
  static constexpr int PAIR = 2 * 4 * 32;
  static constexpr size_t BYTES = (size_t)NW * (ROWS * 32 + PAIR) * sizeof(double);
  // accumulators: lanes 0-15 hold the coefficients 0 .. d of degree d, lanes 16-31 the others; degree
  // d's d + 1 doubles start on a multiple of 8 columns
  __host__ __device__ static constexpr int col(int d) {
    int c = 0;
    for (int k = 0; k < d; k++) c += (2 * (k + 1) + 7) / 8 * 8;
    return c;
  }
  static constexpr int CW = col(Q + 1);  // columns per warp
  static constexpr int TOTAL = CW * ((NW + 3) / 4);
  static constexpr int ALLOC = TOTAL <= 32 ? 32 : TOTAL <= 64 ? 64 : TOTAL <= 128 ? 128 : TOTAL <= 256 ? 256 : 512;
  static_assert(TOTAL <= 512, "M2L accumulators exceed tensor memory");
};

// first slot (double) of degree d's accumulators
__host__ __device__ constexpr int tc_m2lw_slot0(int d) {
  int c = 0;
  for (int k = 0; k < d; k++) c += (2 * (k + 1) + 7) / 8 * 4;
  return c;
}

// n! as a literal of the code: read from constant memory, the compiler may move all of them out of the
// batch loop and spill them
__host__ __device__ constexpr double tc_cfact(int n) {
  double f = 1.0;
  for (int i = 2; i <= n; i++) f *= (double)i;
  return f;
}

// what a pair's work needs besides its registers
struct TcM2LPair {
  const double* Mp;  // packed source expansion
  double* rows;      // this lane's exchange rows, 32 doubles apart
  cd ez, ex;
  double rinv;
  int qb, lane;
  uint32_t tm;  // the warp's accumulators
  bool have, valid, first;
};

// x^E by repeated squaring
template <int E>
__device__ __forceinline__ double tc_powi(double x) {
  if constexpr (E == 0) return 1.0;
  else if constexpr (E == 1) return x;
  else if constexpr (E % 2 == 0) return tc_powi<E / 2>(x * x);
  else return x * tc_powi<E / 2>(x * x);
}

// 8 bytes from global to shared memory without a register
__device__ __forceinline__ void tc_cp8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void tc_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// forward half: degree D of the source (loaded in v), rotated into the pair frame, unscaled, times
// r^-D, to the exchange rows.  The next degree's loads go first; below degree 5 they are all issued at
// once (v then holds the degrees 0 .. D).  A warp without work loads too (the first cell): behind a branch
// the compiler spills a third of the registers.
template <int Q, int D>
__device__ __forceinline__ void tc_m2lw_fwd(const TcM2LPair& g, double* v) {
  using W = TcM2LW<Q>;
  constexpr int K = 2 * D + 1, R = W::R(D), SMALL = 4;
  constexpr int PN = D > SMALL + 1 ? tc_pk_width(D - 1) : tc_pk_off(D);  // what the next degree's v holds
  double next[PN > 0 && D > SMALL ? PN : 1], o[K];
  if constexpr (D > SMALL) {
#pragma unroll
    for (int k = 0; k < PN; k += 4) tc_ld4(g.Mp + (D > SMALL + 1 ? tc_pk_off(D - 1) : 0) + k, next + k);
  }
  if (g.have && D <= g.qb) {
    double* u = D > SMALL ? v : v + tc_pk_off(D);
    tc_rot_fwd<D>(u, g.ez);
    TcSwapPart<D>::template apply<D, D>(u, o);
    tc_rot_fwd<D>(o, g.ex);
    TcSwapPart<D>::template apply<D, R>(o, u);
    const double rk = tc_powi<D>(g.rinv);
#pragma unroll
    for (int m = -R; m <= R; m++)
      g.rows[(W::row(D) + R + m) * 32] = u[D + m] * (rk * (1.0 / (tc_cfact(D + m) * tc_cfact(D - m))));
  }
  if constexpr (D > 0) {
    tc_m2lw_fwd<Q, D - 1>(g, D > SMALL ? next : v);
  }
}

// N doubles of this lane's accumulators, 8 columns at a time
template <int N>
__device__ __forceinline__ void tc_tm_ld8(uint32_t ta, uint32_t* r) {
#pragma unroll
  for (int c = 0; c + 8 <= 2 * N; c += 8) tc_tm_ld_chunk<8>(ta + c, r + c);
  tc_tm_ld<(2 * N) % 8>(ta + 2 * N / 8 * 8, r + 2 * N / 8 * 8);
}
template <int N>
__device__ __forceinline__ void tc_tm_st8(uint32_t ta, const uint32_t* r) {
#pragma unroll
  for (int c = 0; c + 8 <= 2 * N; c += 8) tc_tm_st_chunk<8>(ta + c, r + c);
  tc_tm_st<(2 * N) % 8>(ta + 2 * N / 8 * 8, r + 2 * N / 8 * 8);
}

// the first degree(s) of a packed expansion that the forward half runs (degrees up to 4 come together)
template <int Q>
struct TcM2LFirst {
  static constexpr int OFF = Q > 4 ? tc_pk_off(Q) : 0, N = tc_pk_off(Q + 1) - OFF;
  static __device__ __forceinline__ void load(const double* Mp, double* v) {
#pragma unroll
    for (int k = 0; k < N; k += 4) tc_ld4(Mp + OFF + k, v + k);
  }
};

// backward half: z-translation to output degree N (terms n + k <= qb), rotated back, added to the
// warp's accumulators (read before the arithmetic that hides it)
template <int Q, int N>
__device__ __forceinline__ void tc_m2lw_back(const TcM2LPair& g, const double* nextMp, double* vQ) {
  using W = TcM2LW<Q>;
  constexpr int K = 2 * N + 1, R = W::R(N);
  if constexpr (N == 2) TcM2LFirst<Q>::load(nextMp, vQ);  // the next batch's, behind the small degrees
  // a target's first batch stores every degree, so that no cleared accumulators are needed
  if (g.have && (N <= g.qb || g.first)) {
    uint32_t r[2 * (N + 1)];
    double l[K], o[K + 1], t[N + 1];
    tc_tm_ld8<N + 1>(g.tm + W::col(N), r);
#pragma unroll
    for (int k = 0; k < K; k++) l[k] = 0.0;
#pragma unroll
    for (int k = 0; k <= Q - N; k++) {
      if (k > g.qb - N) break;
      const double* p = g.rows + (W::row(k) + W::R(k)) * 32;
#pragma unroll
      for (int m = -(k < R ? k : R); m <= (k < R ? k : R); m++) l[N + m] = fma(p[m * 32], tc_cfact(N + k), l[N + m]);
    }
    // (-1)^m r^-(N+1); a lane past the list carries a copy of its first pair and adds nothing
    const double f = g.valid ? tc_powi<N + 1>(g.rinv) : 0.0;
#pragma unroll
    for (int m = -R; m <= R; m++) l[N + m] *= (m & 1) ? -f : f;
    TcSwapPart<N>::template apply<R, N>(l, o);
    tc_rot_inv<N>(o, g.ex);
    TcSwapPart<N>::template apply<N, N>(o, l);
    tc_rot_inv<N>(l, g.ez);
    // fold the half-warps: lanes 0-15 keep the coefficients 0 .. N, lanes 16-31 the others
    const bool up = g.lane & 16;
#pragma unroll
    for (int j = 0; j <= N; j++) {
      const double hi = j + N + 1 < K ? l[j + N + 1 < K ? j + N + 1 : 0] : 0.0;
      const double send = up ? l[j] : hi, keep = up ? hi : l[j];
      o[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
    tc_tm_wait_ld();
    tc_tm_to_f64<N + 1>(r, t);
#pragma unroll
    for (int k = 0; k <= N; k++) {
      const double x = g.first ? o[k] : t[k] + o[k];
      r[2 * k] = (uint32_t)__double2loint(x);
      r[2 * k + 1] = (uint32_t)__double2hiint(x);
    }
    tc_tm_st8<N + 1>(g.tm + W::col(N), r);
  }
  if constexpr (N > 0) {
    tc_m2lw_back<Q, N - 1>(g, nextMp, vQ);
  }
}

// The accumulators summed over the lanes and added to the target's local: 16 doubles at a time, four
// halving steps over the 16 lanes leave each lane the sum of one of them.  slot[s]: degree of slot s.
template <int Q>
__device__ __forceinline__ void tc_m2lw_readout(uint32_t tm, const signed char* slot, double* __restrict__ Lt,
                                                int lane) {
#pragma unroll 1
  for (int c = 0; c < TcM2LW<Q>::CW; c += 32) {
    uint32_t r[32];
    double v[16];
#pragma unroll
    for (int k = 0; k < 32; k++) r[k] = 0u;
#pragma unroll
    for (int k = 0; k < 32; k += 8)
      if (c + k < TcM2LW<Q>::CW) tc_tm_ld_chunk<8>(tm + c + k, r + k);
    tc_tm_wait_ld();
    tc_tm_to_f64<16>(r, v);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int j = 0; j < o; j++) {
        const double send = up ? v[j] : v[j + o], keep = up ? v[j + o] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int s = c / 2 + (lane & 15), n = slot[s];
    if (n >= 0) {
      const int j = s - tc_m2lw_slot0(n), k = j + (lane & 16 ? n + 1 : 0);
      if (j <= n && k < 2 * n + 1) atomicAdd(&Lt[n * n + k], v[0]);  // one adder: nothing else writes it now
    }
  }
}

// M2L of order Q over a per-target list (or, with `tend`, one order class's range of it): work item k is
// the expansion k % na (M, Mdot) of target k / na, handed out by `next` (zeroed before the launch);
// adds into L and Ldot, ntp doubles per cell.  np: doubles of a packed expansion.  One CTA per SM,
// which owns the tensor memory it allocates.
template <int Q>
__global__ void __launch_bounds__(TcM2LW<Q>::THREADS, 1)
    k_m2l_warp(const int* __restrict__ tlist, int ntl, const int* __restrict__ tstart, const int* __restrict__ src,
               TcCells c, const double* __restrict__ Mp, int na, int np, int ntp, unsigned* next,
               const unsigned* ntldev, const int* __restrict__ tend) {
  using W = TcM2LW<Q>;
  extern __shared__ __align__(16) unsigned char tc_m2lw_smem[];
  __shared__ uint32_t s_tmem;
  __shared__ signed char s_slot[(W::CW + 31) / 32 * 16];  // degree of an accumulator slot, -1: none
  if (ntldev) ntl = (int)*ntldev;  // device-sized launch (graph)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < (W::CW + 31) / 32 * 16; i += blockDim.x) {
    int d = 0;
    while (d <= Q && tc_m2lw_slot0(d + 1) <= i) d++;
    s_slot[i] = (signed char)(d <= Q ? d : -1);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(&s_tmem)),
                 "r"(W::ALLOC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  TcM2LPair g;
  g.lane = lane;
  // this warp's columns in the lane quarter it may access
  g.tm = s_tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * W::CW);
  double* const sw = reinterpret_cast<double*>(tc_m2lw_smem) + (size_t)warp * (W::ROWS * 32 + W::PAIR);
  g.rows = sw + W::PAIR + lane;
  g.have = false;
  // The next item with work (its target, list range and first pairs) is looked up one load at a time,
  // a step per batch, each step using what the one before asked for: 5 = ready, 6 = no more items.
  const unsigned nitem = (unsigned)ntl * na;
  int stage = 0, nt = 0, nbeg = 0, nend = 0, nsv = 0;
  unsigned nk = 0;
  int ib = 0;  // which of the two pair areas is the current item's
  auto centres = [&](int a, int sv) {  // source centres of the lanes' pairs -> area a
    double* p = sw + a * 128 + 32 + lane;
    const int s = sv & kM2LSrcMask;
    tc_cp8(p, c.X + s);
    tc_cp8(p + 32, c.Y + s);
    tc_cp8(p + 64, c.Z + s);
  };
  auto look = [&]() {
    if (stage == 0) {
      if (lane == 0) nk = atomicAdd(next, 1u);
      stage = 1;
    } else if (stage == 1) {
      nk = __shfl_sync(0xffffffffu, nk, 0);
      stage = nk < nitem ? 2 : 6;
      if (stage == 2) nt = tlist[nk / na];
    } else if (stage == 2) {
      nbeg = tstart[nt];
      nend = tend ? tend[nt] : tstart[nt + 1];
      if (!c.has_sink[nt]) nend = nbeg;
      stage = 3;
    } else if (stage == 3) {
      stage = nend > nbeg ? 4 : 0;
      if (stage == 4) {
        nsv = src[nbeg + lane < nend ? nbeg + lane : nbeg];
        if (lane < 3) tc_cp8(sw + (ib ^ 1) * 128 + lane, (lane == 0 ? c.X : lane == 1 ? c.Y : c.Z) + nt);
      }
    } else if (stage == 4) {
      centres(ib ^ 1, nsv);
      stage = 5;
    }
  };
  int t = 0, arr = 0, s_beg = 0, s_end = 0, b0 = 0, sv = 0;
  auto packed = [&](int sv, int a) { return Mp + ((size_t)(sv & kM2LSrcMask) * na + a) * np; };
  while (stage < 5) look();
  double vQ[TcM2LFirst<Q>::N];
  TcM2LFirst<Q>::load(stage == 5 ? packed(nsv, (int)(nk % na)) : Mp, vQ);
  for (;;) {
    if (!g.have) {
      if (stage == 5) {
        g.have = true;
        t = nt; arr = (int)(nk % na); s_beg = b0 = nbeg; s_end = nend; sv = nsv;
        ib ^= 1;
        g.first = true;
        stage = 0;
      }
    }
    if (!__syncthreads_or(g.have)) break;
    g.valid = b0 + lane < s_end;
    g.qb = Q;
    g.rinv = 0.0;
    g.ez = g.ex = mk(1, 0);
    g.Mp = Mp;
    if (g.have) g.Mp = packed(sv, arr);
    look();
    if (g.have) {
      // a source entry carries its pair's order below Q in its top bits; the batch runs at the largest
      // order of its pairs, a lower order never applied to a pair
      g.qb = Q - (int)__reduce_min_sync(0xffffffffu, g.valid ? (unsigned)sv >> kM2LOrderShift : 31u);
      tc_cp_wait();
      __syncwarp();
      const double* p = sw + ib * 128;
      const TcPairGeo pg = tc_pair_geo(p[0] - p[32 + lane], p[1] - p[64 + lane], p[2] - p[96 + lane]);
      g.ez = pg.ez1;
      g.ex = pg.ex1;
      g.rinv = pg.rinv;
    }
    const bool more = g.have && b0 + 32 < s_end;  // the next batch's pair, loaded behind this one's work
    if (more) sv = src[b0 + 32 + lane < s_end ? b0 + 32 + lane : s_beg];
    tc_m2lw_fwd<Q, Q>(g, vQ);
    if (more) centres(ib, sv);
    look();
    if (!more)
      while (stage < 5) look();
    __syncthreads();  // the warps meet between the halves (and at the top of the loop)
    if (g.have) tc_tm_wait_st();  // earlier accumulator stores
    tc_m2lw_back<Q, Q>(g, more ? packed(sv, arr) : stage == 5 ? packed(nsv, (int)(nk % na)) : Mp, vQ);
    b0 += 32;
    g.first = false;
    if (g.have && !more) {
      tc_tm_wait_st();
      tc_m2lw_readout<Q>(g.tm, s_slot, (arr ? c.Ld : c.L) + (size_t)t * ntp, lane);
      g.have = false;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(W::ALLOC) : "memory");
}

}  // namespace tc
