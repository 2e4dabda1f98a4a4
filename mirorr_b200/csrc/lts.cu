// lts.cu -- the least-trimmed-squares fit on the device.
//
// One launch runs the whole inner loop of OptimizeTransform (classic:
// itkMirorrRegistrationMethod.txx:785-999; symmetric:
// itkSymMirorrRegistrationMethod.txx:771-1442).  Per inner iteration:
//   residuals r_i (FP64) under the current final transform(s);
//   the threshold r_nth: the maximum on the first iteration, otherwise the
//     exact value of rank min(floor(f N), N-1) by a radix select on the
//     residual bit patterns (histograms over narrowing key ranges until at
//     most one CTA's worth of keys is left, then those keys ranked by counting);
//   subset {r_i <= r_nth}: count, first and second moments of the
//     (initial, moved) pairs about the first pair in one sweep, reduced per
//     CTA and summed in a fixed order (deterministic), then centred;
//   the FP64 solve (affine normal equations / Horn quaternion, symmetric
//     half-space algebra) in one warp, and the loop test.
//
// What bounds it is latency: a fit is some 2 to 60 dependent iterations of
// barriers, short passes over a few thousand to a few hundred thousand pairs
// and a serial solve.  So the CTAs of a fit of at most kClusterPairs pairs are
// one thread-block cluster, which meets at the hardware cluster barrier, and a
// batch runs one such cluster per fit; a larger fit spreads over a CTA per SM,
// which meet at a software grid barrier whose wait is bounded (about one
// second; a timeout raises an error flag and every CTA returns).  Per inner
// iteration of a rigid fit: 84K cycles with a software barrier over 2 to 16
// CTAs and the matrices of the solve in local memory, 36K now at 7,300 pairs;
// of a symmetric affine one at 590,000 pairs 150K, now 80K.
#include <mutex>

#include "gridsel.cuh"
#include "kernels.cuh"
#include "keyrange.cuh"

namespace mb2 {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = kKeyBins;
constexpr int kCandMax = kThreads;  // keys left for the final rank (one per thread)
constexpr int kRankMax = 96;  // keys ranked by counting without a further histogram
constexpr int kUnroll = 2;   // pairs a thread has in flight
constexpr int kPartial = 32;  // doubles per CTA partial
constexpr int kSums = 28;     // count, 6 first and 21 second moments
constexpr int kClusterCtas = 8;  // CTAs of a cluster (the portable limit)
// Pairs up to which one cluster is faster than a CTA per SM: an iteration
// (rigid) takes 36K cycles on a cluster at 7,500 pairs, 51K at 25,600 and 64K
// at 47,500, and about 46K on the whole GPU.
constexpr long long kClusterPairs = 16384;
// Pairs up to which one CTA of the cluster runs the fit alone, with the
// histogram, the residuals and the state in its shared memory and no global
// round trips (an iteration at 1,000 pairs 25K cycles against 35K on the
// cluster; equal at about 4,500).
constexpr long long kSinglePairs = 4096;
// Polls of a grid-barrier wait (about 0.84 s with the 100 ns back-off) before
// the wait gives up, raises the error flag and every CTA returns.
constexpr long long kDefaultSpinLimit = 1LL << 23;

struct LtsCtl {
  GridBar bar;
  unsigned long long maxkey;
  unsigned long long ncand;
};

struct LtsArgs {
  LtsState *state;
  const double *init;
  const double *moved;
  const long long *n_dev;
  double *resid;
  double *partial;        // kPartial per CTA: sum q of CTA b at q * CTAs + b
  unsigned int *hist;     // 3 * kBins
  unsigned long long *cand;
  LtsCtl *ctl;
  long long spin_limit;   // polls of a grid-barrier wait before it gives up
};

// How the CTAs of a fit meet.  A cluster's barrier orders their global writes
// at cluster scope and cannot time out (its CTAs are resident together and
// none leaves early).
struct GridSync {
  static constexpr bool single = false;
  LtsCtl *ctl;
  long long spin_limit;
  unsigned int nctas;
  unsigned int round;
  __device__ bool operator()() { return grid_barrier(&ctl->bar, round++, spin_limit, nctas); }
};
struct ClusterSync {
  static constexpr bool single = false;
  __device__ bool operator()() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::
                     : "memory");
    return true;
  }
};

struct SingleSync {
  static constexpr bool single = true;
  __device__ bool operator()() {
    __syncthreads();
    return true;
  }
};

__device__ inline void load_cg(void *dst, const void *src, int bytes) {
  const unsigned long long *s = static_cast<const unsigned long long *>(src);
  unsigned long long *d = static_cast<unsigned long long *>(dst);
  for (int i = threadIdx.x; i < bytes / 8; i += blockDim.x) d[i] = __ldcg(s + i);
}

// Sums each of v[0, kSums) over the CTA; out[q] in shared memory, valid for
// every thread on return.  Within a warp the values are summed by halving:
// at distance 16 a lane sends the half of its values that its partner keeps
// and adds what it gets, then 8, 4, 2, 1, after which lane l holds value l:
// 31 exchanges instead of the 140 of a shuffle tree per value (the shuffle
// unit was the bound).  Then the warps in order.
__device__ inline void block_sums(const double (&v)[kSums], double (*red)[kWarps], double *out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double x[32];
#pragma unroll
  for (int q = 0; q < 32; ++q) x[q] = q < kSums ? v[q] : 0.0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const bool up = (lane & d) != 0;
#pragma unroll
    for (int q = 0; q < d; ++q) {
      const double send = up ? x[q] : x[q + d];
      const double keep = up ? x[q + d] : x[q];
      x[q] = keep + __shfl_xor_sync(0xffffffffu, send, d);
    }
  }
  red[lane][wid] = x[0];
  __syncthreads();
  if (threadIdx.x < kSums) {
    double r = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) r += red[threadIdx.x][w];
    out[threadIdx.x] = r;
  }
  __syncthreads();
}

// out[q] = sum over the fit's CTAs b of part[q * nctas + b], q < kSums: warp
// q % kWarps takes value q, its lanes stride over b, then a shuffle tree (a
// fixed order).  out in shared memory, valid for every thread on return.
__device__ inline void grid_partial_sums(const double *part, double *out, int nctas) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int NQ = (kSums + kWarps - 1) / kWarps;
  double x[NQ];
#pragma unroll
  for (int j = 0; j < NQ; ++j) x[j] = 0.0;
  for (int b0 = lane; b0 < nctas; b0 += 4 * 32) {
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
      const int q = wid + j * kWarps;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int b = b0 + 32 * u;
        if (q < kSums && b < nctas) x[j] += __ldcg(&part[(long long)q * nctas + b]);
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int j = 0; j < NQ; ++j) x[j] += __shfl_down_sync(0xffffffffu, x[j], off);
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < NQ; ++j)
      if (wid + j * kWarps < kSums) out[wid + j * kWarps] = x[j];
  __syncthreads();
}

// Squared distance of the transformed initial point f(x) (matrix f[0..9),
// offset f[9..12)) from y, or from b(y) in the symmetric fit (tfm_apply's
// order of operations).
__device__ inline void apply_rows(const double (&f)[12], const double *x, double *o) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) v += f[3 * i + j] * x[j];
    o[i] = v + f[9 + i];
  }
}
__device__ inline double residual(const double (&f)[12], const double (&b)[12], bool symmetric,
                                  const double *x, const double *y) {
  double p[3], q[3];
  apply_rows(f, x, p);
  if (symmetric) {
    apply_rows(b, y, q);
  } else {
    q[0] = y[0]; q[1] = y[1]; q[2] = y[2];
  }
  double r = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double d = p[i] - q[i];
    r += d * d;
  }
  return r;
}

// f(key) for this thread's residuals' bit patterns, four loads in flight.
template <class F>
__device__ __forceinline__ void for_keys(const double *resid, long long n, long long first,
                                         long long stride, F f) {
  constexpr int U = 4;
  for (long long i0 = first; i0 < n; i0 += U * stride) {
    unsigned long long k[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      k[u] = (unsigned long long)__double_as_longlong(resid[i0 + u * stride < n ? i0 + u * stride : i0]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * stride < n) f(k[u]);
  }
}

// What the solve needs of the subset (shared memory).
struct Subset {
  double mean[6];  // barycentres of the initial and the moved points
  double Z[36];    // second moments about them
  double zn[36];   // Z divided by the subset's size
};

__device__ inline double other_half(double v) { return __shfl_xor_sync(0xffffffffu, v, 4); }

// The solve, by one whole warp.  Every lane runs it: the lanes of a quad hold
// the same values (each takes one of three angles where trigonometric
// functions come in threes), and in the symmetric fit odd quads hold the
// backward half and even quads the forward one.  Lane 0 (and lane 4) write s.
__device__ __noinline__ void solve_classic(LtsState &s, const Subset &m) {
  Tfm T = s.fin;
  double np[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) np[i] = 0.0;
  classic_fit(T, m.mean, m.mean + 3, m.Z, m.zn, np);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    s.fin = T;
    lts_delta(s, np);
  }
}

__device__ __noinline__ void solve_symmetric(LtsState &s, const Subset &m) {
  const int lane = threadIdx.x & 31, h = (lane >> 2) & 1;
  Tfm T = h ? s.finb : s.fin, iT;
  double np[12], inv[9], K[9], ot[3], m12[16];
#pragma unroll
  for (int i = 0; i < 12; ++i) np[i] = 0.0;
  sym_fit(T, h, m.mean, m.mean + 3, m.Z, m.zn, np, inv);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    K[i] = (T.M[i] + other_half(inv[i])) / 2.0;
    const double o = other_half(K[i]);
    if (T.kind == KIND_RIGID && h) K[i] = o;  // both halves take the forward mean
  }
  // (a backward half is left alone when the forward one rejects its matrix)
  const Tfm T0 = T;
  const bool took = sym_mean(T, h, K);
  __syncwarp();
  const unsigned ok = __ballot_sync(0xffffffffu, took);
  if (h && !(ok & 1u)) T = T0;
  sym_to_origin(T, iT);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 9; ++i) K[i] = other_half(iT.M[i]);
#pragma unroll
  for (int i = 0; i < 3; ++i) ot[i] = other_half(iT.t[i]);
  sym_half(T, K, ot, m12);
  __syncwarp();
  const Tfm T1 = T;
  const bool fin = sym_finish(T, m12, false);
  __syncwarp();
  if (!__all_sync(0xffffffffu, fin)) {
    T = T1;
    sym_finish(T, m12, true);
  }
  const double tr[3] = {m12[3], m12[7], m12[11]};
  tfm_set_translation(T, tr);
  __syncwarp();
  if (lane == 0) {
    s.fin = T;
    if ((ok & 0x11u) != 0x11u) s.failed = 1;
    lts_delta(s, np);
  } else if (lane == 4) {
    s.finb = T;
  }
  __syncwarp();
}

// The LTS loop run by `ncta` CTAs (index `cta` among them) that meet at `sync`.
// resid: one double per pair (global scratch; shared memory when one CTA runs
// the fit).
template <class Sync>
__device__ void lts_body(const LtsArgs &a, Sync sync, double *resid, int cta, int ncta) {
  constexpr bool kSingle = Sync::single;
  __shared__ __align__(16) LtsState s;
  __shared__ unsigned int h[kBins];
  __shared__ unsigned long long ck[kCandMax];
  __shared__ double red[32][kWarps];
  __shared__ double s_out[kSums];
  __shared__ Subset sub;
  __shared__ double s_nth;
  __shared__ unsigned long long s_key;
  __shared__ unsigned int s_left;  // keys gathered for the final rank
  __shared__ unsigned long long s_pair[2];
  const long long n = __ldcg(&a.n_dev[0]) + __ldcg(&a.n_dev[1]);
  const long long gstride = (long long)ncta * kThreads;
  const long long gtid = (long long)cta * kThreads + threadIdx.x;

  for (int guard = 0; guard < 200; ++guard) {
    if (!kSingle || guard == 0) load_cg(&s, a.state, sizeof(LtsState));
    for (int i = threadIdx.x; i < kBins; i += kThreads) h[i] = 0;
    if (kSingle && threadIdx.x == 0) {
      s_key = 0;
      s_left = 0;
    }
    if (!kSingle && cta == 0)
      for (int i = threadIdx.x; i < kBins; i += kThreads) a.hist[kBins + i] = 0;  // next pass's
    __syncthreads();
    if (!s.running || n <= 0) break;
    const bool first = s.fraction > 0.99999;
    // ---- residuals (+ max or first histogram) ----------------------------
    unsigned long long kmax = 0;
    // the transforms in registers (in shared memory they would be read again
    // for every pair)
    double ft[12], bt[12];
    const bool symmetric = s.symmetric != 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      ft[i] = i < 9 ? s.fin.M[i < 9 ? i : 0] : s.fin.off[i < 9 ? 0 : i - 9];
      bt[i] = i < 9 ? s.finb.M[i < 9 ? i : 0] : s.finb.off[i < 9 ? 0 : i - 9];
    }
    for (long long i0 = gtid; i0 < n; i0 += kUnroll * gstride) {
      // kUnroll pairs' loads are issued before the first is used
      double x[kUnroll][3], y[kUnroll][3];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const long long i = i0 + u * gstride < n ? i0 + u * gstride : i0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          x[u][c] = __ldcg(&a.init[3 * i + c]);
          y[u][c] = __ldcg(&a.moved[3 * i + c]);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (i0 + u * gstride >= n) break;
        const double r = residual(ft, bt, symmetric, x[u], y[u]);
        resid[i0 + u * gstride] = r;
        const unsigned long long key = (unsigned long long)__double_as_longlong(r);
        if (first) {
          if (key > kmax) kmax = key;
        } else {
          atomicAdd(&h[first_bin(key)], 1u);
        }
      }
    }
    if (first) {
      for (int off = 16; off > 0; off >>= 1) {
        unsigned long long o = __shfl_down_sync(0xffffffffu, kmax, off);
        if (o > kmax) kmax = o;
      }
      if ((threadIdx.x & 31) == 0 && kmax) atomicMax(kSingle ? &s_key : &a.ctl->maxkey, kmax);
    } else if (!kSingle) {
      __syncthreads();
      for (int i = threadIdx.x; i < kBins; i += kThreads)
        if (h[i]) atomicAdd(&a.hist[i], h[i]);
    }
    if (!sync()) return;
    double nth;
    if (first) {
      if (!kSingle) {
        if (threadIdx.x == 0) s_key = __ldcg(&a.ctl->maxkey);
        __syncthreads();
      }
      nth = __longlong_as_double((long long)s_key);
    } else {
      // ---- radix select of rank k ------------------------------------------
      unsigned long long k = (unsigned long long)(unsigned int)(s.fraction * (double)n);
      if (k > (unsigned long long)(n - 1)) k = n - 1;
      unsigned long long lo = 0, hi = 0;  // the keys left lie in [lo, hi]
      int shift = 0, pass = 0;
      while (true) {
        if (!kSingle) {
          // every CTA scans the global histogram of this pass identically
          const unsigned int *gh = a.hist + (pass % 3) * kBins;
          __syncthreads();
          for (int i = threadIdx.x; i < kBins; i += kThreads) h[i] = __ldcg(&gh[i]);
          __syncthreads();
        }
        int d = 0;
        unsigned long long cum = 0;
        find_bucket<kBins, kThreads>(h, k, kBins, s_pair, &d, &cum);
        const unsigned long long bucket = h[d];
        k -= cum;
        if (pass == 0) {
          first_range(d, lo, hi);
        } else {
          range_step(lo, hi, shift, d);
        }
        __syncthreads();
        if (bucket <= (unsigned long long)kCandMax || lo == hi) break;
        // more than one CTA's worth of keys is left: the next histogram, of
        // [lo, hi] in kBins steps
        ++pass;
        shift = range_shift(lo, hi);
        if (!kSingle && cta == 0) {
          unsigned int *zb = a.hist + ((pass + 1) % 3) * kBins;
          for (int i = threadIdx.x; i < kBins; i += kThreads) zb[i] = 0;
        }
        for (int i = threadIdx.x; i < kBins; i += kThreads) h[i] = 0;
        __syncthreads();
        for_keys(resid, n, gtid, gstride, [&](unsigned long long key) {
          if (key >= lo && key <= hi) atomicAdd(&h[(key - lo) >> shift], 1u);
        });
        if (!kSingle) {
          __syncthreads();
          unsigned int *gh2 = a.hist + (pass % 3) * kBins;
          for (int i = threadIdx.x; i < kBins; i += kThreads)
            if (h[i]) atomicAdd(&gh2[i], h[i]);
        }
        if (!sync()) return;
      }
      if (lo == hi) {
        nth = __longlong_as_double((long long)lo);  // the keys left are equal
      } else {
        // ---- gather the keys left (at most one per thread) and rank them
        for_keys(resid, n, gtid, gstride, [&](unsigned long long key) {
          if (key >= lo && key <= hi) {
            if (kSingle) {
              const unsigned int pos = atomicAdd(&s_left, 1u);
              if (pos < (unsigned int)kCandMax) ck[pos] = key;
            } else {
              const unsigned long long pos = atomicAdd(&a.ctl->ncand, 1ULL);
              if (pos < (unsigned long long)kCandMax) a.cand[pos] = key;
            }
          }
        });
        if (!sync()) return;
        unsigned long long mine;
        if (kSingle) {
          mine = ck[threadIdx.x];
          if (threadIdx.x == 0) s_key = s_left;
        } else {
          if (threadIdx.x == 0) s_key = __ldcg(&a.ctl->ncand);
          mine = __ldcg(&a.cand[threadIdx.x]);
        }
        __syncthreads();
        int nc = (int)(s_key < (unsigned long long)kCandMax ? s_key : kCandMax);
        bool have = threadIdx.x < nc;
        unsigned long long kk = k < (unsigned long long)nc ? k : (nc > 0 ? nc - 1 : 0);
        if (nc > kRankMax) {
          // one more histogram, of this CTA alone, so that few keys are ranked
          shift = range_shift(lo, hi);
          for (int i = threadIdx.x; i < kBins; i += kThreads) h[i] = 0;
          __syncthreads();
          if (have) atomicAdd(&h[(mine - lo) >> shift], 1u);
          __syncthreads();
          int d = 0;
          unsigned long long cum = 0;
          find_bucket<kBins, kThreads>(h, kk, kBins, s_pair, &d, &cum);
          kk -= cum;
          nc = (int)h[d];
          have = have && (int)((mine - lo) >> shift) == d;
          if (threadIdx.x == 0) s_pair[0] = 0;
          __syncthreads();
          if (have) ck[atomicAdd(&s_pair[0], 1ULL)] = mine;
        } else if (have) {
          ck[threadIdx.x] = mine;
        }
        __syncthreads();
        // rank by counting: key i has rank kk iff lo_i <= kk < lo_i + eq_i
        if (have) {
          const unsigned long long v = mine;
          int below = 0, eq = 0;
#pragma unroll 8
          for (int j = 0; j < nc; ++j) {
            const unsigned long long u = ck[j];
            below += u < v;
            eq += u == v;
          }
          if ((unsigned long long)below <= kk && kk < (unsigned long long)(below + eq))
            s_nth = __longlong_as_double((long long)v);
        }
        __syncthreads();
        nth = s_nth;
      }
    }
    // ---- subset moments in one sweep: count, first and second moments of
    // the pairs z = (initial, moved) about the first pair z0 (near the data,
    // so centring afterwards loses nothing in FP64) ------------------------
    double z0[6];
    for (int c = 0; c < 3; ++c) {
      z0[c] = __ldg(&a.init[c]);
      z0[3 + c] = __ldg(&a.moved[c]);
    }
    double acc[kSums];
#pragma unroll
    for (int q = 0; q < kSums; ++q) acc[q] = 0.0;
    for (long long i0 = gtid; i0 < n; i0 += kUnroll * gstride) {
      double z[kUnroll][6], r[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const long long i = i0 + u * gstride < n ? i0 + u * gstride : i0;
        r[u] = resid[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          z[u][c] = __ldcg(&a.init[3 * i + c]);
          z[u][3 + c] = __ldcg(&a.moved[3 * i + c]);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (i0 + u * gstride < n && r[u] <= nth) {
#pragma unroll
          for (int c = 0; c < 6; ++c) z[u][c] -= z0[c];
          acc[0] += 1.0;
#pragma unroll
          for (int p = 0; p < 6; ++p) acc[1 + p] += z[u][p];
          int q = 7;
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int c = p; c < 6; ++c) acc[q++] += z[u][p] * z[u][c];
        }
      }
    }
    block_sums(acc, red, s_out);
    if (!kSingle) {
      if (threadIdx.x < kSums) a.partial[(long long)threadIdx.x * ncta + cta] = s_out[threadIdx.x];
      if (!sync()) return;
    }
    if (cta == 0) {
      if (!kSingle) grid_partial_sums(a.partial, s_out, ncta);
      if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        const double cnt = s_out[0];
        // the moments about the barycentres, entry (r, c) of the upper
        // triangle by lane q
        double zz = 0.0;
        int r = 0, c = 0;
        if (l < 21) {
          int q = l;
          while (q >= 6 - r) { q -= 6 - r; ++r; }
          c = r + q;
          zz = s_out[7 + l] - cnt * (s_out[1 + r] / cnt) * (s_out[1 + c] / cnt);
          sub.Z[6 * r + c] = zz;
          sub.Z[6 * c + r] = zz;
          zz /= cnt;
          sub.zn[6 * r + c] = zz;
          sub.zn[6 * c + r] = zz;
        } else if (l < 27) {
          sub.mean[l - 21] =
              (l < 24 ? __ldg(&a.init[l - 21]) : __ldg(&a.moved[l - 24])) + s_out[1 + l - 21] / cnt;
        }
      }
      // (a CTA barrier, after which the solving warp is whole again: run by its
      // lane groups one after another, a solve took three times as long)
      __syncthreads();
      if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        if (s.symmetric) solve_symmetric(s, sub);
        else solve_classic(s, sub);
        __syncwarp();
        if (l == 0) {
          s.fraction = s.lts_keep;
          s.iter += 1;
          s.running = lts_continue(s) ? 1 : 0;
          if (s.iter > 101) s.running = 0;
          if (!kSingle) {  // reset select scratch for the next iteration
            a.ctl->maxkey = 0;
            a.ctl->ncand = 0;
          }
        }
        __syncwarp();
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&s);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(a.state);
        for (int i = l; i < (int)(sizeof(LtsState) / 8); i += 32) dst[i] = src[i];
      } else if (!kSingle) {
        for (int i = threadIdx.x - 32; i < kBins; i += kThreads - 32) a.hist[i] = 0;
      }
    }
    if (!sync()) return;
  }
}

__global__ void __launch_bounds__(kThreads) lts_kernel(LtsArgs a) {
  lts_body(a, GridSync{a.ctl, a.spin_limit, gridDim.x, 0u}, a.resid, blockIdx.x, gridDim.x);
}

// A fit by a cluster, or by its first CTA alone.
__device__ void lts_cluster_body(const LtsArgs &a, int cta) {
  extern __shared__ double s_resid[];  // kSinglePairs
  const long long n = __ldcg(&a.n_dev[0]) + __ldcg(&a.n_dev[1]);
  if (n <= kSinglePairs) {
    if (cta == 0) lts_body(a, SingleSync{}, s_resid, 0, 1);
    return;
  }
  lts_body(a, ClusterSync{}, a.resid, cta, kClusterCtas);
}
constexpr size_t kClusterSmem = sizeof(double) * kSinglePairs;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kThreads)
    lts_cluster_kernel(LtsArgs a) {
  lts_cluster_body(a, blockIdx.x);
}

// Several independent fits in one launch, a cluster each: fit f runs on CTAs
// [f kClusterCtas, (f + 1) kClusterCtas) with its own arguments.
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kThreads)
    lts_batch_kernel(const LtsArgs *args) {
  const LtsArgs a = args[blockIdx.x / kClusterCtas];
  lts_cluster_body(a, blockIdx.x % kClusterCtas);
}

// Zeroes each fit's select control and histograms (CTA f: fit f) so
// a batch's launch sequence has the same nodes whatever the number of fits.
__global__ void lts_batch_zero_kernel(const LtsArgs *args, unsigned long long words) {
  uint4 *p = reinterpret_cast<uint4 *>(args[blockIdx.x].ctl);
  for (unsigned long long i = threadIdx.x; i < words; i += blockDim.x) p[i] = make_uint4(0u, 0u, 0u, 0u);
}

// CTAs of a fit of at most n pairs: one cluster, or up to max_ctas that meet at
// the grid barrier (two pairs a thread).
int fit_ctas(long long n, int max_ctas) {
  if (n <= kClusterPairs) return kClusterCtas;
  const long long want = (n + 2 * kThreads - 1) / (2 * kThreads);
  return (int)(want < max_ctas ? want : max_ctas);
}

mirorr_status launch_fit(LtsArgs &a, long long n, int ctas, cudaStream_t st) {
  if (n <= kClusterPairs) {
    MB2_CUDA_TRY(cudaFuncSetAttribute(lts_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kClusterSmem));
    lts_cluster_kernel<<<kClusterCtas, kThreads, kClusterSmem, st>>>(a);
    MB2_LAUNCH_CHECK();
    return MIRORR_OK;
  }
  void *args[] = {&a};
  MB2_CUDA_TRY(cudaLaunchCooperativeKernel((void *)lts_kernel, dim3(ctas), dim3(kThreads), args, 0, st));
  ++g_launches;
  return MIRORR_OK;
}

}  // namespace

mirorr_status lts_run(LtsWork &w, LtsState &hs, const double *init_dev, const double *moved_dev,
                      const long long *n_dev, long long n, cudaStream_t st, int *inner_iters,
                      long long *n_used, const unsigned int *watch_dev,
                      unsigned int *watch_host) {
  if (watch_host) *watch_host = 0;
  lts_begin(hs);
  if (n <= 0) {
    lts_finish(hs);
    if (inner_iters) *inner_iters = 0;
    if (n_used) *n_used = 0;
    return MIRORR_OK;
  }
  MB2_TRY(lts_issue(w, &hs, init_dev, moved_dev, n_dev, n, st, nullptr, watch_dev));
  MB2_CUDA_TRY(cudaStreamSynchronize(st));
  return lts_collect(w, nullptr, hs, inner_iters, n_used, watch_host);
}

// What lts_issue reads back, in host memory (pinned staging for a captured
// sequence, or the work area's own copy).
struct LtsOut {
  LtsState state;
  LtsCtl ctl;
  long long n[2];
  unsigned int watch;
};

size_t lts_out_bytes() { return sizeof(LtsOut); }

mirorr_status lts_issue(LtsWork &w, const LtsState *state_in, const double *init_dev,
                        const double *moved_dev, const long long *n_dev, long long n,
                        cudaStream_t st, void *out_host, const unsigned int *watch_dev) {
  int dev = 0;
  MB2_CUDA_TRY(cudaGetDevice(&dev));
  if (w.max_ctas == 0) {
    int sms = 0, per = 0, coop = 0;
    MB2_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MB2_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) {
      set_error("device does not support cooperative launches");
      return MIRORR_ECUDA;
    }
    MB2_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lts_kernel, kThreads, 0));
    if (per < 1) {
      set_error("LTS kernel cannot be resident");
      return MIRORR_ECUDA;
    }
    w.max_ctas = sms * (per > 1 ? 1 : per);
  }
  const int grid = fit_ctas(n, w.max_ctas);
  MB2_TRY(w.state.ensure(sizeof(LtsState)));
  MB2_TRY(w.resid.ensure(sizeof(double) * n));
  MB2_TRY(w.partial.ensure(sizeof(double) * kPartial * (size_t)grid));
  MB2_TRY(w.hist.ensure(sizeof(unsigned int) * 3 * kBins));
  MB2_TRY(w.ctrl.ensure(sizeof(LtsCtl)));
  MB2_TRY(w.cand.ensure(sizeof(unsigned long long) * kCandMax));
  if (!out_host) {
    MB2_TRY(w.out.ensure(sizeof(LtsOut)));
    out_host = w.out.ptr;
  }
  LtsOut *o = static_cast<LtsOut *>(out_host);
  MB2_CUDA_TRY(cudaMemcpyAsync(w.state.ptr, state_in, sizeof(LtsState), cudaMemcpyHostToDevice, st));
  MB2_CUDA_TRY(cudaMemsetAsync(w.hist.ptr, 0, sizeof(unsigned int) * 3 * kBins, st));
  MB2_CUDA_TRY(cudaMemsetAsync(w.ctrl.ptr, 0, sizeof(LtsCtl), st));
  LtsArgs a;
  a.state = w.state.as<LtsState>();
  a.init = init_dev;
  a.moved = moved_dev;
  a.n_dev = n_dev;
  a.resid = w.resid.as<double>();
  a.partial = w.partial.as<double>();
  a.hist = w.hist.as<unsigned int>();
  a.cand = w.cand.as<unsigned long long>();
  a.ctl = w.ctrl.as<LtsCtl>();
  a.spin_limit = w.spin_limit > 0 ? w.spin_limit : kDefaultSpinLimit;
  MB2_TRY(launch_fit(a, n, grid, st));
  MB2_CUDA_TRY(cudaMemcpyAsync(&o->state, w.state.ptr, sizeof(LtsState), cudaMemcpyDeviceToHost, st));
  MB2_CUDA_TRY(cudaMemcpyAsync(&o->ctl, w.ctrl.ptr, sizeof(LtsCtl), cudaMemcpyDeviceToHost, st));
  MB2_CUDA_TRY(cudaMemcpyAsync(o->n, n_dev, sizeof(o->n), cudaMemcpyDeviceToHost, st));
  if (watch_dev)
    MB2_CUDA_TRY(cudaMemcpyAsync(&o->watch, watch_dev, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
  else
    o->watch = 0;
  return MIRORR_OK;
}

mirorr_status lts_collect(LtsWork &w, const void *out_host, LtsState &hs, int *inner_iters,
                          long long *n_used, unsigned int *watch_host) {
  const LtsOut *o = static_cast<const LtsOut *>(out_host ? out_host : w.out.ptr);
  hs = o->state;
  if (watch_host) *watch_host = o->watch;
  if (n_used) *n_used = o->n[0] + o->n[1];
  if (o->ctl.bar.err) {
    set_error("LTS grid barrier timed out");
    return MIRORR_ETIMEOUT;
  }
  if (inner_iters) *inner_iters = hs.iter;
  lts_finish(hs);
  return MIRORR_OK;
}

// ---- many fits in one launch ----------------------------------------------------
//
// Each fit is one cluster with its own state, counters and scratch (LtsFit, all
// device pointers); the fits need not be resident together.  The caller has
// run lts_begin on every state it uploaded and runs lts_finish on each after
// reading it back.  A fit whose state is not running returns at once.
size_t lts_args_bytes() { return sizeof(LtsArgs); }

size_t lts_fit_scratch_bytes(long long n_max) {
  const size_t a = 256;
  auto up = [&](size_t v) { return (v + a - 1) / a * a; };
  return up(sizeof(LtsCtl)) + up(sizeof(unsigned int) * 3 * kBins) +
         up(sizeof(unsigned long long) * kCandMax) +
         up(sizeof(double) * kPartial * (size_t)kClusterCtas) +
         up(sizeof(double) * (size_t)(n_max > 0 ? n_max : 1));
}

mirorr_status lts_batch_launch(const LtsFit *fits, int nfits, DevBuf &args_dev,
                               HostBuf &args_host, cudaStream_t st) {
  if (nfits <= 0) return MIRORR_OK;
  MB2_TRY(args_dev.ensure(sizeof(LtsArgs) * nfits));
  MB2_TRY(args_host.ensure(sizeof(LtsArgs) * nfits));
  LtsArgs *ha = args_host.as<LtsArgs>();
  const size_t al = 256;
  auto up = [&](size_t v) { return (v + al - 1) / al * al; };
  for (int f = 0; f < nfits; ++f) {
    unsigned char *p = static_cast<unsigned char *>(fits[f].scratch);
    LtsArgs &a = ha[f];
    a.state = fits[f].state;
    a.init = fits[f].init;
    a.moved = fits[f].moved;
    a.n_dev = fits[f].n_dev;
    a.ctl = reinterpret_cast<LtsCtl *>(p);
    p += up(sizeof(LtsCtl));
    a.hist = reinterpret_cast<unsigned int *>(p);
    p += up(sizeof(unsigned int) * 3 * kBins);
    a.cand = reinterpret_cast<unsigned long long *>(p);
    p += up(sizeof(unsigned long long) * kCandMax);
    a.partial = reinterpret_cast<double *>(p);
    p += up(sizeof(double) * kPartial * (size_t)kClusterCtas);
    a.resid = reinterpret_cast<double *>(p);
    a.spin_limit = 0;  // no fit of a batch waits at the grid barrier
  }
  MB2_CUDA_TRY(cudaMemcpyAsync(args_dev.ptr, ha, sizeof(LtsArgs) * nfits, cudaMemcpyHostToDevice, st));
  const LtsArgs *dargs = args_dev.as<LtsArgs>();
  // zeroed select control and histograms of every fit (the scratch starts 256-byte
  // aligned: the region is whole 16-byte words)
  const size_t zbytes = up(sizeof(LtsCtl)) + up(sizeof(unsigned int) * 3 * kBins);
  lts_batch_zero_kernel<<<nfits, 256, 0, st>>>(dargs, (unsigned long long)(zbytes / 16));
  MB2_LAUNCH_CHECK();
  MB2_CUDA_TRY(cudaFuncSetAttribute(lts_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kClusterSmem));
  lts_batch_kernel<<<nfits * kClusterCtas, kThreads, kClusterSmem, st>>>(dargs);
  MB2_LAUNCH_CHECK();
  return MIRORR_OK;
}

// ---- allocation-free variant ----------------------------------------------------
//
// lts_run_noalloc runs the same kernel with the same grid as lts_run, but every
// scratch buffer lives in one static device array, so the call allocates no
// device memory.  Its address is looked up once per device (the first call on
// that device) with cudaGetSymbolAddress.  Layout, in bytes:
//   [0, 4096)        LtsState (uploaded each call)
//   [4096, 4352)     LtsCtl (zeroed each call)
//   [4352, 4608)     point-pair counters {n, 0} (uploaded each call)
//   [4608, +24 KB)   3 histograms of 2048 bins (zeroed each call)
//   then             512 candidate keys, kNaMaxCtas * 32 partial sums,
//                    MIRORR_LTS_NOALLOC_MAX_POINTS residuals.
// Two calls in flight on one device share the array and race.

namespace {

constexpr int kNaMaxCtas = 256;
constexpr int kNaMaxDevices = 64;
constexpr size_t kNaState = 0;
constexpr size_t kNaCtl = 4096;
constexpr size_t kNaCount = kNaCtl + 256;
constexpr size_t kNaHist = kNaCount + 256;
constexpr size_t kNaCand = kNaHist + sizeof(unsigned int) * 3 * kBins;
constexpr size_t kNaPartial = kNaCand + sizeof(unsigned long long) * kCandMax;
constexpr size_t kNaResid = kNaPartial + sizeof(double) * kPartial * kNaMaxCtas;
constexpr size_t kNaBytes = kNaResid + sizeof(double) * (size_t)MIRORR_LTS_NOALLOC_MAX_POINTS;
static_assert(sizeof(LtsState) <= kNaCtl - kNaState, "LtsState slot");
static_assert(sizeof(LtsCtl) <= kNaCount - kNaCtl, "LtsCtl slot");
static_assert(kNaHist % 256 == 0 && kNaCand % 256 == 0 && kNaPartial % 256 == 0 &&
                  kNaResid % 256 == 0, "slot alignment");

static __device__ __align__(256) unsigned char g_lts_scratch[kNaBytes];

std::mutex g_na_mu;
unsigned char *g_na_ptr[kNaMaxDevices];
int g_na_ctas[kNaMaxDevices];

// One-time set-up per device (the calling thread's current device): the
// scratch address and the co-resident CTA count of the cooperative launch.
mirorr_status na_setup(int dev, unsigned char **ptr, int *ctas) {
  std::lock_guard<std::mutex> lock(g_na_mu);
  if (dev < 0 || dev >= kNaMaxDevices) {
    set_error("device ordinal %d is beyond the %d devices the no-allocation LTS supports", dev,
              kNaMaxDevices);
    return MIRORR_ERANGE;
  }
  if (!g_na_ptr[dev]) {
    int sms = 0, per = 0, coop = 0;
    MB2_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MB2_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) {
      set_error("device does not support cooperative launches");
      return MIRORR_ECUDA;
    }
    MB2_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lts_kernel, kThreads, 0));
    if (per < 1) {
      set_error("LTS kernel cannot be resident");
      return MIRORR_ECUDA;
    }
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_lts_scratch);
    if (e != cudaSuccess || !p) {
      set_error("cudaGetSymbolAddress of the LTS scratch array failed on device %d: %s", dev,
                cudaGetErrorString(e));
      return MIRORR_ECUDA;
    }
    g_na_ctas[dev] = sms * (per > 1 ? 1 : per);
    g_na_ptr[dev] = static_cast<unsigned char *>(p);
  }
  *ptr = g_na_ptr[dev];
  *ctas = g_na_ctas[dev];
  return MIRORR_OK;
}

}  // namespace

mirorr_status lts_run_noalloc(LtsState &hs, const double *init_dev, const double *moved_dev,
                              long long n, cudaStream_t st, int *inner_iters) {
  if (n > (long long)MIRORR_LTS_NOALLOC_MAX_POINTS) {
    set_error("%lld point pairs exceed the no-allocation LTS limit of %d", n,
              (int)MIRORR_LTS_NOALLOC_MAX_POINTS);
    return MIRORR_ERANGE;
  }
  lts_begin(hs);
  if (n <= 0) {
    lts_finish(hs);
    if (inner_iters) *inner_iters = 0;
    return MIRORR_OK;
  }
  int dev = 0;
  MB2_CUDA_TRY(cudaGetDevice(&dev));
  unsigned char *base = nullptr;
  int max_ctas = 0;
  MB2_TRY(na_setup(dev, &base, &max_ctas));
  if (max_ctas > kNaMaxCtas) max_ctas = kNaMaxCtas;
  const int grid = fit_ctas(n, max_ctas);
  long long counts[2] = {n, 0};
  MB2_CUDA_TRY(cudaMemcpyAsync(base + kNaState, &hs, sizeof(LtsState), cudaMemcpyHostToDevice, st));
  MB2_CUDA_TRY(cudaMemcpyAsync(base + kNaCount, counts, sizeof(counts), cudaMemcpyHostToDevice, st));
  MB2_CUDA_TRY(cudaMemsetAsync(base + kNaHist, 0, sizeof(unsigned int) * 3 * kBins, st));
  MB2_CUDA_TRY(cudaMemsetAsync(base + kNaCtl, 0, sizeof(LtsCtl), st));
  LtsArgs a;
  a.state = reinterpret_cast<LtsState *>(base + kNaState);
  a.init = init_dev;
  a.moved = moved_dev;
  a.n_dev = reinterpret_cast<const long long *>(base + kNaCount);
  a.resid = reinterpret_cast<double *>(base + kNaResid);
  a.partial = reinterpret_cast<double *>(base + kNaPartial);
  a.hist = reinterpret_cast<unsigned int *>(base + kNaHist);
  a.cand = reinterpret_cast<unsigned long long *>(base + kNaCand);
  a.ctl = reinterpret_cast<LtsCtl *>(base + kNaCtl);
  a.spin_limit = kDefaultSpinLimit;
  MB2_TRY(launch_fit(a, n, grid, st));
  LtsCtl ctl;
  MB2_CUDA_TRY(cudaMemcpyAsync(&hs, base + kNaState, sizeof(LtsState), cudaMemcpyDeviceToHost, st));
  MB2_CUDA_TRY(cudaMemcpyAsync(&ctl, base + kNaCtl, sizeof(LtsCtl), cudaMemcpyDeviceToHost, st));
  MB2_CUDA_TRY(cudaStreamSynchronize(st));
  if (ctl.bar.err) {
    set_error("LTS grid barrier timed out");
    return MIRORR_ETIMEOUT;
  }
  if (inner_iters) *inner_iters = hs.iter;
  lts_finish(hs);
  return MIRORR_OK;
}

}  // namespace mb2
