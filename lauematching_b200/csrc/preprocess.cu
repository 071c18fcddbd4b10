// Frame preprocessing on the device: the steps of preprocess_image
// (laue_index/preprocess.py:221-338) as the reference runs them with numpy,
// scipy and OpenCV, with identical results:
//
//   background   exact square median (scipy.ndimage.median_filter, mirrored
//                borders).  Frames of whole numbers: tile by tile, window counts
//                below a few thresholds around the tile's medians.  Others: pixels
//                become ranks among the frame's distinct values; one warp per
//                (column, row segment) slides its window down, keeping 8-bit-digit
//                rank histograms level by level and refilling a deeper level only
//                when the digit above it moves.
//   threshold    order statistics (np.median, np.percentile) from a histogram of
//                whole-number values, else by radix selection over
//                order-preserving 64-bit keys, on the device.
//   components   union-find over 8-neighbours (atomicMin on the parent
//                array); OpenCV numbers components by the raster order of
//                the first 2x2 pixel block each touches, so labels come from
//                the ranks of their bits in a map of blocks.
//   centres      integer moments per component (exact), one division each.
//   blur width   closest pair of centres: cell grid, brute force when the
//                pair is farther apart than a cell.
//   blur         separable float64 passes in scipy's summation order.
#include <cub/cub.cuh>

#include <cmath>
#include <cstring>
#include <limits>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "staging.h"

using namespace lmb;

namespace {

constexpr int kT = 256;            // threads of the elementwise kernels
constexpr int kMedWarps = 8;       // warps per median block
constexpr int kMedLevels = 4;      // 8-bit digits of a rank (ranks < 2^32)
constexpr int kCell = 32;          // cell side of the closest-pair grid (pixels)
constexpr int kKeepShift = 40;     // the 8-bit pass that reads the frame and keeps its keys
constexpr int kHist16Threads = 1024;
constexpr size_t kHist16Smem = 32768 * sizeof(unsigned);  // 65536 packed 16-bit counters
constexpr int kPreEvents = 12;
enum PreEv : int {
  EV_SEG0 = 0, EV_SEG_UP, EV_SEG_THR, EV_SEG_CC, EV_BLUR0, EV_BLUR_K, EV_BLUR_DL, EV_MED0, EV_MED_UP,
  EV_MED_RANK, EV_MED_K, EV_MED_PASS
};

enum SelMode : int { SEL_NZ = 0, SEL_ABSDEV = 1, SEL_ALL = 2 };

// ---- small helpers -----------------------------------------------------------
// scipy's 'reflect' border (d c b a | a b c d | d c b a), periodic.
__host__ __device__ __forceinline__ int mirror(int i, int n) {
  if (i >= 0 && i < n) return i;
  if (n == 1) return 0;
  const int p = 2 * n;
  i %= p;
  if (i < 0) i += p;
  return i < n ? i : p - 1 - i;
}

// Order-preserving key of a double (total order; -0 sorts just below +0).
__device__ __forceinline__ unsigned long long okey(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_value(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

// numpy's float64 -> uint16 (x86-64): truncate to int32, keep 16 bits.
__device__ __forceinline__ uint16_t u16_cast(double v) {
  return (uint16_t)((unsigned)x86_trunc_i32(v) & 0xFFFFu);
}

template <typename T>
__device__ __forceinline__ double to_f64(T v) {
  return (double)v;
}

size_t grid_for(size_t n, int num_sms) {
  return std::max<size_t>(1, std::min<size_t>((n + kT - 1) / kT, (size_t)num_sms * 16));
}

// ---- device state of one frame -----------------------------------------------
struct Select {
  unsigned long long n;          // candidates
  unsigned long long k[2];       // residual ranks sought (k[1] = k[0] + 1 when two)
  unsigned long long prefix[2];  // key bits fixed so far
  unsigned long long n_compact;  // candidates kept for the later passes
  unsigned long long kmin[2], kmax[2];  // extremes of the keys under each prefix (this pass)
  int two;
  int valid;
  int done[2];                   // the rank's key is known (all keys under its prefix equal)
  int pad;
};

struct PreState {
  Select sel;
  __align__(16) unsigned int hist[2][256];
  double med;
  double thresh;
  unsigned int blocks_done;  // blocks of the running selection pass that finished
  unsigned int max_bin;      // largest value of the running value histogram
  unsigned int n_fg;         // foreground pixels
  unsigned int nonint;       // a candidate value was not an integer in [0, 65535]
  unsigned int value_path;   // the threshold came from the value histogram
  unsigned int n_comp;      // components
  unsigned int n_labels;    // components + 1
  unsigned int n_keep;      // components with area >= min_area
  unsigned long long best;  // bits of the smallest squared centre distance
};

static_assert(offsetof(PreState, hist) % 16 == 0, "histogram rows are read as 16-byte vectors");

// ---- conversions -------------------------------------------------------------
template <typename T>
__global__ void to_f64_kernel(const T *__restrict__ in, double *__restrict__ out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = to_f64(in[i]);
}

// np.maximum(raw - background, 0.0): NaN stays NaN, -0 stays -0.
template <typename T>
__global__ void subtract_kernel(const T *__restrict__ raw, const double *__restrict__ bg,
                                double *__restrict__ sub, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double d = lmb::dsub(to_f64(raw[i]), bg[i]);
    sub[i] = (d >= 0.0 || isnan(d)) ? d : 0.0;
  }
}

// ---- order statistics ----------------------------------------------------------
__global__ void sel_init_kernel(PreState *st, int mode, unsigned long long n,
                                unsigned long long k0, int two) {
  const int t = threadIdx.x;
  for (int i = t; i < 512; i += blockDim.x) (&st->hist[0][0])[i] = 0;
  if (t == 0) {
    Select &s = st->sel;
    s.n = mode == SEL_ALL ? n : 0;
    s.k[0] = k0;
    s.k[1] = k0 + 1;
    s.prefix[0] = s.prefix[1] = 0;
    s.n_compact = 0;
    s.kmin[0] = s.kmin[1] = ~0ull;
    s.kmax[0] = s.kmax[1] = 0;
    s.done[0] = s.done[1] = 0;
    s.two = mode == SEL_ALL ? two : 0;
    s.valid = 1;
  }
}

// Digit holding residual rank k among 256 bins, lane l holding bins
// 8l..8l+7 in c[]; one warp.
__device__ __forceinline__ unsigned warp_find_in(const unsigned (&c)[8], unsigned long long &k) {
  const int lane = threadIdx.x & 31;
  unsigned long long sum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) sum += c[j];
  unsigned long long incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const unsigned long long excl = incl - sum;
  const unsigned msk = __ballot_sync(0xffffffffu, k < incl);
  const int f = msk ? __ffs(msk) - 1 : 31;
  unsigned digit = 0;
  unsigned long long r = 0;
  if (lane == f) {
    r = k - excl;
    int j = 0;
    while (j < 7 && r >= c[j]) r -= c[j++];
    digit = (unsigned)(lane * 8 + j);
  }
  digit = __shfl_sync(0xffffffffu, digit, f);
  k = __shfl_sync(0xffffffffu, r, f);
  return digit;
}

// The same over a 16-byte aligned shared-memory histogram.
__device__ __forceinline__ unsigned warp_find_digit(const unsigned *h, unsigned long long &k) {
  const int lane = threadIdx.x & 31;
  const uint4 a = reinterpret_cast<const uint4 *>(h)[lane * 2];
  const uint4 b = reinterpret_cast<const uint4 *>(h)[lane * 2 + 1];
  const unsigned c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  return warp_find_in(c, k);
}

// Per-thread run of equal digits, flushed into the block's histogram when the
// digit changes: a frame's values crowd a few bins, so most values only bump
// a register.
struct DigitRun {
  unsigned d = 0x100u, n = 0;
  __device__ __forceinline__ void add(unsigned *hh, unsigned dig) {
    if (dig == d) {
      ++n;
      return;
    }
    if (n) atomicAdd(hh + d, n);
    d = dig;
    n = 1;
  }
  __device__ __forceinline__ void flush(unsigned *hh) {
    if (n) atomicAdd(hh + d, n);
    n = 0;
  }
};

// After a pass (warp 0 of the grid's last block): fix the digit of each
// sought rank and clear the histograms.  Pass 0 also learns the candidate
// count (SEL_NZ / SEL_ABSDEV: the median's ranks, two for an even count).
__device__ void sel_pick(PreState *st, int mode, int shift) {
  Select &s = st->sel;
  const int lane = threadIdx.x & 31;
  unsigned c0[8], c1[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c0[j] = __ldcg(&st->hist[0][lane * 8 + j]);
    c1[j] = __ldcg(&st->hist[1][lane * 8 + j]);
  }
  if (s.valid) {
    for (int L = 0; L < (s.two ? 2 : 1); ++L) {
      if (s.done[L]) continue;
      const int src = L;
      if (s.kmin[src] == s.kmax[src]) {  // every key under the prefix is this one
        if (lane == 0) {
          s.prefix[L] = s.kmin[src];
          s.done[L] = 1;
        }
        __syncwarp();
        continue;
      }
      unsigned long long k = s.k[L];
      const unsigned d = warp_find_in(src == 0 ? c0 : c1, k);
      if (lane == 0) {
        s.k[L] = k;
        s.prefix[L] |= (unsigned long long)d << shift;
      }
      __syncwarp();
    }
  }
  __syncwarp();
  if (lane == 0) {
    s.kmin[0] = s.kmin[1] = ~0ull;
    s.kmax[0] = s.kmax[1] = 0;
  }
  for (int j = lane; j < 512; j += 32) (&st->hist[0][0])[j] = 0;
}

// Key of a selection candidate: non-negative values (every candidate of
// SEL_NZ and SEL_ABSDEV) only need the sign bit set.
__device__ __forceinline__ unsigned long long sel_key(int mode, double v) {
  return mode == SEL_ALL ? okey(v)
                         : ((unsigned long long)__double_as_longlong(v) | 0x8000000000000000ull);
}

// One radix pass: histogram of the digit at `shift` of the candidates whose
// higher digits equal each sought rank's prefix.  Passes 0..2 read the frame
// (pass 2 also keeps the surviving keys), later passes read those keys.  The
// last block to finish picks the digits for the next pass.
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__global__ void __launch_bounds__(kT, 4)
    sel_hist_kernel(const double *frame, size_t n, PreState *st, int mode, int shift,
                    unsigned long long *compact) {
  constexpr int U = 8;  // values per thread per round
  __shared__ unsigned int h[2][256];
  __shared__ Select ss;
  __shared__ bool last;
  __shared__ unsigned long long stage[kT * U];  // kept keys of one round
  __shared__ unsigned n_stage;
  __shared__ unsigned long long base_s;
  __shared__ unsigned long long ext[4][kT / 32];
  for (int i = threadIdx.x; i < 512; i += blockDim.x) (&h[0][0])[i] = 0;
  if (threadIdx.x == 0) {
    ss = st->sel;
    n_stage = 0;
  }
  __syncthreads();
  const Select s = ss;
  const bool two = s.two != 0;
  // ranks whose key is known already need no more passes
  if (!s.valid || (s.done[0] && (!two || s.done[1]))) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool act0 = !s.done[0], act1 = two && !s.done[1];
  const unsigned long long hi = ~0ull << (shift + 8);
  const unsigned long long p0 = s.prefix[0] & hi, p1 = s.prefix[1] & hi;
  const double med = st->med;
  const bool from_frame = shift >= kKeepShift;
  const bool keep = shift == kKeepShift;
  const unsigned m = from_frame ? (unsigned)n : (unsigned)s.n_compact;
  const unsigned stride = gridDim.x * blockDim.x;
  const unsigned rounds = (m + stride * U - 1) / (stride * U);
  DigitRun run0, run1;
  unsigned long long mn0 = ~0ull, mx0 = 0, mn1 = ~0ull, mx1 = 0;
  for (unsigned it = 0; it < rounds; ++it) {
    unsigned long long key[U];
    bool hit0[U], hit1[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = (it * U + u) * stride + blockIdx.x * blockDim.x + threadIdx.x;
      hit0[u] = hit1[u] = false;
      key[u] = 0;
      if (i < m) {
        bool cand = true;
        if (from_frame) {
          const double v = frame[i];
          cand = mode == SEL_ALL || v > 0.0;
          key[u] = sel_key(mode, mode == SEL_ABSDEV ? fabs(lmb::dsub(v, med)) : v);
        } else {
          key[u] = compact[i];
        }
        hit0[u] = cand && act0 && (key[u] & hi) == p0;
        hit1[u] = cand && act1 && (key[u] & hi) == p1;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned d = (unsigned)(key[u] >> shift) & 255u;
      if (hit0[u]) {
        run0.add(h[0], d);
        mn0 = min(mn0, key[u]);
        mx0 = max(mx0, key[u]);
      }
      if (hit1[u]) {
        run1.add(h[1], d);
        mn1 = min(mn1, key[u]);
        mx1 = max(mx1, key[u]);
      }
      if (keep) {  // warp-aggregated slot in the block's staging area
        const bool k = hit0[u] || hit1[u];
        const unsigned msk = __ballot_sync(0xffffffffu, k);
        if (msk) {
          unsigned base = 0;
          if (lane == __ffs(msk) - 1) base = atomicAdd(&n_stage, (unsigned)__popc(msk));
          base = __shfl_sync(0xffffffffu, base, __ffs(msk) - 1);
          if (k) stage[base + __popc(msk & ((1u << lane) - 1u))] = key[u];
        }
      }
    }
    if (keep) {  // one reservation per block and round for the kept keys
      __syncthreads();
      const unsigned ns = n_stage;
      if (threadIdx.x == 0 && ns) base_s = atomicAdd(&st->sel.n_compact, (unsigned long long)ns);
      __syncthreads();
      for (unsigned q = threadIdx.x; q < ns; q += blockDim.x) compact[base_s + q] = stage[q];
      __syncthreads();
      if (threadIdx.x == 0) n_stage = 0;
      __syncthreads();
    }
  }
  run0.flush(h[0]);
  run1.flush(h[1]);
  mn0 = warp_min_u64(mn0);
  mx0 = warp_max_u64(mx0);
  mn1 = warp_min_u64(mn1);
  mx1 = warp_max_u64(mx1);
  if (lane == 0) {
    ext[0][warp] = mn0;
    ext[1][warp] = mx0;
    ext[2][warp] = mn1;
    ext[3][warp] = mx1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kT / 32; ++w) {
      mn0 = min(mn0, ext[0][w]);
      mx0 = max(mx0, ext[1][w]);
      mn1 = min(mn1, ext[2][w]);
      mx1 = max(mx1, ext[3][w]);
    }
    if (mn0 != ~0ull) {
      atomicMin(&st->sel.kmin[0], mn0);
      atomicMax(&st->sel.kmax[0], mx0);
    }
    if (mn1 != ~0ull) {
      atomicMin(&st->sel.kmin[1], mn1);
      atomicMax(&st->sel.kmax[1], mx1);
    }
  }
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const unsigned v = (&h[0][0])[i];
    if (v) atomicAdd(&(&st->hist[0][0])[i], v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && threadIdx.x < 32) {
    __threadfence();
    sel_pick(st, mode, shift);
    if (threadIdx.x == 0) st->blocks_done = 0;
  }
}

// ---- first selection pass: 16-bit digits --------------------------------------
// The top 16 key bits (sign, exponent, 4 mantissa bits) of every candidate are
// counted in 65536 packed 16-bit counters in shared memory (a block handles at
// most 65535 values), flushed to a 65536-bin histogram in global memory; the
// grid's last block finds the bins of the sought ranks with all its threads.
struct Digit16Run {
  unsigned d = 0xffffffffu, n = 0;
  __device__ __forceinline__ void add(unsigned *words, unsigned dig) {
    if (dig == d) {
      ++n;
      return;
    }
    flush(words);
    d = dig;
    n = 1;
  }
  __device__ __forceinline__ void flush(unsigned *words) {
    if (n) atomicAdd(words + (d >> 1), n << (16 * (d & 1)));
    n = 0;
  }
};

__device__ __forceinline__ unsigned key16(int mode, double v) {
  return (unsigned)(sel_key(mode, v) >> 48);
}

// Block of 1024 threads: each owns 64 consecutive bins.
__device__ void sel_pick16(PreState *st, unsigned *g16, int mode) {
  __shared__ unsigned long long warp_tot[32];
  __shared__ unsigned long long total_s;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint4 *src = reinterpret_cast<const uint4 *>(g16 + t * 64);
  unsigned long long mine = 0;
  {
    uint4 q[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) q[j] = __ldcg(src + j);
#pragma unroll
    for (int j = 0; j < 16; ++j) mine += (unsigned long long)q[j].x + q[j].y + q[j].z + q[j].w;
  }
  unsigned long long incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    unsigned long long v = warp_tot[lane], x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += u;
    }
    warp_tot[lane] = x - v;  // exclusive prefix of the warps
    if (lane == 31) total_s = x;
  }
  __syncthreads();
  const unsigned long long excl = warp_tot[w] + incl - mine;
  Select &s = st->sel;
  if (t == 0) {
    const unsigned long long tot = total_s;
    if (mode != SEL_ALL) {
      s.n = tot;
      s.k[0] = tot ? (tot - 1) / 2 : 0;
      s.k[1] = s.k[0] + 1;
      s.two = tot > 0 && (tot % 2) == 0;
    }
    if (s.n == 0) s.valid = 0;
  }
  __syncthreads();
  const unsigned long long kk[2] = {s.k[0], s.k[1]};
  __syncthreads();  // the owner of a rank's bin replaces the rank below
  if (s.valid) {
    for (int L = 0; L < (s.two ? 2 : 1); ++L) {
      const unsigned long long k = kk[L];
      if (k >= excl && k < excl + mine) {
        unsigned long long r = k - excl;
        int jj = 63;
        for (int j = 0; j < 16 && jj == 63; ++j) {
          const uint4 q = __ldcg(src + j);
          const unsigned cc[4] = {q.x, q.y, q.z, q.w};
          for (int e = 0; e < 4; ++e) {
            if (4 * j + e == 63) break;
            if (r < cc[e]) {
              jj = 4 * j + e;
              break;
            }
            r -= cc[e];
          }
        }
        s.k[L] = r;
        s.prefix[L] = (unsigned long long)(t * 64 + jj) << 48;
      }
    }
  }
  __syncthreads();
  uint4 *dst = reinterpret_cast<uint4 *>(g16 + t * 64);
#pragma unroll
  for (int j = 0; j < 16; ++j) dst[j] = make_uint4(0, 0, 0, 0);
}

// Pass A over the subtracted frame.
__global__ void __launch_bounds__(kHist16Threads, 1)
    sel_hist16_kernel(const double *__restrict__ sub, unsigned n, PreState *st, unsigned *g16,
                      int mode) {
  extern __shared__ unsigned words[];
  __shared__ bool last;
  for (int i = threadIdx.x; i < 32768; i += blockDim.x) words[i] = 0;
  __syncthreads();
  const double med = st->med;
  Digit16Run run;
  constexpr int U = 4;
  const unsigned stride = gridDim.x * blockDim.x;
  const unsigned rounds = (n + stride * U - 1) / (stride * U);
  for (unsigned it = 0; it < rounds; ++it) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = (it * U + u) * stride + blockIdx.x * blockDim.x + threadIdx.x;
      v[u] = i < n ? sub[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = (it * U + u) * stride + blockIdx.x * blockDim.x + threadIdx.x;
      if (i < n && (mode == SEL_ALL || v[u] > 0.0))
        run.add(words, key16(mode, mode == SEL_ABSDEV ? fabs(lmb::dsub(v[u], med)) : v[u]));
    }
  }
  run.flush(words);
  __syncthreads();
  for (int wd = threadIdx.x; wd < 32768; wd += blockDim.x) {
    const unsigned x = words[wd];
    if (x & 0xffffu) atomicAdd(g16 + 2 * wd, x & 0xffffu);
    if (x >> 16) atomicAdd(g16 + 2 * wd + 1, x >> 16);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) {
    __threadfence();
    sel_pick16(st, g16, mode);
    if (threadIdx.x == 0) st->blocks_done = 0;
  }
}

// ---- threshold statistics of integer-valued frames ---------------------------------
// A detector frame minus a median background holds integers.  When every
// candidate value is an integer in [0, 65535], one pass counts the values
// themselves (65536 packed 16-bit counters per block, flushed into the global
// histogram); the grid's last block turns the histogram into prefix sums and
// finds the order statistics by binary search: np.median / np.percentile
// directly, and the median of |v - median| as the smallest distance d with
// more than k values within d of the median.  Any other value (fraction,
// negative zero, NaN, above 65535) leaves the work to the radix selection.
// Prefix sums P[0..top] of the histogram: values at most v.
struct ValueCounts {
  const unsigned *P;
  int top;
  __device__ __forceinline__ unsigned long long le(int v) const {
    return v < 0 ? 0ull : (unsigned long long)P[min(v, top)];
  }
};

// Smallest x in [lo, hi] with pred(x), pred monotone and true at hi; the
// whole warp probes 32 points per round.
template <typename Pred>
__device__ long long warp_search(long long lo, long long hi, Pred pred) {
  const int lane = threadIdx.x & 31;
  while (hi - lo + 1 > 32) {
    const long long step = (hi - lo + 1 + 31) / 32;
    long long x = lo + (long long)(lane + 1) * step - 1;
    if (x > hi) x = hi;
    const unsigned m = __ballot_sync(0xffffffffu, pred(x));
    const int f = __ffs(m) - 1;
    long long nhi = lo + (long long)(f + 1) * step - 1;
    if (nhi > hi) nhi = hi;
    lo = lo + (long long)f * step;
    hi = nhi;
  }
  const long long x = lo + lane;
  const unsigned m = __ballot_sync(0xffffffffu, x <= hi && pred(x));
  return lo + __ffs(m) - 1;
}

// Smallest value v >= lo with more than r values in [lo, v].
__device__ int vh_rank(const ValueCounts &c, int lo, unsigned long long r) {
  const unsigned long long base = c.le(lo - 1);
  return (int)warp_search(lo, max(lo, c.top), [&](long long v) { return c.le((int)v) - base > r; });
}

// Values in [lo, 65535] within t/2 of med.
__device__ unsigned long long vh_within(const ValueCounts &c, int lo, double med, long long t) {
  const double h = 0.5 * (double)t;
  long long a = (long long)ceil(med - h), b = (long long)floor(med + h);
  if (a < lo) a = lo;
  if (b > 65535) b = 65535;
  if (b < a) return 0ull;
  return c.le((int)b) - c.le((int)a - 1);
}

// Smallest distance (a multiple of 1/2) with more than r values within it.
__device__ double vh_dist(const ValueCounts &c, int lo, double med, unsigned long long r) {
  const long long t = warp_search(0, 2 * ((long long)c.top + 1), [&](long long x) {
    return vh_within(c, lo, med, x) > r;
  });
  return 0.5 * (double)t;
}

constexpr int kVhLocal = 4096;
constexpr int kVhThreads = 256;

// Last block: prefix sums of bins [0, top] -- in shared memory (h, kVhLocal bins)
// when they fit, in place otherwise --, the threshold (warp 0), and the global
// histogram empty again.
__device__ void vh_finish(PreState *st, unsigned *g16, unsigned *h, int top, int mode,
                          unsigned long long k0, int two, double gamma) {
  __shared__ unsigned warp_tot[kVhThreads / 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const bool local = top < kVhLocal;
  unsigned *P = local ? h : g16;
  const int per = ((top + kVhThreads) / kVhThreads + 3) / 4 * 4;  // bins per thread
  const int b0 = t * per, b1 = min(b0 + per, top + 1);
  if (local) {
    for (int b = t; b <= top; b += kVhThreads) h[b] = __ldcg(g16 + b);
    __syncthreads();
  }
  unsigned mine = 0;  // counts fit 32 bits (frames < 2^31 pixels)
  for (int b = b0; b < b1; ++b) mine += local ? h[b] : __ldcg(g16 + b);
  unsigned incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  unsigned run = incl - mine;
  for (int j = 0; j < w; ++j) run += warp_tot[j];
  for (int b = b0; b < b1; ++b) {
    run += local ? h[b] : __ldcg(g16 + b);
    P[b] = run;
  }
  __threadfence_block();
  __syncthreads();
  if (w == 0) {
    const ValueCounts c{P, top};
    double thresh;
    if (mode == SEL_ALL) {  // np.percentile over every pixel
      const double a = (double)vh_rank(c, 0, k0);
      const double b = two ? (double)vh_rank(c, 0, k0 + 1) : a;
      const double diff = lmb::dsub(b, a);
      thresh = lmb::dadd(a, lmb::dmul(diff, gamma));
      if (gamma >= 0.5) thresh = lmb::dsub(b, lmb::dmul(diff, lmb::dsub(1.0, gamma)));
    } else {  // the adaptive noise floor over the nonzero pixels
      const unsigned long long n = c.le(65535) - c.le(0);
      if (n == 0) {
        thresh = 1.0;
      } else {
        const unsigned long long k = (n - 1) / 2;
        const bool even = (n % 2) == 0;
        const double a = (double)vh_rank(c, 1, k);
        const double med =
            even ? lmb::ddiv(lmb::dadd(a, (double)vh_rank(c, 1, k + 1)), 2.0) : a;
        const double m1 = vh_dist(c, 1, med, k);
        const double md = even ? lmb::ddiv(lmb::dadd(m1, vh_dist(c, 1, med, k + 1)), 2.0) : m1;
        const double mad = lmb::dmul(1.4826, md);
        const double thr = lmb::dadd(med, lmb::dmul(4.0, mad));
        thresh = (1.0 > thr) ? 1.0 : thr;
      }
    }
    if (lane == 0) {
      st->thresh = thresh;
      st->value_path = 1;
    }
  }
  __syncthreads();
  for (int b = t; b <= top; b += kVhThreads) g16[b] = 0u;
}

// Eight neighbouring pixels of an 8- or 16-bit frame as 16-bit pairs.
__device__ __forceinline__ uint4 load_eight(const uint16_t *raw, unsigned q) {
  return reinterpret_cast<const uint4 *>(raw)[q];
}
__device__ __forceinline__ uint4 load_eight(const uint8_t *raw, unsigned q) {
  const uint2 b = reinterpret_cast<const uint2 *>(raw)[q];
  return make_uint4(__byte_perm(b.x, 0, 0x4140), __byte_perm(b.x, 0, 0x4342),
                    __byte_perm(b.y, 0, 0x4140), __byte_perm(b.y, 0, 0x4342));
}

// A frame and a background of 8- or 16-bit whole numbers: differences (not below
// zero) eight pixels at a time in integers, zeros counted in a register.
template <typename T>
__device__ __forceinline__ void value_hist_whole(const T *__restrict__ raw, const uint16_t *__restrict__ bg16,
                                                 uint16_t *__restrict__ sub16, unsigned n, unsigned *g16,
                                                 int mode, unsigned *h, DigitRun &run, unsigned &most) {
  unsigned zeros = 0;
  auto count = [&](unsigned b) {
    if (b == 0) {
      ++zeros;
      return;
    }
    most = max(most, b);
    if (b < (unsigned)kVhLocal) run.add(h, b);
    else atomicAdd(g16 + b, 1u);
  };
  const unsigned groups = n / 8, stride = gridDim.x * blockDim.x;
  const unsigned first = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int U = 2;
  for (unsigned q0 = first; q0 < groups; q0 += U * stride) {
    uint4 a[U], b[U];
    bool in[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned q = q0 + u * stride;
      in[u] = u == 0 || q < groups;
      if (in[u]) {
        a[u] = load_eight(raw, q);
        b[u] = reinterpret_cast<const uint4 *>(bg16)[q];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!in[u]) continue;
      const uint4 d = make_uint4(__vsubus2(a[u].x, b[u].x), __vsubus2(a[u].y, b[u].y),
                                 __vsubus2(a[u].z, b[u].z), __vsubus2(a[u].w, b[u].w));
      reinterpret_cast<uint4 *>(sub16)[q0 + u * stride] = d;
      for (unsigned w : {d.x, d.y, d.z, d.w}) {
        count(w & 0xFFFFu);
        count(w >> 16);
      }
    }
  }
  for (unsigned i = groups * 8 + first; i < n; i += stride) {  // up to seven pixels
    const unsigned r = raw[i], g = bg16[i], d = r > g ? r - g : 0u;
    sub16[i] = (uint16_t)d;
    count(d);
  }
  zeros = __reduce_add_sync(0xffffffffu, zeros);
  if (mode == SEL_ALL && (threadIdx.x & 31) == 0 && zeros) atomicAdd(h, zeros);
}

// Subtraction fused with the value histogram (see above); the differences are
// kept as 16-bit values.  The background is whole numbers (bg16).  Each block counts
// values below kVhLocal in shared memory (runs of equal values in registers) and
// adds larger ones straight into the global 65536-bin histogram.  8- and 16-bit
// frames have whole differences, all of it is integers; a float frame with another
// value leaves the value path, and the host takes the radix selection.  Measured on
// B200 (cold caches), 2048^2 uint16 frame: 70.7 us with the background and the
// differences as float64 and the last block's search over all 65536 bins in global
// memory, 34.3 us with one pixel at a time in float64; in integers the whole
// threshold stage takes 36-43 us instead of 49-50 (a frame into its slot 333 -> 322
// us).
template <typename T>
__global__ void __launch_bounds__(kVhThreads, 4)
    value_hist_kernel(const T *__restrict__ raw, const uint16_t *__restrict__ bg16,
                      uint16_t *__restrict__ sub16, unsigned n, PreState *st, unsigned *g16, int mode,
                      unsigned long long k0, int two, double gamma) {
  __shared__ unsigned h[kVhLocal];
  __shared__ bool last;
  __shared__ unsigned max_s;
  for (int i = threadIdx.x; i < kVhLocal; i += blockDim.x) h[i] = 0;
  if (threadIdx.x == 0) max_s = 0;
  __syncthreads();
  DigitRun run;  // bins below kVhLocal
  bool nonint = false;
  unsigned most = 0;
  if constexpr (std::is_same_v<T, uint16_t> || std::is_same_v<T, uint8_t>) {
    value_hist_whole(raw, bg16, sub16, n, g16, mode, h, run, most);
  } else {
    constexpr int U = 8;
    const unsigned stride = gridDim.x * blockDim.x;
    const unsigned rounds = (n + stride * U - 1) / (stride * U);
    for (unsigned it = 0; it < rounds; ++it) {
      double v[U];
      bool in[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned i = (it * U + u) * stride + blockIdx.x * blockDim.x + threadIdx.x;
        in[u] = i < n;
        v[u] = 0.0;
        if (in[u]) {
          const double d = lmb::dsub(to_f64(raw[i]), (double)bg16[i]);
          v[u] = (d >= 0.0 || isnan(d)) ? d : 0.0;
          sub16[i] = (uint16_t)((unsigned)x86_trunc_i32(v[u]) & 0xFFFFu);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!in[u] || !(mode == SEL_ALL || v[u] > 0.0)) continue;
        const double x = v[u];
        if (x == trunc(x) && x <= 65535.0 && !signbit(x)) {
          const unsigned b = (unsigned)x;
          most = max(most, b);
          if (b < (unsigned)kVhLocal) run.add(h, b);
          else atomicAdd(g16 + b, 1u);
        } else {
          nonint = true;  // also NaN: every comparison with it is false
        }
      }
    }
  }
  run.flush(h);
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most) atomicMax(&max_s, most);
  if (__syncthreads_or(nonint) && threadIdx.x == 0) atomicOr(&st->nonint, 1u);
  if (threadIdx.x == 0) atomicMax(&st->max_bin, max_s);
  for (int b = threadIdx.x; b < kVhLocal; b += blockDim.x)
    if (h[b]) atomicAdd(g16 + b, h[b]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) {
    __threadfence();
    const int top = (int)__ldcg(&st->max_bin);
    if (__ldcg(&st->nonint) == 0) {
      vh_finish(st, g16, h, top, mode, k0, two, gamma);
    } else {  // leave an empty histogram for the radix selection
      for (int b = threadIdx.x; b <= top; b += kVhThreads) g16[b] = 0u;
      if (threadIdx.x == 0) st->value_path = 0;
    }
    if (threadIdx.x == 0) {
      st->blocks_done = 0;
      st->nonint = 0;
      st->max_bin = 0;
    }
  }
}

__device__ __forceinline__ double sel_value(const Select &s, int L) {
  return okey_value(s.prefix[L]);
}

// np.median of the candidates: the middle one, or the mean of the two.
__device__ __forceinline__ double sel_median(const Select &s) {
  const double a = sel_value(s, 0);
  return s.two ? lmb::ddiv(lmb::dadd(a, sel_value(s, 1)), 2.0) : a;
}

__global__ void finish_median_kernel(PreState *st) {
  st->med = st->sel.valid ? sel_median(st->sel) : 0.0;
}

// thresholds.py:35-45: max(med + 4 * (1.4826 * mad), 1.0); 1.0 without candidates.
__global__ void finish_adaptive_kernel(PreState *st) {
  if (!st->sel.valid) {
    st->thresh = 1.0;
    return;
  }
  const double mad = lmb::dmul(1.4826, sel_median(st->sel));
  const double t = lmb::dadd(st->med, lmb::dmul(4.0, mad));
  st->thresh = (1.0 > t) ? 1.0 : t;
}

// numpy's _lerp(a, b, gamma) of the two order statistics.
__global__ void finish_percentile_kernel(PreState *st, double gamma) {
  const Select &s = st->sel;
  const double a = sel_value(s, 0);
  const double b = s.two ? sel_value(s, 1) : a;
  const double diff = lmb::dsub(b, a);
  double r = lmb::dadd(a, lmb::dmul(diff, gamma));
  if (gamma >= 0.5) r = lmb::dsub(b, lmb::dmul(diff, lmb::dsub(1.0, gamma)));
  st->thresh = r;
}

__global__ void set_thresh_kernel(PreState *st, double t) { st->thresh = t; }

__global__ void reset_counts_kernel(PreState *st) {
  st->n_fg = 0;
  st->n_comp = 0;
  st->best = 0x7ff0000000000000ull;  // +inf
}

// ---- threshold, uint16, components ---------------------------------------------
// Where a frame's thresholded uint16 pixels come from (thresholds.py:29-32,
// preprocess.py:291): the subtracted frame in float64 or as whole numbers and the
// threshold, or the thresholded frame itself.
__device__ __forceinline__ uint16_t over(double v, double thr) {
  return (v <= thr) ? (uint16_t)0 : u16_cast(v);
}
struct FromSub {
  const double *sub;
  static constexpr bool kStored = false;
  __device__ __forceinline__ uint16_t at(size_t i, double thr) const { return over(sub[i], thr); }
  __device__ __forceinline__ void four(size_t q, double thr, uint16_t (&u)[4]) const {
    const double2 a = reinterpret_cast<const double2 *>(sub)[2 * q];
    const double2 b = reinterpret_cast<const double2 *>(sub)[2 * q + 1];
    u[0] = over(a.x, thr);
    u[1] = over(a.y, thr);
    u[2] = over(b.x, thr);
    u[3] = over(b.y, thr);
  }
};
struct FromSub16 {
  const uint16_t *sub;
  static constexpr bool kStored = false;
  static __device__ __forceinline__ uint16_t pass(uint16_t v, double thr) {
    return ((double)v <= thr) ? (uint16_t)0 : v;
  }
  __device__ __forceinline__ uint16_t at(size_t i, double thr) const { return pass(sub[i], thr); }
  __device__ __forceinline__ void four(size_t q, double thr, uint16_t (&u)[4]) const {
    const ushort4 a = reinterpret_cast<const ushort4 *>(sub)[q];
    u[0] = pass(a.x, thr);
    u[1] = pass(a.y, thr);
    u[2] = pass(a.z, thr);
    u[3] = pass(a.w, thr);
  }
};
struct FromThresholded {
  const uint16_t *t16;
  static constexpr bool kStored = true;
  __device__ __forceinline__ uint16_t at(size_t i, double) const { return t16[i]; }
  __device__ __forceinline__ void four(size_t q, double, uint16_t (&u)[4]) const {
    const ushort4 a = reinterpret_cast<const ushort4 *>(t16)[q];
    u[0] = a.x;
    u[1] = a.y;
    u[2] = a.z;
    u[3] = a.w;
  }
};

// One pass over the frame: the thresholded pixels, the filtered frame cleared, and
// of the foreground pixels (in any order: components are numbered by their first
// block, sums are exact) the list and the union-find parents along row runs: a
// foreground pixel points at its left neighbour when that one is foreground too.
// Also clears the cell grid and the tile flags of the later kernels.  V pixels per
// thread at a time (V = 4 needs n a multiple of 4).
template <int V, typename Src>
__global__ void foreground_kernel(const Src src, PreState *st, uint16_t *__restrict__ t16,
                                  uint16_t *__restrict__ filt, int *__restrict__ par,
                                  unsigned *__restrict__ fg, int nx, size_t n, int *__restrict__ head,
                                  int cells, uint8_t *__restrict__ tiles, int ntiles) {
  const double thr = st->thresh;
  const int lane = threadIdx.x & 31;
  const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = first; i < (size_t)cells; i += stride) head[i] = -1;
  for (size_t i = first; i < (size_t)ntiles; i += stride) tiles[i] = 0;
  const size_t nv = n / V, rounds = (nv + stride - 1) / stride;
  for (size_t it = 0; it < rounds; ++it) {  // whole warps
    const size_t q = it * stride + first, i0 = q * V;
    uint16_t u[V];
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < V; ++j) u[j] = 0;
    if (q < nv) {
      if constexpr (V == 4)
        src.four(q, thr, u);
      else
        u[0] = src.at(q, thr);
    }
#pragma unroll
    for (int j = 0; j < V; ++j) bits |= u[j] ? 1u << j : 0u;
    if (q < nv) {
      if constexpr (V == 4) {
        if (!Src::kStored)
          reinterpret_cast<ushort4 *>(t16)[q] = make_ushort4(u[0], u[1], u[2], u[3]);
        reinterpret_cast<ushort4 *>(filt)[q] = make_ushort4(0, 0, 0, 0);
      } else {
        if (!Src::kStored) t16[q] = u[0];
        filt[q] = 0;
      }
    }
    if (!__any_sync(0xffffffffu, bits != 0u)) continue;
    const int cnt = __popc(bits);
    int x = cnt;  // the warp's places in the list
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    unsigned base = 0;
    if (lane == 31) base = atomicAdd(&st->n_fg, (unsigned)x);
    base = __shfl_sync(0xffffffffu, base, 31) + (unsigned)(x - cnt);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if (!u[j]) continue;
      const size_t i = i0 + j;
      fg[base++] = (unsigned)i;
      const bool left = i % nx != 0 && (j > 0 ? u[j > 0 ? j - 1 : 0] != 0 : src.at(i - 1, thr) != 0);
      par[i] = left ? (int)i - 1 : (int)i;
    }
  }
}

__device__ __forceinline__ int uf_find(int *L, int x) {
  int p = __ldcg(L + x);
  while (p != x) {
    x = p;
    p = __ldcg(L + x);
  }
  return x;
}

// Hang the larger root under the smaller; retry when another thread moved it.
__device__ void uf_union(int *L, int a, int b) {
  for (;;) {
    a = uf_find(L, a);
    b = uf_find(L, b);
    if (a == b) return;
    if (a > b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(L + b, a);
    if (old == b) return;
    b = old;
  }
}

// Joins each row run S = [s, e] to every run R of the row above that touches
// it (8-connectivity).  Row runs are already chained, so one join per pair
// suffices: at q, the leftmost pixel of R within [s-1, e+1], from the pixel
// max(s, q-1) of S.  Seen from a pixel x of S: the upper-left neighbour when
// x = s; the upper one when x = s and the upper-left is background; the
// upper-right one when the upper one is background.
__global__ void merge_kernel(const uint16_t *t16, int *L, int nx, const unsigned *fg,
                             const PreState *st) {
  const unsigned nf = st->n_fg;
  for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    const unsigned i = fg[f];
    const int y = (int)(i / nx), x = (int)(i % nx);
    if (y == 0) continue;
    const int p = (int)i;
    const bool left = x > 0 && t16[i - 1];
    const uint16_t *up = t16 + (i - nx);
    const bool ul = x > 0 && up[-1], uc = up[0], ur = x + 1 < nx && up[1];
    if (ul && !left) uf_union(L, p, p - nx - 1);
    if (uc && !left && !ul) uf_union(L, p, p - nx);
    if (ur && !uc) uf_union(L, p, p - nx + 1);
  }
}


struct Comps {
  int *area, *x0, *y0, *x1, *y1;
  unsigned *fb;  // first 2x2 block (raster index)
  unsigned long long *sw, *swx, *swy;
  int *label, *keep;
};

// Every foreground pixel points straight at its root; each root takes the
// next component id.
__global__ void compress_kernel(int *L, int *cid, PreState *st, Comps c, const unsigned *fg) {
  const unsigned nf = st->n_fg;
  for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    const unsigned i = fg[f];
    const int r = uf_find(L, (int)i);
    if (r != (int)i) {
      L[i] = r;
      continue;
    }
    const unsigned id = atomicAdd(&st->n_comp, 1u);
    cid[i] = (int)id;
    c.area[id] = 0;
    c.x0[id] = INT_MAX;
    c.y0[id] = INT_MAX;
    c.x1[id] = -1;
    c.y1[id] = -1;
    c.fb[id] = 0xffffffffu;
    c.sw[id] = c.swx[id] = c.swy[id] = 0;
  }
}

__global__ void moments_kernel(const int *L, const int *cid, const uint16_t *t16, Comps c, int nx,
                               const unsigned *fg, const PreState *st) {
  const unsigned nf = st->n_fg;
  const unsigned bw = (unsigned)(nx + 1) / 2;
  for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    const unsigned i = fg[f];
    const int r = L[i];
    const int id = cid[r];
    const int y = (int)(i / nx), x = (int)(i % nx);
    const unsigned long long w = t16[i];
    atomicAdd(c.area + id, 1);
    atomicMin(c.x0 + id, x);
    atomicMin(c.y0 + id, y);
    atomicMax(c.x1 + id, x);
    atomicMax(c.y1 + id, y);
    atomicMin(c.fb + id, (unsigned)(y >> 1) * bw + (unsigned)(x >> 1));
    atomicAdd(c.sw + id, w);
    atomicAdd(c.swx + id, w * (unsigned long long)x);
    atomicAdd(c.swy + id, w * (unsigned long long)y);
  }
}

// OpenCV numbers components by their first 2x2 block in raster order: a bit per
// block that is some component's first (and in a second map, some kept one's), the
// bits before each of 1024 segments of a map, and a component's number is the
// bits before its own.
__global__ void flags_kernel(const PreState *st, Comps c, int min_area, unsigned *bits,
                             unsigned *keep_bits) {
  const size_t nc = st->n_comp;
  for (size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x; id < nc;
       id += (size_t)gridDim.x * blockDim.x) {
    const unsigned fb = c.fb[id], bit = 1u << (fb & 31u);
    atomicOr(bits + (fb >> 5), bit);
    if (c.area[id] >= min_area) atomicOr(keep_bits + (fb >> 5), bit);
  }
}

constexpr int kSegs = 1024;
// Blocks 0 and 1: the two maps.  seg[s] = bits before segment s of len words;
// totals into the state.
__global__ void __launch_bounds__(kSegs) rank_bits_kernel(PreState *st, const unsigned *bits,
                                                          const unsigned *keep_bits, unsigned nwords,
                                                          unsigned len, unsigned *seg,
                                                          unsigned *keep_seg) {
  __shared__ unsigned warp_tot[kSegs / 32];
  const unsigned *b = blockIdx.x ? keep_bits : bits;
  unsigned *out = blockIdx.x ? keep_seg : seg;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned w0 = min((unsigned)t * len, nwords), w1 = min(w0 + len, nwords);
  unsigned mine = 0;
  unsigned k = w0;
  for (; k + 4 <= w1; k += 4) {  // len and the map's start are multiples of 4 words
    const uint4 v = *reinterpret_cast<const uint4 *>(b + k);
    mine += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
  }
  for (; k < w1; ++k) mine += __popc(b[k]);
  unsigned incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  unsigned before = incl - mine, total = 0;
  for (int j = 0; j < kSegs / 32; ++j) {
    if (j < w) before += warp_tot[j];
    total += warp_tot[j];
  }
  out[t] = before;
  if (t == 0) {
    if (blockIdx.x)
      st->n_keep = total;
    else
      st->n_labels = total + 1u;
  }
}

__device__ __forceinline__ unsigned bits_before(const unsigned *bits, const unsigned *seg, unsigned len,
                                                unsigned fb) {
  const unsigned w = fb >> 5, s = w / len;
  unsigned n = seg[s];
  for (unsigned k = s * len; k < w; ++k) n += __popc(bits[k]);
  return n + __popc(bits[w] & ((1u << (fb & 31u)) - 1u));
}

// Labels, boxes and centres; a kept component's centre joins its cell of the
// closest-pair grid.
__global__ void label_kernel(const PreState *st, Comps c, int min_area, const unsigned *bits,
                             const unsigned *keep_bits, const unsigned *seg, const unsigned *keep_seg,
                             unsigned len, double *centres, int *stats, int *head, int *next, int gcx,
                             int gcy) {
  const size_t nc = st->n_comp;
  for (size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x; id < nc;
       id += (size_t)gridDim.x * blockDim.x) {
    const unsigned fb = c.fb[id];
    const int label = (int)bits_before(bits, seg, len, fb) + 1;
    const bool keep = c.area[id] >= min_area;
    c.label[id] = label;
    const int x0 = c.x0[id], y0 = c.y0[id];
    int *sr = stats + (size_t)(label - 1) * 5;
    sr[0] = x0;
    sr[1] = y0;
    sr[2] = c.x1[id] - x0 + 1;
    sr[3] = c.y1[id] - y0 + 1;
    sr[4] = c.area[id];
    if (keep) {
      const int k = (int)bits_before(keep_bits, keep_seg, len, fb);
      c.keep[id] = k;
      const unsigned long long sw = c.sw[id];
      const double rx = (double)(c.swx[id] - (unsigned long long)x0 * sw);
      const double ry = (double)(c.swy[id] - (unsigned long long)y0 * sw);
      double *cr = centres + (size_t)k * 4;
      cr[0] = (double)label;
      cr[1] = lmb::dadd(lmb::ddiv(rx, (double)sw), (double)x0);
      cr[2] = lmb::dadd(lmb::ddiv(ry, (double)sw), (double)y0);
      cr[3] = (double)c.area[id];
      const int cx = min(max((int)(cr[1] / kCell), 0), gcx - 1);
      const int cy = min(max((int)(cr[2] / kCell), 0), gcy - 1);
      next[k] = atomicExch(head + cy * gcx + cx, k);
    } else {
      c.keep[id] = -1;
    }
  }
}

// Labels of all and of the kept components over zeroed frames (built only
// when a caller asks for them).
__global__ void labels_kernel(const int *__restrict__ L, const int *__restrict__ cid, Comps c,
                              int *__restrict__ labels, int *__restrict__ flabels,
                              const unsigned *fg, const PreState *st) {
  const unsigned nf = st->n_fg;
  for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    const unsigned i = fg[f];
    const int id = cid[L[i]];
    const int lab = c.label[id];
    labels[i] = lab;
    if (c.keep[id] >= 0) flabels[i] = lab;
  }
}

// ---- closest pair of centres (blur width) ---------------------------------------
__device__ __forceinline__ double pair_d2(const double *a, const double *b) {
  const double dx = lmb::dsub(a[1], b[1]), dy = lmb::dsub(a[2], b[2]);
  return lmb::dadd(lmb::dmul(dx, dx), lmb::dmul(dy, dy));
}

// Smallest double over the warp, one atomic per warp that found a pair.
__device__ __forceinline__ void warp_min_to(unsigned long long *dst, double v) {
  for (int o = 16; o; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0 && v < __longlong_as_double(0x7ff0000000000000ll))
    atomicMin(dst, (unsigned long long)__double_as_longlong(v));
}

// Every pair of kept centres, a warp of the grid for each first one.
__device__ __forceinline__ double all_pairs(const double *centres, unsigned n) {
  const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
  double best = __longlong_as_double(0x7ff0000000000000ll);
  for (unsigned i = warp; i < n; i += warps)
    for (unsigned j = i + 1 + (threadIdx.x & 31u); j < n; j += 32)
      best = fmin(best, pair_d2(centres + (size_t)i * 4, centres + (size_t)j * 4));
  return best;
}

constexpr int kBlurTile = 32;  // side of a blur tile
// Up to this many centres every pair is taken at once, by the whole grid: 28 pairs a
// thread at most, where the cells' lists are two dependent loads a centre.
constexpr unsigned kAllPairs = 2048;

// After the labels: the filtered frame (kept components' pixels over a cleared
// frame) with the blur tiles it touches, the closest pair of centres within
// neighbouring cells (of few centres, all pairs), and the first-block maps empty
// again.  Pairs in cells that are not neighbours lie more than a cell apart, so the
// cells' answer is exact when it is within a cell; otherwise the host, which reads it,
// has brute_pairs_kernel take every pair.  Measured on B200, 2048^2 frames of isolated
// spots, the component stage: 50 / 1000 / 2000 / 3500 of them 42 / 52 / 56 / 93 us; with
// the pairs in the last block of the cells' search 50 / 206 / 640 / 1760, in a kernel of
// one thread a centre, after slower ones, 93 / 214 / 384 / 644.
__global__ void finish_kernel(PreState *st, Comps c, const int *__restrict__ L,
                              const int *__restrict__ cid, const uint16_t *__restrict__ t16,
                              uint16_t *__restrict__ filt, const unsigned *fg, int nx,
                              uint8_t *__restrict__ tiles, int tiles_x, unsigned *bits,
                              unsigned *keep_bits, const double *centres, const int *head,
                              const int *next, int gcx, int gcy) {
  const unsigned first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const unsigned nf = st->n_fg, nc = st->n_comp, n = st->n_keep;
  for (unsigned f = first; f < nf; f += stride) {
    const unsigned i = fg[f];
    if (c.keep[cid[L[i]]] < 0) continue;
    filt[i] = t16[i];
    tiles[(i / nx / kBlurTile) * tiles_x + i % nx / kBlurTile] = 1;
  }
  for (unsigned id = first; id < nc; id += stride) {
    const unsigned w = c.fb[id] >> 5;
    bits[w] = 0u;
    keep_bits[w] = 0u;
  }
  if (n <= kAllPairs) {
    warp_min_to(&st->best, all_pairs(centres, n));
    return;
  }
  double best = __longlong_as_double(0x7ff0000000000000ll);
  for (unsigned i = first; i < n; i += stride) {
    const double *a = centres + (size_t)i * 4;
    const int cx = min(max((int)(a[1] / kCell), 0), gcx - 1);
    const int cy = min(max((int)(a[2] / kCell), 0), gcy - 1);
    for (int y = max(cy - 1, 0); y <= min(cy + 1, gcy - 1); ++y)
      for (int x = max(cx - 1, 0); x <= min(cx + 1, gcx - 1); ++x)
        for (int j = head[y * gcx + x]; j >= 0; j = next[j])
          if ((unsigned)j > i) best = fmin(best, pair_d2(a, centres + (size_t)j * 4));
  }
  warp_min_to(&st->best, best);
}

__global__ void brute_pairs_kernel(PreState *st, const double *centres) {
  warp_min_to(&st->best, all_pairs(centres, st->n_keep));
}

// ---- Gaussian blur ---------------------------------------------------------------
// scipy's symmetric correlation: w_c*x_0, then + (x_-j + x_+j) * w_j from the
// outermost pair inwards, every operation rounded on its own.
template <typename TIn>
__global__ void blur_rows_kernel(const TIn *in, const double *wts, int r, int ny, int nx,
                                 double *out) {
  extern __shared__ double w[];
  for (int j = threadIdx.x; j <= 2 * r; j += blockDim.x) w[j] = wts[j];
  __syncthreads();
  const size_t n = (size_t)ny * nx;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int y = (int)(i / nx), x = (int)(i % nx);
    double acc = lmb::dmul(to_f64(in[i]), w[r]);
    for (int j = r; j >= 1; --j) {
      const double a = to_f64(in[(size_t)mirror(y - j, ny) * nx + x]);
      const double b = to_f64(in[(size_t)mirror(y + j, ny) * nx + x]);
      acc = lmb::dadd(acc, lmb::dmul(lmb::dadd(a, b), w[r - j]));
    }
    out[i] = acc;
  }
}

template <typename TOut>
__global__ void blur_cols_kernel(const double *in, const double *wts, int r, int ny, int nx,
                                 TOut *out) {
  extern __shared__ double w[];
  for (int j = threadIdx.x; j <= 2 * r; j += blockDim.x) w[j] = wts[j];
  __syncthreads();
  const size_t n = (size_t)ny * nx;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const double *row = in + (i - x);
    double acc = lmb::dmul(row[x], w[r]);
    for (int j = r; j >= 1; --j)
      acc = lmb::dadd(acc, lmb::dmul(lmb::dadd(row[mirror(x - j, nx)], row[mirror(x + j, nx)]), w[r - j]));
    out[i] = (TOut)acc;
  }
}

// Both passes for a 32x32 output tile: the mirrored input tile with its halo
// in shared memory, the axis-0 pass over the tile's rows and halo columns,
// then the axis-1 pass; the same operations in the same order as the two
// separate passes, without the float64 intermediate in global memory.
constexpr int kBlurTileMaxR = 32;

size_t blur_tile_smem(int r) {
  const int W = kBlurTile + 2 * r;
  return (size_t)(2 * r + 1 + kBlurTile * W) * sizeof(double) + (size_t)W * W * sizeof(uint16_t);
}

template <typename TOut>
__global__ void __launch_bounds__(256)
    blur_tile_kernel(const uint16_t *__restrict__ in, const double *__restrict__ wts, int r, int ny,
                     int nx, TOut *__restrict__ out) {
  extern __shared__ double sm[];
  const int W = kBlurTile + 2 * r;
  double *w = sm;
  double *vert = sm + (2 * r + 1);
  uint16_t *tile = reinterpret_cast<uint16_t *>(vert + kBlurTile * W);
  const int x0 = blockIdx.x * kBlurTile, y0 = blockIdx.y * kBlurTile;
  const int tid = threadIdx.x;
  for (int j = tid; j <= 2 * r; j += blockDim.x) w[j] = wts[j];
  for (int idx = tid; idx < W * W; idx += blockDim.x) {
    const int ty = idx / W, tx = idx - ty * W;
    tile[idx] = in[(size_t)mirror(y0 - r + ty, ny) * nx + mirror(x0 - r + tx, nx)];
  }
  __syncthreads();
  for (int idx = tid; idx < kBlurTile * W; idx += blockDim.x) {
    const int ty = idx / W, tx = idx - ty * W;
    const uint16_t *col = tile + (ty + r) * W + tx;
    double acc = lmb::dmul((double)col[0], w[r]);
    for (int j = r; j >= 1; --j)
      acc = lmb::dadd(acc, lmb::dmul(lmb::dadd((double)col[-j * W], (double)col[j * W]), w[r - j]));
    vert[idx] = acc;
  }
  __syncthreads();
  for (int idx = tid; idx < kBlurTile * kBlurTile; idx += blockDim.x) {
    const int ty = idx / kBlurTile, tx = idx - ty * kBlurTile;
    const int gy = y0 + ty, gx = x0 + tx;
    if (gy >= ny || gx >= nx) continue;
    const double *row = vert + ty * W + tx + r;
    double acc = lmb::dmul(row[0], w[r]);
    for (int j = r; j >= 1; --j) acc = lmb::dadd(acc, lmb::dmul(lmb::dadd(row[-j], row[j]), w[r - j]));
    out[(size_t)gy * nx + gx] = (TOut)acc;
  }
}

// The same for radius R known at compile time (1..8; sigma 1 gives R = 4):
// each thread keeps a 4-output segment of a column (axis-0 pass) and then of
// a row (axis-1 pass) in registers, 4 + 2R inputs, each converted once.
constexpr int kBlurFixedMaxR = 8;

// tiles, unless null: the 32 x 32 tiles that hold a positive pixel.  A tile with
// none there nor in its eight neighbours (most of a filtered frame; a reach of R <=
// 8 pixels, mirrored or not, stays among them) is all zero: tiles is given when the
// weights are finite and not negative, so that no term has a sign.
// max_bits, unless null, takes the bits of the frame's largest positive value.
// Measured on B200 (cold caches), 2048^2 frame of 50 spots, float32 result: 37.4 us
// with every tile computed (FP64 issue), 25.3 us with empty tiles found by loading
// them, 14.2 us by the flags.
struct BlurWeights {
  double w[2 * kBlurFixedMaxR + 1];
};

template <int R, typename TOut>
__global__ void __launch_bounds__(256)
    blur_tile_r_kernel(const uint16_t *__restrict__ in, const BlurWeights wts, int ny, int nx,
                       const uint8_t *__restrict__ tiles, unsigned long long *__restrict__ max_bits,
                       TOut *__restrict__ out) {
  constexpr int W = kBlurTile + 2 * R;
  __shared__ double w[2 * R + 1];
  __shared__ double vert[kBlurTile * W];
  __shared__ uint16_t tile[W * W];
  const int x0 = blockIdx.x * kBlurTile, y0 = blockIdx.y * kBlurTile;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (tiles) {
    const int tx = (int)blockIdx.x + t % 3 - 1, ty = (int)blockIdx.y + t / 3 - 1;
    const bool any = t < 9 && tx >= 0 && tx < (int)gridDim.x && ty >= 0 && ty < (int)gridDim.y &&
                     tiles[ty * (int)gridDim.x + tx];
    if (!__syncthreads_or(any)) {
      if (x0 + kBlurTile <= nx && nx % 4 == 0) {  // 16-byte stores
        constexpr int kPer = 16 / sizeof(TOut), kRow = kBlurTile / kPer;
        for (int i = t; i < kBlurTile * kRow; i += 256) {
          const int gy = y0 + i / kRow;
          if (gy < ny)
            *reinterpret_cast<uint4 *>(out + (size_t)gy * nx + x0 + i % kRow * kPer) =
                make_uint4(0u, 0u, 0u, 0u);
        }
      } else {
        for (int row = warp; row < kBlurTile; row += 8)
          if (y0 + row < ny && x0 + lane < nx) out[(size_t)(y0 + row) * nx + x0 + lane] = (TOut)0;
      }
      return;
    }
  }
  if (t <= 2 * R) w[t] = wts.w[t];
  // mirrored source columns of this lane (W <= 48 < 64)
  const int c0 = mirror(x0 - R + lane, nx);
  const int c1 = lane + 32 < W ? mirror(x0 - R + lane + 32, nx) : 0;
  for (int row = warp; row < W; row += 8) {
    const uint16_t *src = in + (size_t)mirror(y0 - R + row, ny) * nx;
    tile[row * W + lane] = src[c0];
    if (lane + 32 < W) tile[row * W + lane + 32] = src[c1];
  }
  __syncthreads();
  double most = 0.0;
  // axis 0: task = (group of 4 output rows, tile column)
  for (int task = t; task < 8 * W; task += 256) {
    const int rg = task / W, col = task - rg * W;
    double v[4 + 2 * R];
#pragma unroll
    for (int q = 0; q < 4 + 2 * R; ++q) v[q] = (double)tile[(rg * 4 + q) * W + col];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      double acc = lmb::dmul(v[o + R], w[R]);
#pragma unroll
      for (int j = R; j >= 1; --j)
        acc = lmb::dadd(acc, lmb::dmul(lmb::dadd(v[o + R - j], v[o + R + j]), w[R - j]));
      vert[(rg * 4 + o) * W + col] = acc;
    }
  }
  __syncthreads();
  // axis 1: task = (output row, group of 4 output columns)
  {
    const int row = t >> 3, cg = (t & 7) * 4;
    const double *src = vert + row * W + cg;
    double v[4 + 2 * R];
#pragma unroll
    for (int q = 0; q < 4 + 2 * R; ++q) v[q] = src[q];
    const int gy = y0 + row;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      double acc = lmb::dmul(v[o + R], w[R]);
#pragma unroll
      for (int j = R; j >= 1; --j)
        acc = lmb::dadd(acc, lmb::dmul(lmb::dadd(v[o + R - j], v[o + R + j]), w[R - j]));
      const int gx = x0 + cg + o;
      if (gy < ny && gx < nx) {
        out[(size_t)gy * nx + gx] = (TOut)acc;
        if ((double)(TOut)acc > most) most = (double)(TOut)acc;
      }
    }
  }
  if (max_bits) {  // non-negative doubles order like their bits
    const unsigned long long b = warp_max_u64((unsigned long long)__double_as_longlong(most));
    if (lane == 0 && b) atomicMax(max_bits, b);
  }
}

template <typename TOut>
void blur_tile_r_launch(int r, dim3 grid, const uint16_t *in, const BlurWeights &w, int ny, int nx,
                        const uint8_t *tiles, unsigned long long *max_bits, TOut *out,
                        cudaStream_t st) {
#define LMB_BLUR_R(R)                                                                       \
  case R:                                                                                   \
    blur_tile_r_kernel<R, TOut><<<grid, 256, 0, st>>>(in, w, ny, nx, tiles, max_bits, out); \
    break;
  switch (r) {
    LMB_BLUR_R(1) LMB_BLUR_R(2) LMB_BLUR_R(3) LMB_BLUR_R(4)
    LMB_BLUR_R(5) LMB_BLUR_R(6) LMB_BLUR_R(7) LMB_BLUR_R(8)
  }
#undef LMB_BLUR_R
}

// ---- median ------------------------------------------------------------------------
__global__ void rank_keys_kernel(const double *img, unsigned long long *keys, unsigned *idx,
                                 size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    keys[i] = okey(img[i]);
    idx[i] = (unsigned)i;
  }
}

__global__ void rank_flags_kernel(const unsigned long long *keys, unsigned *flag, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    flag[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

__global__ void rank_scatter_kernel(const unsigned long long *keys, const unsigned *idx,
                                    const unsigned *flag, const unsigned *incl, unsigned *rank,
                                    double *vals, unsigned *n_distinct, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const unsigned r = incl[i] - 1u;
    rank[idx[i]] = r;
    if (flag[i]) vals[r] = okey_value(keys[i]);
    if (i == n - 1) *n_distinct = incl[i];
  }
}

__device__ __forceinline__ unsigned med_digit(unsigned r, int l, int L) {
  return (r >> (8 * (L - 1 - l))) & 255u;
}
__device__ __forceinline__ unsigned med_prefix(unsigned r, int l, int L) {
  const int sh = 8 * (L - l);
  return sh >= 32 ? 0u : (r >> sh);
}

// Add `delta` for rank r to every level whose path prefix it follows, and
// count it into `below` of the levels where its digit lies under the path's.
__device__ __forceinline__ void med_update(unsigned *h, const unsigned (&pp)[kMedLevels],
                                           const int (&path)[kMedLevels], int (&below)[kMedLevels],
                                           int L, unsigned r, int delta) {
#pragma unroll
  for (int l = 0; l < kMedLevels; ++l) {
    if (l >= L || med_prefix(r, l, L) != pp[l]) break;
    const unsigned d = med_digit(r, l, L);
    atomicAdd(h + l * 256 + d, (unsigned)delta);
    below[l] += (int)d < path[l] ? delta : 0;
  }
}

// Fill level l from the whole window (ranks whose digits above l equal pp).
__device__ void med_fill(unsigned *h, int l, int L, unsigned pp, const unsigned *rk, int ny,
                         int nx, int x, int y, int lo, int hi) {
  const int lane = threadIdx.x & 31;
  for (int j = lane; j < 256; j += 32) h[l * 256 + j] = 0;
  __syncwarp();
  for (int dy = -lo; dy <= hi; ++dy) {
    const unsigned *row = rk + (size_t)mirror(y + dy, ny) * nx;
    for (int dx = -lo + lane; dx <= hi; dx += 32) {
      const unsigned r = row[mirror(x + dx, nx)];
      if (l == 0 || med_prefix(r, l, L) == pp) atomicAdd(h + l * 256 + med_digit(r, l, L), 1u);
    }
  }
  __syncwarp();
}

// One warp per (column x, segment of rows): the window's ranks are kept as
// per-level histograms of 8-bit digits.  Level 0 counts every rank; level l
// counts the ranks whose higher digits equal the median's path so far, and
// below[l] how many of those have a smaller digit at l than the path.  When
// the window slides down one row, the leaving and entering rows update both.
// The median's digit at a level is kept while below <= k < below + count
// (the common case: a background changes slowly); otherwise a short walk
// over neighbouring bins or a scan of the level finds it, and the levels
// under a moved digit are refilled from the whole window.
__global__ void __launch_bounds__(kMedWarps * 32, 4)
    median_kernel(const unsigned *rk, const double *vals, const unsigned *n_distinct, int ny, int nx,
                  int s, int seg, double *out) {
  __shared__ __align__(16) unsigned hist[kMedWarps][kMedLevels * 256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nseg = (ny + seg - 1) / seg;
  const long long task = (long long)blockIdx.x * kMedWarps + warp;
  if (task >= (long long)nx * nseg) return;
  const int x = (int)(task % nx), sg = (int)(task / nx);
  const int y0 = sg * seg, y1 = min(ny, y0 + seg);
  const unsigned D = *n_distinct;
  const int bits = D <= 1 ? 1 : 32 - __clz(D - 1);
  const int L = (bits + 7) / 8;
  unsigned *h = hist[warp];
  int path[kMedLevels], below[kMedLevels];
  unsigned pp[kMedLevels];
#pragma unroll
  for (int l = 0; l < kMedLevels; ++l) {
    path[l] = -1;
    below[l] = 0;
    pp[l] = 0xffffffffu;
  }
  pp[0] = 0;
  const int lo = s / 2, hi = s - 1 - lo;
  const unsigned long long k = ((unsigned long long)s * s) / 2;
  med_fill(h, 0, L, 0, rk, ny, nx, x, y0, lo, hi);
  int rb = 0;  // shallowest level whose digit must be found by a full scan
  for (int y = y0; y < y1; ++y) {
    if (y > y0) {
      int mine[kMedLevels];
#pragma unroll
      for (int l = 0; l < kMedLevels; ++l) mine[l] = 0;
      const unsigned *ro = rk + (size_t)mirror(y - 1 - lo, ny) * nx;
      const unsigned *ri = rk + (size_t)mirror(y + hi, ny) * nx;
      for (int dx = -lo + lane; dx <= hi; dx += 32) {
        const int c = mirror(x + dx, nx);
        med_update(h, pp, path, mine, L, ro[c], -1);
        med_update(h, pp, path, mine, L, ri[c], 1);
      }
#pragma unroll
      for (int l = 0; l < kMedLevels; ++l)
        if (l < L) below[l] += __reduce_add_sync(0xffffffffu, mine[l]);
      __syncwarp();
    }
    unsigned long long kres = k;
    unsigned rank = 0;
#pragma unroll
    for (int l = 0; l < kMedLevels; ++l) {
      if (l >= L) break;
      const unsigned *hl = h + l * 256;
      bool found = false;
      if (l < rb) {
        // keep the digit, or walk a few bins from it
        long long b = below[l];
        int d = path[l];
        for (int step = 0; step < 8; ++step) {
          const long long c = hl[d];
          if ((long long)kres < b) {
            if (d == 0) break;
            --d;
            b -= hl[d];
          } else if ((long long)kres >= b + c) {
            if (d == 255) break;
            b += c;
            ++d;
          } else {
            found = true;
            break;
          }
        }
        if (found) {
          kres -= (unsigned long long)b;
          below[l] = (int)b;
          if (d != path[l]) {
            path[l] = d;
            if (rb > l + 1) rb = l + 1;
          }
        }
      } else if (l > 0) {
        med_fill(h, l, L, pp[l], rk, ny, nx, x, y, lo, hi);
      }
      if (!found) {
        const unsigned long long k0 = kres;
        const int d = (int)warp_find_digit(hl, kres);
        below[l] = (int)(k0 - kres);
        if (d != path[l]) {
          path[l] = d;
          if (rb > l + 1) rb = l + 1;
        }
        if (rb <= l) rb = l + 1;
      }
      rank = (rank << 8) | (unsigned)path[l];
      if (l + 1 < kMedLevels) pp[l + 1] = rank;
    }
    // a rank outside the distinct values would mean inconsistent histograms
    if (lane == 0)
      out[(size_t)y * nx + x] = rank < D ? vals[rank] : __longlong_as_double(0x7ff8000000000000ll);
  }
}

// Median of a frame of whole numbers (0..65535), tile by tile.
//
// A background changes slowly: the medians of the 64 x 32 windows around a tile are
// a handful of neighbouring values.  For one threshold t the number of values below
// t in every window of the tile comes from two sliding sums over the tile and its
// halo (in shared memory), and median >= t exactly when that number is at most
// k = s * s / 2.  A block starts at the median of 256 of its values and moves t by
// doubling steps, then by halves, until every pixel has count(m) <= k <
// count(m + 1): about one threshold for each value among the tile's medians, and a
// few more.  How many there are shows early: the range of the counts in the tile,
// divided by what a step of one adds to them.  A tile with more than kMedMost by the
// thresholds kMedLook and 0 (four times as many by 3 and 0), or one that kMedTries
// have not resolved, is counted in *unresolved and the frame takes the rank path; other
// blocks see that when they start and every eight thresholds.  A block's threshold
// takes 5 to 15 us, mostly latency.  Measured on B200, 2048^2 frames, ranks and median:
// a detector frame, s = 101, 2.75 ms on the rank path, 0.19 ms here; frames that end on
// the rank path (a steep background, s = 101; noise of standard deviation 1000, s = 31;
// random words, s = 31, three passes), whole call: 5.89, 2.96, 15.2 ms there alone,
// 7.34, 4.05, 18.4 with all 48 thresholds of every tile first, 6.02, 3.06, 15.4 as it
// is.  Values with gaps can look wilder than they are: multiples of 16, s = 31, are
// given up (2.19 ms) where 48 thresholds would do (1.03; s = 101 is not).
constexpr int kMtX = 64, kMtY = 32, kMtThreads = 256;
constexpr int kMedTries = 48;
constexpr int kMedLook = 5;   // the last threshold that the estimate is made from
constexpr int kMedMost = 40;  // as many values take some 48 thresholds (1.2 each and a few)
constexpr int kMedTileMaxS = 255;  // a column sum is a byte

size_t median_tile_smem(int s) {
  const size_t cols = kMtX + s - 1, rows = kMtY + s - 1;
  // values | column sums | per warp the prefix sums of a row | the sample
  return (rows * cols * 2 + 15) / 16 * 16 + (kMtY * cols + 15) / 16 * 16 +
         (kMtThreads / 32) * (cols + 1) * 4 + kMtThreads * 4;
}

// 48 registers: five blocks an SM where the window leaves room for them.
__global__ void __launch_bounds__(kMtThreads, 5)
    median_tile_kernel(const uint16_t *__restrict__ img, int ny, int nx, int s, double *__restrict__ out,
                       uint16_t *__restrict__ out16, unsigned *__restrict__ unresolved) {
  extern __shared__ __align__(16) double sm[];  // (declared as the blur's)
  const int cols = kMtX + s - 1, rows = kMtY + s - 1;
  uint16_t *val = reinterpret_cast<uint16_t *>(sm);
  unsigned char *csum = reinterpret_cast<unsigned char *>(sm) + ((size_t)rows * cols * 2 + 15) / 16 * 16;
  unsigned *pre_all = reinterpret_cast<unsigned *>(csum + ((size_t)kMtY * cols + 15) / 16 * 16);
  unsigned *sample = pre_all + (kMtThreads / 32) * (cols + 1);
  __shared__ unsigned key_s, guess_s;
  __shared__ unsigned least_s, most_s, sum_s;  // of the tile's counts below a threshold
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned lost = t == 0 ? __ldcg(unresolved) : 0u;
  unsigned *pre = pre_all + warp * (cols + 1);
  const int lo = s / 2;
  const int x0 = blockIdx.x * kMtX, y0 = blockIdx.y * kMtY;
  for (int r = warp; r < rows; r += kMtThreads / 32) {
    const uint16_t *src = img + (size_t)mirror(y0 - lo + r, ny) * nx;
    for (int c = lane; c < cols; c += 32) val[r * cols + c] = src[mirror(x0 - lo + c, nx)];
  }
  if (t == 0) guess_s = 0u;
  if (__syncthreads_or(lost != 0u)) return;
  // the median of 256 values spread over tile and halo
  sample[t] = val[(int)((long long)(2 * t + 1) * rows * cols / (2 * kMtThreads))];
  __syncthreads();
  {
    const unsigned mine = sample[t];
    int below = 0;
    for (int j = 0; j < kMtThreads; j++) below += sample[j] < mine ? 1 : 0;
    // the largest value with at most half of the sample below it
    if (below <= kMtThreads / 2) atomicMax(&guess_s, mine);
  }
  __syncthreads();
  // this thread's pixels: columns lane and lane + 32 of rows warp, warp + 8, ...
  constexpr int kRows = kMtY / (kMtThreads / 32), kOwn = 2 * kRows;
  unsigned L[kOwn], H[kOwn];  // L <= median < H
#pragma unroll
  for (int i = 0; i < kOwn; i++) {
    const int gx = x0 + lane + 32 * (i & 1), gy = y0 + warp + (i >> 1) * (kMtThreads / 32);
    L[i] = 0u;
    H[i] = gx < nx && gy < ny ? 65536u : 1u;  // outside the frame: nothing to find
  }
  const unsigned k = (unsigned)s * (unsigned)s / 2u;
  const int per = (cols + 31) / 32;
  unsigned thr = guess_s;
  unsigned step_up = 1u, step_down = 1u;
  unsigned thr0 = 0, sum0 = 0;  // the first threshold and its counts
  float medians = 1e30f;        // estimate of the values among the tile's medians
  bool found = false;
  for (int round = 0; round < kMedTries; round++) {
    const bool poll = (round & 7) == 7, look = round == 0 || round == 3 || round == kMedLook;
    if (poll && t == 0) lost = __ldcg(unresolved);
    unsigned least = 0xffffffffu, largest = 0u, sum_all = 0u;
    if (thr > 0u) {
      // values below thr: column sums of s rows, for every row of the tile
      for (int c = t; c < cols; c += kMtThreads) {
        const uint16_t *col = val + c;
        unsigned n = 0;
        for (int r = 0; r < s; r++) n += col[r * cols] < thr ? 1u : 0u;
        csum[c] = (unsigned char)n;
#pragma unroll 4
        for (int r = 1; r < kMtY; r++) {
          n += (col[(r + s - 1) * cols] < thr ? 1u : 0u) - (col[(r - 1) * cols] < thr ? 1u : 0u);
          csum[r * cols + c] = (unsigned char)n;
        }
      }
      if (t == 0) {
        key_s = least_s = 0xffffffffu;
        most_s = sum_s = 0u;
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kRows; q++) {
        const unsigned char *row = csum + (warp + q * (kMtThreads / 32)) * cols;
        unsigned sum = 0;
        for (int j = 0; j < per; j++) {
          const int c = lane * per + j;
          sum += c < cols ? row[c] : 0u;
        }
        unsigned run = sum;  // exclusive prefix sum over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned y = __shfl_up_sync(0xffffffffu, run, o);
          if (lane >= o) run += y;
        }
        run -= sum;
        for (int j = 0; j < per; j++) {
          const int c = lane * per + j;
          if (c > cols) break;
          pre[c] = run;
          run += c < cols ? row[c] : 0u;
        }
        if (lane == 31 && 32 * per <= cols) pre[cols] = run;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int x = lane + 32 * h;
          const unsigned cnt = pre[x + s] - pre[x];
          const int i = 2 * q + h;
          least = min(least, cnt);
          largest = max(largest, cnt);
          sum_all += cnt;
          if (cnt <= k)
            L[i] = max(L[i], thr);
          else
            H[i] = min(H[i], thr);
        }
        __syncwarp();
      }
    } else {
      if (t == 0) {
        key_s = least_s = 0xffffffffu;
        most_s = sum_s = 0u;
      }
      __syncthreads();
    }
    // the lowest interval still open: its ends say where to look next
    unsigned key = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < kOwn; i++)
      if (H[i] > L[i] + 1u) key = min(key, (L[i] << 16) | (H[i] - 1u));
    key = __reduce_min_sync(0xffffffffu, key);
    if (lane == 0 && key != 0xffffffffu) atomicMin(&key_s, key);
    if (look && thr > 0u) {  // uniform in the block
      least = __reduce_min_sync(0xffffffffu, least);
      largest = __reduce_max_sync(0xffffffffu, largest);
      sum_all = __reduce_add_sync(0xffffffffu, sum_all);
      if (lane == 0) {
        atomicMin(&least_s, least);
        atomicMax(&most_s, largest);
        atomicAdd(&sum_s, sum_all);
      }
    }
    const bool leave = poll ? __syncthreads_or(lost != 0u) : (__syncthreads(), false);
    const unsigned open = key_s, range = most_s - least_s, sum = sum_s;
    __syncthreads();  // before the next round's reset
    if (open == 0xffffffffu) {
      found = true;
      break;
    }
    if (leave) return;
    if (look && thr > 0u) {
      if (thr0 == 0u) {
        thr0 = thr;
        sum0 = sum;
      } else if (sum != sum0) {
        // values among the medians: the range over what a unit of threshold adds.  The
        // least of the estimates: frames whose values have gaps look wilder the further
        // the threshold moves without meeting one.
        const float units = thr > thr0 ? (float)(thr - thr0) : (float)(thr0 - thr);
        const float added = (sum > sum0 ? (float)(sum - sum0) : (float)(sum0 - sum)) / (kMtX * kMtY);
        medians = fminf(medians, (float)range * units / added);
      }
      if (medians < 1e30f && medians > (float)(round == kMedLook ? kMedMost : 4 * kMedMost)) break;
    }
    const unsigned l = open >> 16, h = (open & 0xFFFFu) + 1u;
    if (l == 0u && h == 65536u) {  // nothing known: only thr = 0 comes here
      thr = 1u;
    } else if (h == 65536u) {  // no upper end yet
      thr = min(l + step_up, 65535u);
      step_up *= 2u;
    } else if (l == 0u && h > step_down) {  // no lower end yet
      thr = h - step_down;
      step_down *= 2u;
    } else {
      thr = (l + h) / 2u;
    }
  }
  if (!found && t == 0) atomicAdd(unresolved, 1u);
#pragma unroll
  for (int i = 0; i < kOwn; i++) {
    const int gx = x0 + lane + 32 * (i & 1), gy = y0 + warp + (i >> 1) * (kMtThreads / 32);
    if (gx < nx && gy < ny) {
      out[(size_t)gy * nx + gx] = (double)L[i];
      out16[(size_t)gy * nx + gx] = (uint16_t)L[i];
    }
  }
}

// A frame as 16-bit whole numbers; *other is set when a value is not one.
template <typename T>
__global__ void whole_kernel(const T *__restrict__ in, uint16_t *__restrict__ out,
                             unsigned *__restrict__ other, size_t n) {
  bool bad = false;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double v = to_f64(in[i]);
    const bool ok = v >= 0.0 && v <= 65535.0 && v == trunc(v) && !signbit(v);
    bad |= !ok;
    out[i] = ok ? (uint16_t)v : (uint16_t)0;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(other, 1u);
}

}  // namespace

// ---- handle ------------------------------------------------------------------------
struct lmb_pre {
  int device = 0, ny = 0, nx = 0, num_sms = 148;
  size_t npx = 0, nblocks = 0;
  cudaStream_t st = nullptr;
  void *d_raw = nullptr;
  double *d_bg = nullptr, *d_sub = nullptr, *d_tmp = nullptr;
  void *d_out = nullptr;
  uint16_t *d_t16 = nullptr, *d_filt = nullptr;
  int *d_par = nullptr, *d_cid = nullptr, *d_lab = nullptr, *d_flab = nullptr;
  Comps c{};
  unsigned long long *d_compact = nullptr;
  unsigned *d_bits = nullptr;  // first-block maps (all, kept) and their segments' counts
  unsigned nwords = 0, seg_len = 4;
  uint16_t *d_sub16 = nullptr, *d_bg16 = nullptr;  // whole-number differences, background
  unsigned *d_bg_other = nullptr;                  // the background is no whole numbers,
  unsigned bg_other = 0;                           // on the host
  uint8_t *d_tiles = nullptr;                      // blur tiles with a positive pixel
  int tiles_x = 1, tiles_y = 1;
  unsigned *d_hist16 = nullptr;  // 65536-bin histogram of the first selection pass
  unsigned *d_fg = nullptr;  // foreground pixel list
  bool labels_ready = false;  // label images of the last segment built
  double *d_centres = nullptr, *d_w = nullptr;
  unsigned long long *d_max = nullptr;  // maximum of the blurred frame in d_out
  int *d_stats = nullptr, *d_head = nullptr, *d_next = nullptr;
  int gcx = 1, gcy = 1;
  PreState *d_state = nullptr, *h_state = nullptr;
  Staging staging;  // results into ordinary memory
  // median scratch, allocated on first use
  unsigned long long *m_keys = nullptr, *m_keys2 = nullptr;
  unsigned *m_idx = nullptr, *m_idx2 = nullptr, *m_flag = nullptr, *m_incl = nullptr,
           *m_rank = nullptr, *m_nd = nullptr;
  double *m_vals = nullptr, *m_img = nullptr;
  void *m_cub = nullptr;
  size_t m_cub_bytes = 0;
  // medians of whole numbers: frame and result as uint16 (taken in turn), and what
  // sends a frame to the rank path (not whole numbers, unresolved tiles)
  uint16_t *m_v16[2] = {nullptr, nullptr};
  unsigned *m_flag16 = nullptr;
  bool segmented = false;
  lmb_pre_counts last{};
  // stage events: frame upload, threshold, components, blur, download, median ranks, median
  cudaEvent_t ev[kPreEvents] = {};
  float ms[LMB_PRE_STAGES] = {};
  // blurred frame handed to an engine: ready on this stream, free once the
  // engine's quantisation has read it
  cudaEvent_t ev_out_ready = nullptr, ev_out_free = nullptr;
  bool out_in_use = false;
  bool blur_untimed = false;  // the last blur's events have not been read
};

namespace {

int check_pre(lmb_pre *p) {
  if (!p) {
    set_error("null preprocessing handle");
    return LMB_ERR_INVALID;
  }
  LMB_CUDA(cudaSetDevice(p->device));
  return LMB_OK;
}

void free_pre(lmb_pre *p) {
  if (!p) return;
  cudaSetDevice(p->device);
  if (p->st) cudaStreamSynchronize(p->st);
  if (p->out_in_use) cudaEventSynchronize(p->ev_out_free);  // an engine may still read d_out
  void *bufs[] = {p->d_raw, p->d_bg, p->d_sub, p->d_tmp, p->d_out, p->d_t16, p->d_filt, p->d_par,
                  p->d_cid, p->d_lab, p->d_flab, p->c.area, p->c.x0, p->c.y0, p->c.x1, p->c.y1,
                  p->c.fb, p->c.sw, p->c.swx, p->c.swy, p->c.label, p->c.keep, p->d_bits,
                  p->d_sub16, p->d_bg16, p->d_bg_other, p->d_tiles, p->d_compact, p->d_centres, p->d_w,
                  p->d_max, p->d_stats, p->d_head, p->d_next,
                  p->d_state, p->d_hist16, p->d_fg, p->m_keys, p->m_keys2, p->m_idx, p->m_idx2, p->m_flag,
                  p->m_incl, p->m_rank, p->m_nd, p->m_vals, p->m_img, p->m_cub,
                  p->m_v16[0], p->m_v16[1], p->m_flag16};
  for (void *b : bufs)
    if (b) cudaFree(b);
  if (p->h_state) cudaFreeHost(p->h_state);
  for (auto &e : p->ev)
    if (e) cudaEventDestroy(e);
  if (p->ev_out_ready) cudaEventDestroy(p->ev_out_ready);
  if (p->ev_out_free) cudaEventDestroy(p->ev_out_free);
  if (p->st) cudaStreamDestroy(p->st);
  delete p;
}

template <typename T>
int alloc(T **ptr, size_t count) {
  LMB_CUDA(cudaMalloc(reinterpret_cast<void **>(ptr), std::max<size_t>(count, 1) * sizeof(T)));
  return LMB_OK;
}

size_t pre_dtype_bytes(int dtype) {
  return dtype == LMB_F64 ? 8 : dtype == LMB_F32 ? 4 : dtype == LMB_U16 ? 2 : 1;
}

template <typename F>
int by_dtype(int dtype, F &&f) {
  switch (dtype) {
    case LMB_F64: return f((const double *)nullptr);
    case LMB_F32: return f((const float *)nullptr);
    case LMB_U16: return f((const uint16_t *)nullptr);
    case LMB_U8: return f((const uint8_t *)nullptr);
  }
  set_error("unknown dtype %d", dtype);
  return LMB_ERR_INVALID;
}

int upload_frame(lmb_pre *p, const void *frame, int dtype) {
  LMB_REQUIRE(frame, "null frame");
  LMB_CUDA(cudaMemcpyAsync(p->d_raw, frame, p->npx * pre_dtype_bytes(dtype),
                           cudaMemcpyHostToDevice, p->st));
  return LMB_OK;
}

// Blocks of the 16-bit pass: each handles at most 65535 values.
unsigned hist16_grid(const lmb_pre *p) {
  return (unsigned)std::max<size_t>((size_t)p->num_sms, p->npx / 60000 + 1);
}

// One order-statistic search.  The 16-bit first pass has run (fused with
// the subtraction, or launched here when `first_pass`); the 8-bit passes
// follow, the first over the frame, the rest over the keys it kept.
int run_select(lmb_pre *p, int mode, bool first_pass) {
  if (first_pass)
    sel_hist16_kernel<<<hist16_grid(p), kHist16Threads, kHist16Smem, p->st>>>(
        p->d_sub, (unsigned)p->npx, p->d_state, p->d_hist16, mode);
  for (int shift = kKeepShift; shift >= 0; shift -= 8) {
    // one wave of blocks over the frame; the kept keys' count is on the device
    const unsigned gp = (unsigned)(p->num_sms * (shift == kKeepShift ? 4 : 2));
    sel_hist_kernel<<<gp, kT, 0, p->st>>>(p->d_sub, p->npx, p->d_state, mode, shift, p->d_compact);
  }
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

// Subtraction fused with the value histogram, over a background of whole numbers.
// *whole: every candidate is a whole number in [0, 65535] and the threshold is set.
// 8- and 16-bit frames always are; of a float frame the host asks the device.  Not
// asking, and segmenting again when it was none, gave a fractional frame all the
// component kernels twice (2048^2 float32 call on B200: 1.23 ms, asking 1.19; a whole
// frame pays 0.95 -> 0.97).
int value_select(lmb_pre *p, int dtype, int mode, unsigned long long k0, int two, double gamma,
                 bool *whole) {
  int rc = by_dtype(dtype, [&](auto tag) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(tag)>>;
    value_hist_kernel<T><<<(unsigned)(p->num_sms * 4), kVhThreads, 0, p->st>>>(
        static_cast<const T *>(p->d_raw), p->d_bg16, p->d_sub16, (unsigned)p->npx, p->d_state,
        p->d_hist16, mode, k0, two, gamma);
    return LMB_OK;
  });
  if (rc) return rc;
  LMB_CUDA(cudaGetLastError());
  *whole = dtype == LMB_U8 || dtype == LMB_U16;
  if (*whole) return LMB_OK;
  LMB_CUDA(cudaMemcpyAsync(&p->h_state->value_path, &p->d_state->value_path, sizeof(unsigned),
                           cudaMemcpyDeviceToHost, p->st));
  LMB_CUDA(cudaStreamSynchronize(p->st));
  *whole = p->h_state->value_path != 0;
  return LMB_OK;
}

int subtract(lmb_pre *p, int dtype) {
  return by_dtype(dtype, [&](auto tag) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(tag)>>;
    subtract_kernel<T><<<(unsigned)grid_for(p->npx, p->num_sms), kT, 0, p->st>>>(
        static_cast<const T *>(p->d_raw), p->d_bg, p->d_sub, p->npx);
    return LMB_OK;
  });
}

// The background as 16-bit whole numbers, where it is; h_state->nonint says whether
// once the stream has been waited for.
int background_changed(lmb_pre *p) {
  LMB_CUDA(cudaMemsetAsync(p->d_bg_other, 0, sizeof(unsigned), p->st));
  whole_kernel<double><<<(unsigned)grid_for(p->npx, p->num_sms), kT, 0, p->st>>>(
      p->d_bg, p->d_bg16, p->d_bg_other, p->npx);
  LMB_CUDA(cudaGetLastError());
  LMB_CUDA(cudaMemcpyAsync(&p->h_state->nonint, p->d_bg_other, sizeof(unsigned), cudaMemcpyDeviceToHost,
                           p->st));
  return LMB_OK;
}

// np.percentile's order statistics and weight for n values (linear method).
void percentile_plan(size_t n, double pct, unsigned long long *k0, int *two, double *gamma) {
  const double q = pct / 100.0;
  const double vi = (double)(n - 1) * q;
  double prev = std::floor(vi);
  if (vi >= (double)(n - 1)) {
    *k0 = n - 1;
    *two = 0;
    prev = -1.0;
  } else if (vi < 0) {
    *k0 = 0;
    *two = 0;
    prev = 0.0;
  } else {
    *k0 = (unsigned long long)prev;
    *two = 1;
  }
  *gamma = vi - prev;
}

// Thresholded pixels, components, centres, filtered frame and closest pair; then
// the state on the host.
template <typename Src>
int segment_tail(lmb_pre *p, const Src &src, int min_area, lmb_pre_counts *counts) {
  cudaStream_t st = p->st;
  // kernels over the foreground list: its length is on the device
  const unsigned g = (unsigned)p->num_sms * 4;
  reset_counts_kernel<<<1, 1, 0, st>>>(p->d_state);
  const int cells = p->gcx * p->gcy, ntiles = p->tiles_x * p->tiles_y;
  if (p->npx % 4 == 0)
    foreground_kernel<4, Src><<<(unsigned)grid_for(p->npx / 4, p->num_sms), kT, 0, st>>>(
        src, p->d_state, p->d_t16, p->d_filt, p->d_par, p->d_fg, p->nx, p->npx, p->d_head, cells,
        p->d_tiles, ntiles);
  else
    foreground_kernel<1, Src><<<(unsigned)grid_for(p->npx, p->num_sms), kT, 0, st>>>(
        src, p->d_state, p->d_t16, p->d_filt, p->d_par, p->d_fg, p->nx, p->npx, p->d_head, cells,
        p->d_tiles, ntiles);
  LMB_CUDA(cudaEventRecord(p->ev[EV_SEG_THR], st));
  merge_kernel<<<g, kT, 0, st>>>(p->d_t16, p->d_par, p->nx, p->d_fg, p->d_state);
  compress_kernel<<<g, kT, 0, st>>>(p->d_par, p->d_cid, p->d_state, p->c, p->d_fg);
  moments_kernel<<<g, kT, 0, st>>>(p->d_par, p->d_cid, p->d_t16, p->c, p->nx, p->d_fg, p->d_state);
  unsigned *bits = p->d_bits, *keep_bits = bits + p->nwords;
  unsigned *seg = keep_bits + p->nwords, *keep_seg = seg + kSegs;
  flags_kernel<<<g, kT, 0, st>>>(p->d_state, p->c, min_area, bits, keep_bits);
  rank_bits_kernel<<<2, kSegs, 0, st>>>(p->d_state, bits, keep_bits, p->nwords, p->seg_len, seg,
                                        keep_seg);
  label_kernel<<<g, kT, 0, st>>>(p->d_state, p->c, min_area, bits, keep_bits, seg, keep_seg,
                                 p->seg_len, p->d_centres, p->d_stats, p->d_head, p->d_next, p->gcx,
                                 p->gcy);
  finish_kernel<<<(unsigned)p->num_sms * 2, kT, 0, st>>>(
      p->d_state, p->c, p->d_par, p->d_cid, p->d_t16, p->d_filt, p->d_fg, p->nx, p->d_tiles,
      p->tiles_x, bits, keep_bits, p->d_centres, p->d_head, p->d_next, p->gcx, p->gcy);
  p->labels_ready = false;
  LMB_CUDA(cudaGetLastError());
  LMB_CUDA(cudaEventRecord(p->ev[EV_SEG_CC], st));
  PreState *hs = p->h_state;
  LMB_CUDA(cudaMemcpyAsync(hs, p->d_state, sizeof(PreState), cudaMemcpyDeviceToHost, st));
  LMB_CUDA(cudaStreamSynchronize(st));
  if (hs->n_keep > kAllPairs &&
      __builtin_bit_cast(double, hs->best) > (double)kCell * (double)kCell) {
    brute_pairs_kernel<<<p->num_sms * 2, kT, 0, st>>>(p->d_state, p->d_centres);
    LMB_CUDA(cudaGetLastError());
    LMB_CUDA(cudaEventRecord(p->ev[EV_SEG_CC], st));
    LMB_CUDA(cudaMemcpyAsync(hs, p->d_state, sizeof(PreState), cudaMemcpyDeviceToHost, st));
    LMB_CUDA(cudaStreamSynchronize(st));
  }
  lmb_pre_counts out{};
  out.threshold = hs->thresh;
  out.n_labels = (int32_t)hs->n_labels;
  out.n_centres = (int32_t)hs->n_keep;
  double best;
  memcpy(&best, &hs->best, sizeof(best));
  out.min_dist2 = hs->n_keep >= 2 ? best : std::numeric_limits<double>::infinity();
  p->last = out;
  p->segmented = true;
  if (counts) *counts = out;
  return LMB_OK;
}

// Elapsed device time between two recorded events (the stream is synchronised).
int stage_times(lmb_pre *p, int a, int b, int slot) {
  float ms = 0.f;
  LMB_CUDA(cudaEventElapsedTime(&ms, p->ev[a], p->ev[b]));
  p->ms[slot] = ms;
  return LMB_OK;
}

int ensure_median_scratch(lmb_pre *p) {
  if (p->m_keys) return LMB_OK;
  int rc;
  if ((rc = alloc(&p->m_keys, p->npx)) || (rc = alloc(&p->m_keys2, p->npx)) ||
      (rc = alloc(&p->m_idx, p->npx)) || (rc = alloc(&p->m_idx2, p->npx)) ||
      (rc = alloc(&p->m_flag, p->npx)) || (rc = alloc(&p->m_incl, p->npx)) ||
      (rc = alloc(&p->m_rank, p->npx)) || (rc = alloc(&p->m_nd, 1)) ||
      (rc = alloc(&p->m_vals, p->npx)) || (rc = alloc(&p->m_img, p->npx)))
    return rc;
  size_t a = 0, b = 0;
  LMB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, a, p->m_keys, p->m_keys2, p->m_idx, p->m_idx2,
                                           (int)p->npx));
  LMB_CUDA(cub::DeviceScan::InclusiveSum(nullptr, b, p->m_flag, p->m_incl, (int)p->npx));
  p->m_cub_bytes = std::max(a, b);
  LMB_CUDA(cudaMalloc(&p->m_cub, p->m_cub_bytes));
  return LMB_OK;
}

// One median pass of d_in into d_out (both float64 on the device).
int median_pass(lmb_pre *p, const double *d_in, double *d_out, int size) {
  cudaStream_t st = p->st;
  const unsigned g = (unsigned)grid_for(p->npx, p->num_sms);
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_PASS], st));
  rank_keys_kernel<<<g, kT, 0, st>>>(d_in, p->m_keys, p->m_idx, p->npx);
  size_t tb = p->m_cub_bytes;
  LMB_CUDA(cub::DeviceRadixSort::SortPairs(p->m_cub, tb, p->m_keys, p->m_keys2, p->m_idx,
                                           p->m_idx2, (int)p->npx, 0, 64, st));
  rank_flags_kernel<<<g, kT, 0, st>>>(p->m_keys2, p->m_flag, p->npx);
  tb = p->m_cub_bytes;
  LMB_CUDA(cub::DeviceScan::InclusiveSum(p->m_cub, tb, p->m_flag, p->m_incl, (int)p->npx, st));
  rank_scatter_kernel<<<g, kT, 0, st>>>(p->m_keys2, p->m_idx2, p->m_flag, p->m_incl, p->m_rank,
                                        p->m_vals, p->m_nd, p->npx);
  // row segments: enough warps to fill every SM several times over
  const long long want = (long long)p->num_sms * 64 * 2;
  int seg = (int)std::max<long long>(16, ((long long)p->ny * p->nx + want - 1) / want);
  seg = std::min(seg, p->ny);
  const long long tasks = (long long)p->nx * ((p->ny + seg - 1) / seg);
  const unsigned blocks = (unsigned)((tasks + kMedWarps - 1) / kMedWarps);
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_RANK], st));
  median_kernel<<<blocks, kMedWarps * 32, 0, st>>>(p->m_rank, p->m_vals, p->m_nd, p->ny, p->nx,
                                                   size, seg, d_out);
  LMB_CUDA(cudaGetLastError());
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_K], st));
  return LMB_OK;
}

// All median passes of a frame of whole numbers; *done = false when it is none or a
// tile was not resolved (the rank path then starts again from the frame).  The last
// pass leaves the background as whole numbers too.
int median_whole(lmb_pre *p, int dtype, int size, int passes, bool *done) {
  *done = false;
  if (size > kMedTileMaxS) return LMB_OK;
  cudaStream_t st = p->st;
  const size_t smem = median_tile_smem(size);
  if (!p->m_flag16) {
    int rc;
    if ((rc = alloc(&p->m_v16[0], p->npx)) || (rc = alloc(&p->m_v16[1], p->npx)) ||
        (rc = alloc(&p->m_flag16, 1)))
      return rc;
  }
  LMB_CUDA(cudaFuncSetAttribute(median_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)median_tile_smem(kMedTileMaxS)));
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_PASS], st));
  LMB_CUDA(cudaMemsetAsync(p->m_flag16, 0, sizeof(unsigned), st));
  const unsigned g = (unsigned)grid_for(p->npx, p->num_sms);
  const uint16_t *in = p->m_v16[0];
  if (dtype == LMB_U16) {
    in = static_cast<const uint16_t *>(p->d_raw);
  } else {
    const int rc = by_dtype(dtype, [&](auto tag) {
      using T = std::remove_const_t<std::remove_pointer_t<decltype(tag)>>;
      whole_kernel<T><<<g, kT, 0, st>>>(static_cast<const T *>(p->d_raw), p->m_v16[0], p->m_flag16,
                                        p->npx);
      return LMB_OK;
    });
    if (rc) return rc;
  }
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_RANK], st));
  const dim3 tiles((p->nx + kMtX - 1) / kMtX, (p->ny + kMtY - 1) / kMtY);
  for (int i = 0; i < passes; ++i) {
    uint16_t *to = i + 1 < passes ? p->m_v16[(i + 1) & 1] : p->d_bg16;  // the background as whole numbers
    median_tile_kernel<<<tiles, kMtThreads, smem, st>>>(in, p->ny, p->nx, size, p->d_bg, to,
                                                        p->m_flag16);
    in = to;
  }
  LMB_CUDA(cudaGetLastError());
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_K], st));
  LMB_CUDA(cudaMemcpyAsync(&p->h_state->n_comp, p->m_flag16, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
  LMB_CUDA(cudaStreamSynchronize(st));
  *done = p->h_state->n_comp == 0;
  return LMB_OK;
}

}  // namespace

extern "C" {

int lmb_pre_create(int32_t device, int32_t nr_px_y, int32_t nr_px_x, lmb_pre **out) {
  LMB_REQUIRE(out, "null output");
  *out = nullptr;
  LMB_REQUIRE(nr_px_y > 0 && nr_px_x > 0, "frame size %d x %d", nr_px_y, nr_px_x);
  LMB_REQUIRE((long long)nr_px_y * nr_px_x < (1ll << 31), "frame of %lld pixels is too large",
              (long long)nr_px_y * nr_px_x);
  LMB_CUDA(cudaSetDevice(device));
  lmb_pre *p = new lmb_pre();
  p->device = device;
  p->ny = nr_px_y;
  p->nx = nr_px_x;
  p->npx = (size_t)nr_px_y * nr_px_x;
  p->nblocks = (size_t)((nr_px_y + 1) / 2) * ((nr_px_x + 1) / 2);
  p->gcx = (nr_px_x + kCell - 1) / kCell;
  p->gcy = (nr_px_y + kCell - 1) / kCell;
  p->tiles_x = (nr_px_x + kBlurTile - 1) / kBlurTile;
  p->tiles_y = (nr_px_y + kBlurTile - 1) / kBlurTile;
  // a map's words, and its segments' lengths, in multiples of 4
  p->nwords = (unsigned)((p->nblocks + 127) / 128 * 4);
  p->seg_len = std::max(4u, ((p->nwords + kSegs - 1) / kSegs + 3) / 4 * 4);
  cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, device);
  int rc = LMB_OK;
  auto fail = [&](int r) {
    free_pre(p);
    return r;
  };
  if (cudaStreamCreateWithFlags(&p->st, cudaStreamNonBlocking) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cudaStreamCreate", __FILE__, __LINE__));
  const size_t n = p->npx, nb = p->nblocks;
  if ((rc = alloc(reinterpret_cast<double **>(&p->d_raw), n)) || (rc = alloc(&p->d_bg, n)) ||
      (rc = alloc(&p->d_sub, n)) || (rc = alloc(&p->d_tmp, n)) ||
      (rc = alloc(reinterpret_cast<double **>(&p->d_out), n)) || (rc = alloc(&p->d_t16, n)) ||
      (rc = alloc(&p->d_filt, n)) || (rc = alloc(&p->d_par, n)) || (rc = alloc(&p->d_cid, n)) ||
      (rc = alloc(&p->d_lab, n)) || (rc = alloc(&p->d_flab, n)) || (rc = alloc(&p->c.area, nb)) ||
      (rc = alloc(&p->c.x0, nb)) || (rc = alloc(&p->c.y0, nb)) || (rc = alloc(&p->c.x1, nb)) ||
      (rc = alloc(&p->c.y1, nb)) || (rc = alloc(&p->c.fb, nb)) || (rc = alloc(&p->c.sw, nb)) ||
      (rc = alloc(&p->c.swx, nb)) || (rc = alloc(&p->c.swy, nb)) ||
      (rc = alloc(&p->c.label, nb)) || (rc = alloc(&p->c.keep, nb)) ||
      (rc = alloc(&p->d_bits, 2 * (size_t)p->nwords + 2 * kSegs)) || (rc = alloc(&p->d_sub16, n)) ||
      (rc = alloc(&p->d_bg16, n)) || (rc = alloc(&p->d_bg_other, 1)) ||
      (rc = alloc(&p->d_tiles, (size_t)p->tiles_x * p->tiles_y)) ||
      (rc = alloc(&p->d_compact, n)) || (rc = alloc(&p->d_centres, nb * 4)) ||
      (rc = alloc(&p->d_w, 1024)) || (rc = alloc(&p->d_max, 1)) || (rc = alloc(&p->d_stats, nb * 5)) ||
      (rc = alloc(&p->d_head, (size_t)p->gcx * p->gcy)) || (rc = alloc(&p->d_next, nb)) ||
      (rc = alloc(&p->d_state, 1)) || (rc = alloc(&p->d_hist16, 65536)) ||
      (rc = alloc(&p->d_fg, n)))
    return fail(rc);
  if (cudaMemset(p->d_hist16, 0, 65536 * sizeof(unsigned)) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cudaMemset", __FILE__, __LINE__));
  {
    // the 16-bit selection pass uses 128 KiB of shared memory per block
    const int b = (int)kHist16Smem;
    cudaError_t e = cudaFuncSetAttribute(sel_hist16_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaFuncSetAttribute", __FILE__, __LINE__));
  }
  for (auto &e : p->ev)
    if (cudaEventCreate(&e) != cudaSuccess)
      return fail(cuda_fail(cudaGetLastError(), "cudaEventCreate", __FILE__, __LINE__));
  if (cudaEventCreateWithFlags(&p->ev_out_ready, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&p->ev_out_free, cudaEventDisableTiming) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cudaEventCreate", __FILE__, __LINE__));
  if (cudaMallocHost(&p->h_state, sizeof(PreState)) != cudaSuccess)
    return fail(cuda_fail(cudaErrorMemoryAllocation, "cudaMallocHost", __FILE__, __LINE__));
  memset(p->h_state, 0, sizeof(PreState));
  p->h_state->best = 0x7ff0000000000000ull;
  if (cudaMemset(p->d_bg, 0, n * sizeof(double)) != cudaSuccess ||
      cudaMemset(p->d_bg16, 0, n * sizeof(uint16_t)) != cudaSuccess ||
      cudaMemset(p->d_bg_other, 0, sizeof(unsigned)) != cudaSuccess ||
      cudaMemset(p->d_bits, 0, 2 * (size_t)p->nwords * sizeof(unsigned)) != cudaSuccess ||
      cudaMemset(p->d_state, 0, sizeof(PreState)) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cudaMemset", __FILE__, __LINE__));
  *out = p;
  return LMB_OK;
}

int lmb_pre_destroy(lmb_pre *p) {
  if (!p) return LMB_OK;
  free_pre(p);
  return LMB_OK;
}

int lmb_pre_set_background(lmb_pre *p, const double *background) {
  int rc = check_pre(p);
  if (rc) return rc;
  p->bg_other = 1;  // until it has been looked at
  if (background)
    LMB_CUDA(cudaMemcpyAsync(p->d_bg, background, p->npx * sizeof(double), cudaMemcpyHostToDevice,
                             p->st));
  else
    LMB_CUDA(cudaMemsetAsync(p->d_bg, 0, p->npx * sizeof(double), p->st));
  if ((rc = background_changed(p))) return rc;
  LMB_CUDA(cudaStreamSynchronize(p->st));
  p->bg_other = p->h_state->nonint;
  return LMB_OK;
}

int lmb_pre_get_background(lmb_pre *p, double *out) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(out, "null output");
  return p->staging.download(out, p->d_bg, p->npx * sizeof(double), p->st);
}

int lmb_pre_median(lmb_pre *p, const void *frame, int32_t dtype, int32_t size, int32_t passes,
                   double *out) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(size >= 1, "median size %d", size);
  LMB_REQUIRE(!(p->ny > 1 && size >= 8 * p->ny) && !(p->nx > 1 && size >= 8 * p->nx),
              "median size %d reaches 8x the %d x %d frame", size, p->ny, p->nx);
  p->bg_other = 1;  // until it has been looked at
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED0], p->st));
  if ((rc = upload_frame(p, frame, dtype))) return rc;
  LMB_CUDA(cudaEventRecord(p->ev[EV_MED_UP], p->st));
  bool done = false;
  if (size > 1 && passes > 0 && (rc = median_whole(p, dtype, size, passes, &done))) return rc;
  if (!done && (rc = ensure_median_scratch(p))) return rc;
  const unsigned g = (unsigned)grid_for(p->npx, p->num_sms);
  if (!done) rc = by_dtype(dtype, [&](auto tag) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(tag)>>;
    to_f64_kernel<T><<<g, kT, 0, p->st>>>(static_cast<const T *>(p->d_raw), p->d_bg, p->npx);
    return LMB_OK;
  });
  if (rc) return rc;
  if (size > 1 && !done) {
    for (int i = 0; i < passes; ++i) {
      LMB_CUDA(cudaMemcpyAsync(p->m_img, p->d_bg, p->npx * sizeof(double),
                               cudaMemcpyDeviceToDevice, p->st));
      if ((rc = median_pass(p, p->m_img, p->d_bg, size))) return rc;
    }
  }
  if (!done && (rc = background_changed(p))) return rc;
  if (out && (rc = p->staging.download(out, p->d_bg, p->npx * sizeof(double), p->st))) return rc;
  LMB_CUDA(cudaStreamSynchronize(p->st));
  p->bg_other = done ? 0u : p->h_state->nonint;
  if (size > 1 && passes > 0)
    return stage_times(p, EV_MED0, EV_MED_UP, 5) || stage_times(p, EV_MED_PASS, EV_MED_RANK, 6) ||
           stage_times(p, EV_MED_RANK, EV_MED_K, 7);
  return stage_times(p, EV_MED0, EV_MED_UP, 5);
}

int lmb_pre_segment(lmb_pre *p, const void *frame, int32_t dtype, const lmb_pre_params *prm,
                    lmb_pre_counts *counts) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(prm, "null parameters");
  LMB_CUDA(cudaEventRecord(p->ev[EV_SEG0], p->st));
  if ((rc = upload_frame(p, frame, dtype))) return rc;
  LMB_CUDA(cudaEventRecord(p->ev[EV_SEG_UP], p->st));
  if (prm->override_thresh > 0 || prm->threshold_method == LMB_THR_FIXED) {
    if ((rc = subtract(p, dtype))) return rc;
    set_thresh_kernel<<<1, 1, 0, p->st>>>(
        p->d_state, prm->override_thresh > 0 ? prm->override_thresh : prm->threshold_value);
    rc = segment_tail(p, FromSub{p->d_sub}, prm->min_area, counts);
  } else {
    const bool pct = prm->threshold_method == LMB_THR_PERCENTILE;
    LMB_REQUIRE(pct || prm->threshold_method == LMB_THR_ADAPTIVE, "threshold method %d",
                prm->threshold_method);
    unsigned long long k0 = 0;
    int two = 0;
    double gamma = 0.0;
    if (pct) {
      LMB_REQUIRE(prm->threshold_percentile >= 0.0 && prm->threshold_percentile <= 100.0,
                  "Percentiles must be in the range [0, 100]");
      percentile_plan(p->npx, prm->threshold_percentile, &k0, &two, &gamma);
    }
    bool whole = false;  // a fractional background leaves hardly a whole difference
    if (!p->bg_other && (rc = value_select(p, dtype, pct ? SEL_ALL : SEL_NZ, k0, two, gamma, &whole)))
      return rc;
    if (whole) {
      rc = segment_tail(p, FromSub16{p->d_sub16}, prm->min_area, counts);
    } else {
      if ((rc = subtract(p, dtype))) return rc;
      if (pct) {
        sel_init_kernel<<<1, kT, 0, p->st>>>(p->d_state, SEL_ALL, p->npx, k0, two);
        if ((rc = run_select(p, SEL_ALL, true))) return rc;
        finish_percentile_kernel<<<1, 1, 0, p->st>>>(p->d_state, gamma);
      } else {
        sel_init_kernel<<<1, kT, 0, p->st>>>(p->d_state, SEL_NZ, p->npx, 0, 0);
        if ((rc = run_select(p, SEL_NZ, true))) return rc;
        finish_median_kernel<<<1, 1, 0, p->st>>>(p->d_state);
        sel_init_kernel<<<1, kT, 0, p->st>>>(p->d_state, SEL_ABSDEV, p->npx, 0, 0);
        if ((rc = run_select(p, SEL_ABSDEV, true))) return rc;
        finish_adaptive_kernel<<<1, 1, 0, p->st>>>(p->d_state);
      }
      rc = segment_tail(p, FromSub{p->d_sub}, prm->min_area, counts);
    }
  }
  if (rc) return rc;
  return stage_times(p, EV_SEG0, EV_SEG_UP, 0) || stage_times(p, EV_SEG_UP, EV_SEG_THR, 1) ||
         stage_times(p, EV_SEG_THR, EV_SEG_CC, 2);
}

int lmb_pre_segment_thresholded(lmb_pre *p, const uint16_t *thresholded, int32_t min_area,
                                lmb_pre_counts *counts) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(thresholded, "null frame");
  LMB_CUDA(cudaMemcpyAsync(p->d_t16, thresholded, p->npx * sizeof(uint16_t),
                           cudaMemcpyHostToDevice, p->st));
  set_thresh_kernel<<<1, 1, 0, p->st>>>(p->d_state, 0.0);
  LMB_CUDA(cudaGetLastError());
  return segment_tail(p, FromThresholded{p->d_t16}, min_area, counts);
}

int lmb_pre_centres(lmb_pre *p, double *centres, int32_t cap) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(p->segmented, "no frame segmented yet");
  const int n = std::min(cap, p->last.n_centres);
  LMB_REQUIRE(centres || n == 0, "null output");
  if (n > 0)
    LMB_CUDA(cudaMemcpy(centres, p->d_centres, (size_t)n * 4 * sizeof(double),
                        cudaMemcpyDeviceToHost));
  return LMB_OK;
}

int lmb_pre_stats(lmb_pre *p, int32_t *stats, int32_t cap) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(p->segmented, "no frame segmented yet");
  const int n = std::min(cap, p->last.n_labels - 1);
  LMB_REQUIRE(stats || n == 0, "null output");
  if (n > 0)
    LMB_CUDA(cudaMemcpy(stats, p->d_stats, (size_t)n * 5 * sizeof(int32_t),
                        cudaMemcpyDeviceToHost));
  return LMB_OK;
}

int lmb_pre_images(lmb_pre *p, uint16_t *thresholded, int32_t *labels, uint16_t *filt_img,
                   int32_t *filt_labels) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(p->segmented, "no frame segmented yet");
  const size_t n = p->npx;
  if ((labels || filt_labels) && !p->labels_ready) {
    LMB_CUDA(cudaMemsetAsync(p->d_lab, 0, n * sizeof(int), p->st));
    LMB_CUDA(cudaMemsetAsync(p->d_flab, 0, n * sizeof(int), p->st));
    labels_kernel<<<(unsigned)grid_for(n, p->num_sms), kT, 0, p->st>>>(
        p->d_par, p->d_cid, p->c, p->d_lab, p->d_flab, p->d_fg, p->d_state);
    LMB_CUDA(cudaGetLastError());
    p->labels_ready = true;
  }
  const struct {
    void *to;
    const void *from;
    size_t bytes;
  } frames[] = {{thresholded, p->d_t16, n * 2}, {labels, p->d_lab, n * 4}, {filt_img, p->d_filt, n * 2},
                {filt_labels, p->d_flab, n * 4}};
  for (const auto &f : frames)
    if (f.to && (rc = p->staging.download(f.to, f.from, f.bytes, p->st))) return rc;
  return LMB_OK;
}

}  // extern "C"

namespace {

// Both blur passes of the last segment's filtered frame into p->d_out; with
// want_max and a radius whose kernel finds it, the frame's maximum into p->d_max
// (*have_max).
int blur_launch(lmb_pre *p, const double *weights, int32_t radius, int32_t out_dtype,
                bool want_max = false, bool *have_max = nullptr) {
  LMB_REQUIRE(p->segmented, "no frame segmented yet");
  LMB_REQUIRE(weights, "null weights");
  LMB_REQUIRE(radius >= 0 && 2 * radius + 1 <= 1024, "blur radius %d outside 0..511", radius);
  LMB_REQUIRE(out_dtype == LMB_F64 || out_dtype == LMB_F32, "blur output dtype %d", out_dtype);
  if (p->out_in_use) {  // an engine may still be reading the previous blurred frame
    LMB_CUDA(cudaStreamWaitEvent(p->st, p->ev_out_free, 0));
    p->out_in_use = false;
  }
  LMB_CUDA(cudaEventRecord(p->ev[EV_BLUR0], p->st));
  const bool fixed = radius >= 1 && radius <= kBlurFixedMaxR;
  if (!fixed)
    LMB_CUDA(cudaMemcpyAsync(p->d_w, weights, (size_t)(2 * radius + 1) * sizeof(double),
                             cudaMemcpyHostToDevice, p->st));
  const unsigned g = (unsigned)grid_for(p->npx, p->num_sms);
  if (fixed) {
    const dim3 tg((unsigned)p->tiles_x, (unsigned)p->tiles_y);
    bool skip_zero = p->nx >= 2 * kBlurTile && p->ny >= 2 * kBlurTile;
    BlurWeights bw{};
    for (int j = 0; j <= 2 * radius; j++) {
      bw.w[j] = weights[j];
      if (!(std::isfinite(weights[j]) && !std::signbit(weights[j]))) skip_zero = false;
    }
    const uint8_t *tiles = skip_zero ? p->d_tiles : nullptr;
    if (want_max) LMB_CUDA(cudaMemsetAsync(p->d_max, 0, sizeof(unsigned long long), p->st));
    unsigned long long *mx = want_max ? p->d_max : nullptr;
    if (out_dtype == LMB_F64)
      blur_tile_r_launch<double>(radius, tg, p->d_filt, bw, p->ny, p->nx, tiles, mx,
                                 static_cast<double *>(p->d_out), p->st);
    else
      blur_tile_r_launch<float>(radius, tg, p->d_filt, bw, p->ny, p->nx, tiles, mx,
                                static_cast<float *>(p->d_out), p->st);
    if (have_max) *have_max = want_max;
  } else if (radius <= kBlurTileMaxR) {
    const dim3 tg((p->nx + kBlurTile - 1) / kBlurTile, (p->ny + kBlurTile - 1) / kBlurTile);
    const size_t tsm = blur_tile_smem(radius);
    if (out_dtype == LMB_F64)
      blur_tile_kernel<double><<<tg, 256, tsm, p->st>>>(p->d_filt, p->d_w, radius, p->ny, p->nx,
                                                        static_cast<double *>(p->d_out));
    else
      blur_tile_kernel<float><<<tg, 256, tsm, p->st>>>(p->d_filt, p->d_w, radius, p->ny, p->nx,
                                                       static_cast<float *>(p->d_out));
  } else {
    const size_t sm = (size_t)(2 * radius + 1) * sizeof(double);
    blur_rows_kernel<uint16_t><<<g, kT, sm, p->st>>>(p->d_filt, p->d_w, radius, p->ny, p->nx,
                                                     p->d_tmp);
    if (out_dtype == LMB_F64)
      blur_cols_kernel<double><<<g, kT, sm, p->st>>>(p->d_tmp, p->d_w, radius, p->ny, p->nx,
                                                     static_cast<double *>(p->d_out));
    else
      blur_cols_kernel<float><<<g, kT, sm, p->st>>>(p->d_tmp, p->d_w, radius, p->ny, p->nx,
                                                    static_cast<float *>(p->d_out));
  }
  LMB_CUDA(cudaGetLastError());
  LMB_CUDA(cudaEventRecord(p->ev[EV_BLUR_K], p->st));
  return LMB_OK;
}

}  // namespace

extern "C" {

int lmb_pre_blur(lmb_pre *p, const double *weights, int32_t radius, void *out, int32_t out_dtype) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(out, "null output");
  if ((rc = blur_launch(p, weights, radius, out_dtype))) return rc;
  rc = p->staging.download(out, p->d_out, p->npx * (out_dtype == LMB_F64 ? 8 : 4), p->st);
  if (rc) return rc;
  LMB_CUDA(cudaEventRecord(p->ev[EV_BLUR_DL], p->st));
  LMB_CUDA(cudaStreamSynchronize(p->st));
  p->blur_untimed = false;
  return stage_times(p, EV_BLUR0, EV_BLUR_K, 3) || stage_times(p, EV_BLUR_K, EV_BLUR_DL, 4);
}

int lmb_pre_blur_to_slot(lmb_pre *p, const double *weights, int32_t radius, lmb_engine *e,
                         int32_t slot, int32_t frame_dtype, double *im_scale) {
  int rc = check_pre(p);
  if (rc) return rc;
  LMB_REQUIRE(e, "null engine");
  LMB_REQUIRE(engine_device(e) == p->device, "engine on device %d, preprocessing on device %d",
              engine_device(e), p->device);
  bool have_max = false;
  if ((rc = blur_launch(p, weights, radius, frame_dtype, true, &have_max))) return rc;
  LMB_CUDA(cudaEventRecord(p->ev_out_ready, p->st));
  rc = engine_load_device_frame(e, slot, p->d_out, frame_dtype, p->ny, p->nx,
                                have_max ? p->d_max : nullptr, p->ev_out_ready, p->ev_out_free,
                                im_scale);
  if (rc) return rc;
  p->out_in_use = true;
  // The blur need not be waited for: the engine's stream waits for it, and what comes
  // next on this one follows it.  Small radii take their weights with the launch; for
  // others the caller's array must have been read.
  if (radius < 1 || radius > kBlurFixedMaxR) LMB_CUDA(cudaStreamSynchronize(p->st));
  p->blur_untimed = true;
  return LMB_OK;
}

int lmb_pre_timings(lmb_pre *p, float *ms, int32_t n) {
  LMB_REQUIRE(p && ms, "null argument");
  if (p->blur_untimed) {
    LMB_CUDA(cudaSetDevice(p->device));
    LMB_CUDA(cudaEventSynchronize(p->ev[EV_BLUR_K]));
    const int rc = stage_times(p, EV_BLUR0, EV_BLUR_K, 3);
    if (rc) return rc;
    p->blur_untimed = false;
  }
  for (int i = 0; i < n && i < LMB_PRE_STAGES; ++i) ms[i] = p->ms[i];
  return LMB_OK;
}

}  // extern "C"
