// DB build: forward simulation of the orientation DB on the device.
//
// Restates the per-orientation loop of LaueMatchingCPU.c:595-667 (the only
// implementation in the reference, copied at LaueMatchingGPU.cu:478-614 and
// LaueMatchingGPUStream.cu:854-946).  One thread owns one orientation and
// walks the HKL list in file order, appending on-detector, in-band,
// not-yet-seen pixels until MaxNrLaueSpots are taken.
//
// Arithmetic.  FP64 in the reference's exact operation order and rounding (no
// FMA; C truncation of the pixel coordinate as x86 performs it) alone decides
// acceptance and the pixel, so the records are the reference's, byte for byte.
// FP32 screens before it only REJECT, with margins above their error bounds:
//
//   band      E = (hc / 4 pi) |q|^2 / (-q_z) and sin(theta) = -q_z / |q|, and |q| of
//             an HKL is the same for every rotation: the energy band and the
//             scattering angles that the detector covers are an interval of |q_z|
//             per HKL, known on the host.  HKLs whose interval is empty are left
//             out of the build (of 1240 fcc HKLs at 5-30 keV a detector normal to
//             the beam at 500 mm can see 88, of 7790 hexagonal ones 256); the
//             others cost three FMAs and two comparisons, one test for h and -h
//             together (they differ in the sign of q_z, which says which of the two
//             has a positive energy; both reflect the same way).
//   detector  of those: z > 0 and the pixel inside the frame as linear
//             inequalities in the direction, without a division or a square root.
//             The list holds unit vectors, so a coordinate is one dot product and
//             one FMA (about 25 operations; |q|^2 and scaled margins per unit took
//             40).
//
// The HKLs that can be seen are taken in chunks of file order.  Each thread owns one orientation
// and keeps a bit per unit (a pair h, -h of the chunk, or a single HKL) that
// passed the band test, then a bit per HKL that passed both; it walks its own
// set bits, so the lanes of a warp stay busy over a whole chunk although they
// keep different HKLs.  FP64 then takes an orientation's HKLs in file order.
// The band test is bound by instruction issue (about 10 per unit and warp), the
// other two by the lane with the most bits of its warp.  Measured on B200 at 1e8
// synthetic orientations (whole build, one warp-wide FP32 test of energy and
// detector per HKL before): fcc beam-normal 644 -> 39 ms, tilted 34-ID-E detector
// 890 -> 234 ms, hexagonal beam-normal 3250 -> 66 ms; with unit vectors and
// chunks of 384 HKLs instead of 512 (six blocks per SM fit instead of five), 3e7
// orientations: tilted 60.8 -> 52.6 ms (of them FP64 20, detector test 27 before and
// about 20 now), hexagonal 13.5 -> 12.1, fcc 8.9 -> 8.0.  Chunks of 256: tilted 59.7
// where 384 gave 57.9, the lanes' numbers of bits being less equal.
//
// A matrix that is no rotation (rounded to a few digits, scaled, strained) has
// another |q| than the list says: its HKLs are all screened one by one, with |q|
// taken from the matrix.  2e5 matrices of 3 digits, B200, normal / tilted: 1.6 / 2.0
// ms, 4.6 / 5.0 with FP64 for every HKL.  A build flag (exact_all) and geometry
// outside the screens' assumptions take FP64 for every HKL.
//
// Layout.  Blocks of TB orientations; accepted pixels live in shared memory as
// [spot][thread] so the de-duplication scan is bank-conflict free; the block's
// records (contiguous in the DB) are written with coalesced stores.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <limits>
#include <map>
#include <tuple>
#include <vector>

#include "kernels.cuh"

namespace lmb {

struct BuildGeo {
  double recip[9], rt[9];
  double p0, p1, p2, px_x, px_y, cx, cy, elo, ehi;
  int W, H, S, R;
  // detector screen, direction d = (x, y, z) of a unit reflection vector q as
  // d = (-2 q_z) u + rt2, u = detector rotation . q: X = a x / tol = q_z (su u_x) + c and
  // the frame's edges as X + b0 z > 0, X + b1 z < 0 (b / tol), the same for y; z itself
  float sux, suy, cx2, cy2, cz2, bx0, bx1, by0, by1;
  float hc, elof, ehif;  // hc / 4 pi and the energies, for matrices that are no rotations
};

static constexpr double kHcKeVnm = 1.2398419739;              // LaueMatchingHeaders.h:41
static constexpr double kFourPi = 4.0 * 3.14159265358979323846;  // 4 * M_PI as C folds it
static constexpr int kHklChunk = 384;                // HKLs per chunk
static constexpr int kChunkWords = kHklChunk / 32;
static constexpr double kRotTol = 1e-4;  // a rotation: |OM^T OM - 1| below this
static constexpr double kBandTol = 4e-4;  // relative margin of |q| and |q|^2 (3 kRotTol and rounding)

// The units of a chunk: hkl / |q| (as floats) and the interval of |q_z| / |q| it can
// be seen in, as two bf16 (the lower bound in the high half, rounded down; the upper
// one rounded up); the error of its unit direction; the chunk positions of h (taken
// when q_z < 0) and of -h (q_z > 0), 0xFFFF for none.
struct BuildUnits {
  float4 hkl_band[kHklChunk];
  float eps[kHklChunk];
  uint32_t pos[kHklChunk];
};

// FP64 evaluation in the reference's exact order (LaueMatchingCPU.c:605-636,
// MatrixMultF LaueMatchingHeaders.h:361-369).  Returns acceptance and pixel.
__device__ __forceinline__ bool exact_spot(const double T[9], const int4 hk, const BuildGeo &g,
                                           int &ipx, int &ipy) {
  const double h = (double)hk.x, k = (double)hk.y, l = (double)hk.z;
  const double q0 = dadd(dadd(dadd(0.0, dmul(T[0], h)), dmul(T[1], k)), dmul(T[2], l));
  const double q1 = dadd(dadd(dadd(0.0, dmul(T[3], h)), dmul(T[4], k)), dmul(T[5], l));
  const double q2 = dadd(dadd(dadd(0.0, dmul(T[6], h)), dmul(T[7], k)), dmul(T[8], l));
  const double ql = dsqrt(dadd(dadd(dmul(q0, q0), dmul(q1, q1)), dmul(q2, q2)));
  if (ql == 0.0) return false;
  const double h0 = ddiv(q0, ql), h1 = ddiv(q1, ql), h2 = ddiv(q2, ql);
  const double td = dmul(2.0, h2);
  const double k0 = dsub(0.0, dmul(td, h0));
  const double k1 = dsub(0.0, dmul(td, h1));
  const double k2 = dsub(1.0, dmul(td, h2));
  const double x = dadd(dadd(dadd(0.0, dmul(g.rt[0], k0)), dmul(g.rt[1], k1)), dmul(g.rt[2], k2));
  const double y = dadd(dadd(dadd(0.0, dmul(g.rt[3], k0)), dmul(g.rt[4], k1)), dmul(g.rt[5], k2));
  const double z = dadd(dadd(dadd(0.0, dmul(g.rt[6], k0)), dmul(g.rt[7], k1)), dmul(g.rt[8], k2));
  if (z <= 0.0) return false;
  const double xp = dsub(ddiv(dmul(x, g.p2), z), g.p0);
  const double yp = dsub(ddiv(dmul(y, g.p2), z), g.p1);
  const int ix = x86_trunc_i32(dadd(ddiv(xp, g.px_x), g.cx));
  if (ix < 0 || ix > g.W - 1) return false;
  const int iy = x86_trunc_i32(dadd(ddiv(yp, g.px_y), g.cy));
  if (iy < 0 || iy > g.H - 1) return false;
  const double e = ddiv(dmul(kHcKeVnm, ql), dmul(kFourPi, -h2));
  if (e < g.elo || e > g.ehi) return false;
  ipx = ix;
  ipy = iy;
  return true;
}

constexpr float kUnitErr = 256.f / 16777216.f;  // BuildUnits::eps: this times sum |column| |h| / |q|
constexpr float kUnitErr0 = 4e-6f;              // ... and this

template <bool kExactAll>
__global__ void __launch_bounds__(128, 6) dbbuild_kernel(const double *__restrict__ om, uint64_t n,
                                                      const int4 *__restrict__ hkl,
                                                      const float4 *__restrict__ hklf, int nh,
                                                      const int4 *__restrict__ seen, int nseen,
                                                      const BuildUnits *__restrict__ units,
                                                      const uint32_t *__restrict__ unit_count,
                                                      const __grid_constant__ BuildGeo g,
                                                      uint16_t *__restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int TB = blockDim.x;
  BuildUnits *su = reinterpret_cast<BuildUnits *>(smem);
  uint32_t *sh_list = reinterpret_cast<uint32_t *>(smem + sizeof(BuildUnits));
  uint32_t *sh_cnt = sh_list + (size_t)g.S * TB;
  uint32_t *band = sh_cnt + TB;              // [kChunkWords][TB] units inside their band
  uint32_t *keep = band + kChunkWords * TB;  // [kChunkWords][TB] HKLs for FP64

  const int t = threadIdx.x;
  const uint64_t base = (uint64_t)blockIdx.x * TB;
  const uint64_t oid = base + t;
  const bool valid = oid < n;

  double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  float U[9];           // detector rotation . T, rows scaled (BuildGeo)
  float t0 = 0, t1 = 0, t2 = 0;  // T's last row
  bool regular = true;
  if (valid) {
    double m[9];
#pragma unroll
    for (int i = 0; i < 9; i++) m[i] = __ldg(om + oid * 9 + i);
    // thisOrient = OM . recip  (MatrixMultF33, LaueMatchingHeaders.h:349-357)
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int c = 0; c < 3; c++)
        T[r * 3 + c] = dadd(dadd(dmul(m[r * 3 + 0], g.recip[0 * 3 + c]),
                                 dmul(m[r * 3 + 1], g.recip[1 * 3 + c])),
                            dmul(m[r * 3 + 2], g.recip[2 * 3 + c]));
    if (!kExactAll) {
      // the band screen holds for rotations (NaN: not one)
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
          const double d = m[i] * m[j] + m[3 + i] * m[3 + j] + m[6 + i] * m[6 + j] - (i == j ? 1.0 : 0.0);
          regular = regular && fabs(d) <= kRotTol;
        }
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++)
          U[r * 3 + c] = (float)(g.rt[r * 3] * T[c] + g.rt[r * 3 + 1] * T[3 + c] + g.rt[r * 3 + 2] * T[6 + c]) *
                         (r == 0 ? g.sux : r == 1 ? g.suy : -2.f);
      t0 = (float)T[6];
      t1 = (float)T[7];
      t2 = (float)T[8];
    }
  }
  int cnt = 0;
  bool done = !valid || g.S <= 0;
  auto take = [&](const int4 h) {  // one HKL in FP64
    int ix = 0, iy = 0;
    if (!exact_spot(T, h, g, ix, iy)) return;
    const uint32_t key = (uint32_t)(ix & 0xFFFF) | ((uint32_t)(iy & 0xFFFF) << 16);
    bool dup = false;
    for (int s = 0; s < cnt; s++) dup |= (sh_list[(size_t)s * TB + t] == key);
    if (dup) return;
    sh_list[(size_t)cnt * TB + t] = key;
    done = ++cnt == g.S;
  };
  // The detector screen of a unit reflection vector (q_z, and u scaled as in BuildGeo)
  // with error m; nothing is off when m is NaN.
  auto off_detector = [&](float qz, float u0, float u1, float u2, float m) {
    const float x = fmaf(qz, u0, g.cx2), y = fmaf(qz, u1, g.cy2), z = fmaf(qz, u2, g.cz2);
    return z < -m || fmaf(g.bx0, z, x) < -m || fmaf(g.bx1, z, x) > m || fmaf(g.by0, z, y) < -m ||
           fmaf(g.by1, z, y) > m;
  };
  if (kExactAll) {
    for (int i = 0; i < nh && !done; i++) take(__ldg(hkl + i));
    done = true;
  } else if (!regular) {
    // No rotation: the whole list, a chunk's worth of bits at a time, with |q| from the
    // matrix.  Not a number anywhere: nothing is rejected.
    float col[3];
#pragma unroll
    for (int j = 0; j < 3; j++)
      col[j] = 1.00001f * (float)sqrt(T[j] * T[j] + T[3 + j] * T[3 + j] + T[6 + j] * T[6 + j]);
    const float a0 = (float)T[0], a1 = (float)T[1], a2 = (float)T[2];
    const float b0 = (float)T[3], b1 = (float)T[4], b2 = (float)T[5];
    float qz, rq, m;  // of an HKL: q_z and 1 / |q|, error of the unit vector
    auto reflect = [&](const float4 h) {
      qz = fmaf(t0, h.x, fmaf(t1, h.y, t2 * h.z));
      const float qx = fmaf(a0, h.x, fmaf(a1, h.y, a2 * h.z)), qy = fmaf(b0, h.x, fmaf(b1, h.y, b2 * h.z));
      const float ql2 = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
      rq = ql2 > 1e-20f && ql2 < 1e20f ? rsqrtf(ql2) : __int_as_float(0x7fc00000);
      const float sum = fmaf(col[0], fabsf(h.x), fmaf(col[1], fabsf(h.y), col[2] * fabsf(h.z)));
      m = fmaf(kUnitErr, sum * rq, kUnitErr0);
      return ql2 * rq;
    };
    for (int c0 = 0; c0 < nh && !done; c0 += kHklChunk) {
      const int cn = min(kHklChunk, nh - c0), words = (cn + 31) / 32;
      for (int w = 0; w < words; w++) {  // energy = hc |q| / (4 pi s), s = -q_z / |q|
        uint32_t bits = 0u;
        for (int b = 0; b < 32 && w * 32 + b < cn; b++) {
          const float e = g.hc * reflect(__ldg(hklf + c0 + w * 32 + b)), s = -qz * rq;
          const bool out = s < -m || e * (1.f - 2.f * m) > g.ehif * (s + m) ||
                           e * (1.f + 2.f * m) < g.elof * (s - m);
          if (!out) bits |= 1u << b;
        }
        band[w * TB + t] = bits;
      }
      for (int w = 0; w < words; w++) {
        uint32_t kept = 0u;
        for (uint32_t bits = band[w * TB + t]; bits; bits &= bits - 1u) {
          const int b = __ffs(bits) - 1;
          const float4 h = __ldg(hklf + c0 + w * 32 + b);
          reflect(h);
          const float u0 = fmaf(U[0], h.x, fmaf(U[1], h.y, U[2] * h.z)) * rq;
          const float u1 = fmaf(U[3], h.x, fmaf(U[4], h.y, U[5] * h.z)) * rq;
          const float u2 = fmaf(U[6], h.x, fmaf(U[7], h.y, U[8] * h.z)) * rq;
          if (!off_detector(qz * rq, u0, u1, u2, m)) kept |= 1u << b;
        }
        keep[w * TB + t] = kept;
      }
      int w = -1;
      uint32_t bits = 0u;
      while (!done) {
        while (bits == 0u && ++w < words) bits = keep[w * TB + t];
        if (w >= words) break;
        const int i = c0 + w * 32 + __ffs(bits) - 1;
        bits &= bits - 1u;
        take(__ldg(hkl + i));
      }
    }
    done = true;
  }
  for (int c0 = 0, chunk = 0; !kExactAll && c0 < nseen; c0 += kHklChunk, chunk++) {
    const int words = (min(kHklChunk, nseen - c0) + 31) / 32;
    const int nu = (int)unit_count[chunk];  // a multiple of 32, the rest never passes
    __syncthreads();
    const BuildUnits *src = units + chunk;
    for (int i = t; i < nu; i += TB) {
      su->hkl_band[i] = src->hkl_band[i];
      su->eps[i] = src->eps[i];
      su->pos[i] = src->pos[i];
    }
    __syncthreads();
    if (!done) {
      for (int w = 0; w < words; w++) keep[w * TB + t] = 0u;
      const int uw = nu / 32;
      for (int w = 0; w < uw; w++) {
        uint32_t bits = 0u;
#pragma unroll
        for (int b = 0; b < 32; b++) {
          const float4 h = su->hkl_band[w * 32 + b];
          const float q = fabsf(fmaf(t0, h.x, fmaf(t1, h.y, t2 * h.z)));
          const float lo = __uint_as_float(__float_as_uint(h.w) & 0xFFFF0000u);
          const float hi = __uint_as_float(__float_as_uint(h.w) << 16);
          if (!(q < lo) && !(q > hi)) bits |= 1u << b;
        }
        band[w * TB + t] = bits;
      }
      // detector
      int w = -1;
      uint32_t bits = 0u;
      for (;;) {
        while (bits == 0u && ++w < uw) bits = band[w * TB + t];
        if (w >= uw) break;
        const int u = w * 32 + __ffs(bits) - 1;
        bits &= bits - 1u;
        const float4 h = su->hkl_band[u];
        const float m = su->eps[u];  // error of the unit direction
        const uint32_t pos = su->pos[u];
        const float qz = fmaf(t0, h.x, fmaf(t1, h.y, t2 * h.z));
        const float u0 = fmaf(U[0], h.x, fmaf(U[1], h.y, U[2] * h.z));
        const float u1 = fmaf(U[3], h.x, fmaf(U[4], h.y, U[5] * h.z));
        const float u2 = fmaf(U[6], h.x, fmaf(U[7], h.y, U[8] * h.z));
        if (off_detector(qz, u0, u1, u2, m)) continue;
        const bool either = !(fabsf(qz) > m);  // q_z may have either sign (or m is NaN)
        const uint32_t i = pos & 0xFFFFu, j = pos >> 16;
        if ((qz < 0.f || either) && i != 0xFFFFu) keep[(i >> 5) * TB + t] |= 1u << (i & 31u);
        if ((!(qz < 0.f) || either) && j != 0xFFFFu) keep[(j >> 5) * TB + t] |= 1u << (j & 31u);
      }
      // FP64 over the kept HKLs in file order
      w = -1;
      bits = 0u;
      while (!done) {
        while (bits == 0u && ++w < words) bits = keep[w * TB + t];
        if (w >= words) break;
        const int i = c0 + w * 32 + __ffs(bits) - 1;
        bits &= bits - 1u;
        take(__ldg(seen + i));
      }
    }
    if (__syncthreads_and(done)) break;
  }
  sh_cnt[t] = (uint32_t)cnt;
  __syncthreads();
  // Coalesced store of this block's records: [count, x0, y0, ...] zero padded.
  if (base >= n) return;
  const uint32_t nvalid = (uint32_t)min((uint64_t)TB, n - base);
  const uint32_t R = (uint32_t)g.R;
  const uint32_t total = nvalid * R;
  uint16_t *dst = out + base * R;
  auto field = [&](uint32_t o, uint32_t f) -> uint32_t {
    if (f == 0) return sh_cnt[o];
    const uint32_t s = (f - 1) >> 1;
    if (s >= sh_cnt[o]) return 0u;
    const uint32_t key = sh_list[(size_t)s * TB + o];
    return (f & 1) ? key & 0xFFFFu : key >> 16;
  };
  // two fields per store: a block's records start on a 4-byte boundary (TB is even)
  const uint32_t step_o = 2u * TB / R, step_f = 2u * TB - step_o * R;
  uint32_t o = 2u * t / R, f = 2u * t - o * R;
  for (uint32_t w = 2u * t; w < total; w += 2u * TB) {
    const uint32_t lo = field(o, f);
    const bool wrap = f + 1 == R;
    if (w + 1 < total)
      *reinterpret_cast<uint32_t *>(dst + w) = lo | field(wrap ? o + 1 : o, wrap ? 0u : f + 1) << 16;
    else
      dst[w] = (uint16_t)lo;
    o += step_o;
    f += step_f;
    if (f >= R) {
      f -= R;
      o++;
    }
  }
}

// Synthetic orientations: Shoemake's uniform rotations from a counter-based
// generator (SplitMix64 finaliser of counter*golden + seed*constant), the
// same uniforms as lauematching_b200/synth.py.
__device__ __forceinline__ double u01(uint64_t seed, uint64_t c) {
  uint64_t z = c * 0x9E3779B97F4A7C15ull + seed * 0xD1B54A32D192ED03ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// Symmetry quaternions (w, x, y, z), normalised, of a fundamental-zone
// reduction of the synthetic orientations (nsym = 0: none).
struct SynthSym {
  int nsym;
  double q[24][4];
};

__global__ void synth_orient_kernel(uint64_t seed, uint64_t first, uint64_t n,
                                    double *__restrict__ out, const SynthSym sym) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t id = first + i;
    const double u1 = u01(seed, id * 3 + 0), u2 = u01(seed, id * 3 + 1),
                 u3 = u01(seed, id * 3 + 2);
    const double a = sqrt(1.0 - u1), b = sqrt(u1);
    double s2, c2, s3, c3;
    sincospi(2.0 * u2, &s2, &c2);
    sincospi(2.0 * u3, &s3, &c3);
    double x = a * s2, y = a * c2, z = b * s3, w = b * c3;
    if (sym.nsym > 0) {
      // of the equivalent rotations r (x) q keep the one with the largest
      // |scalar part| (the first such), scalar part made non-negative and
      // renormalised: the operator order and product of
      // LaueMatchingHeaders.h:111-122,166-178, as synth.hexagonal_fundamental_zone
      int best = 0;
      double bw = -1.0;
      for (int k = 0; k < sym.nsym; k++) {
        const double *r = sym.q[k];
        const double wk = fabs(r[0] * w - r[1] * x - r[2] * y - r[3] * z);
        if (wk > bw) {
          bw = wk;
          best = k;
        }
      }
      const double *r = sym.q[best];
      double Q0 = r[0] * w - r[1] * x - r[2] * y - r[3] * z;
      double Q1 = r[1] * w + r[0] * x + r[3] * y - r[2] * z;
      double Q2 = r[2] * w + r[0] * y + r[1] * z - r[3] * x;
      double Q3 = r[3] * w + r[0] * z + r[2] * x - r[1] * y;
      const double sg = Q0 < 0 ? -1.0 : 1.0;
      const double inv = sg / sqrt(Q0 * Q0 + Q1 * Q1 + Q2 * Q2 + Q3 * Q3);
      w = Q0 * inv;
      x = Q1 * inv;
      y = Q2 * inv;
      z = Q3 * inv;
    }
    double *o = out + i * 9;
    o[0] = 1.0 - 2.0 * (y * y + z * z);
    o[1] = 2.0 * (x * y - z * w);
    o[2] = 2.0 * (x * z + y * w);
    o[3] = 2.0 * (x * y + z * w);
    o[4] = 1.0 - 2.0 * (x * x + z * z);
    o[5] = 2.0 * (y * z - x * w);
    o[6] = 2.0 * (x * z - y * w);
    o[7] = 2.0 * (y * z + x * w);
    o[8] = 1.0 - 2.0 * (x * x + y * y);
  }
}

static BuildGeo make_build_geo(const lmb_geometry &geo) {
  BuildGeo g;
  for (int i = 0; i < 9; i++) {
    g.recip[i] = geo.recip[i];
    g.rt[i] = geo.rot_t[i];
  }
  g.p0 = geo.p[0];
  g.p1 = geo.p[1];
  g.p2 = geo.p[2];
  g.px_x = geo.px_x;
  g.px_y = geo.px_y;
  g.cx = 0.5 * (geo.nr_px_x - 1);
  g.cy = 0.5 * (geo.nr_px_y - 1);
  g.elo = geo.elo;
  g.ehi = geo.ehi;
  g.W = geo.nr_px_x;
  g.H = geo.nr_px_y;
  g.S = geo.max_nr_spots;
  g.R = 1 + 2 * geo.max_nr_spots;
  // pixel * z = a * x + b * z must lie in (-z, N z); an error m of x and z is one of
  // tol * m in that
  const double ax = g.p2 / g.px_x, bx = g.cx - g.p0 / g.px_x;
  const double ay = g.p2 / g.px_y, by = g.cy - g.p1 / g.px_y;
  const double tolx = std::fabs(ax) + std::max(std::fabs(bx + 1.0), std::fabs(bx - g.W));
  const double toly = std::fabs(ay) + std::max(std::fabs(by + 1.0), std::fabs(by - g.H));
  g.sux = (float)(-2.0 * ax / tolx);
  g.suy = (float)(-2.0 * ay / toly);
  g.cx2 = (float)(ax / tolx * g.rt[2]);
  g.cy2 = (float)(ay / toly * g.rt[5]);
  g.cz2 = (float)g.rt[8];
  g.bx0 = (float)((bx + 1.0) / tolx);
  g.bx1 = (float)((bx - g.W) / tolx);
  g.by0 = (float)((by + 1.0) / toly);
  g.by1 = (float)((by - g.H) / toly);
  g.hc = (float)(kHcKeVnm / kFourPi);
  g.elof = (float)g.elo;
  g.ehif = (float)g.ehi;
  return g;
}

// The screens assume finite values in FP32 range, an orthonormal detector
// rotation and a band of non-negative energies.
static bool screen_sound(const lmb_geometry &geo) {
  auto ok = [](double v) { return std::isfinite(v) && std::fabs(v) < 1e15; };
  for (int i = 0; i < 9; i++)
    if (!ok(geo.rot_t[i]) || !ok(geo.recip[i])) return false;
  for (int i = 0; i < 3; i++)
    for (int j = i; j < 3; j++) {
      double d = i == j ? -1.0 : 0.0;
      for (int k = 0; k < 3; k++) d += geo.rot_t[3 * i + k] * geo.rot_t[3 * j + k];
      if (!(std::fabs(d) < 1e-9)) return false;
    }
  for (int i = 0; i < 3; i++)
    if (!ok(geo.p[i])) return false;
  if (!ok(geo.px_x) || !ok(geo.px_y) || geo.px_x == 0 || geo.px_y == 0) return false;
  for (double v : {geo.p[2] / geo.px_x, geo.p[2] / geo.px_y, geo.p[0] / geo.px_x, geo.p[1] / geo.px_y})
    if (!ok(v)) return false;
  return ok(geo.elo) && ok(geo.ehi) && geo.elo >= 0.0 && geo.ehi > 0.0;
}

// sin(theta) of the directions that reach the detector (with a pixel to spare on
// every side), from a grid of cells of the detector plane at z = 1: a cell's
// directions lie within its half diagonal of its centre's (an angle is at most
// the distance in that plane).
static void detector_angles(const lmb_geometry &geo, double *smin, double *smax) {
  *smin = 0.0;
  *smax = 1.0;
  if (geo.p[2] == 0.0) return;
  const double xa = ((-1.0 - 0.5 * (geo.nr_px_x - 1)) * geo.px_x + geo.p[0]) / geo.p[2];
  const double xb = ((geo.nr_px_x - 0.5 * (geo.nr_px_x - 1)) * geo.px_x + geo.p[0]) / geo.p[2];
  const double ya = ((-1.0 - 0.5 * (geo.nr_px_y - 1)) * geo.px_y + geo.p[1]) / geo.p[2];
  const double yb = ((geo.nr_px_y - 0.5 * (geo.nr_px_y - 1)) * geo.px_y + geo.p[1]) / geo.p[2];
  const int kCells = 64;
  const double dx = (xb - xa) / kCells, dy = (yb - ya) / kCells;
  const double r = 0.5 * std::sqrt(dx * dx + dy * dy) * (1.0 + 1e-9) + 1e-9;
  double lo = 4.0, hi = -4.0;  // 2 theta
  for (int i = 0; i < kCells; i++)
    for (int j = 0; j < kCells; j++) {
      const double x = xa + (i + 0.5) * dx, y = ya + (j + 0.5) * dy;
      const double k = (geo.rot_t[2] * x + geo.rot_t[5] * y + geo.rot_t[8]) / std::sqrt(x * x + y * y + 1.0);
      const double a = std::acos(std::max(-1.0, std::min(1.0, k)));
      lo = std::min(lo, a - r);
      hi = std::max(hi, a + r);
    }
  const double pi = kFourPi / 4.0;
  if (lo > 0.0 && lo < pi) *smin = std::sin(0.5 * lo) * (1.0 - 1e-6);
  if (hi > 0.0 && hi < pi) *smax = std::min(1.0, std::sin(0.5 * hi) * (1.0 + 1e-6));
}

// A bf16 not above (down) or not below v >= 0, as its 16 bits.
static uint32_t bf16_bound(double v, bool down) {
  float f = (float)std::min(v, 3e38);
  if (down && (double)f > v) f = std::nextafter(f, 0.f);
  if (!down && (double)f < v) f = std::nextafter(f, std::numeric_limits<float>::infinity());
  uint32_t b;
  memcpy(&b, &f, 4);
  return (down ? b : b + 0xFFFFu) >> 16;
}

// The HKLs that some rotation can put on the detector within the energy band, in
// file order, and their units, chunk by chunk.  Errors: the FP32 q_z of a rotation
// is within 10 x 2^-24 of sum |recip column| |h| (rounded inputs, one product, two
// FMAs); eps bounds that of x, y and z for the unit vector (4 such products and a few
// roundings, with a factor of 4 to spare) and its length, which is 1 within kBandTol
// (|q| is taken from the list, the matrix is a rotation within kRotTol).
static void build_units(const lmb_geometry &geo, const int4 *hkl, int nh, std::vector<int4> *seen,
                        std::vector<BuildUnits> *units, std::vector<uint32_t> *count) {
  const double c = kHcKeVnm / kFourPi, ulp = std::ldexp(1.0, -24);
  double col[3], smin, smax;
  for (int j = 0; j < 3; j++)
    col[j] = std::sqrt(geo.recip[j] * geo.recip[j] + geo.recip[3 + j] * geo.recip[3 + j] +
                       geo.recip[6 + j] * geo.recip[6 + j]);
  detector_angles(geo, &smin, &smax);
  std::map<std::tuple<int, int, int>, std::vector<int>> open;  // units still without their -h
  int nu = 0;
  auto close_chunk = [&]() {
    if (units->empty()) return;
    BuildUnits &bu = units->back();
    for (; nu % 32; nu++) {  // padding: an empty interval, no HKL
      const uint32_t none = 0x7F800000u;  // +inf, 0
      memcpy(&bu.hkl_band[nu].w, &none, 4);
      bu.eps[nu] = 1.f;
      bu.pos[nu] = 0xFFFFFFFFu;
    }
    count->push_back((uint32_t)nu);
  };
  for (int n = 0; n < nh; n++) {
    const int4 h = hkl[n];
    double q2 = 0.0;
    for (int r = 0; r < 3; r++) {
      const double q = geo.recip[3 * r] * h.x + geo.recip[3 * r + 1] * h.y + geo.recip[3 * r + 2] * h.z;
      q2 += q * q;
    }
    const double sum = col[0] * std::fabs((double)h.x) + col[1] * std::fabs((double)h.y) +
                       col[2] * std::fabs((double)h.z);
    const double err = 10.0 * ulp * sum, q = std::sqrt(q2);
    const bool plain = q2 > 1e-20 && q2 < 1e20 && sum < 1e15;  // else FP64 decides
    double lo = 0.0, hi = 3e38;
    if (plain) {
      lo = std::max(0.0, std::max(c * q2 / geo.ehi, q * smin) * (1.0 - kBandTol) - err);
      hi = std::min(geo.elo > 0 ? c * q2 / geo.elo : 3e38, q * smax) * (1.0 + kBandTol) + err;
      if (lo > hi) continue;  // no rotation puts it on the detector
    }
    const int i = (int)(seen->size() % kHklChunk);
    if (i == 0) {
      close_chunk();
      units->push_back(BuildUnits{});
      open.clear();
      nu = 0;
    }
    BuildUnits &bu = units->back();
    seen->push_back(h);
    auto it = open.find(std::make_tuple(-h.x, -h.y, -h.z));
    const bool zero = h.x == 0 && h.y == 0 && h.z == 0;
    if (!zero && it != open.end() && !it->second.empty()) {
      uint32_t &pos = bu.pos[it->second.back()];
      pos = (pos & 0xFFFFu) | ((uint32_t)i << 16);
      it->second.pop_back();
      continue;
    }
    // NaN eps: every comparison of the detector screen fails, so it rejects nothing
    const double len = plain ? q : 1.0;
    const uint32_t band =
        plain ? bf16_bound(lo / len, true) << 16 | bf16_bound(hi / len, false) : 0x00007F80u;
    float w;
    memcpy(&w, &band, 4);
    bu.hkl_band[nu] = make_float4((float)(h.x / len), (float)(h.y / len), (float)(h.z / len), w);
    bu.eps[nu] = plain ? (float)((double)kUnitErr * sum / q + (double)kUnitErr0 + kBandTol)
                       : std::numeric_limits<float>::quiet_NaN();
    bu.pos[nu] = (uint32_t)i | 0xFFFF0000u;
    open[std::make_tuple(h.x, h.y, h.z)].push_back(nu);
    nu++;
  }
  close_chunk();
}

// Threads per block so that the [S][TB] pixel lists fit in shared memory.
static int build_block(int S) {
  int tb = 128;
  while (tb > 32 && (size_t)S * tb * 4 > 160 * 1024) tb /= 2;
  return tb;
}

static size_t dbbuild_smem_bytes(int S) {
  const int tb = build_block(S);
  // a chunk's units, pixel lists, counts, two bit maps
  return sizeof(BuildUnits) + (size_t)tb * 4 * ((size_t)S + 1 + 2 * kChunkWords);
}

// The HKL list with its screens on the device, for the builds of one call.
struct BuildTables {
  int4 *hkl = nullptr, *seen = nullptr;
  float4 *hklf = nullptr;  // hkl as floats
  BuildUnits *units = nullptr;
  uint32_t *count = nullptr;
  BuildGeo g{};
  int nh = 0, nseen = 0;
  bool all = false;  // FP64 for every pair
};

int dbbuild_tables(const lmb_geometry &geo, const int32_t *hkls, int nh, bool exact_all,
                   cudaStream_t st, BuildTables **out) {
  const int S = geo.max_nr_spots;
  LMB_REQUIRE(S >= 1 && (size_t)S * 32 * 4 <= 160 * 1024,
              "MaxNrLaueSpots=%d outside the supported range 1..1280", S);
  BuildTables *t = new BuildTables();
  t->g = make_build_geo(geo);
  t->nh = nh;
  t->all = exact_all || !screen_sound(geo);
  std::vector<int4> h((size_t)std::max(nh, 1));
  for (int i = 0; i < nh; i++) h[i] = make_int4(hkls[3 * i], hkls[3 * i + 1], hkls[3 * i + 2], 0);
  std::vector<int4> seen;
  std::vector<BuildUnits> units;
  std::vector<uint32_t> count;
  if (!t->all) build_units(geo, h.data(), nh, &seen, &units, &count);
  t->nseen = (int)seen.size();
  // one allocation and one copy: HKLs | seen HKLs | units | unit counts
  std::vector<unsigned char> host;
  auto part = [&](const void *src, size_t bytes) {  // 256-byte aligned parts
    const size_t at = host.size();
    host.resize(at + (bytes + 255) / 256 * 256);
    std::copy_n(static_cast<const unsigned char *>(src), bytes, host.begin() + (ptrdiff_t)at);
    return at;
  };
  std::vector<float4> hf(h.size());
  for (size_t i = 0; i < h.size(); i++) hf[i] = make_float4((float)h[i].x, (float)h[i].y, (float)h[i].z, 0.f);
  const size_t oh = part(h.data(), h.size() * sizeof(int4));
  const size_t of = part(hf.data(), hf.size() * sizeof(float4));
  const size_t os = part(seen.data(), seen.size() * sizeof(int4));
  const size_t ou = part(units.data(), units.size() * sizeof(BuildUnits));
  const size_t oc = part(count.data(), count.size() * sizeof(uint32_t));
  unsigned char *d = nullptr;
  cudaError_t ce = cudaMalloc(&d, host.size());
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(d, host.data(), host.size(), cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  const void *fn = t->all ? (const void *)dbbuild_kernel<true> : (const void *)dbbuild_kernel<false>;
  if (ce == cudaSuccess)
    ce = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)dbbuild_smem_bytes(S));
  if (ce != cudaSuccess) {
    cudaFree(d);
    delete t;
    return cuda_fail(ce, "DB build tables", __FILE__, __LINE__);
  }
  t->hkl = reinterpret_cast<int4 *>(d + oh);  // oh = 0: the allocation itself
  t->hklf = reinterpret_cast<float4 *>(d + of);
  t->seen = reinterpret_cast<int4 *>(d + os);
  t->units = reinterpret_cast<BuildUnits *>(d + ou);
  t->count = reinterpret_cast<uint32_t *>(d + oc);
  *out = t;
  return LMB_OK;
}

void dbbuild_tables_free(BuildTables *t) {
  if (!t) return;
  cudaFree(t->hkl);
  delete t;
}

int dbbuild_launch(const double *d_om, uint64_t n, const BuildTables *t, uint16_t *d_out,
                   cudaStream_t st) {
  if (n == 0) return LMB_OK;
  const int tb = build_block(t->g.S);
  const size_t smem = dbbuild_smem_bytes(t->g.S);
  const uint64_t blocks = (n + tb - 1) / tb;
  LMB_REQUIRE(blocks < (1ull << 31), "too many orientations (%llu)", (unsigned long long)n);
  if (t->all)
    dbbuild_kernel<true><<<(unsigned)blocks, tb, smem, st>>>(d_om, n, t->hkl, t->hklf, t->nh, t->seen, t->nseen,
                                                             t->units, t->count, t->g, d_out);
  else
    dbbuild_kernel<false><<<(unsigned)blocks, tb, smem, st>>>(d_om, n, t->hkl, t->hklf, t->nh, t->seen, t->nseen,
                                                              t->units, t->count, t->g, d_out);
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

// The 12 operators of the hexagonal (622) group, LaueMatchingHeaders.h:111-122
// (5-decimal values, normalised here).
static const double kHexSym[12][4] = {
    {1, 0, 0, 0},          {0.86603, 0, 0, 0.5},  {0.5, 0, 0, 0.86603},  {0, 0, 0, 1},
    {0.5, 0, 0, -0.86603}, {0.86603, 0, 0, -0.5}, {0, 1, 0, 0},          {0, 0.86603, 0.5, 0},
    {0, 0.5, 0.86603, 0},  {0, 0, 1, 0},          {0, -0.5, 0.86603, 0}, {0, -0.86603, 0.5, 0}};

int synth_orient_launch(uint64_t seed, uint64_t first, uint64_t n, double *d_out,
                        cudaStream_t st, uint32_t flags) {
  if (n == 0) return LMB_OK;
  SynthSym sym{};
  if (flags & LMB_BUILD_SYNTH_HEX_FZ) {
    sym.nsym = 12;
    for (int k = 0; k < 12; k++) {
      const double *q = kHexSym[k];
      const double nrm = std::sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
      for (int j = 0; j < 4; j++) sym.q[k][j] = q[j] / nrm;
    }
  }
  const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 148ull * 32);
  synth_orient_kernel<<<(unsigned)blocks, 256, 0, st>>>(seed, first, n, d_out, sym);
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

}  // namespace lmb
