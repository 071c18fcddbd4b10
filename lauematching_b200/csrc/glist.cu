// Records grouped by their number of on-detector spots.
//
// A record can only pass when it has at least MinNrSpots spots on the detector
// (LaueMatchingCPU.c:671-683), so a pass needs the records of the large counts
// alone.  `perm` lists the record numbers by falling count (within one count tile by
// tile of kGlTile records, in no order within a tile: its warps race for places, so
// two builds of one DB may differ there; survivors are ordered by ID after the pass),
// so the records with at least m spots are its first entries whatever m is.  Each count starts at a multiple of 32
// (places without a record hold kNoRecord): a chunk of 32 places has one count.
// 4 bytes per record, made once per DB by a counting sort on the device: 6 to 7 ms
// to the end of the first pass at 1e8 records of 122 bytes on B200, where packing
// the tiled compact layout (clist.cu) on the host took 42 to 490 ms.
#include "kernels.cuh"

namespace lmb {

// Spots of each record (0..S) and, per tile of kGlTile records, how many records
// have each count: bh[c * ntiles + tile].  on_detector: every stored spot lies on
// the detector (a DB made by the build kernel), so the count word alone is read.
__global__ void __launch_bounds__(256) glist_count_kernel(const uint16_t *__restrict__ db, uint64_t n,
                                                          int R, int S, int W, int H, int on_detector,
                                                          uint32_t ntiles, uint8_t *__restrict__ cnt,
                                                          uint32_t *__restrict__ bh) {
  __shared__ unsigned int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t first = (uint64_t)blockIdx.x * kGlTile;
  for (uint32_t k = threadIdx.x; k < kGlTile; k += 256) {
    const uint64_t i = first + k;
    if (i >= n) break;
    const uint16_t *rec = db + i * (uint64_t)R;
    int c = min((int)rec[0], S);
    if (!on_detector) {
      int on = 0;
      for (int s = 0; s < c; s++) on += (rec[1 + 2 * s] < W && rec[2 + 2 * s] < H) ? 1 : 0;
      c = on;
    }
    cnt[i] = (uint8_t)c;
    atomicAdd(&h[c], 1u);
  }
  __syncthreads();
  bh[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Total of each count (one block per count).
__global__ void __launch_bounds__(256) glist_total_kernel(const uint32_t *__restrict__ bh, uint32_t ntiles,
                                                          unsigned long long *__restrict__ hist) {
  __shared__ unsigned long long part[8];
  unsigned long long v = 0;
  for (uint32_t t = threadIdx.x; t < ntiles; t += 256) v += bh[(uint64_t)blockIdx.x * ntiles + t];
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) v += part[w];
    hist[blockIdx.x] = v;
  }
}

// bh becomes the first position of each (count, tile) in perm (one block per
// count; counts from the largest down).
__global__ void __launch_bounds__(1024) glist_scan_kernel(uint32_t *__restrict__ bh, uint32_t ntiles,
                                                          const unsigned long long *__restrict__ hist) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (hist[blockIdx.x] == 0) return;
  if (threadIdx.x == 0) {
    unsigned long long base = 0;
    for (int c = 255; c > (int)blockIdx.x; c--) base += (hist[c] + 31) / 32 * 32;
    carry = (uint32_t)base;
  }
  __syncthreads();
  uint32_t *row = bh + (uint64_t)blockIdx.x * ntiles;
  for (uint32_t t0 = 0; t0 < ntiles; t0 += 1024) {
    const uint32_t t = t0 + threadIdx.x;
    const uint32_t v = t < ntiles ? row[t] : 0;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t s = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      warp_sum[lane] = s;
    }
    __syncthreads();
    const uint32_t before = carry + (warp ? warp_sum[warp - 1] : 0);
    if (t < ntiles) row[t] = before + x - v;
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_sum[31];
    __syncthreads();
  }
}

// Record numbers to their places; the lanes of a warp with equal counts take
// consecutive ones.
__global__ void __launch_bounds__(256) glist_scatter_kernel(const uint8_t *__restrict__ cnt, uint64_t n,
                                                            uint32_t ntiles,
                                                            const uint32_t *__restrict__ bh,
                                                            uint32_t *__restrict__ perm) {
  __shared__ uint32_t pos[256];
  pos[threadIdx.x] = bh[(uint64_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t first = (uint64_t)blockIdx.x * kGlTile;
  for (uint32_t k = threadIdx.x; k < kGlTile; k += 256) {  // whole warps
    const uint64_t i = first + k;
    const int c = i < n ? cnt[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    uint32_t at = 0;
    if (c >= 0 && lane == __ffs(same) - 1) at = atomicAdd(&pos[c], (uint32_t)__popc(same));
    at = __shfl_sync(0xffffffffu, at, __ffs(same) - 1);
    if (c >= 0) perm[at + __popc(same & ((1u << lane) - 1u))] = (uint32_t)i;
  }
}

// Cell codes of the records of one count (c >= 1), perm[0, 32 chunks): a spot's
// cell of cw x ch pixels, 16 bits each, two to a unit.  A chunk's codes are ceil(c /
// 2) units per lane: pairs of them as [pair][lane][2], so that a warp reads four
// spots of its 32 records with one 8-byte load per lane, and an odd last one as
// [lane].  Codes past the last spot, and of places without a record, are `none`, the
// code of a cell that is never marked.
//
// The order of a record's codes is free, and the filter's lanes look up their
// k-th codes together: for records of up to 32 spots the k-th codes of a chunk are
// chosen to spread over the shared-memory banks (two cells per 4-byte word).  A lane
// offers the banks of the spots it has left, three rounds hand every bank to at most
// two lanes that ask for it, and the lanes that got none take any spot.  (At most one
// lane per bank leaves more lanes without: 2.9 wavefronts a look-up instead of 2.3,
// 3.7 unordered.)
__global__ void __launch_bounds__(256) glist_code_kernel(const uint16_t *__restrict__ db, int R, int S,
                                                         int W, int H,
                                                         const uint32_t *__restrict__ perm,
                                                         uint32_t chunks, int c, int cw, int ch,
                                                         int cells_x, uint32_t none,
                                                         uint32_t *__restrict__ codes) {
  constexpr int kMost = 32;  // spots of a record whose codes are ordered
  __shared__ uint16_t held[8][kMost][33];
  const uint32_t chunk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (chunk >= chunks) return;  // whole warps
  const int units = (c + 1) / 2;
  uint32_t *out = codes + (uint64_t)chunk * units * 32;
  const uint32_t id = perm[chunk * 32 + lane];
  const uint16_t *rec = db + (id != kNoRecord ? (uint64_t)id * R : 0);
  const int stored = id != kNoRecord ? min((int)rec[0], S) : 0;
  uint32_t four[4] = {none, none, none, none};
  int k = 0;
  auto flush = [&](int first) {  // the unit `first` and the next
    if (first + 1 < units)
      *reinterpret_cast<uint2 *>(out + first * 32 + 2 * lane) =
          make_uint2(four[0] | four[1] << 16, four[2] | four[3] << 16);
    else
      out[first * 32 + lane] = four[0] | four[1] << 16;
#pragma unroll
    for (int j = 0; j < 4; j++) four[j] = none;
  };
  auto put = [&](uint32_t q) {
#pragma unroll
    for (int j = 0; j < 4; j++)
      if ((k & 3) == j) four[j] = q;
    if ((++k & 3) == 0) flush(k / 2 - 2);
  };
  uint16_t(*mine)[33] = held[threadIdx.x >> 5];
  int n = 0;
  for (int s = 0; s < stored && n < c; s++) {
    const uint32_t x = rec[1 + 2 * s], y = rec[2 + 2 * s];
    if (x >= (uint32_t)W || y >= (uint32_t)H) continue;
    const uint32_t q = (y / (uint32_t)ch) * (uint32_t)cells_x + x / (uint32_t)cw;
    if (c <= kMost)
      mine[n][lane] = (uint16_t)q;
    else
      put(q);
    n++;
  }
  if (c <= kMost) {
    unsigned left = n >= 32 ? ~0u : (1u << n) - 1u, banks = 0u;
    for (int j = 0; j < n; j++) banks |= 1u << ((mine[j][lane] >> 1) & 31);
    const unsigned all = 0xffffffffu;
    for (int step = 0; step < c; step++) {
      unsigned once = 0u, full = 0u;  // banks handed to one lane, to two
      int bank = -1;
      const int turn = (lane + 11 * step) & 31;  // where a lane starts looking
      for (int round = 0; round < 3; round++) {
        const unsigned free = bank < 0 ? banks & ~full : 0u;
        const int ask = free ? (__ffs(__funnelshift_r(free, free, turn)) - 1 + turn) & 31 : -1;
        const unsigned same = __match_any_sync(all, ask);
        const int room = ask >= 0 ? 2 - (int)(once >> ask & 1u) : 0;
        if (__popc(same & ((1u << lane) - 1u)) < room) bank = ask;
        // the first lane that asks says what becomes of the bank
        const bool speaks = ask >= 0 && lane == __ffs(same) - 1;
        const bool fills = __popc(same) >= room;
        once |= __reduce_or_sync(all, speaks && !fills ? 1u << ask : 0u);
        full |= __reduce_or_sync(all, speaks && fills ? 1u << ask : 0u);
      }
      if (bank < 0 && banks) bank = (__ffs(__funnelshift_r(banks, banks, turn)) - 1 + turn) & 31;
      if (bank >= 0) {  // the lane's spot of that bank; the banks of the others
        int pick = -1;
        banks = 0u;
        for (unsigned m = left; m; m &= m - 1u) {
          const int j = __ffs(m) - 1;
          const int b = (mine[j][lane] >> 1) & 31;
          if (pick < 0 && b == bank)
            pick = j;
          else
            banks |= 1u << b;
        }
        left &= ~(1u << pick);
        put(mine[pick][lane]);
      } else {
        put(none);
      }
    }
  }
  for (int u = k / 4 * 2; u < units; u += 2) flush(u);
}

int glist_code_launch(const uint16_t *d_db, int R, int S, int W, int H, const uint32_t *d_perm, int c,
                      uint32_t chunks, const GroupCells &cells, uint32_t *d_codes, cudaStream_t st) {
  if (chunks == 0) return LMB_OK;
  glist_code_kernel<<<(chunks + 7) / 8, 256, 0, st>>>(d_db, R, S, W, H, d_perm, chunks, c, cells.cw,
                                                      cells.ch, cells.nx, cells.n, d_codes);
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int glist_count_launch(const uint16_t *d_db, uint64_t n, int R, int S, int W, int H, bool on_detector,
                       uint8_t *d_cnt, uint32_t *d_bh, unsigned long long *d_hist, cudaStream_t st) {
  LMB_REQUIRE(S <= 255 && n > 0 && n < kGlMost, "records cannot be grouped by count");
  const uint32_t nt = glist_tiles(n);
  glist_count_kernel<<<nt, 256, 0, st>>>(d_db, n, R, S, W, H, on_detector ? 1 : 0, nt, d_cnt, d_bh);
  glist_total_kernel<<<256, 256, 0, st>>>(d_bh, nt, d_hist);
  glist_scan_kernel<<<256, 1024, 0, st>>>(d_bh, nt, d_hist);
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int glist_scatter_launch(const uint8_t *d_cnt, uint64_t n, const uint32_t *d_bh, uint32_t *d_perm,
                         cudaStream_t st) {
  const uint32_t nt = glist_tiles(n);
  LMB_CUDA(cudaMemsetAsync(d_perm, 0xff, glist_places(n) * sizeof(uint32_t), st));
  glist_scatter_kernel<<<nt, 256, 0, st>>>(d_cnt, n, nt, d_bh, d_perm);
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

}  // namespace lmb
