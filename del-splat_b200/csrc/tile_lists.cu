// tile_lists.cu -- stage 2 of the tile-list builder (reference-format output
// only): the superblock lists of tiles.cu split into per-tile lists
// tile2idx / idx2pnt.
//
// Bound: the pairs' 4-byte stores and the 8-byte entries read twice.  A
// superblock's list is cut into segments of kSegEntries entries at multiples
// of kSegEntries in the whole list, so that the work is spread over the GPU
// whatever the lists' lengths (one block per superblock left the long lists
// of the view's middle to a few blocks: 1308 us for 1,048,576 Gaussians at
// 1920x1080 and 16x16 tiles, 510 superblocks; by segments 137 us):
//   k_seg_count    per (segment, tile) entry counts;
//   k_seg_scan     per superblock: each tile's counts become exclusive
//                  prefixes over its segments, their sum the tile's length;
//   (exclusive scan of the lengths -> tile2idx)
//   k_seg_scatter  every pair to tile2idx[tile] + its segment's prefix +
//                  lower entries of the segment.
// A warp takes 32 consecutive entries at a time, one ballot per tile says
// which cover it (tile order outside, entries inside, so the stores of a
// ballot are consecutive words) and list order is kept.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace dsplat {

constexpr int kSegThreads = 256;
constexpr int kSegWarps = kSegThreads / 32;
constexpr int kSegRounds = 4;
constexpr uint32_t kSegEntries = kSegThreads * kSegRounds;  // 1024

// Segment ids: superblock sb meets the aligned pieces floor(s / S) ..
// floor((e - 1) / S) of the list; piece + sb numbers the (piece, superblock)
// meetings uniquely and in list order (some ids belong to no entry).  A block
// takes a run of consecutive ids and searches for the superblock of the first
// only.
size_t tile_seg_slots(uint64_t capacity, uint32_t num_sb) { return size_t(capacity / kSegEntries) + num_sb + 1; }

__device__ __forceinline__ uint32_t sb_begin(const uint32_t* __restrict__ off1, uint32_t nchunk, uint64_t capacity,
                                             uint32_t sb) {
  return uint32_t(min(uint64_t(off1[size_t(sb) * nchunk]), capacity));
}

struct SegWalk {
  uint32_t id, id_end;  // this block's ids [id, id_end)
  uint32_t sb, s, e;    // the superblock of id and its entries
  const uint32_t* off1;
  uint32_t nchunk, num_sb;
  uint64_t capacity;

  __device__ __forceinline__ SegWalk(const uint32_t* off1_, uint32_t nchunk_, uint64_t cap_, uint32_t num_sb_)
      : off1(off1_), nchunk(nchunk_), num_sb(num_sb_), capacity(cap_) {
    const uint32_t count = sb_begin(off1, nchunk, capacity, num_sb) / kSegEntries + num_sb;
    const uint32_t per = (count + gridDim.x - 1) / gridDim.x;
    id = min(count, blockIdx.x * per);
    id_end = min(count, id + per);
    uint32_t lo = 0, hi = num_sb - 1;  // last superblock whose first id is <= id
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) / 2;
      if (sb_begin(off1, nchunk, capacity, mid) / kSegEntries + mid <= id) lo = mid;
      else hi = mid - 1;
    }
    sb = lo;
    s = sb_begin(off1, nchunk, capacity, sb);
    e = sb_begin(off1, nchunk, capacity, sb + 1);
  }
  // the next superblock begins at id e / S + sb + 1
  __device__ __forceinline__ void next() {
    ++id;
    while (sb + 1 < num_sb && e / kSegEntries + sb + 1 <= id) {
      ++sb;
      s = e;
      e = sb_begin(off1, nchunk, capacity, sb + 1);
    }
  }
  __device__ __forceinline__ uint32_t lo() const { return max(s, (id - sb) * kSegEntries); }
  __device__ __forceinline__ uint32_t hi() const { return uint32_t(min(uint64_t(e), uint64_t(id - sb + 1) * kSegEntries)); }
};

// Tiles k = y * side + x of a superblock of side 1 << SL that an entry's
// local span (local_rect in tiles.cu) covers, as a bit mask: the row's x bits
// repeated on every row, rows y0 .. y1 kept.
template <int SL>
struct Cover {
  typedef typename std::conditional<SL == 3, unsigned long long, uint32_t>::type mask_t;
  static constexpr int SIDE = 1 << SL, TILES = SIDE * SIDE;
  static __device__ __forceinline__ mask_t below(int bits) {  // the lowest `bits` bits
    return bits >= int(8 * sizeof(mask_t)) ? ~mask_t(0) : (mask_t(1) << bits) - 1;
  }
  static __device__ __forceinline__ mask_t of(uint32_t lr) {
    const int x0 = lr & 15, y0 = (lr >> 4) & 15, x1 = (lr >> 8) & 15, y1 = (lr >> 12) & 15;
    const mask_t row = below(x1) & ~below(x0);
    const mask_t repeat = SL == 0 ? 1u : SL == 1 ? 0x5u : SL == 2 ? 0x1111u : mask_t(0x0101010101010101ull);
    return row * repeat & below(y1 << SL) & ~below(y0 << SL);
  }
};

// The segment's entries, kSegRounds per thread (warp w takes entries
// lo + 128 w .. of the segment in rounds of 32): masks[w][r][k] the lanes of
// round r that cover tile k, cnt[w][k] the warp's count.
template <int SL>
struct SegShared {
  static constexpr int T = 1 << (2 * SL);
  uint32_t masks[kSegWarps][kSegRounds][T];
  uint32_t cnt[kSegWarps][T];
};

template <int SL>
__device__ __forceinline__ void seg_ballots(const uint2* __restrict__ list1, uint32_t lo, uint32_t hi, int warp,
                                            int lane, SegShared<SL>& sh, uint32_t* g) {
  constexpr int T = Cover<SL>::TILES;
  typename Cover<SL>::mask_t cov[kSegRounds];
#pragma unroll
  for (int k = 0; k < kSegRounds; ++k) {
    const uint32_t off = uint32_t(warp * kSegRounds + k) * 32 + lane;
    uint2 en = make_uint2(0u, 0u);  // empty span
    if (off < hi - lo) en = list1[size_t(lo) + off];
    g[k] = en.x;
    cov[k] = Cover<SL>::of(en.y);
  }
  uint32_t c0 = 0, c1 = 0;
#pragma unroll
  for (int k = 0; k < kSegRounds; ++k) {
    uint32_t m0 = 0, m1 = 0;  // lane t keeps tiles t and t + 32
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const uint32_t m = __ballot_sync(0xffffffffu, (cov[k] >> t) & 1u);
      if ((t & 31) == lane) (t < 32 ? m0 : m1) = m;
    }
    if (lane < T) sh.masks[warp][k][lane] = m0;
    if (T > 32) sh.masks[warp][k][(lane + 32) % T] = m1;
    c0 += __popc(m0);
    c1 += __popc(m1);
  }
  if (lane < T) sh.cnt[warp][lane] = c0;
  if (T > 32) sh.cnt[warp][(lane + 32) % T] = c1;
}

template <int SL>
__global__ void __launch_bounds__(kSegThreads) k_seg_count(const uint2* __restrict__ list1,
                                                           const uint32_t* __restrict__ off1, uint32_t nchunk,
                                                           uint64_t capacity, uint32_t num_sb,
                                                           uint32_t* __restrict__ segcnt) {
  constexpr int T = Cover<SL>::TILES;
  __shared__ SegShared<SL> sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (SegWalk w(off1, nchunk, capacity, num_sb); w.id < w.id_end; w.next()) {
    uint32_t g[kSegRounds];
    seg_ballots<SL>(list1, w.lo(), max(w.lo(), w.hi()), warp, lane, sh, g);
    __syncthreads();
    if (threadIdx.x < T) {
      uint32_t c = 0;
#pragma unroll
      for (int i = 0; i < kSegWarps; ++i) c += sh.cnt[i][threadIdx.x];
      segcnt[size_t(w.id) * T + threadIdx.x] = c;
    }
    __syncthreads();
  }
}

// The tile of a superblock (its item in the view), or -1 outside the view.
__device__ __forceinline__ int64_t tile_of(const ViewDev& vd, uint32_t sb, int t) {
  const int sl = vd.sb_log2, side = 1 << sl;
  const uint32_t sbw = uint32_t(sb_cols(vd));
  const int x = int(sb % sbw) * side + (t & (side - 1)), y = int(sb / sbw) * side + (t >> sl);
  return x < vd.tile_w && y < vd.tile_h ? int64_t(y) * vd.tile_w + x : -1;
}

// One block per superblock, its tiles times 256 / tiles runs of segments.
__global__ void __launch_bounds__(kSegThreads) k_seg_scan(const uint32_t* __restrict__ off1, uint32_t nchunk,
                                                          uint64_t capacity, const ViewDev vd,
                                                          uint32_t* __restrict__ segcnt, uint32_t* __restrict__ tcnt) {
  __shared__ uint32_t sums[kSegThreads];
  const uint32_t sb = blockIdx.x;
  const int tiles = 1 << (2 * vd.sb_log2), parts = kSegThreads / tiles;
  const int t = int(threadIdx.x) & (tiles - 1), part = int(threadIdx.x) / tiles;
  const uint32_t s = sb_begin(off1, nchunk, capacity, sb), e = sb_begin(off1, nchunk, capacity, sb + 1);
  uint32_t* const mine = segcnt + (size_t(s / kSegEntries) + sb) * tiles + t;  // this superblock's first id
  const uint32_t nseg = e > s ? (e - 1) / kSegEntries - s / kSegEntries + 1 : 0u;
  const uint32_t per = (nseg + parts - 1) / parts, p0 = min(nseg, part * per), p1 = min(nseg, p0 + per);
  uint32_t acc = 0;
  for (uint32_t i = p0; i < p1; ++i) acc += mine[size_t(i) * tiles];
  sums[threadIdx.x] = acc;
  __syncthreads();
  uint32_t run = 0, total = 0;
  const uint32_t used = per ? (nseg + per - 1) / per : 0u;  // runs that hold segments
  for (uint32_t p = 0; p < used; ++p) {
    const uint32_t c = sums[p * tiles + t];
    if (int(p) < part) run += c;
    total += c;
  }
  for (uint32_t i = p0; i < p1; ++i) {
    const uint32_t c = mine[size_t(i) * tiles];
    mine[size_t(i) * tiles] = run;
    run += c;
  }
  if (part == 0) {
    const int64_t item = tile_of(vd, sb, t);
    if (item >= 0) tcnt[item] = total;
  }
}

// out_tile (nullable) receives each pair's tile.
template <int SL>
__global__ void __launch_bounds__(kSegThreads) k_seg_scatter(const uint2* __restrict__ list1,
                                                             const uint32_t* __restrict__ off1, uint32_t nchunk,
                                                             uint64_t capacity, uint32_t num_sb, const ViewDev vd,
                                                             const uint32_t* __restrict__ segcnt,
                                                             const uint32_t* __restrict__ item_start,
                                                             uint32_t* __restrict__ idx2pnt,
                                                             uint32_t* __restrict__ out_tile,
                                                             uint32_t* __restrict__ flags) {
  constexpr int T = Cover<SL>::TILES;
  __shared__ SegShared<SL> sh;
  __shared__ uint32_t item[T];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (SegWalk w(off1, nchunk, capacity, num_sb); w.id < w.id_end; w.next()) {
    uint32_t g[kSegRounds];
    seg_ballots<SL>(list1, w.lo(), max(w.lo(), w.hi()), warp, lane, sh, g);
    __syncthreads();
    if (threadIdx.x < T) {  // each warp's first slot of every tile (tiles outside the view have no entries)
      const int64_t it = tile_of(vd, w.sb, threadIdx.x);
      item[threadIdx.x] = it >= 0 ? uint32_t(it) : 0u;
      uint32_t run = it >= 0 ? item_start[it] + segcnt[size_t(w.id) * T + threadIdx.x] : 0u;
#pragma unroll
      for (int i = 0; i < kSegWarps; ++i) {
        const uint32_t c = sh.cnt[i][threadIdx.x];
        sh.cnt[i][threadIdx.x] = run;
        run += c;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < T; ++t) {
      uint32_t base = sh.cnt[warp][t];
#pragma unroll
      for (int k = 0; k < kSegRounds; ++k) {
        const uint32_t m = sh.masks[warp][k][t];
        if ((m >> lane) & 1u) {
          const uint32_t slot = base + __popc(m & lt);
          if (slot < capacity) {
            idx2pnt[slot] = g[k];
            if (out_tile) out_tile[slot] = item[t];
          } else {
            set_flag(flags, kFlagPairOverflow);
          }
        }
        base += __popc(m);
      }
    }
    __syncthreads();
  }
}

namespace {
// Blocks of a kernel over the segments: more of them even out what the
// segments take (how many tiles their entries cover), each pays for the search
// of its first segment.  1,048,576 Gaussians at 1920x1080, us for 8, 24, 32,
// 64 and 256 blocks per SM: scatter 105, 94, 94, 97, 150; count, whose
// segments all take the same, 40, 40 (12 per SM), 43 (32).
constexpr size_t kSegCountBlocks = 148 * 8, kSegScatterBlocks = 148 * 24;
unsigned seg_grid(uint64_t capacity, uint32_t num_sb, size_t most) {
  return unsigned(std::min<size_t>(tile_seg_slots(capacity, num_sb), most));
}
}  // namespace

// Both take the lists of a single view (view 0 of b).  segcnt holds
// tile_seg_slots() times the superblock's tile count words (64 at most).
cudaError_t split_tile_lists(cudaStream_t st, const uint2* list1, const uint32_t* off1, uint32_t nchunk,
                             uint64_t capacity, const ViewBatch& b, uint32_t* segcnt, uint32_t* tcnt) {
  const unsigned grid = seg_grid(capacity, b.num_sb, kSegCountBlocks);
  switch (b.v[0].sb_log2) {
    case 0: k_seg_count<0><<<grid, kSegThreads, 0, st>>>(list1, off1, nchunk, capacity, b.num_sb, segcnt); break;
    case 1: k_seg_count<1><<<grid, kSegThreads, 0, st>>>(list1, off1, nchunk, capacity, b.num_sb, segcnt); break;
    case 2: k_seg_count<2><<<grid, kSegThreads, 0, st>>>(list1, off1, nchunk, capacity, b.num_sb, segcnt); break;
    default: k_seg_count<3><<<grid, kSegThreads, 0, st>>>(list1, off1, nchunk, capacity, b.num_sb, segcnt); break;
  }
  count_launch();
  k_seg_scan<<<b.num_sb, kSegThreads, 0, st>>>(off1, nchunk, capacity, b.v[0], segcnt, tcnt);
  count_launch();
  return cudaGetLastError();
}

cudaError_t scatter_tile_lists(cudaStream_t st, const uint2* list1, const uint32_t* off1, uint32_t nchunk,
                               uint64_t capacity, const ViewBatch& b, const uint32_t* segcnt,
                               const uint32_t* item_start, uint32_t* idx2pnt, uint32_t* out_tile, uint32_t* flags) {
  const unsigned grid = seg_grid(capacity, b.num_sb, kSegScatterBlocks);
#define X(SL)                                                                                                       \
  k_seg_scatter<SL><<<grid, kSegThreads, 0, st>>>(list1, off1, nchunk, capacity, b.num_sb, b.v[0], segcnt,           \
                                                  item_start, idx2pnt, out_tile, flags)
  switch (b.v[0].sb_log2) {
    case 0: X(0); break;
    case 1: X(1); break;
    case 2: X(2); break;
    default: X(3); break;
  }
#undef X
  count_launch();
  return cudaGetLastError();
}

}  // namespace dsplat
