// tiles.cu -- tile-pair construction: device scan, stable LSD radix sort,
// rank-ordered pair emission and per-tile range finding.
//
// Reference counterpart: del-splat-cudarc/src/splat_gauss.rs:96-195 (count ->
// two exclusive scans -> D2H read of the pair total -> fill_index_info ->
// radix_sort_by_key_u64_u32 on 64-bit (tile << 32 | depth bits) keys), with
// scan and sort taken from the absent del-cudarc-sys crate.
//
// Design here (same result, fewer bytes moved):
//   1. depth sort: each view's N depth keys are sorted once by a stable
//      segmented LSD radix sort (equal depths stay in point-index order) ->
//      the points of every view in rank order;
//   2. stage 1: a stable multisplit of that rank sequence into superblock
//      lists (square blocks of 1, 2, 4 or 8 tiles per side, chosen per view):
//      per (chunk, superblock) counts, one exclusive scan, then a scatter
//      whose in-warp slots come from ballots; an entry is (point, its tile
//      span clipped to the superblock).  The batched rasteriser walks these
//      lists directly, filtering by tile;
//   3. stage 2 (reference-format output only, tile_lists.cu): the superblock
//      lists split into per-tile lists with ballot ranking -> tile2idx/idx2pnt.
// Filtering a rank-ordered superblock list by tile keeps rank order, so every
// tile list is the reference's order, (tile, depth bits, point index)
// ascending, bit for bit; no 64-bit pair key is sorted.
#include <algorithm>

#include "common.cuh"

namespace dsplat {

// ---------------------------------------------------------------------------
// Exclusive scan of u32 (two kernels: block totals, then each block adds the
// earlier blocks' totals to its own scan; any length).
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Block-wide exclusive scan of one value per thread; returns the prefix and
// writes the block total.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  uint32_t inc = warp_incl_scan(x, lane);
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < nwarps ? warp_sums[lane] : 0u;
    uint32_t si = warp_incl_scan(s, lane);
    if (lane < nwarps) warp_sums[lane] = si - s;
    if (lane == nwarps - 1) *total = si;
  }
  __syncthreads();
  uint32_t r = warp_sums[warp] + inc - x;
  __syncthreads();
  return r;
}

// This thread's kScanItems words from `base` on (base is a multiple of 8, in
// 16-byte aligned), zero from n on.
__device__ __forceinline__ void scan_load(const uint32_t* __restrict__ in, size_t base, size_t n, uint32_t* v) {
  if (base + kScanItems <= n) {
    const uint4 a = *reinterpret_cast<const uint4*>(in + base), c = *reinterpret_cast<const uint4*>(in + base + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
  } else {
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) v[i] = base + i < n ? in[base + i] : 0u;
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const uint32_t* __restrict__ in, size_t n,
                                                              uint32_t* __restrict__ sums) {
  uint32_t v[kScanItems], s = 0;
  scan_load(in, size_t(blockIdx.x) * kScanTile + size_t(threadIdx.x) * kScanItems, n, v);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) s += v[i];
  __shared__ uint32_t tot;
  block_excl_scan(s, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// out[i] = sum of in[0, i) for i in [0, n], at most limit; a total above limit
// sets the overflow flag.
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint32_t* __restrict__ in,
                                                             uint32_t* __restrict__ out, size_t n,
                                                             const uint32_t* __restrict__ sums, uint32_t limit,
                                                             uint32_t* __restrict__ flags) {
  const size_t base = size_t(blockIdx.x) * kScanTile + size_t(threadIdx.x) * kScanItems;
  uint32_t v[kScanItems], s = 0;
  scan_load(in, base, n, v);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) s += v[i];
  __shared__ uint32_t carry, tot;
  uint32_t p = block_excl_scan(s, &tot);
  if (blockIdx.x > 0) {
    // the earlier blocks' totals, summed by every block itself (a few hundred
    // words for the scans here, so no separate pass scans them)
    uint32_t part = 0;
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kScanThreads) part += sums[i];
    block_excl_scan(part, &carry);
    p += carry;
  }
  uint32_t o[kScanItems];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    o[i] = min(p, limit);
    if (base + i == n && p > limit) set_flag(flags, kFlagPairOverflow);
    p += v[i];
  }
  if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
    *reinterpret_cast<uint4*>(out + base) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4*>(out + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
  } else {
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
      if (base + i <= n) out[base + i] = o[i];
  }
}

size_t scan_tmp_words(size_t n) { return n / kScanTile + 2; }

// out[0, n] <- exclusive sums of in[0, n) and their total (one launch up to
// kScanTile - 1 words); out may be in when the total is not wanted there.
cudaError_t exclusive_scan(cudaStream_t st, const uint32_t* in, uint32_t* out, size_t n, uint32_t* tmp,
                           uint32_t limit, uint32_t* flags) {
  const uint32_t nb = uint32_t(n / kScanTile + 1);
  if (nb > 1) {
    k_scan_reduce<<<nb, kScanThreads, 0, st>>>(in, n, tmp);
    count_launch();
  }
  k_scan_apply<<<nb, kScanThreads, 0, st>>>(in, out, n, tmp, limit, flags);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (u32 key, u32 value), 8-bit digits.
// Each block owns a tile of 4096 consecutive elements, or of 2048.  Segmented
// form: with nb_seg blocks per segment the histogram is laid out (segment,
// digit, block) so that one exclusive scan yields every block's output offset
// per digit and segments never mix.
//   upsweep:   16-byte key loads, per-warp shared histograms;
//   downsweep: warp w ranks its elements (16 or 8 rounds of 32, in index
//              order) with ballots against its running digit counts; the
//              block turns the counts into local digit offsets, scatters
//              (key, value) into shared memory in digit order, and writes each
//              digit's run to its global offset with consecutive threads on
//              consecutive addresses.
// Short sorts are bound by the chain of launches and, in each, by the chain of
// rounds (us of all sort and scan launches of one sort below, before -> after):
//   up to kRsShortBlocks tiles of 2048 (two for each SM) the tiles are 2048:
//   half the rounds, and every block still resident at once.  16,384 keys 46
//   -> 35, 50,021 50 -> 37, 262,144 72 -> 66; from 8 x 100,003 on the halved
//   tiles only add histograms (66 with tiles of 4096, 72 with 2048; 16 x
//   1,048,576: 550 and 645);
//   up to kRsFewRows rows of counts read by all blocks together (blocks per
//   segment x blocks) the downsweep sums its segment's counts itself: no scan,
//   8 launches instead of 16.  One row per block then, so that the reads are
//   coalesced.  262,144 keys 66 -> 42, 1,048,576 92 -> 77, 8 x 262,144 110 ->
//   104; past the limit the rows take as long as the scans (2 x 1,048,576:
//   72 + 32 for downsweeps and scans, 110 + 7 with rows);
//   up to 8192 elements per segment one block sorts it in shared memory, all
//   four digits in one launch (1,000 elements 34 us in 16 launches -> 10 in
//   one; 3,000 -> 16).
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsRounds = 16;
constexpr int kRsShortRounds = 8;

// FEW: a row of 256 counts per block, otherwise a row of nb_seg per digit
template <int ROUNDS, bool FEW>
__global__ void __launch_bounds__(kRsThreads) k_radix_upsweep(const uint32_t* __restrict__ keys, int shift,
                                                              uint32_t nb_seg, uint32_t* __restrict__ hist) {
  constexpr int kRsTile = kRsThreads * ROUNDS;
  __shared__ uint32_t h[kRsWarps][256];
  for (int i = threadIdx.x; i < kRsWarps * 256; i += kRsThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  const uint4* k4 = reinterpret_cast<const uint4*>(keys + size_t(blockIdx.x) * kRsTile);
#pragma unroll
  for (int r = 0; r < kRsTile / 4 / kRsThreads; ++r) {
    const uint4 q = k4[r * kRsThreads + threadIdx.x];
    atomicAdd(&h[warp][(q.x >> shift) & 255u], 1u);
    atomicAdd(&h[warp][(q.y >> shift) & 255u], 1u);
    atomicAdd(&h[warp][(q.z >> shift) & 255u], 1u);
    atomicAdd(&h[warp][(q.w >> shift) & 255u], 1u);
  }
  __syncthreads();
  uint32_t sum = 0;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) sum += h[w][threadIdx.x];
  const uint32_t seg = blockIdx.x / nb_seg, b = blockIdx.x % nb_seg;
  hist[FEW ? size_t(blockIdx.x) * 256 + threadIdx.x : (size_t(seg) * 256 + threadIdx.x) * nb_seg + b] = sum;
}

// lanes of the warp whose 8-bit digit equals this lane's (one ballot per bit)
__device__ __forceinline__ uint32_t peers_of_digit(uint32_t d) {
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int bit = 0; bit < 8; ++bit) {
    const uint32_t b = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
    m &= ((d >> bit) & 1u) ? b : ~b;
  }
  return m;
}

// This element's rank among its warp's elements of the same digit so far
// (counts[d] of them in earlier rounds), which it joins.
__device__ __forceinline__ uint32_t warp_digit_rank(uint32_t* counts, uint32_t d, int lane, uint32_t lt) {
  const uint32_t peers = peers_of_digit(d);
  const uint32_t before = counts[d];
  __syncwarp();
  if (lane == __ffs(peers) - 1) counts[d] = before + __popc(peers);
  __syncwarp();
  return before + __popc(peers & lt);
}

constexpr uint64_t kRsFewRows = 1u << 16;
constexpr uint32_t kRsShortBlocks = 296;
constexpr uint32_t kRsSumRows = 8;  // in flight per thread (4: 63 us for 57 with 256 rows, 16: the same)

// FEW: offs holds the blocks' counts, which every block sums for itself;
// otherwise their exclusive scan.
template <int ROUNDS, bool FEW>
__global__ void __launch_bounds__(kRsThreads, FEW ? 2 : 3) k_radix_downsweep(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, int shift, uint32_t nb_seg, const uint32_t* __restrict__ offs, int write_keys,
    const uint2* __restrict__ gather_src, uint32_t gather_n, uint2* __restrict__ gather_dst, uint32_t iota_n) {
  constexpr int kRsTile = kRsThreads * ROUNDS;
  static_assert(kRsTile >= 8 * 256, "sk holds eight rows of sums");
  __shared__ uint32_t wc[kRsWarps][256];
  __shared__ uint32_t dstart[256];
  __shared__ uint32_t goff[256];
  __shared__ __align__(16) uint32_t sk[kRsTile];
  __shared__ uint32_t sv[kRsTile];
  __shared__ uint32_t block_total;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) wc[w][threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const size_t base = size_t(blockIdx.x) * kRsTile + size_t(warp) * (ROUNDS * 32);
  uint32_t k[ROUNDS], v[ROUNDS];
  // vin null (first pass of a sort of the identity permutation): an
  // element's value is its index in its segment, 0xffffffff from iota_n on
  if (vin) {
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      k[r] = kin[base + r * 32 + lane];
      v[r] = vin[base + r * 32 + lane];
    }
  } else {
    const uint32_t local0 = (blockIdx.x % nb_seg) * kRsTile + uint32_t(warp) * (ROUNDS * 32) + uint32_t(lane);
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      k[r] = kin[base + r * 32 + lane];
      const uint32_t local = local0 + uint32_t(r) * 32u;
      v[r] = local < iota_n ? local : 0xffffffffu;
    }
  }
  // FEW: the digits' counts in the segment's blocks, all and those before this
  // one; threads 64 g .. take every fourth row, four digits each, and leave
  // their sums in sk until phase 2
  if (FEW) {
    const uint32_t b = blockIdx.x % nb_seg, g = threadIdx.x >> 6, q = threadIdx.x & 63u;
    const uint4* h = reinterpret_cast<const uint4*>(offs) + size_t(blockIdx.x - b) * 64 + q;
    uint4 before = make_uint4(0u, 0u, 0u, 0u), all = before;
    for (uint32_t i0 = g; i0 < nb_seg; i0 += 4 * kRsSumRows)
#pragma unroll
      for (uint32_t j = 0; j < kRsSumRows; ++j) {
        const uint32_t i = i0 + 4 * j;
        const uint4 c = i < nb_seg ? h[size_t(i) * 64] : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t m = i < b ? 0xffffffffu : 0u;
        before.x += c.x & m;
        before.y += c.y & m;
        before.z += c.z & m;
        before.w += c.w & m;
        all.x += c.x;
        all.y += c.y;
        all.z += c.z;
        all.w += c.w;
      }
    reinterpret_cast<uint4*>(sk)[g * 64 + q] = all;
    reinterpret_cast<uint4*>(sk)[256 + g * 64 + q] = before;
  }
  // phase 1: ranks inside the warp, per-warp digit counts
  uint32_t rank[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) rank[r] = warp_digit_rank(wc[warp], (k[r] >> shift) & 255u, lane, lt);
  __syncthreads();
  // phase 2: block-local digit starts, warp bases, global digit offsets
  {
    const uint32_t d = threadIdx.x;
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) tot += wc[w][d];
    uint32_t run = block_excl_scan(tot, &block_total);
    dstart[d] = run;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
      const uint32_t t = wc[w][d];
      wc[w][d] = run;
      run += t;
    }
    const uint32_t seg = blockIdx.x / nb_seg, b = blockIdx.x % nb_seg;
    if (FEW) {
      const uint32_t all = sk[d] + sk[256 + d] + sk[512 + d] + sk[768 + d];
      const uint32_t before = sk[1024 + d] + sk[1280 + d] + sk[1536 + d] + sk[1792 + d];
      goff[d] = seg * nb_seg * kRsTile + block_excl_scan(all, &block_total) + before;
    } else {
      goff[d] = offs[(size_t(seg) * 256 + d) * nb_seg + b];
    }
  }
  __syncthreads();
  // phase 3: stable scatter into shared memory, digit-major
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const uint32_t lp = wc[warp][(k[r] >> shift) & 255u] + rank[r];
    sk[lp] = k[r];
    sv[lp] = v[r];
  }
  __syncthreads();
  // phase 4: digit runs to their global offsets
#pragma unroll 4
  for (int i = threadIdx.x; i < kRsTile; i += kRsThreads) {
    const uint32_t key = sk[i];
    const uint32_t d = (key >> shift) & 255u;
    const uint32_t pos = goff[d] + (uint32_t(i) - dstart[d]);
    const uint32_t val = sv[i];
    if (write_keys) kout[pos] = key;
    vout[pos] = val;
    // optional: the value's record gathered into sorted order (segment-major
    // source, one row of gather_n records per segment; values >= gather_n
    // are padding and get an empty record)
    if (gather_dst) {
      const uint32_t seg = blockIdx.x / nb_seg;
      gather_dst[pos] = val < gather_n ? gather_src[size_t(seg) * gather_n + val] : make_uint2(0u, 0u);
    }
  }
}

// n: keys of all segments together
static int radix_rounds(size_t n) {
  return n <= size_t(kRsThreads) * kRsShortRounds * kRsShortBlocks ? kRsShortRounds : kRsRounds;
}
// (a workspace of n keys also serves fewer)
size_t radix_hist_words(size_t n) {
  const size_t shrt = std::min<size_t>((n + kRsThreads * kRsShortRounds - 1) / (kRsThreads * kRsShortRounds),
                                       kRsShortBlocks);
  return std::max(shrt, (n + kRsThreads * kRsRounds - 1) / (kRsThreads * kRsRounds)) * 256 + 1;
}

// One block sorts a whole segment of up to THREADS * kBsRounds elements in
// shared memory: the same ranking, four digits one after the other, every
// warp with the same number of rounds of 32 consecutive elements.
constexpr int kBsRounds = 8;

template <int THREADS>
struct BlockSortShared {
  uint32_t keys[THREADS * kBsRounds];
  uint16_t idx[THREADS * kBsRounds];
  uint32_t wc[THREADS / 32][256];
  uint32_t total;
};

template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_block_sort(const uint32_t* __restrict__ kin, uint32_t n, uint32_t npad,
                                                        uint32_t* __restrict__ vout,
                                                        const uint2* __restrict__ gather_src,
                                                        uint2* __restrict__ gather_dst) {
  extern __shared__ __align__(16) unsigned char bs_raw[];
  BlockSortShared<THREADS>& sh = *reinterpret_cast<BlockSortShared<THREADS>*>(bs_raw);
  constexpr int WARPS = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, seg = blockIdx.x;
  const uint32_t rounds = (n + THREADS - 1) / THREADS;  // of this segment
  const uint32_t place0 = uint32_t(warp) * rounds * 32 + lane;
  // places from n on hold all-ones keys, which stay behind every element
  uint32_t k[kBsRounds], v[kBsRounds];  // v: index << 16 | rank
#pragma unroll
  for (int r = 0; r < kBsRounds; ++r) {
    const uint32_t i = place0 + 32 * r;
    k[r] = uint32_t(r) < rounds && i < n ? kin[size_t(seg) * npad + i] : 0xffffffffu;
    v[r] = i << 16;
  }
#pragma unroll 1
  for (int shift = 0; shift < 32; shift += 8) {
    for (int i = threadIdx.x; i < WARPS * 256; i += THREADS) (&sh.wc[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kBsRounds; ++r)
      if (uint32_t(r) < rounds) v[r] |= warp_digit_rank(sh.wc[warp], (k[r] >> shift) & 255u, lane, lt);
    __syncthreads();
    uint32_t c[WARPS], tot = 0;  // digit threadIdx.x's counts, warp by warp
    if (threadIdx.x < 256) {
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        c[w] = sh.wc[w][threadIdx.x];
        tot += c[w];
      }
    }
    uint32_t run = block_excl_scan(tot, &sh.total);
    if (threadIdx.x < 256) {
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        sh.wc[w][threadIdx.x] = run;
        run += c[w];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kBsRounds; ++r)
      if (uint32_t(r) < rounds) {
        const uint32_t lp = sh.wc[warp][(k[r] >> shift) & 255u] + (v[r] & 0xffffu);
        sh.keys[lp] = k[r];
        sh.idx[lp] = uint16_t(v[r] >> 16);
      }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kBsRounds; ++r)
      if (uint32_t(r) < rounds) {
        k[r] = sh.keys[place0 + 32 * r];
        v[r] = uint32_t(sh.idx[place0 + 32 * r]) << 16;
      }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < npad; i += THREADS) {
    const uint32_t idx = i < rounds * THREADS ? sh.idx[i] : 0xffffu;
    const bool real = idx < n;
    vout[size_t(seg) * npad + i] = real ? idx : 0xffffffffu;
    gather_dst[size_t(seg) * npad + i] = real ? gather_src[size_t(seg) * n + idx] : make_uint2(0u, 0u);
  }
}

template <int THREADS>
static cudaError_t block_sort(cudaStream_t st, const uint32_t* keys, uint32_t n, uint32_t npad, uint32_t nseg,
                              uint32_t* vout, const uint2* gather_src, uint2* gather_dst) {
  constexpr int smem = int(sizeof(BlockSortShared<THREADS>));
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_block_sort<THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  k_block_sort<THREADS><<<nseg, THREADS, smem, st>>>(keys, n, npad, vout, gather_src, gather_dst);
  count_launch();
  return cudaGetLastError();
}

template <int ROUNDS>
static cudaError_t radix_sort(cudaStream_t st, uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb, uint32_t npad,
                              uint32_t nseg, uint32_t* hist, uint32_t* scan_tmp, const uint2* gather_src, uint32_t n,
                              uint2* gather_dst) {
  const uint32_t nb_seg = npad / (kRsThreads * ROUNDS), nblocks = nb_seg * nseg;
  const bool few = uint64_t(nb_seg) * nblocks <= kRsFewRows;
  for (int pass = 0; pass < 4; ++pass) {
    const uint32_t* ki = pass & 1 ? kb : ka;
    const uint32_t* vi = pass == 0 ? nullptr : pass & 1 ? vb : va;  // the first pass forms the indices
    uint32_t* ko = pass & 1 ? ka : kb;
    uint32_t* vo = pass & 1 ? va : vb;
    (few ? k_radix_upsweep<ROUNDS, true> : k_radix_upsweep<ROUNDS, false>)<<<nblocks, kRsThreads, 0, st>>>(
        ki, 8 * pass, nb_seg, hist);
    count_launch();
    if (!few) {
      const cudaError_t e = exclusive_scan(st, hist, hist, size_t(nblocks) * 256, scan_tmp, 0xffffffffu, nullptr);
      if (e != cudaSuccess) return e;
    }
    const bool last = pass == 3;  // its keys are not needed
    (few ? k_radix_downsweep<ROUNDS, true> : k_radix_downsweep<ROUNDS, false>)<<<nblocks, kRsThreads, 0, st>>>(
        ki, vi, ko, vo, 8 * pass, nb_seg, hist, last ? 0 : 1, gather_src, n, last ? gather_dst : nullptr, n);
    count_launch();
  }
  return cudaGetLastError();
}

// Stable order of every segment's n elements by their 32-bit keys in ka
// ([nseg][npad], all-ones from n on; ka, kb and vb are scratch after): va gets
// the elements' indices in their segment, 0xffffffff for the padding, and
// gather_dst gather_src's record of each ([nseg][n], an empty one for the
// padding).  npad is a multiple of 4096.
cudaError_t depth_sort(cudaStream_t st, uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb, uint32_t npad,
                       uint32_t nseg, uint32_t* hist, uint32_t* scan_tmp, const uint2* gather_src, uint32_t n,
                       uint2* gather_dst) {
  if (npad == 0 || npad % (kRsThreads * kRsRounds) != 0 || nseg == 0) return cudaErrorInvalidValue;
  if (n <= 512 * kBsRounds) return block_sort<512>(st, ka, n, npad, nseg, va, gather_src, gather_dst);
  if (n <= 1024 * kBsRounds) return block_sort<1024>(st, ka, n, npad, nseg, va, gather_src, gather_dst);
  if (radix_rounds(size_t(npad) * nseg) == kRsShortRounds)
    return radix_sort<kRsShortRounds>(st, ka, va, kb, vb, npad, nseg, hist, scan_tmp, gather_src, n, gather_dst);
  return radix_sort<kRsRounds>(st, ka, va, kb, vb, npad, nseg, hist, scan_tmp, gather_src, n, gather_dst);
}

// ---------------------------------------------------------------------------
// Rank order helpers
// ---------------------------------------------------------------------------
// superblock span of a tile span (superblocks of 1 << sl tiles per side);
// empty if no tile
__device__ __forceinline__ bool sb_span(uint2 rc, int sl, int* sx0, int* sy0, int* sx1, int* sy1) {
  const int x0 = rc.x & 0xffff, y0 = rc.x >> 16, x1 = rc.y & 0xffff, y1 = rc.y >> 16;
  if (x1 <= x0 || y1 <= y0) return false;
  *sx0 = x0 >> sl;
  *sy0 = y0 >> sl;
  *sx1 = ((x1 - 1) >> sl) + 1;
  *sy1 = ((y1 - 1) >> sl) + 1;
  return true;
}

// tile span clipped to superblock (sx, sy), in local tile coordinates
// 0..(1 << sl): x0 | y0 << 4 | x1 << 8 | y1 << 12
__device__ __forceinline__ uint32_t local_rect(uint2 rc, int sl, int sx, int sy) {
  const int side = 1 << sl, bx = sx << sl, by = sy << sl;
  const int x0 = max(int(rc.x & 0xffff), bx) - bx, x1 = min(int(rc.y & 0xffff), bx + side) - bx;
  const int y0 = max(int(rc.x >> 16), by) - by, y1 = min(int(rc.y >> 16), by + side) - by;
  return uint32_t(x0) | uint32_t(y0) << 4 | uint32_t(x1) << 8 | uint32_t(y1) << 12;
}

constexpr int kMsThreads = 256;
constexpr int kMsWarps = kMsThreads / 32;

// ---------------------------------------------------------------------------
// Stage 1a: per (chunk, superblock) counts.  Block = one chunk of ranks (512
// to 4096, choose_chunk in capi.cu) of one view.  Output layout cnt[(sb_base[v] + s) * nchunk + c] so that an
// exclusive scan in index order yields (view, superblock, rank) positions.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kMsThreads) k_sb_count(const uint32_t* __restrict__ order,
                                                         const uint2* __restrict__ srect, uint32_t chunk, uint32_t npad,
                                                         const ViewBatch b,
                                                         uint32_t* __restrict__ cnt,
                                                         unsigned long long* __restrict__ totals) {
  extern __shared__ uint32_t hist[];
  const uint32_t nchunk = npad / chunk;
  const uint32_t v = blockIdx.x / nchunk, c = blockIdx.x % nchunk;
  const ViewDev& vd = b.v[v];
  const int sl = vd.sb_log2, sbw = sb_cols(vd), sbh = sb_rows(vd);
  const int nsb = sbw * sbh;
  for (int i = threadIdx.x; i < nsb; i += kMsThreads) hist[i] = 0;
  __syncthreads();
  const size_t base = size_t(v) * npad + size_t(c) * chunk;
  unsigned long long pairs = 0, entries = 0;
  for (uint32_t i = threadIdx.x; i < chunk; i += kMsThreads) {
    const uint2 rc = srect[base + i];
    int sx0, sy0, sx1, sy1;
    if (!sb_span(rc, sl, &sx0, &sy0, &sx1, &sy1)) continue;
    pairs += (unsigned long long)((rc.y & 0xffff) - (rc.x & 0xffff)) * ((rc.y >> 16) - (rc.x >> 16));
    entries += (unsigned long long)(sx1 - sx0) * (sy1 - sy0);
    for (int sy = sy0; sy < sy1; ++sy)
      for (int sx = sx0; sx < sx1; ++sx) atomicAdd(&hist[sy * sbw + sx], 1u);
  }
  // exact 64-bit totals of tile pairs (tile-span areas) and superblock
  // entries, known even when a later stage overflows or a 32-bit list offset
  // wraps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    entries += __shfl_xor_sync(0xffffffffu, entries, o);
  }
  if ((threadIdx.x & 31) == 0 && entries) {
    atomicAdd(&totals[0], pairs);
    atomicAdd(&totals[1], entries);
  }
  __syncthreads();
  const uint32_t sb0 = vd.sb_base;
  for (int i = threadIdx.x; i < nsb; i += kMsThreads) cnt[(size_t(sb0) + i) * nchunk + c] = hist[i];
}

// ---------------------------------------------------------------------------
// Stage 1b: stable scatter of point indices into superblock lists.  Warp w
// owns an eighth of the chunk's ranks in rounds of 32.  In a round,
// each lane sets its bit in a shared mask per superblock column and row its
// span covers; the lanes covering superblock (x, y) are then
// colmask[x] & rowmask[y], and a lane's slot is its popcount among them.
// ---------------------------------------------------------------------------
// Flags a capacity overflow when the superblock lists need more entries than
// the capacity (the 64-bit total also catches a wrapped 32-bit offset scan).
__device__ __forceinline__ void check_capacity(uint64_t capacity, uint32_t* __restrict__ flags) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && *reinterpret_cast<const unsigned long long*>(flags + 8) > capacity)
    set_flag(flags, kFlagPairOverflow);
}

__global__ void __launch_bounds__(kMsThreads) k_sb_scatter(const uint32_t* __restrict__ order,
                                                           const uint2* __restrict__ srect, uint32_t chunk, uint32_t npad,
                                                           const ViewBatch b,
                                                           const uint32_t* __restrict__ off, uint64_t capacity,
                                                           uint2* __restrict__ list1, uint32_t* __restrict__ flags) {
  check_capacity(capacity, flags);
  extern __shared__ uint32_t smem_ms[];  // [kMsWarps][nsb] counters, then [kMsWarps][2 * side] masks
  const uint32_t nchunk = npad / chunk;
  const uint32_t v = blockIdx.x / nchunk, c = blockIdx.x % nchunk;
  const ViewDev& vd = b.v[v];
  const int sl = vd.sb_log2, sbw = sb_cols(vd), sbh = sb_rows(vd);
  const int nsb = sbw * sbh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t rounds = chunk / kMsThreads;  // of 32 ranks per warp
  uint32_t* wc = smem_ms;
  const uint32_t side = b.max_sb_side;
  uint32_t* colmask = smem_ms + kMsWarps * b.max_sb + warp * 2 * side;
  uint32_t* rowmask = colmask + side;
  for (int i = threadIdx.x; i < kMsWarps * nsb; i += kMsThreads) wc[i] = 0;
  __syncthreads();
  const size_t base = size_t(v) * npad + size_t(c) * chunk + size_t(warp) * (rounds * 32);
  uint32_t* my = wc + warp * nsb;
  // phase 1: per-warp counts
  for (uint32_t r = 0; r < rounds; ++r) {
    int sx0, sy0, sx1, sy1;
    if (sb_span(srect[base + r * 32 + lane], sl, &sx0, &sy0, &sx1, &sy1))
      for (int sy = sy0; sy < sy1; ++sy)
        for (int sx = sx0; sx < sx1; ++sx) atomicAdd(&my[sy * sbw + sx], 1u);
  }
  __syncthreads();
  // phase 2: warp bases = chunk offset + earlier warps
  const uint32_t sb0 = vd.sb_base;
  for (int i = threadIdx.x; i < nsb; i += kMsThreads) {
    uint32_t run = off[(size_t(sb0) + i) * nchunk + c];
    for (int w = 0; w < kMsWarps; ++w) {
      const uint32_t t = wc[w * nsb + i];
      wc[w * nsb + i] = run;
      run += t;
    }
  }
  __syncthreads();
  // phase 3: stable scatter, round by round
  for (uint32_t r = 0; r < rounds; ++r) {
    const uint32_t g = order[base + r * 32 + lane];
    int sx0 = 0, sy0 = 0, sx1 = 0, sy1 = 0;
    const uint2 rc = srect[base + r * 32 + lane];
    const bool has = sb_span(rc, sl, &sx0, &sy0, &sx1, &sy1);
    // the round's column / row coverage masks: every lane clears, then sets
    // its bit in, the entries of the columns and rows its span covers
    if (has) {
      for (int x = sx0; x < sx1; ++x) colmask[x] = 0u;
      for (int y = sy0; y < sy1; ++y) rowmask[y] = 0u;
    }
    __syncwarp();
    if (has) {
      for (int x = sx0; x < sx1; ++x) atomicOr(&colmask[x], 1u << lane);
      for (int y = sy0; y < sy1; ++y) atomicOr(&rowmask[y], 1u << lane);
    }
    __syncwarp();
    for (int sy = sy0; sy < sy1; ++sy) {
      const uint32_t rm = rowmask[sy];
      for (int sx = sx0; sx < sx1; ++sx) {
        const uint32_t m = colmask[sx] & rm;
        const uint32_t dst = my[sy * sbw + sx] + uint32_t(__popc(m & lt));
        if (dst < capacity) list1[dst] = make_uint2(g, local_rect(rc, sl, sx, sy));
        else set_flag(flags, kFlagPairOverflow);
      }
    }
    __syncwarp();
    // the highest lane covering a superblock advances the warp's counter
    for (int sy = sy0; sy < sy1; ++sy) {
      const uint32_t rm = rowmask[sy];
      for (int sx = sx0; sx < sx1; ++sx) {
        const uint32_t m = colmask[sx] & rm;
        if ((m >> lane) == 1u) my[sy * sbw + sx] += uint32_t(__popc(m));
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Stage 1b, staged: the same result as k_sb_scatter with coalesced stores and
// its work spread over entries instead of ranks.  The chunk is taken in
// sub-passes of kSubRanks consecutive ranks, a sub-pass in pieces of at most
// kPiece entries:
//   expand   every rank writes its superblocks, in order, to its place in the
//            piece (ranks and places from a block-wide scan of the counts);
//   rank     warp w takes an eighth of the piece's entries, 32 at a time: the
//            lanes of the same superblock come from one ballot per bit of its
//            number, earlier rounds from the warp's counters;
//   bases    one block-wide scan over the view's superblocks;
//   stage    the entries in superblock order in shared memory;
//   store    each superblock's run to its contiguous range of the list (the
//            block's cursor for it advances piece by piece).
// Bound: the latency between its barriers, at 3 blocks per SM (4, by fewer
// registers, were slower).  us, against every lane looping over its own rank's
// span with coverage masks: 16 views of 1,048,576 points 816 -> 762, 8 of
// 4,194,304 1800 -> 1650, one 76 -> 68, one of 16,384 17 -> 13.  Unrolling the
// ballots, match.any and ranking all rounds before counting were slower (822,
// 861, 868).
// Shared memory: see SbScatterShared.
// ---------------------------------------------------------------------------
constexpr int kSubRanks = 2 * kMsThreads;  // 512 ranks per sub-pass, two per thread
constexpr int kPieceRounds = 12;
constexpr uint32_t kPiece = kMsThreads * kPieceRounds;  // 3072 entries

struct SbScatterShared {
  uint2 stage[kPiece];         // the piece's entries in superblock order
  union {
    uint32_t ent[kPiece];      // superblock x | y << 8 | rank of the sub-pass << 16, in list order
    uint16_t stage_sb[kPiece];
  };
  uint2 rect[kSubRanks];       // the sub-pass's spans
  uint32_t point[kSubRanks];   // and points
  uint32_t first[kSubRanks + 1];  // and first entries
  uint32_t total;
  // then uint32_t cur[max_sb], sbase[max_sb + 1], uint16_t wc[kMsWarps][max_sb]
};

size_t sb_scatter_staged_smem(uint32_t max_sb) {
  return sizeof(SbScatterShared) + (2 * size_t(max_sb) + 1) * 4 + size_t(kMsWarps) * max_sb * 2;
}

__global__ void __launch_bounds__(kMsThreads, 3) k_sb_scatter_staged(const uint32_t* __restrict__ order,
                                                                  const uint2* __restrict__ srect, uint32_t chunk,
                                                                  uint32_t npad, const ViewBatch b,
                                                                  const uint32_t* __restrict__ off, uint64_t capacity,
                                                                  uint2* __restrict__ list1,
                                                                  uint32_t* __restrict__ flags) {
  check_capacity(capacity, flags);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SbScatterShared& sh = *reinterpret_cast<SbScatterShared*>(smem_raw);
  const uint32_t nchunk = npad / chunk;
  const uint32_t v = blockIdx.x / nchunk, c = blockIdx.x % nchunk;
  const ViewDev& vd = b.v[v];
  const int sl = vd.sb_log2, sbw = sb_cols(vd), nsb = sbw * sb_rows(vd);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* const cur = reinterpret_cast<uint32_t*>(smem_raw + sizeof(SbScatterShared));
  uint32_t* const sbase = cur + b.max_sb;
  uint16_t* const wc = reinterpret_cast<uint16_t*>(sbase + b.max_sb + 1);
  uint16_t* const my = wc + warp * nsb;
  int bits = 1;  // of a superblock's number
  while ((1 << bits) < nsb) ++bits;
  for (int i = threadIdx.x; i < nsb; i += kMsThreads) cur[i] = off[(size_t(vd.sb_base) + i) * nchunk + c];
  const int seg = (nsb + kMsThreads - 1) / kMsThreads;
  const int s_lo = min(nsb, int(threadIdx.x) * seg), s_hi = min(nsb, s_lo + seg);
  for (uint32_t sub = 0; sub < chunk / kSubRanks; ++sub) {
    const size_t base = size_t(v) * npad + size_t(c) * chunk + size_t(sub) * kSubRanks + 2 * threadIdx.x;
    // this thread's two ranks
    const uint4 rr = *reinterpret_cast<const uint4*>(srect + base);
    const uint2 pp = *reinterpret_cast<const uint2*>(order + base);
    const uint2 rc[2] = {make_uint2(rr.x, rr.y), make_uint2(rr.z, rr.w)};
    int sx0[2], sy0[2], sx1[2], sy1[2];
    uint32_t count[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
      count[k] = sb_span(rc[k], sl, &sx0[k], &sy0[k], &sx1[k], &sy1[k])
                     ? uint32_t(sx1[k] - sx0[k]) * uint32_t(sy1[k] - sy0[k]) : 0u;
    const uint32_t first = block_excl_scan(count[0] + count[1], &sh.total);
    *reinterpret_cast<uint4*>(&sh.rect[2 * threadIdx.x]) = rr;
    *reinterpret_cast<uint2*>(&sh.point[2 * threadIdx.x]) = pp;
    sh.first[2 * threadIdx.x] = first;
    sh.first[2 * threadIdx.x + 1] = first + count[0];
    if (threadIdx.x == 0) sh.first[kSubRanks] = sh.total;
    __syncthreads();
    const uint32_t total = sh.total;
    // pieces of whole ranks: a rank has at most nsb <= kPiece entries
    for (uint32_t r0 = 0, e0 = 0; e0 < total;) {
      uint32_t r1 = kSubRanks, e1 = total;
      if (total - e0 > kPiece) {  // the last rank that still fits, the same search in every thread
        uint32_t lo = r0 + 1, hi = kSubRanks;
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) / 2;
          if (sh.first[mid] - e0 <= kPiece) lo = mid;
          else hi = mid - 1;
        }
        r1 = lo;
        e1 = sh.first[r1];
      }
      for (int i = threadIdx.x; i < (kMsWarps * nsb + 1) / 2; i += kMsThreads) reinterpret_cast<uint32_t*>(wc)[i] = 0;
      uint32_t at = first - e0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t rank = 2 * threadIdx.x + k;
        if (count[k] && rank >= r0 && rank < r1) {
          uint32_t o = at;
          for (int sy = sy0[k]; sy < sy1[k]; ++sy)
            for (int sx = sx0[k]; sx < sx1[k]; ++sx) sh.ent[o++] = uint32_t(sx) | uint32_t(sy) << 8 | rank << 16;
        }
        at += count[k];
      }
      __syncthreads();
      const uint32_t n_piece = e1 - e0, rounds = (n_piece + kMsThreads - 1) / kMsThreads;
      const uint32_t i0 = uint32_t(warp) * rounds * 32 + lane;
      uint32_t e[kPieceRounds], place[kPieceRounds];  // place: superblock << 16 | rank among the warp's of it
#pragma unroll
      for (int r = 0; r < kPieceRounds; ++r) {
        if (uint32_t(r) >= rounds) break;
        const bool in = i0 + 32 * r < n_piece;
        e[r] = in ? sh.ent[i0 + 32 * r] : 0u;
        const uint32_t sb = in ? ((e[r] >> 8) & 255u) * uint32_t(sbw) + (e[r] & 255u) : 0u;
        uint32_t peers = __ballot_sync(0xffffffffu, in);
        for (int bit = 0; bit < bits; ++bit) {
          const uint32_t m = __ballot_sync(0xffffffffu, (sb >> bit) & 1u);
          peers &= ((sb >> bit) & 1u) ? m : ~m;
        }
        uint32_t before = 0;
        if (in) before = my[sb];
        __syncwarp();
        if (in && lane == __ffs(peers) - 1) my[sb] = uint16_t(before + __popc(peers));
        __syncwarp();
        place[r] = sb << 16 | (before + __popc(peers & lt));
      }
      __syncthreads();
      // stage layout: superblock-major, then warp (= list order)
      uint32_t loc = 0;
      for (int sb = s_lo; sb < s_hi; ++sb)
#pragma unroll
        for (int w = 0; w < kMsWarps; ++w) loc += wc[w * nsb + sb];
      uint32_t run = block_excl_scan(loc, &sh.total);
      for (int sb = s_lo; sb < s_hi; ++sb) {
        sbase[sb] = run;
#pragma unroll
        for (int w = 0; w < kMsWarps; ++w) {
          const uint32_t t = wc[w * nsb + sb];
          wc[w * nsb + sb] = uint16_t(run);
          run += t;
        }
      }
      if (threadIdx.x == 0) sbase[nsb] = n_piece;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kPieceRounds; ++r) {
        if (uint32_t(r) >= rounds) break;
        if (i0 + 32 * r < n_piece) {
          const uint32_t sb = place[r] >> 16, rank = e[r] >> 16, pos = my[sb] + (place[r] & 0xffffu);
          sh.stage[pos] = make_uint2(sh.point[rank], local_rect(sh.rect[rank], sl, int(e[r] & 255u),
                                                                int((e[r] >> 8) & 255u)));
          sh.stage_sb[pos] = uint16_t(sb);
        }
      }
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < n_piece; i += kMsThreads) {
        const int sb = sh.stage_sb[i];
        const uint64_t dst = uint64_t(cur[sb]) + (i - sbase[sb]);
        if (dst < capacity) list1[dst] = sh.stage[i];
        else set_flag(flags, kFlagPairOverflow);
      }
      __syncthreads();
      for (int sb = threadIdx.x; sb < nsb; sb += kMsThreads) cur[sb] += sbase[sb + 1] - sbase[sb];
      r0 = r1;
      e0 = e1;
      __syncthreads();
    }
  }
}

cudaError_t sb_scatter_staged(cudaStream_t st, unsigned grid, const uint32_t* order, const uint2* srect, uint32_t chunk,
                              uint32_t npad, const ViewBatch& b, const uint32_t* off, uint64_t capacity, uint2* list1,
                              uint32_t* flags) {
  const size_t smem = sb_scatter_staged_smem(b.max_sb);
  if (smem > 48 * 1024) {  // the same limit in every call (see kSbScatterMost in capi.cu)
    const cudaError_t e =
        cudaFuncSetAttribute(k_sb_scatter_staged, cudaFuncAttributeMaxDynamicSharedMemorySize, kSbStagedMost);
    if (e != cudaSuccess) return e;
  }
  k_sb_scatter_staged<<<grid, kMsThreads, smem, st>>>(order, srect, chunk, npad, b, off, capacity, list1, flags);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Longest-first task order for the rasterisers: items bucketed by floor(log2)
// of their cost, heaviest bucket first, so the tail of the persistent launch
// is made of short tasks.  The cost is that of the item's longest walk in the
// last forward (measured, kept in the workspace) or, where none is recorded
// yet, its superblock-list length; the workspace's mark (*cost_tag == tag) says
// whether a forward of this layout has measured at all.  Only the schedule
// depends on it, never the results.  sched: see kSchedCost in common.cuh.
//
// Heavy items: a task whose cost is a good part of what every resident warp
// has to do (total / warps) ends after the others, and the GPU waits for it
// -- the tiles of a scene's rim, whose pixels never saturate, walk ten times
// the mean list.  The items of the buckets above that share are walked in 8x8
// blocks (about 15% more instructions, so short tasks stay whole).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t item_cost(const ViewBatch& b, uint32_t item, const uint32_t* off1, uint32_t nchunk,
                                              const uint32_t* cost, bool measured) {
  int v = 0;
  for (int k = 1; k < b.num_views; ++k)
    if (item >= b.v[k].item_base) v = k;
  const ViewDev& vd = b.v[v];
  const uint32_t t = item - vd.item_base;
  const uint32_t tx = t % uint32_t(vd.tile_w), ty = t / uint32_t(vd.tile_w);
  // 8x8 tiles: the leftmost tile of a run carries the task of both
  if (b.ts == 8 && tx % min(2u, 1u << vd.sb_log2)) return 0u;
  const uint32_t c = measured ? cost[item] : 0u;
  if (c) return c;
  const uint32_t sb = vd.sb_base + (ty >> vd.sb_log2) * uint32_t(sb_cols(vd)) + (tx >> vd.sb_log2);
  return off1[size_t(sb + 1) * nchunk] - off1[size_t(sb) * nchunk];
}

__global__ void k_order_hist(const ViewBatch b, const uint32_t* __restrict__ off1, uint32_t nchunk,
                             const uint32_t* __restrict__ cost, const unsigned long long* __restrict__ cost_tag,
                             unsigned long long tag, uint32_t* __restrict__ sched) {
  __shared__ uint32_t h[33];
  const bool measured = *cost_tag == tag;
  if (blockIdx.x == 0 && threadIdx.x == 0) sched[kSchedMeasured] = measured;
  if (threadIdx.x < 33) h[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long sum = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < b.num_items; i += gridDim.x * blockDim.x) {
    const uint32_t c = item_cost(b, i, off1, nchunk, cost, measured);
    atomicAdd(&h[__clz(c)], 1u);
    sum += c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(reinterpret_cast<unsigned long long*>(sched + kSchedCost), sum);
  __syncthreads();
  if (threadIdx.x < 33 && h[threadIdx.x]) atomicAdd(&sched[threadIdx.x], h[threadIdx.x]);
}

// Scatter into bucket order: each block ranks its items in shared memory and
// takes one range per bucket from the global cursors (one global atomic per
// bucket and block instead of one per item on 33 hot counters); every block
// forms the buckets' starts from the counts itself.  heavy_share: an item
// is heavy when its cost times that is above the total cost.
// The costs are set to zero for this forward to measure, and marked as its.
__global__ void k_order_scatter(const ViewBatch b, const uint32_t* __restrict__ off1, uint32_t nchunk,
                                uint32_t* __restrict__ cost, unsigned long long* __restrict__ cost_tag,
                                unsigned long long tag, float heavy_share, uint32_t* __restrict__ sched,
                                uint32_t* __restrict__ order) {
  const bool measured = sched[kSchedMeasured] != 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0) *cost_tag = tag;
  __shared__ uint32_t cnt[33], base[33], start[33];
  if (threadIdx.x == 0) {
    const float total = float(*reinterpret_cast<const unsigned long long*>(sched + kSchedCost));
    uint32_t run = 0, heavy = 0;
    for (int k = 0; k < 33; ++k) {
      start[k] = run;
      run += sched[k];
      // bucket k holds the costs from 2^(31 - k) on
      if (k < 32 && exp2f(float(31 - k)) * heavy_share > total) heavy = run;
    }
    if (blockIdx.x == 0) sched[kSchedHeavy] = heavy;
  }
  __syncthreads();
  const uint32_t per_block = (b.num_items + gridDim.x - 1) / gridDim.x;
  const uint32_t lo = blockIdx.x * per_block, hi = min(b.num_items, lo + per_block);
  for (uint32_t i0 = lo; i0 < hi; i0 += blockDim.x) {
    if (threadIdx.x < 33) cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t i = i0 + threadIdx.x;
    uint32_t bucket = 0, slot = 0;
    if (i < hi) {
      bucket = uint32_t(__clz(item_cost(b, i, off1, nchunk, cost, measured)));
      cost[i] = 0u;
      slot = atomicAdd(&cnt[bucket], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 33 && cnt[threadIdx.x])
      base[threadIdx.x] = start[threadIdx.x] + atomicAdd(&sched[40 + threadIdx.x], cnt[threadIdx.x]);
    __syncthreads();
    if (i < hi) order[base[bucket] + slot] = i;
    __syncthreads();
  }
}


// keys for the drop-in API: idx2tiledepth = (tile << 32) | depth bits of the
// point, recomputed from pnt2pixxydepth
__global__ void k_make_keys64(const uint32_t* __restrict__ tile, const uint32_t* __restrict__ pnt,
                              const float* __restrict__ xyd, const unsigned long long* __restrict__ count_ptr,
                              uint64_t capacity, uint64_t* __restrict__ out) {
  const uint64_t cnt = *count_ptr < capacity ? uint64_t(*count_ptr) : capacity;
  for (size_t p = size_t(blockIdx.x) * blockDim.x + threadIdx.x; p < cnt; p += size_t(gridDim.x) * blockDim.x)
    out[p] = (uint64_t(tile[p]) << 32) | depth_bits(xyd[3 * size_t(pnt[p]) + 2]);
}

}  // namespace dsplat
