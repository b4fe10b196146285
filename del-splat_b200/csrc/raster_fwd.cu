// raster_fwd.cu -- the forward rasterisers (see raster_common.cuh).
//
// The blend must perform del-splat-cpu's operations one IEEE rounding at a
// time.  The file is built with -fmad=false (no scalar multiply-add is
// contracted), and every packed product whose result feeds an add is formed
// with mul2_rn (an fma with a runtime -0 addend, kernel argument nz), because
// the assembler contracts packed mul/add pairs regardless of that flag.  The
// fused multiply-adds the exponential wants are written out (fma2) and stay
// fused.
#include <algorithm>

#include "raster_block.cuh"
#include "raster_common.cuh"

namespace dsplat {

uint32_t raster_slabs_per_tile(int ts, int ppl);

// The L2 loss is summed in units of 8 columns and as many rows, 8 or, where a
// slab has only four, 4, in the same order of pixels in a slab as in an 8x8
// block, so that its bits do not depend on the shape an item is walked in.
__host__ __device__ constexpr int loss_rows(int slab_rows) { return slab_rows < 8 ? slab_rows : 8; }

// ---------------------------------------------------------------------------
// Forward walk of one slab by one warp over the list range [s, e).  Slot k of
// every lane lies in the same row pair of the slab, so the per-slot skips
// (pixel done, row outside the entry's box) are uniform across the warp most
// of the time.
// ---------------------------------------------------------------------------
// SPLIT (a 16x8 task of two 8x8 tiles, 4 slots per lane): lane L covers
// column L % 8 of both tiles at rows L / 8 and L / 8 + 4, slot pair 0 in the
// left tile and pair 1 in the right one, so that an entry whose box meets
// one tile keeps every lane of the warp busy on one pair and skips the
// other pair warp-wide.  Otherwise lane L covers column L % TS, slot k at
// row L / TS + k (32 / TS).
template <int TS, int PPL_, bool SPLIT, class Walk, class Src, class Loss>
__device__ __forceinline__ uint32_t fwd_slab(const Walk& walk, const Src& src, EntP* sm, float4* park,
                                         uint32_t* park_pos, const float* tab, float nz,
                                         uint32_t s, uint32_t e, int px0, int py0, int w, int h, int xend,
                                         float* __restrict__ out_rgb, size_t pix_base, float* __restrict__ out_T,
                                         float* __restrict__ out_alpha, uint32_t* __restrict__ out_last,
                                         const float* __restrict__ target,
                                         float* __restrict__ grad_pix, const Loss& loss) {
  using G = Geo<TS, PPL_>;
  constexpr int PPL = G::PPL;
  static_assert(PPL % 2 == 0, "pixel slots are evaluated in pairs");
  constexpr int NP = PPL / 2;
  static_assert(!SPLIT || (TS == 16 && PPL == 4), "split lanes: two 8-wide tiles, two slot pairs");
  constexpr int COLS = SPLIT ? TS / 2 : TS;
  constexpr int RSTEP = SPLIT ? 4 : G::ROW_STEP;
  const int lane = threadIdx.x & 31;
  const int col = lane % COLS, row0 = lane / COLS;
  auto slot_x = [&](int k) { return px0 + col + (SPLIT ? (k / 2) * COLS : 0); };
  auto slot_y = [&](int k) { return py0 + row0 + (SPLIT ? k % 2 : k) * RSTEP; };
  float fxp[NP];  // column centre of each slot pair
#pragma unroll
  for (int q = 0; q < NP; ++q) fxp[q] = float(slot_x(2 * q)) + 0.5f;
  float T[PPL], as[PPL], c0[PPL], c1[PPL], c2[PPL], fy[PPL];
  uint32_t live = 0;
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    const int ix = slot_x(k), iy = slot_y(k);
    fy[k] = float(iy) + 0.5f;
    T[k] = 1.f;
    as[k] = 0.f;
    c0[k] = c1[k] = c2[k] = 0.f;
    if (ix < xend && iy < h) {
      live |= 1u << k;
    }
  }
  // slot pairs (2p, 2p+1) in packed registers during the walk
  f2 T2[NP], as2[NP], c02[NP], c12[NP], c22[NP], fy2[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    T2[q] = f2_make(T[2 * q], T[2 * q + 1]);
    as2[q] = f2_make(as[2 * q], as[2 * q + 1]);
    c02[q] = f2_make(c0[2 * q], c0[2 * q + 1]);
    c12[q] = f2_make(c1[2 * q], c1[2 * q + 1]);
    c22[q] = f2_make(c2[2 * q], c2[2 * q + 1]);
    fy2[q] = f2_make(fy[2 * q], fy[2 * q + 1]);
  }
  const f2 nz2 = f2_dup(nz);  // (-0, -0), a runtime value (see mul2_rn)
  // a slot that stops parks its final values in the warp's shared area
  // (park[k][lane] = T, r, g, b; park_pos[k][lane] = its stop position); its
  // registers are no longer read, and the outputs are written after the walk
  const uint32_t inside = live;
  // centres of the slab's first and last rows (the same for every lane)
  const float fy_first = float(py0) + 0.5f, fy_last = float(py0 + G::SLAB_ROWS - 1) + 0.5f;
  uint32_t hi = e, cost = 0;
  uint2 en = hi > s ? walk.load(hi - 1u - uint32_t(lane), uint32_t(lane) < hi - s) : make_uint2(0u, 0u);
  while (hi > s) {
    const int cnt = int(min(32u, hi - s));
    const int k_staged = walk.stage(src, sm, en, hi - 1u - uint32_t(lane), lane < cnt, lane);
    {  // the next batch's list words arrive while this batch is blended
      const uint32_t hn = hi - uint32_t(cnt);
      if (hn > s) en = walk.load(hn - 1u - uint32_t(lane), uint32_t(lane) < hn - s);
    }
    __syncwarp();
    if (live) {
      for (int j = 0; j < k_staged; ++j) {
        const float4 ee = sm[j].e;
        // column tests: the slot pairs' columns (one column unless SPLIT)
        const bool cin0 = ee.x <= fxp[0] && fxp[0] <= ee.y;
        const bool cin1 = SPLIT ? (ee.x <= fxp[NP - 1] && fxp[NP - 1] <= ee.y) : cin0;
        if (!(cin0 || cin1)) continue;
        const ulonglong2 qa = *reinterpret_cast<const ulonglong2*>(&sm[j].a);  // (py,py) (2B,2B)
        const ulonglong2 qb = *reinterpret_cast<const ulonglong2*>(&sm[j].b);  // (C,C) (op,op)
        const ulonglong2 qc = *reinterpret_cast<const ulonglong2*>(&sm[j].c);  // (r,r) (g,g)
        const float4 ed = sm[j].d;                                             // b, b, px, A
        const f2 qbl = f2_make(ed.x, ed.y);
        const float2 ef = *reinterpret_cast<const float2*>(&sm[j].f);
        // -q/2 with q = A dx dx + B (dx dy + dy dx) + C dy dy in the
        // reference's order (mat2_sym::mult_vec_from_both_sides), from the
        // conic staged times -1/2; dx is fixed per slot pair, so (A dx) dx
        // is formed once per entry and column, and B (dx dy + dy dx) is
        // (2B)(dx dy) exactly
        auto col_terms = [&](float fxq, f2* adxdx2, f2* dx2) {
          const float dx = fs(fxq, ed.z);
          *adxdx2 = f2_dup(__fmaf_rn(fm(ed.w, dx), dx, nz));
          *dx2 = f2_dup(dx);
        };
        f2 adxdx2_1 = 0, dx2_1 = 0;  // the lane's column (all pairs) unless SPLIT
        if (!SPLIT) col_terms(fxp[0], &adxdx2_1, &dx2_1);
        const uint32_t pos = __float_as_uint(ef.y);
        // all instances compute the same bits: `inrange` skips expf_cr's
        // range check and the care for colours that are not finite (proven by
        // the entry's staged flag), `rows` the row test of an entry whose box
        // holds every row of the slab
        auto blend_slots = [&](auto inrange, auto rows) {
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            // a slot is one row of the slab across the warp: the skips are
            // warp-uniform in practice
            const int k0 = 2 * q, k1 = 2 * q + 1;
            if (SPLIT && !(q == 0 ? cin0 : cin1)) continue;
            // a0/a1: the slot's row lies in the box.  A stopped slot's
            // registers are no longer read (its outputs are written), so only
            // the row test masks the update
            const bool a0 = decltype(rows)::value || (ee.z <= fy[k0] && fy[k0] <= ee.w);
            const bool a1 = decltype(rows)::value || (ee.z <= fy[k1] && fy[k1] <= ee.w);
            if (!((((live >> k0) & 1u) && a0) || (((live >> k1) & 1u) && a1))) continue;
            f2 adxdx2 = adxdx2_1, dx2 = dx2_1;
            if (SPLIT) col_terms(fxp[q], &adxdx2, &dx2);
            const f2 dy2 = sub2(fy2[q], qa.x);
            const f2 qf = add2(add2(adxdx2, mul2_rn(qa.y, mul2(dx2, dy2), nz2)),
                               mul2_rn(mul2(qb.x, dy2), dy2, nz2));
            const f2 g2 = expf_cr2<!decltype(inrange)::value>(qf, tab);
            const f2 al = mul2_rn(g2, qb.y, nz2);
            // a live slot whose row is outside the box takes alpha 0: its
            // state is unchanged
            const f2 e2 = decltype(rows)::value ? al : f2_make(a0 ? f2_lo(al) : 0.f, a1 ? f2_hi(al) : 0.f);
            const f2 eo2 = mul2_rn(T2[q], e2, nz2);
            // of an entry that may have an infinite colour, a pixel outside
            // the box takes colour 0
            auto colour = [&](f2 c) {
              return decltype(inrange)::value || decltype(rows)::value
                         ? c : f2_make(a0 ? f2_lo(c) : 0.f, a1 ? f2_hi(c) : 0.f);
            };
            c02[q] = add2(c02[q], mul2_rn(colour(qc.x), eo2, nz2));
            c12[q] = add2(c12[q], mul2_rn(colour(qc.y), eo2, nz2));
            c22[q] = add2(c22[q], mul2_rn(colour(qbl), eo2, nz2));
            T2[q] = mul2(T2[q], sub2(f2_dup(1.f), e2));
            as2[q] = add2(as2[q], eo2);
            // a stopped slot's alpha sum is parked at -inf (it stays -inf
            // or NaN, which no test passes), and a live slot keeps a sum at
            // or below the threshold until it stops, so one test of the
            // pair's larger sum finds every slot that stops at this entry
            const float amax = fmaxf(f2_lo(as2[q]), f2_hi(as2[q]));
            if (amax > kAlphaStop) {  // rare
              float s0 = f2_lo(as2[q]), s1 = f2_hi(as2[q]);
              if (s0 > kAlphaStop) {
                live &= ~(1u << k0);
                park[k0 * 32 + lane] = make_float4(f2_lo(T2[q]), f2_lo(c02[q]), f2_lo(c12[q]), f2_lo(c22[q]));
                park_pos[k0 * 32 + lane] = pos;
                s0 = -INFINITY;
              }
              if (s1 > kAlphaStop) {
                live &= ~(1u << k1);
                park[k1 * 32 + lane] = make_float4(f2_hi(T2[q]), f2_hi(c02[q]), f2_hi(c12[q]), f2_hi(c22[q]));
                park_pos[k1 * 32 + lane] = pos;
                s1 = -INFINITY;
              }
              as2[q] = f2_make(s0, s1);
            }
          }
        };
        const bool all_rows = ee.z <= fy_first && fy_last <= ee.w;
        if (__float_as_uint(ef.x)) {
          if (all_rows)
            blend_slots(std::true_type{}, std::true_type{});
          else
            blend_slots(std::true_type{}, std::false_type{});
        } else {
          if (all_rows)
            blend_slots(std::false_type{}, std::true_type{});
          else
            blend_slots(std::false_type{}, std::false_type{});
        }
        if (!live) break;
      }
    }
    hi -= uint32_t(cnt);
    cost += kCostBatch + uint32_t(k_staged) * kCostEntry;
    if (!__any_sync(0xffffffffu, live != 0u)) break;
    __syncwarp();
  }
  // slots still walking at the end walked the whole list (stop position s)
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    if ((live >> (2 * q)) & 1u) {
      park[2 * q * 32 + lane] = make_float4(f2_lo(T2[q]), f2_lo(c02[q]), f2_lo(c12[q]), f2_lo(c22[q]));
      park_pos[2 * q * 32 + lane] = s;
    }
    if ((live >> (2 * q + 1)) & 1u) {
      park[(2 * q + 1) * 32 + lane] = make_float4(f2_hi(T2[q]), f2_hi(c02[q]), f2_hi(c12[q]), f2_hi(c22[q]));
      park_pos[(2 * q + 1) * 32 + lane] = s;
    }
  }
  float l[PPL] = {};
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    if (!((inside >> k) & 1u)) continue;
    const float4 o = park[k * 32 + lane];
    const size_t p = pix_base + size_t(slot_y(k)) * w + slot_x(k);
    out_rgb[3 * p] = o.y;
    out_rgb[3 * p + 1] = o.z;
    out_rgb[3 * p + 2] = o.w;
    if (out_T) out_T[p] = o.x;
    if (out_alpha) out_alpha[p] = 1.f - o.x;
    if (out_last) out_last[p] = park_pos[k * 32 + lane];
    if (target) {
      const float d0 = o.y - target[3 * p], d1 = o.z - target[3 * p + 1], d2 = o.w - target[3 * p + 2];
      grad_pix[3 * p] = 2.f * d0;
      grad_pix[3 * p + 1] = 2.f * d1;
      grad_pix[3 * p + 2] = 2.f * d2;
      l[k] = d0 * d0 + d1 * d1 + d2 * d2;
    }
  }
  if (target) {  // the loss units, each summed in a block's order
    constexpr int ROWS = loss_rows(G::SLAB_ROWS);
    if (SPLIT) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float v = l[2 * q] + l[2 * q + 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) loss(q, v);
      }
    } else {
      constexpr int SLOTS = ROWS / G::ROW_STEP;  // of a unit
#pragma unroll
      for (int u = 0; u < PPL / SLOTS; ++u) {
        // row r and, in a unit of 8, r + 4; then r ^ 2, r ^ 1 and the columns
        float v[4 / G::ROW_STEP];
#pragma unroll
        for (int k = 0; k < 4 / G::ROW_STEP; ++k) {
          v[k] = l[u * SLOTS + k];
          if (ROWS == 8) v[k] += l[u * SLOTS + k + 4 / G::ROW_STEP];
        }
        float sum;
        if (G::ROW_STEP == 1) {
          sum = (v[0] + v[2 % (4 / G::ROW_STEP)]) + (v[1] + v[3 % (4 / G::ROW_STEP)]);
        } else {
          sum = v[0] + v[1];
          sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane % 8 == 0 && lane < TS) loss(u * (TS / 8) + lane / 8, sum);
      }
    }
  }
  return cost;
}

// A task's loss from which on one of its upstream gradients 2 (image - target)
// can be above kBwdLarge.
constexpr float kLargeLoss = 0.25f * kBwdLarge * kBwdLarge;

// ---------------------------------------------------------------------------
// Fused-path forward: persistent, per-warp work stealing, walking each tile's
// entries out of its superblock list.  The first sched[kSchedHeavy] items of
// the order are walked in 8x8 blocks (raster_block.cuh), the others in tasks
// of TaskGeo.  No block count is asked of the compiler: it takes 80 registers
// by itself (6 blocks of 4 warps per SM), and 10% more instructions when told
// to (16 views of 1,048,576 Gaussians 2890 -> 3210 us).  unit_loss: the items'
// loss units, row by row in a tile, those inside the view.
// ---------------------------------------------------------------------------
template <int TS, int PPL, int NT>
__global__ void __launch_bounds__(32 * kRasterWarps) k_raster_fwd(
    const ViewBatch b, uint32_t n, const float4* __restrict__ rec, const uint2* __restrict__ list1,
    const uint32_t* __restrict__ off1, uint32_t nchunk, uint64_t capacity, const uint32_t* __restrict__ order,
    uint32_t* __restrict__ sched, uint32_t* __restrict__ work_counter, float* __restrict__ out_rgb,
    float* __restrict__ out_T, float* __restrict__ out_alpha, uint32_t* __restrict__ out_last,
    const float* __restrict__ target, float* __restrict__ grad_pix, float* __restrict__ unit_loss, uint32_t* __restrict__ item_cost,
    float nz) {
  using G = TaskGeo<TS, PPL, NT>;
  static_assert(sizeof(EntB) >= sizeof(EntP), "the warps' entries of either form share their place");
  __shared__ EntB ent_all[kRasterWarps][32];
  __shared__ float4 park_all[kRasterWarps][G::PPL * 32];
  __shared__ uint32_t park_pos_all[kRasterWarps][G::PPL * 32];
  __shared__ float tab[256];
  load_exp_table(tab);
  EntB* const ent = ent_all[threadIdx.x >> 5];
  float4* const park = park_all[threadIdx.x >> 5];
  uint32_t* const park_pos = park_pos_all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(work_counter, 1u);
    const Task t(b, __shfl_sync(0xffffffffu, i, 0), order, sched, G::SLABS);
    if (t.none) return;
    const ItemGeo ig = item_geo(b, t.item, off1, nchunk, capacity);
    const ViewDev& vd = b.v[ig.v];
    const PackedSrc src{rec + 3 * size_t(ig.v) * n};
    // tiles of the item's tasks (NT > 1: a run of a superblock row, see
    // k_raster_bwd, carried by its leftmost tile)
    uint32_t nx = 1;
    if (NT > 1) {
      nx = min(uint32_t(NT), 1u << vd.sb_log2);
      if (ig.lx % nx) continue;
    }
    // unit u of a tile of the run
    constexpr int ROWS = loss_rows(G::SLAB_ROWS), UNITS = TS * TS / (8 * ROWS);
    auto loss = [&](uint32_t tile, uint32_t u, float l) {
      unit_loss[size_t(t.item + tile) * UNITS + u] = l;
      if (!(l <= kLargeLoss)) sched[kSchedOdd] = 1u;
    };
    uint32_t cost;
    if (t.block) {
      auto block_loss = [&](int k, float l) {
        constexpr uint32_t SIDE = TS / 8;
        if (TS == 8) loss(t.sub, k, l);
        else loss(0, ROWS == 8 ? t.sub : (2 * (t.sub / SIDE) + k) * SIDE + t.sub % SIDE, l);
      };
      BlockPlace p;
      if (!block_place(b, ig, t.sub, nx, &p)) continue;
      const FwdOut out{out_rgb, out_T, out_alpha, out_last, target, grad_pix};
      cost = blend_block<false, ROWS>(SbWords{list1, p.lx, ig.ly, ig.lx, nx}, PackedBlockSrc{src.rec}, ent, park, park_pos, tab, nz,
                                      ig.s, ig.e, p.px0, p.py0, vd.w, vd.w, vd.h, false, vd.pix_base, out, block_loss);
    } else {
      SbWalkSpan walk{list1, ig.lx, ig.ly, nx};
      const int xend = min(vd.w, ig.px0 + int(nx) * TS);
      cost = fwd_slab<G::GX, G::PPL, NT == 2 && G::PPL == 4>(
          walk, src, reinterpret_cast<EntP*>(ent), park, park_pos, tab, nz, ig.s, ig.e, ig.px0,
          ig.py0 + int(t.sub) * G::SLAB_ROWS, vd.w, vd.h, xend, out_rgb, vd.pix_base, out_T, out_alpha, out_last, target,
          grad_pix, [&](int k, float l) {
            constexpr uint32_t PER_SLAB = UNITS / G::SLABS;
            if (TS > 8) loss(0, t.sub * PER_SLAB + k, l);
            else if (ig.px0 + 8 * k < xend) loss(k, t.sub, l);
          });
    }
    // scheduling hint for the backward and the next forward
    if (lane == 0 && cost) atomicMax(&item_cost[t.item], cost);
    __syncwarp();
  }
}

// Drop-in forward (splat_gauss.rs:46-94): AoS inputs and per-tile lists,
// accumulates into pix2rgb; in 8x8 blocks (raster_block.cuh).
template <bool CUDA_STOP>
__global__ void __launch_bounds__(32 * kRasterWarps, 6) k_raster_fwd_aos(
    int w, int h, int ts, int tile_w, uint32_t num_tasks, float* __restrict__ pix2rgb, AosBlockSrc src,
    const uint32_t* __restrict__ tile2idx, const uint32_t* __restrict__ idx2pnt, float* __restrict__ out_T,
    uint32_t* __restrict__ out_last, float nz) {
  __shared__ EntB ent[kRasterWarps][32];
  __shared__ float4 park[kRasterWarps][64];
  __shared__ uint32_t park_pos[kRasterWarps][64];
  __shared__ float tab[256];
  load_exp_table(tab);
  const int warp = threadIdx.x >> 5;
  const uint32_t task = blockIdx.x * kRasterWarps + (threadIdx.x >> 5);
  if (task >= num_tasks) return;
  const uint32_t side = uint32_t(ts) / kBlock, tile = task / (side * side), blk = task % (side * side);
  const int px0 = int(tile % uint32_t(tile_w)) * ts + int(blk % side) * kBlock;
  const int py0 = int(tile / uint32_t(tile_w)) * ts + int(blk / side) * kBlock;
  if (px0 >= w || py0 >= h) return;
  const FwdOut out{pix2rgb, out_T, nullptr, out_last, nullptr, nullptr};
  blend_block<CUDA_STOP, 8>(TileWords{idx2pnt}, src, ent[warp], park[warp], park_pos[warp], tab, nz, tile2idx[tile],
                         tile2idx[tile + 1], px0, py0, w, w, h, true, 0, out, [](int, float) {});
}

// Units of a tile's slab (8x8 tiles: the slabs' slots are the units').
uint32_t loss_units_per_slab(int ts, int ppl) {
  const int slab_rows = ts == 8 ? 4 * ppl : 32 * ppl / ts;
  return uint32_t(ts / 8 * (slab_rows / loss_rows(slab_rows)));
}

// A slab's loss: its units' in order, those outside the view (not written by
// blocks) left out.
__global__ void __launch_bounds__(256) k_slab_loss(const ViewBatch b, const float* __restrict__ unit_loss, int slab_rows,
                                                   float* __restrict__ slab_loss) {
  const uint32_t slabs = uint32_t(b.ts / slab_rows), i = blockIdx.x * 256u + threadIdx.x;
  if (i >= b.num_items * slabs) return;
  const uint32_t item = i / slabs;
  const ViewDev& vd = b.v[view_of_item(b, item)];
  const uint32_t t = item - vd.item_base;
  const int px0 = int(t % uint32_t(vd.tile_w)) * b.ts, py0 = int(t / uint32_t(vd.tile_w)) * b.ts + int(i % slabs) * slab_rows;
  const int rows = loss_rows(slab_rows), cols = b.ts / 8, units = cols * (slab_rows / rows);
  float sum = 0.f;
  for (int k = 0; k < units; ++k)
    if (px0 + 8 * (k % cols) < vd.w && py0 + rows * (k / cols) < vd.h) sum += unit_loss[size_t(i) * units + k];
  slab_loss[i] = sum;
}

template <int TS, int PPL>
static cudaError_t launch_fwd(cudaStream_t st, const ViewBatch& b, const FwdArgs& a) {
  constexpr int NT = TS == 8 ? kFwdGroup8 : 1;
  k_raster_fwd<TS, PPL, NT>
      <<<persistent_grid(k_raster_fwd<TS, PPL, NT>, max_tasks(b, TaskGeo<TS, PPL, NT>::SLABS)), 32 * kRasterWarps, 0,
         st>>>(b, a.n, a.rec, a.list1, a.off1, a.nchunk, a.capacity, a.order, a.sched, a.counter, a.out_rgb, a.out_T,
               a.out_alpha, a.out_last, a.target, a.grad_pix, TS == 8 ? a.slab_loss : a.unit_loss, a.item_cost, -0.f);
  count_launch();
  if (TS > 8 && a.target) {
    constexpr int SLAB_ROWS = TaskGeo<TS, PPL, NT>::SLAB_ROWS;
    const uint32_t slabs = b.num_items * uint32_t(TS / SLAB_ROWS);
    k_slab_loss<<<(slabs + 255) / 256, 256, 0, st>>>(b, a.unit_loss, SLAB_ROWS, a.slab_loss);
    count_launch();
  }
  return cudaGetLastError();
}

cudaError_t raster_fwd(cudaStream_t st, const ViewBatch& b, const FwdArgs& a) {
#define X(T, P) \
  if (b.ts == T && b.ppl == P) return launch_fwd<T, P>(st, b, a);
  DSPLAT_RASTER_CONFIGS(X)
#undef X
  return cudaErrorInvalidValue;
}

cudaError_t raster_fwd_aos(cudaStream_t st, int ts, int w, int h, float* pix2rgb, const float* xyd, const float* conic,
                           const float* aabb, const float* opacity, const float* rgb, const uint32_t* tile2idx,
                           const uint32_t* idx2pnt, float* out_T, uint32_t* out_last, bool cuda_stop) {
  if (w <= 0 || h <= 0) return cudaSuccess;
  const AosBlockSrc src{xyd, conic, aabb, opacity, rgb};
  const uint32_t side = uint32_t(ts) / kBlock;
  const int tw = (w + ts - 1) / ts, th = (h + ts - 1) / ts;
  const uint32_t tasks = uint32_t(tw) * uint32_t(th) * side * side;
  const unsigned grid = (tasks + kRasterWarps - 1) / kRasterWarps;
  if (cuda_stop)
    k_raster_fwd_aos<true><<<grid, 32 * kRasterWarps, 0, st>>>(w, h, ts, tw, tasks, pix2rgb, src, tile2idx, idx2pnt,
                                                               out_T, out_last, -0.f);
  else
    k_raster_fwd_aos<false><<<grid, 32 * kRasterWarps, 0, st>>>(w, h, ts, tw, tasks, pix2rgb, src, tile2idx, idx2pnt,
                                                                out_T, out_last, -0.f);
  count_launch();
  return cudaGetLastError();
}

// expf_cr elementwise (exposed so that it can be checked against a
// correctly rounded reference on every float).
__global__ void k_expf_cr(size_t n, const float* __restrict__ x, float* __restrict__ y) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) y[i] = expf_cr(x[i]);
}

cudaError_t expf_cr_launch(cudaStream_t st, size_t n, const float* x, float* y) {
  if (n == 0) return cudaSuccess;
  k_expf_cr<<<unsigned((n + 255) / 256), 256, 0, st>>>(n, x, y);
  count_launch();
  return cudaGetLastError();
}

}  // namespace dsplat
