// raster.cu -- the backward rasteriser, the circle tile painter and the
// raster configuration queries (see raster_common.cuh; the forward lives in
// raster_fwd.cu).
#include "raster_common.cuh"

namespace dsplat {

// ---------------------------------------------------------------------------
// Fused-path backward.  grad2d[(v*N+g)*3 + k] float4:
//   (d px, d py, d A, d B) (d C, d opacity, d r, d g) (d b, 0, 0, 0)
// exp and 1/(1-alpha) use the hardware approximations: gradients need not
// reproduce the forward bit for bit (the discrete structure -- boxes, stop
// positions -- comes from the forward).
// ---------------------------------------------------------------------------
// Per-entry sums over the warp: the nine per-lane values of an entry go to
// shared memory as nine rows of 32, and every kRedEntries entries the rows
// are summed eight to an entry, one lane each, with 16-byte reads (rows are
// 36 words apart, so the eight lanes of a read phase meet 32 different
// banks).  A transposed shuffle butterfly per entry (14 shuffles with their
// selects, 2 more for the mean, the output arithmetic in one lane group at a
// time) cost about 72 of 240 warp-instructions per entry; with the rows and
// the pixels in packed pairs an entry takes 189 (1,048,576 Gaussians at
// 1920x1080, 8x8 tiles, counted by ncu).  The kernel then waits on its
// dependency chains instead of issue slots (68% busy, was 76%): 16 views of
// 1,048,576 Gaussians 3579 -> 3440 us, 8 at 1920x1080 of 4,194,304 6958 ->
// 6770, one at 1280x720 of 262,144 337 -> 300.  80 registers (6 blocks of 4
// warps per SM) are the best cap: at 72 the spills cost more than the warps
// give (3810), at 96 the warps are missed (3590).
constexpr int kRedEntries = 4;
struct __align__(16) RedBuf {
  float row[kRedEntries][9][36];
};

// base: the view's first record; touched: the marks of those that got a
// gradient.
__device__ __forceinline__ void red_flush(const RedBuf* red, int held, int lane, size_t base,
                                          float4* __restrict__ grad2d, uint8_t* __restrict__ touched) {
  __syncwarp();
  const int slot = lane >> 3, k = lane & 7;
  const ulonglong2* r = reinterpret_cast<const ulonglong2*>(red->row[slot][k]);
  f2 s0 = r[0].x, s1 = r[0].y;
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    const ulonglong2 q = r[i];
    s0 = add2(s0, q.x);
    s1 = add2(s1, q.y);
  }
  s0 = add2(s0, s1);
  const float sum = f2_lo(s0) + f2_hi(s0);
  // the ninth row, a quarter word per lane
  const float4 q8 = *reinterpret_cast<const float4*>(&red->row[slot][8][4 * k]);
  float gb = (q8.x + q8.y) + (q8.z + q8.w);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) gb += __shfl_xor_sync(0xffffffffu, gb, o);
  const float m0 = __shfl_sync(0xffffffffu, sum, lane & 24), m1 = __shfl_sync(0xffffffffu, sum, (lane & 24) | 1);
  const float4 c = *reinterpret_cast<const float4*>(&red->row[slot][0][32]);
  const uint32_t g = __float_as_uint(red->row[slot][1][32]);
  // with the w moments m_i = -op/2 (t moments): d px = -2 (A m0 + B m1),
  // d py = -2 (B m0 + C m1), d A = m2, d B = 2 m3, d C = m4 (raw conic
  // recovered from the staged one)
  const float A = c.x * kInvNegHalfLog2e, B = c.y * (0.5f * kInvNegHalfLog2e), C = c.z * kInvNegHalfLog2e;
  float out = sum;
  if (k == 0) out = -2.f * (A * m0 + B * m1);
  if (k == 1) out = -2.f * (B * m0 + C * m1);
  if (k == 3) out = 2.f * sum;
  if (k < 5) out *= 0.5f * c.w;  // the moments of t become moments of w = dL/dq (c.w = -opacity)
  if (k > 5) out = -out;
  if (slot < held) {
    float* dst = reinterpret_cast<float*>(grad2d) + 12 * (base + g);
    atomicAdd(dst + k, out);
    if (k == 0) {
      atomicAdd(dst + 8, -gb);
      touched[base + g] = 1;
    }
  }
  __syncwarp();
}

// NT > 1 (8x8 tiles): one task covers NT horizontally adjacent tiles of one
// superblock row (fewer where the superblock is narrower), NT x as wide with
// NT x the pixels per lane, so that the per-entry warp reduction serves NT x
// the pixels.  The run's leftmost tile leads the task; the other tiles' tasks
// are empty.  The walk keeps entries whose span meets any of the tiles and
// every pixel still tests the entry's box, which contains the pixel only if
// the entry is in that pixel's own tile list, so each pixel sees exactly its
// tile's entries (and its stop position is a position in the shared
// superblock list).  The forward groups tiles the same way.
// Units of work as in the forward: heavy items in 8x8 blocks, two pixels per
// lane (BlockGeo), the others in tasks of TaskGeo.  The walks of a block are
// half as long per entry, the warp reductions of an entry serve half the
// pixels: every unit a block, 3,000 Gaussians at 96x80 in 16x16 tiles 228 ->
// 108 us, 262,144 at 1280x720 327 -> 233, 16 views of 1,048,576 3440 -> 4180.
struct BlockGeo {
  static constexpr int GX = 8, PPL = 2, ROW_STEP = 4;
};

// One task: 32 lanes over GX columns at (px0, py0), columns below xend.
// A pair's arithmetic runs over both of its pixels, one that the entry does not
// reach with a zero alpha.  That leaves the pixel as it is only while all is
// finite; the CAREFUL form takes every pixel by itself.  It has a launch of its
// own, which does all the work of a batch with something odd in it (kSchedOdd)
// and else returns at once (2 us): beside the plain form in one kernel its
// registers cost the walk 3 to 10%, a look at the values in every task and batch
// 1 to 8%, one at every four entries' sums (walking a task again where they are
// not finite) 2 to 5%.
template <class GEO, bool CAREFUL>
__device__ __forceinline__ void bwd_task(const SbWalkSpan& walk, const PackedSrc& src, Ent* sm, RedBuf* red,
                                         const ViewDev& vd, uint32_t s, uint32_t e, int px0, int py0, int xend,
                                         const float* __restrict__ grad_pix, const float* __restrict__ pix_T,
                                         const uint32_t* __restrict__ pix_last, size_t base,
                                         float4* __restrict__ grad2d, uint8_t* __restrict__ touched) {
  constexpr int PPL = GEO::PPL, NP = PPL / 2;
  static_assert(PPL % 2 == 0, "pixels are evaluated in pairs");
  const int lane = threadIdx.x & 31;
  const int ix = px0 + lane % GEO::GX, iy0 = py0 + lane / GEO::GX;
  const bool col_in = ix < xend;
  const float fx = float(ix) + 0.5f;
  // per pixel pair: T in front of the current entry, nS = -(d . colour
  // behind it), d = dL/dpixel; per pixel the stop position
  f2 Tc[NP], nS[NP], d0[NP], d1[NP], d2[NP], fy2[NP];
  uint32_t last[PPL];
  uint32_t lo_min = e;
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    float t[2] = {1.f, 1.f}, g0[2] = {0.f, 0.f}, g1[2] = {0.f, 0.f}, g2[2] = {0.f, 0.f}, y[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = 2 * q + h, iy = iy0 + k * GEO::ROW_STEP;
      y[h] = float(iy) + 0.5f;
      last[k] = e;  // outside pixels process nothing
      if (col_in && ix < vd.w && iy < vd.h) {
        const size_t p = size_t(vd.pix_base) + size_t(iy) * vd.w + ix;
        t[h] = pix_T[p];
        last[k] = pix_last[p];
        g0[h] = grad_pix[3 * p];
        g1[h] = grad_pix[3 * p + 1];
        g2[h] = grad_pix[3 * p + 2];
        lo_min = min(lo_min, last[k]);
      }
    }
    Tc[q] = f2_make(t[0], t[1]);
    nS[q] = f2_make(0.f, 0.f);
    d0[q] = f2_make(g0[0], g0[1]);
    d1[q] = f2_make(g1[0], g1[1]);
    d2[q] = f2_make(g2[0], g2[1]);
    fy2[q] = f2_make(y[0], y[1]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lo_min = min(lo_min, __shfl_xor_sync(0xffffffffu, lo_min, o));
  const uint32_t lo0 = max(s, lo_min);
  int held = 0;  // entries waiting in red
  uint2 en = lo0 < e ? walk.load(lo0 + uint32_t(lane), uint32_t(lane) < e - lo0) : make_uint2(0u, 0u);
  for (uint32_t lo = lo0; lo < e; lo += 32) {
    const int cnt = int(min(32u, e - lo));
    int k_staged;
    if (GEO::GX == 8) {  // of the tiles' entries those whose box reaches the block's pixel centres
      const float cx = float(px0) + 4.f, cy = float(py0) + 4.f;
      bool hit = lane < cnt && walk.hit(en);
      if (hit) {
        const float4 r0 = __ldg(src.rec + 3 * size_t(en.x)), r2 = __ldg(src.rec + 3 * size_t(en.x) + 2);
        hit = fabsf(r0.x - cx) <= r2.y + 4.f && fabsf(r0.y - cy) <= r2.z + 4.f;
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        Ent* dst = &sm[__popc(bal & ((1u << lane) - 1u))];
        src.stage(dst, en.x);
        dst->set_pos(lo + uint32_t(lane));
      }
      k_staged = __popc(bal);
    } else {
      k_staged = walk.stage(src, sm, en, lo + uint32_t(lane), lane < cnt, lane);
    }
    // the next batch's list words arrive while this batch is processed
    if (lo + 32u < e) en = walk.load(lo + 32u + uint32_t(lane), uint32_t(lane) < e - (lo + 32u));
    __syncwarp();
    for (int j = 0; j < k_staged; ++j) {
      const float4 ed = sm[j].d, ee = sm[j].e;
      const uint32_t pos = __float_as_uint(sm[j].f.x);
      // this lane's sums over its pixels, pair halves apart: t = G dL/dalpha
      // (its sum is dL/dop; w = dL/dq = -op/2 t), t dy, t dy^2, and the
      // negated dL/dcolour
      f2 st = 0, sty = 0, styy = 0, nr = 0, ng = 0, nb = 0;
      bool any = false;
      const float dx = fx - ed.x;
      if (ee.x <= fx && fx <= ee.y) {
        const ulonglong2 qa = *reinterpret_cast<const ulonglong2*>(&sm[j].a);
        const ulonglong2 qb = *reinterpret_cast<const ulonglong2*>(&sm[j].b);
        const ulonglong2 qc = *reinterpret_cast<const ulonglong2*>(&sm[j].c);
        const f2 kadxdx = f2_dup(ed.y * dx * dx), kb2dx = f2_dup(ed.z * dx);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const float fy0 = f2_lo(fy2[q]), fy1 = f2_hi(fy2[q]);
          const bool in0 = pos >= last[2 * q] && ee.z <= fy0 && fy0 <= ee.w;
          const bool in1 = pos >= last[2 * q + 1] && ee.z <= fy1 && fy1 <= ee.w;
          if (!(in0 || in1)) continue;
          any = true;
          const f2 dy = sub2(fy2[q], qa.x);
          const f2 y = fma2(fma2(qa.y, dy, kb2dx), dy, kadxdx);  // k q
          if (CAREFUL) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {  // the same operations, one pixel
              if (!(i ? in1 : in0)) continue;
              auto at = [&](f2 x) { return i ? f2_hi(x) : f2_lo(x); };
              auto put = [&](f2& x, float v) { x = i ? f2_make(f2_lo(x), v) : f2_make(v, f2_hi(x)); };
              const float G = ex2_approx(at(y)), na = G * at(qb.x), iom = rcp_approx(fmaxf(1.f + na, 1e-7f));
              const float T = at(Tc[q]) * iom, nw = na * T, S = at(nS[q]);
              const float drgb = fmaf(at(d2[q]), at(qc.y), fmaf(at(d1[q]), at(qc.x), at(d0[q]) * at(qb.y)));
              const float t = G * fmaf(iom, S, T * drgb), ty = t * at(dy);
              put(Tc[q], T);
              put(nS[q], fmaf(nw, drgb, S));
              put(nr, fmaf(nw, at(d0[q]), at(nr)));
              put(ng, fmaf(nw, at(d1[q]), at(ng)));
              put(nb, fmaf(nw, at(d2[q]), at(nb)));
              put(st, at(st) + t);
              put(sty, at(sty) + ty);
              put(styy, fmaf(ty, at(dy), at(styy)));
            }
            continue;
          }
          // a pixel outside the box or past its stop takes G = 0: alpha 0,
          // 1 / (1 - alpha) = 1, every sum unchanged while all is finite
          const f2 Gv = f2_make(in0 ? ex2_approx(f2_lo(y)) : 0.f, in1 ? ex2_approx(f2_hi(y)) : 0.f);
          const f2 nal = mul2(Gv, qb.x);  // -alpha
          // alpha < 1 is a precondition (opacity < 1); the floor only
          // keeps gradients finite if an input breaks it
          const f2 om = add2(nal, f2_dup(1.f));
          const f2 iom = f2_make(rcp_approx(fmaxf(f2_lo(om), 1e-7f)), rcp_approx(fmaxf(f2_hi(om), 1e-7f)));
          Tc[q] = mul2(Tc[q], iom);
          const f2 nw = mul2(nal, Tc[q]);  // -alpha T
          const f2 drgb = fma2(d2[q], qc.y, fma2(d1[q], qc.x, mul2(d0[q], qb.y)));
          const f2 dLde = fma2(iom, nS[q], mul2(Tc[q], drgb));
          nS[q] = fma2(nw, drgb, nS[q]);
          nr = fma2(nw, d0[q], nr);
          ng = fma2(nw, d1[q], ng);
          nb = fma2(nw, d2[q], nb);
          const f2 t = mul2(Gv, dLde);
          st = add2(st, t);
          const f2 ty = mul2(t, dy);
          sty = add2(sty, ty);
          styy = fma2(ty, dy, styy);
        }
      }
      if (__any_sync(0xffffffffu, any)) {
        const float s_t = f2_lo(st) + f2_hi(st), s_ty = f2_lo(sty) + f2_hi(sty), s_tx = s_t * dx;
        red->row[held][0][lane] = s_tx;
        red->row[held][1][lane] = s_ty;
        red->row[held][2][lane] = s_tx * dx;
        red->row[held][3][lane] = s_ty * dx;
        red->row[held][4][lane] = f2_lo(styy) + f2_hi(styy);
        red->row[held][5][lane] = s_t;
        red->row[held][6][lane] = f2_lo(nr) + f2_hi(nr);
        red->row[held][7][lane] = f2_lo(ng) + f2_hi(ng);
        red->row[held][8][lane] = f2_lo(nb) + f2_hi(nb);
        // what the flush needs of the entry, in the rows' padding (every
        // lane stores the same words)
        *reinterpret_cast<float4*>(&red->row[held][0][32]) = make_float4(ed.y, ed.z, sm[j].a.z, sm[j].b.x);
        red->row[held][1][32] = ed.w;
        if (++held == kRedEntries) {
          red_flush(red, held, lane, base, grad2d, touched);
          held = 0;
        }
      }
    }
    __syncwarp();
  }
  if (held) red_flush(red, held, lane, base, grad2d, touched);
}

template <int TS, int PPL_, int NT, bool CAREFUL>
__global__ void __launch_bounds__(32 * kRasterWarps, NT * PPL_ <= 4 ? 6 : 4) k_raster_bwd(
    const ViewBatch b, uint32_t n, const float4* __restrict__ rec, const uint2* __restrict__ list1,
    const uint32_t* __restrict__ off1, uint32_t nchunk, uint64_t capacity, const uint32_t* __restrict__ order,
    const uint32_t* __restrict__ sched, uint32_t* __restrict__ work_counter, const float* __restrict__ grad_pix,
    const float* __restrict__ pix_T, const uint32_t* __restrict__ pix_last, float4* __restrict__ grad2d,
    uint8_t* __restrict__ touched) {
  using G = TaskGeo<TS, PPL_, NT>;
  if ((sched[kSchedOdd] != 0u) != CAREFUL) return;
  __shared__ Ent sm_all[kRasterWarps][32];
  __shared__ RedBuf red_all[kRasterWarps];
  Ent* sm = sm_all[threadIdx.x >> 5];
  RedBuf* red = &red_all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(work_counter, 1u);
    const Task t(b, __shfl_sync(0xffffffffu, i, 0), order, sched, G::SLABS);
    if (t.none) return;
    const ItemGeo ig = item_geo(b, t.item, off1, nchunk, capacity);
    const ViewDev& vd = b.v[ig.v];
    // tiles of the item's tasks: 1, or 2 when the superblock holds the right
    // neighbour; the run's leftmost tile carries them
    uint32_t nx = 1;
    if (NT > 1) {
      nx = min(uint32_t(NT), 1u << vd.sb_log2);
      if (ig.lx % nx) continue;
    }
    const PackedSrc src{rec + 3 * size_t(ig.v) * n};
    const size_t base = size_t(ig.v) * n;
    if (t.block) {
      BlockPlace p;
      if (!block_place(b, ig, t.sub, nx, &p)) continue;
      bwd_task<BlockGeo, CAREFUL>(SbWalkSpan{list1, p.lx, ig.ly, 1u}, src, sm, red, vd, ig.s, ig.e, p.px0, p.py0, vd.w,
                                  grad_pix, pix_T, pix_last, base, grad2d, touched);
    } else {
      bwd_task<G, CAREFUL>(SbWalkSpan{list1, ig.lx, ig.ly, nx}, src, sm, red, vd, ig.s, ig.e, ig.px0,
                           ig.py0 + int(t.sub) * G::SLAB_ROWS, min(vd.w, ig.px0 + int(nx) * TS), grad_pix, pix_T, pix_last,
                           base, grad2d, touched);
    }
  }
}

// ---------------------------------------------------------------------------
// Circle tile painter (splat_circle.cu:93-132): ascending walk, the last
// covering entry wins; covered iff sqrt(dx^2+dy^2) <= rad.
// ---------------------------------------------------------------------------
template <int TS>
__global__ void __launch_bounds__(TS* TS) k_circle_splat_tiles(int w, int h, int tile_w, float* __restrict__ pix2rgb,
                                                              const float* __restrict__ xyd,
                                                              const float* __restrict__ rad,
                                                              const float* __restrict__ rgb,
                                                              const uint32_t* __restrict__ tile2idx,
                                                              const uint32_t* __restrict__ idx2pnt) {
  constexpr int NT = TS * TS;
  __shared__ float s_x[NT], s_y[NT], s_r[NT];
  __shared__ uint32_t s_g[NT];
  const int tid = threadIdx.x;
  const uint32_t tile = blockIdx.y * uint32_t(tile_w) + blockIdx.x;
  const int ix = int(blockIdx.x) * TS + (tid % TS), iy = int(blockIdx.y) * TS + (tid / TS);
  const bool inside = ix < w && iy < h;
  const float fx = float(ix) + 0.5f, fy = float(iy) + 0.5f;
  const uint32_t s = tile2idx[tile], e = tile2idx[tile + 1];
  int64_t win = -1;
  for (uint32_t lo = s; lo < e; lo += NT) {
    const int cnt = int(min(uint32_t(NT), e - lo));
    if (tid < cnt) {
      const uint32_t g = idx2pnt[lo + uint32_t(tid)];
      s_x[tid] = xyd[3 * size_t(g)];
      s_y[tid] = xyd[3 * size_t(g) + 1];
      s_r[tid] = rad[g];
      s_g[tid] = g;
    }
    __syncthreads();
    for (int j = 0; j < cnt; ++j) {
      const float dx = fs(s_x[j], fx), dy = fs(s_y[j], fy);
      const float dist = sqrtf(fa(fm(dx, dx), fm(dy, dy)));
      if (!(dist > s_r[j])) win = s_g[j];
    }
    __syncthreads();
  }
  if (inside && win >= 0) {
    const size_t pix = size_t(iy) * w + ix;
    pix2rgb[3 * pix] = rgb[3 * size_t(win)];
    pix2rgb[3 * pix + 1] = rgb[3 * size_t(win) + 1];
    pix2rgb[3 * pix + 2] = rgb[3 * size_t(win) + 2];
  }
}

bool raster_config_ok(int ts, int ppl) {
  return (ts == 8 && (ppl == 1 || ppl == 2)) || (ts == 16 && (ppl == 2 || ppl == 4 || ppl == 8)) ||
         (ts == 32 && (ppl == 4 || ppl == 8));
}
int raster_default_ppl(int ts) { return ts == 8 ? 2 : 4; }
uint32_t raster_slabs_per_tile(int ts, int ppl) { return uint32_t(ts * ts / (32 * ppl)); }

template <int TS, int PPL>
static cudaError_t launch_bwd(cudaStream_t st, const ViewBatch& b, const BwdArgs& a) {
  constexpr int NT = TS == 8 ? kBwdGroup8 : 1;
  const int grid = persistent_grid(k_raster_bwd<TS, PPL, NT, false>, max_tasks(b, TaskGeo<TS, PPL, NT>::SLABS));
#define X(CAREFUL)                                                                                                  \
  k_raster_bwd<TS, PPL, NT, CAREFUL><<<grid, 32 * kRasterWarps, 0, st>>>(                                           \
      b, a.n, a.rec, a.list1, a.off1, a.nchunk, a.capacity, a.order, a.sched, a.counter, a.grad_pix, a.pix_T,       \
      a.pix_last, a.grad2d, a.touched);                                                                             \
  count_launch();
  X(false) X(true)
#undef X
  return cudaGetLastError();
}

cudaError_t raster_bwd(cudaStream_t st, const ViewBatch& b, const BwdArgs& a) {
#define X(T, P) \
  if (b.ts == T && b.ppl == P) return launch_bwd<T, P>(st, b, a);
  DSPLAT_RASTER_CONFIGS(X)
#undef X
  return cudaErrorInvalidValue;
}

cudaError_t circle_splat_tiles(cudaStream_t st, int ts, int w, int h, float* pix2rgb, const float* xyd,
                               const float* rad, const float* rgb, const uint32_t* tile2idx, const uint32_t* idx2pnt) {
  const int tw = (w + ts - 1) / ts, th = (h + ts - 1) / ts;
  if (tw == 0 || th == 0) return cudaSuccess;
  switch (ts) {
    case 8:
      k_circle_splat_tiles<8><<<dim3(tw, th), 64, 0, st>>>(w, h, tw, pix2rgb, xyd, rad, rgb, tile2idx, idx2pnt);
      break;
    case 16:
      k_circle_splat_tiles<16><<<dim3(tw, th), 256, 0, st>>>(w, h, tw, pix2rgb, xyd, rad, rgb, tile2idx, idx2pnt);
      break;
    case 32:
      k_circle_splat_tiles<32><<<dim3(tw, th), 1024, 0, st>>>(w, h, tw, pix2rgb, xyd, rad, rgb, tile2idx, idx2pnt);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  count_launch();
  return cudaGetLastError();
}

}  // namespace dsplat
