// raster_block.cuh -- the forward's walk of an 8x8-pixel block (raster_fwd.cu,
// which also has the rule for its use and the blend's arithmetic rules).
//
// Bound: the walk's length.  A tile of a scene's rim, whose pixels never
// saturate, walks ten times the mean list, and a warp alone on its scheduler
// issues an instruction every four to five cycles, so a batch that does not
// fill the GPU many times over takes as long as its longest tasks.  A block
// has a pair of pixels per lane: half the instructions per entry of the 16x8
// tasks and twice the tasks, for about 15% more instructions in all.
// Measured (us, every task 16x8 -> every task a block): 3,000 Gaussians at
// 96x80 in 16x16 tiles 200 -> 80, 262,144 at 1280x720 288 -> 211; the drop-in
// forward (16x16 tiles): 1,000 at 96x64 73 -> 34, 16,384 at 256x256 127 -> 72,
// 1,048,576 at 1920x1080 644 -> 601.  Two entries at a time, so that their
// exponentials overlap, were no faster for the short batches and slower for
// the others.
#pragma once
#include "raster_common.cuh"

namespace dsplat {

// The task: a block of 8x8 pixels, lane L at column L % 8 and rows
// L / 8 and L / 8 + 4 (its two pixel slots), for every tile size.
constexpr int kBlock = 8;

// bits [0, n), n clamped to [0, 32]
__device__ __forceinline__ uint32_t low_bits(int n) { return n <= 0 ? 0u : 0xffffffffu >> (32 - min(n, 32)); }

// First and one past the last pixel i in [0, n) with lo <= i + origin + 0.5
// <= hi, by the same exact comparisons: with f = floor(lo), i + 0.5 >= lo
// from i = f on if lo - f <= 0.5, else from f + 1; i + 0.5 <= hi up to f if
// hi - f >= 0.5, else f - 1.  NaN bounds give an empty range.
__device__ __forceinline__ void pixel_range(float lo, float hi, int origin, int n, int* i0, int* i1) {
  const float fl = floorf(lo), fh = floorf(hi), o = float(origin);
  const float a = (lo - fl <= 0.5f ? fl : fl + 1.f) - o, b = (hi - fh >= 0.5f ? fh : fh - 1.f) - o;
  *i0 = a > 0.f ? int(fminf(a, float(n))) : 0;
  *i1 = b < float(n) ? int(fmaxf(b, -1.f)) + 1 : n;
  if (!(lo <= hi)) *i1 = 0;
}

// The lanes whose pixel of slot 0 and slot 1 lies in a box, one bit each, for
// the block at (px0, py0).
__device__ __forceinline__ uint2 block_masks(float x0, float y0, float x1, float y1, int px0, int py0) {
  int c0, c1, r0, r1;
  pixel_range(x0, x1, px0, kBlock, &c0, &c1);
  pixel_range(y0, y1, py0, kBlock, &r0, &r1);
  const uint32_t cols = (low_bits(c1) & ~low_bits(c0)) * 0x01010101u;  // on every row of a slot
  return make_uint2(cols & low_bits(8 * r1) & ~low_bits(8 * r0),
                    cols & low_bits(8 * r1 - 32) & ~low_bits(8 * r0 - 32));
}

// A staged entry for the forward, whose two pixel slots are evaluated as a
// pair with packed two-wide FP32: every value the pair uses is stored twice,
// so a 64-bit shared load yields the packed operand.  px and A enter through
// the per-lane column term.  112 bytes, a stride of 28 words, keep the staging
// lanes' 16-byte stores free of bank conflicts.
struct EntB {  // conic (A, B, C) staged times -1/2 (see make_entb)
  float4 a;    // py, py, -B, -B
  float4 b;    // -C/2, -C/2, opacity, opacity
  float4 c;    // r, r, g, g
  float4 d;    // b, b, px, -A/2
  float2 tie;  // expf_cr2's tie, twice
  uint32_t pos, pad0;
  uint2 mask;  // block_masks
  uint32_t pad1[6];
};

// Returns whether a colour is infinite or NaN.
__device__ __forceinline__ bool make_entb(EntB* dst, uint32_t pos, uint2 mask, float px, float py, float A, float B,
                                          float C, float op, float r, float g, float b, float x0, float y0, float x1,
                                          float y1) {
  // q = A dx^2 + 2B dx dy + C dy^2 of every pixel centre in the box is
  // bounded in magnitude by the same sum of absolute terms at the box's
  // farthest corner; below 170 (rounding adds far less than the margin to
  // 174) every exponent -q/2 of the entry lies in expf_cr's fast range and
  // the per-pixel range check is skipped.  NaN or infinite terms fail it.
  //
  // The conic is staged times -1/2 (exact), so that the walk forms the
  // exponent -q/2 directly: every product and sum of q scaled by -1/2 is the
  // scaled rounding of the same operation on the unscaled values, except
  // where an operand is subnormal -- and then |q| < 2^-100 and e^(-q/2)
  // rounds to 1 either way.
  const float B2 = fa(B, B);
  const float dxm = fmaxf(fabsf(x0 - px), fabsf(x1 - px)), dym = fmaxf(fabsf(y0 - py), fabsf(y1 - py));
  const float mag = fabsf(A) * dxm * dxm + fabsf(B2) * dxm * dym + fabsf(C) * dym * dym;
  const float hA = fm(A, -0.5f), hB2 = fm(B2, -0.5f), hC = fm(C, -0.5f);
  const float tie = mag < 170.f ? kExpTie : __int_as_float(0x7f800000);
  dst->a = make_float4(py, py, hB2, hB2);
  dst->b = make_float4(hC, hC, op, op);
  dst->c = make_float4(r, r, g, g);
  dst->d = make_float4(b, b, px, hA);
  *reinterpret_cast<float4*>(&dst->tie) = make_float4(tie, tie, __uint_as_float(pos), 0.f);
  dst->mask = mask;
  return !(fabsf(r) < INFINITY && fabsf(g) < INFINITY && fabsf(b) < INFINITY);
}

// Sources of the forward's entries: an entry's box (loaded first, and with
// it whether the entry meets the block at all), then the rest of it.
struct AosBlockSrc {
  const float *xyd, *conic, *aabb, *opacity, *rgb;
  __device__ __forceinline__ uint2 masks(uint32_t g, int px0, int py0) const {
    const size_t i = g;
    return block_masks(aabb[4 * i], aabb[4 * i + 1], aabb[4 * i + 2], aabb[4 * i + 3], px0, py0);
  }
  __device__ __forceinline__ bool stage(EntB* dst, uint32_t g, uint32_t pos, uint2 mask) const {
    const size_t i = g;
    return make_entb(dst, pos, mask, xyd[3 * i], xyd[3 * i + 1], conic[3 * i], conic[3 * i + 1], conic[3 * i + 2], opacity[i],
              rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], aabb[4 * i], aabb[4 * i + 1], aabb[4 * i + 2],
              aabb[4 * i + 3]);
  }
};

struct PackedBlockSrc {
  const float4* rec;
  __device__ __forceinline__ uint2 masks(uint32_t g, int px0, int py0) const {
    const float4 r0 = __ldg(rec + 3 * size_t(g)), r2 = __ldg(rec + 3 * size_t(g) + 2);
    return block_masks(fs(r0.x, r2.y), fs(r0.y, r2.z), fa(r0.x, r2.y), fa(r0.y, r2.z), px0, py0);
  }
  __device__ __forceinline__ bool stage(EntB* dst, uint32_t g, uint32_t pos, uint2 mask) const {
    const float4 r0 = __ldg(rec + 3 * size_t(g));
    const float4 r1 = __ldg(rec + 3 * size_t(g) + 1);
    const float4 r2 = __ldg(rec + 3 * size_t(g) + 2);
    return make_entb(dst, pos, mask, r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, fs(r0.x, r2.y), fs(r0.y, r2.z),
              fa(r0.x, r2.y), fa(r0.y, r2.z));
  }
};

// List words of the two forms of tile lists: load() reads a lane's word ahead
// of time, point() and hit() are its point and whether its entry lies in the
// block's tile, counts() whether a whole task of the item would stage it.
struct TileWords {  // a per-tile list (tile2idx / idx2pnt)
  typedef uint32_t word;
  const uint32_t* idx2pnt;
  __device__ __forceinline__ word load(uint32_t pos) const { return idx2pnt[pos]; }
  static __device__ __forceinline__ uint32_t point(word w) { return w; }
  __device__ __forceinline__ bool hit(word) const { return true; }
  static constexpr bool kMeasured = false;  // nobody asks for the walk's cost
  __device__ __forceinline__ bool counts(word) const { return false; }
};

// A superblock list filtered to the block's tile (lx, ly); the item's tasks
// take the nx tiles from run on.
struct SbWords {
  typedef uint2 word;
  const uint2* list1;
  uint32_t lx, ly, run, nx;
  __device__ __forceinline__ word load(uint32_t pos) const { return list1[pos]; }
  static __device__ __forceinline__ uint32_t point(word w) { return w.x; }
  __device__ __forceinline__ bool meets(word w, uint32_t x, uint32_t n) const {
    const uint32_t lr = w.y;
    return x < ((lr >> 8) & 15u) && x + n > (lr & 15u) && ly >= ((lr >> 4) & 15u) && ly < (lr >> 12);
  }
  __device__ __forceinline__ bool hit(word w) const { return meets(w, lx, 1u); }
  static constexpr bool kMeasured = true;
  __device__ __forceinline__ bool counts(word w) const { return meets(w, run, nx); }
};

// ---------------------------------------------------------------------------
// Forward walk of one 8x8-pixel block by one warp over the list range [s, e),
// from its end.  A lane owns two pixels (four rows apart), evaluated as a
// packed pair.
// CUDA_STOP: the stop test of the reference's CUDA kernel (alpha_sum >=
// 0.999f, its double comparison) instead of del-splat-cpu's (> 0.999f).
// Returns the cost of the walk in a whole task's measure (kCostBatch and
// kCostEntry for what such a task would stage), so that an item's cost, the
// largest of its tasks' or blocks', is the same in either shape and the schedule
// of the same inputs does not swing between the two.
// ---------------------------------------------------------------------------
struct FwdOut {  // where a block's results go
  float* rgb;
  float* T;         // nullable
  float* alpha;     // nullable: 1 - T
  uint32_t* last;   // nullable
  const float* target;  // nullable; with it grad_pix and the loss
  float* grad_pix;
};

// ent, park (T, r, g, b of a stopped pixel) and park_pos (its stop position),
// 32, 64 and 64 of them, are the warp's in shared memory; loss(k, l) takes the
// L2 loss of the block's loss unit k (one, or an upper and a lower half: see
// loss_rows in raster_fwd.cu).
template <bool CUDA_STOP, int LOSS_ROWS, class Walk, class Src, class Loss>
__device__ __forceinline__ uint32_t blend_block(const Walk& walk, const Src& src, EntB* ent_sm, float4* park,
                                              uint32_t* park_pos, const float* tab, float nz,
                                              uint32_t s, uint32_t e, int px0, int py0, int w, int xend, int yend,
                                              bool accumulate, size_t pix_base, const FwdOut& out, const Loss& loss) {
  const int lane = threadIdx.x & 31;
  const uint32_t bit = 1u << lane;
  const int ix = px0 + (lane & 7), iy = py0 + (lane >> 3);
  const float fx = float(ix) + 0.5f;
  const f2 fy2 = f2_make(float(iy) + 0.5f, float(iy + 4) + 0.5f);
  const f2 nz2 = f2_dup(nz);  // (-0, -0), a runtime value (see mul2_rn)
  // live: this lane's bit (as in the entries' masks) while the pixel is in
  // the view and has not stopped, else 0
  const bool in0 = ix < xend && iy < yend, in1 = ix < xend && iy + 4 < yend;
  uint32_t live0 = in0 ? bit : 0u, live1 = in1 ? bit : 0u;
  const size_t p0 = pix_base + size_t(iy) * w + ix, p1 = p0 + 4 * size_t(w);
  f2 T2 = f2_dup(1.f), as2 = f2_dup(0.f), c0 = as2, c1 = as2, c2 = as2;
  if (accumulate) {
    float q[2][3] = {};
    for (int i = 0; i < 3; ++i) {
      if (in0) q[0][i] = out.rgb[3 * p0 + i];
      if (in1) q[1][i] = out.rgb[3 * p1 + i];
    }
    c0 = f2_make(q[0][0], q[1][0]);
    c1 = f2_make(q[0][1], q[1][1]);
    c2 = f2_make(q[0][2], q[1][2]);
  }
  // One entry and one pixel at a time, the same operations: for batches with
  // an infinite or NaN colour, which must not meet the alpha of 0 that the
  // pairs below give to a pixel outside a box.
  auto blend_one = [&](const EntB& ent, int k) {
    float T = k ? f2_hi(T2) : f2_lo(T2), a = k ? f2_hi(as2) : f2_lo(as2);
    float r = k ? f2_hi(c0) : f2_lo(c0), g = k ? f2_hi(c1) : f2_lo(c1), b = k ? f2_hi(c2) : f2_lo(c2);
    const float dx = fs(fx, ent.d.z), dy = fs(k ? f2_hi(fy2) : f2_lo(fy2), ent.a.x);
    const float x = fa(fa(fm(fm(ent.d.w, dx), dx), fm(ent.a.z, fm(dx, dy))), fm(fm(ent.b.x, dy), dy));
    const float al = fm(expf_cr(x), ent.b.z), eo = fm(T, al);
    r = fa(r, fm(ent.c.x, eo));
    g = fa(g, fm(ent.c.z, eo));
    b = fa(b, fm(ent.d.x, eo));
    T = fm(T, fs(1.f, al));
    a = fa(a, eo);
    if (CUDA_STOP ? a >= kAlphaStop : a > kAlphaStop) {
      (k ? live1 : live0) = 0u;
      park[32 * k + lane] = make_float4(T, r, g, b);
      park_pos[32 * k + lane] = ent.pos;
      a = -INFINITY;
    }
    T2 = k ? f2_make(f2_lo(T2), T) : f2_make(T, f2_hi(T2));
    as2 = k ? f2_make(f2_lo(as2), a) : f2_make(a, f2_hi(as2));
    c0 = k ? f2_make(f2_lo(c0), r) : f2_make(r, f2_hi(c0));
    c1 = k ? f2_make(f2_lo(c1), g) : f2_make(g, f2_hi(c1));
    c2 = k ? f2_make(f2_lo(c2), b) : f2_make(b, f2_hi(c2));
  };
  uint32_t hi = e, cost = 0;
  typename Walk::word en{};
  if (hi > s && uint32_t(lane) < hi - s) en = walk.load(hi - 1u - uint32_t(lane));
  while (hi > s) {
    const uint32_t cnt = min(32u, hi - s);
    // stage the batch's entries that hold a pixel of the block, in order
    bool hit = uint32_t(lane) < cnt && walk.hit(en);
    const uint32_t counted =
        Walk::kMeasured ? __ballot_sync(0xffffffffu, uint32_t(lane) < cnt && walk.counts(en)) : 0u;
    const uint32_t g = walk.point(en);
    uint2 mask = make_uint2(0u, 0u);
    if (hit) {
      mask = src.masks(g, px0, py0);
      hit = (mask.x | mask.y) != 0u;
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, hit);
    int staged = __popc(bal);
    bool odd = false;
    if (hit) odd = src.stage(&ent_sm[__popc(bal & (bit - 1u))], g, hi - 1u - uint32_t(lane), mask);
    const bool odd_colour = __any_sync(0xffffffffu, odd);
    hi -= cnt;
    cost += kCostBatch + uint32_t(__popc(counted)) * kCostEntry;
    // the next batch's list words arrive while this batch is blended
    if (hi > s && uint32_t(lane) < hi - s) en = walk.load(hi - 1u - uint32_t(lane));
    __syncwarp();
    if (odd_colour) {
      for (int j = 0; j < staged; ++j) {
        const EntB& ent = ent_sm[j];
        if (ent.mask.x & live0) blend_one(ent, 0);
        if (ent.mask.y & live1) blend_one(ent, 1);
      }
      staged = 0;
    }
    for (int j = 0; j < staged; ++j) {
      const EntB& ent = ent_sm[j];
      // which of the lane's pixels the entry's box holds and that still blend
      const bool a0 = (ent.mask.x & live0) != 0u, a1 = (ent.mask.y & live1) != 0u;
      if (!(a0 || a1)) continue;
      // -q/2 with q = A dx dx + B (dx dy + dy dx) + C dy dy in the
      // reference's order (mat2_sym::mult_vec_from_both_sides), from the
      // conic staged times -1/2; dx is the lane's, so (A dx) dx is formed
      // once per entry, and B (dx dy + dy dx) is (2B)(dx dy) exactly
      const ulonglong2 qa = *reinterpret_cast<const ulonglong2*>(&ent.a);  // (py,py) (2B,2B)
      const ulonglong2 qb = *reinterpret_cast<const ulonglong2*>(&ent.b);  // (C,C) (op,op)
      const ulonglong2 qc = *reinterpret_cast<const ulonglong2*>(&ent.c);  // (r,r) (g,g)
      const float4 d = ent.d;                                              // b, b, px, A
      const float dx = fs(fx, d.z);
      const f2 dx2 = f2_dup(dx), adxdx2 = f2_dup(__fmaf_rn(fm(d.w, dx), dx, nz));
      const f2 dy2 = sub2(fy2, qa.x);
      const f2 x = add2(add2(adxdx2, mul2_rn(qa.y, mul2(dx2, dy2), nz2)), mul2_rn(mul2(qb.x, dy2), dy2, nz2));
      const f2 al = mul2_rn(expf_cr2_want(x, *reinterpret_cast<const f2*>(&ent.tie), a0, a1, tab), qb.y, nz2);
      // a pixel that the box does not hold takes alpha 0: its state is
      // unchanged (a stopped pixel's registers are never read again)
      const f2 e2 = f2_make(a0 ? f2_lo(al) : 0.f, a1 ? f2_hi(al) : 0.f);
      const f2 eo2 = mul2_rn(T2, e2, nz2);
      c0 = add2(c0, mul2_rn(qc.x, eo2, nz2));
      c1 = add2(c1, mul2_rn(qc.y, eo2, nz2));
      c2 = add2(c2, mul2_rn(f2_make(d.x, d.y), eo2, nz2));
      T2 = mul2(T2, sub2(f2_dup(1.f), e2));
      as2 = add2(as2, eo2);
      // a stopped pixel's alpha sum is held at -inf (it stays -inf or NaN,
      // which no test passes), and a live one keeps a sum at or below the
      // threshold until it stops, so one test of the larger sum finds every
      // pixel that stops at this entry
      const float amax = fmaxf(f2_lo(as2), f2_hi(as2));
      if (CUDA_STOP ? amax >= kAlphaStop : amax > kAlphaStop) {  // rare
        float s0 = f2_lo(as2), s1 = f2_hi(as2);
        if (CUDA_STOP ? s0 >= kAlphaStop : s0 > kAlphaStop) {
          live0 = 0u;
          park[lane] = make_float4(f2_lo(T2), f2_lo(c0), f2_lo(c1), f2_lo(c2));
          park_pos[lane] = ent.pos;
          s0 = -INFINITY;
        }
        if (CUDA_STOP ? s1 >= kAlphaStop : s1 > kAlphaStop) {
          live1 = 0u;
          park[32 + lane] = make_float4(f2_hi(T2), f2_hi(c0), f2_hi(c1), f2_hi(c2));
          park_pos[32 + lane] = ent.pos;
          s1 = -INFINITY;
        }
        as2 = f2_make(s0, s1);
      }
    }
    if (!__any_sync(0xffffffffu, (live0 | live1) != 0u)) break;
    __syncwarp();
  }
  // pixels still walking at the end walked the whole list (stop position s)
  if (live0) {
    park[lane] = make_float4(f2_lo(T2), f2_lo(c0), f2_lo(c1), f2_lo(c2));
    park_pos[lane] = s;
  }
  if (live1) {
    park[32 + lane] = make_float4(f2_hi(T2), f2_hi(c0), f2_hi(c1), f2_hi(c2));
    park_pos[32 + lane] = s;
  }
  float l[2] = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!(k ? in1 : in0)) continue;
    const float4 o = park[32 * k + lane];
    const size_t p = k ? p1 : p0;
    out.rgb[3 * p] = o.y;
    out.rgb[3 * p + 1] = o.z;
    out.rgb[3 * p + 2] = o.w;
    if (out.T) out.T[p] = o.x;
    if (out.alpha) out.alpha[p] = 1.f - o.x;
    if (out.last) out.last[p] = park_pos[32 * k + lane];
    if (out.target) {
      const float d0 = o.y - out.target[3 * p], d1 = o.z - out.target[3 * p + 1], d2 = o.w - out.target[3 * p + 2];
      out.grad_pix[3 * p] = 2.f * d0;
      out.grad_pix[3 * p + 1] = 2.f * d1;
      out.grad_pix[3 * p + 2] = 2.f * d2;
      l[k] = d0 * d0 + d1 * d1 + d2 * d2;
    }
  }
  if (out.target) {
    constexpr int units = 8 / LOSS_ROWS;
    if (units == 1) l[0] += l[1];
#pragma unroll
    for (int k = 0; k < units; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) l[k] += __shfl_xor_sync(0xffffffffu, l[k], o);
      if (lane == 0) loss(k, l[k]);
    }
  }
  __syncwarp();
  return cost;
}

}  // namespace dsplat
