// Forward / backward / fused tile compositing kernels.
//
// A tile of TS x TS pixels is walked by NW warps (one or more CTAs); each thread
// owns 2 pixels (4 rows apart) of a compact 8x8 warp footprint, so that a
// primitive's square cull is mostly warp-uniform and the warp's texel
// fetches stay close together in the atlas.
//
// Every warp walks the tile's primitive list on its own, without CTA
// barriers: it stages 32 list entries at a time into a warp-private shared
// buffer (lane i loads entry i's 64-byte PrimInfo record, runs the
// warp-footprint cull and the grid tests for it, and stores it behind the
// survivors before it), and composites the survivors, in list order in the
// forward walk and in reverse order in the backward walk.  Per entry a thread
// first computes the texel coordinates of all its pixels and issues their
// texel loads (addresses of pixels without a fragment are redirected to texel
// 0 of the template, so every load is in bounds), then composites them
// branch-free.  A warp stops when all its pixels are below t_stop; the
// backward walk of a warp starts at its own last contributor and adds its
// warp-reduced per-primitive sums straight into the FP64 accumulator.  A
// thread's two pixels go through the arithmetic as one float2 of packed FP32x2
// instructions, and the forward walk issues the texel loads of two entries
// before compositing either.
#include "dbmp_internal.cuh"

namespace dbmp {

constexpr int kChunk = 32;   // list entries staged per warp at a time (one per lane)
constexpr unsigned kFull = 0xffffffffu;

// A warp footprint reaches 3.5 pixels from its centre (cx, cy); the cull tests
// of whole footprints take 1 px more for rounding.
constexpr float kReach = 4.5f;

// Conservative warp-uniform rejection: true when the primitive's cull square
// misses every pixel of the warp footprint (1 px margin for rounding; NaN
// never rejects, matching the reference's cull).
__device__ __forceinline__ bool footprint_miss(const float4& g0, float cx, float cy) {
  return (g0.x - g0.z > cx + kReach) || (g0.x + g0.z < cx - kReach) || (g0.y - g0.w > cy + kReach) ||
         (g0.y + g0.w < cy - kReach);
}

// Warp-uniform: true when every pixel of the warp footprint passes the
// primitive's square cull with a 1 px margin, so the per-pixel cull can be
// skipped (false for NaN geometry, which then takes the per-pixel path).
__device__ __forceinline__ bool footprint_inside(const float4& g0, float cx, float cy) {
  return (g0.x - g0.z <= cx - kReach) && (g0.x + g0.z >= cx + kReach) && (g0.y - g0.w <= cy - kReach) &&
         (g0.y + g0.w >= cy + kReach);
}

// Grid cell (within the template's cells) of the warp footprint's centre
// (cx, cy): its texel coordinate clamped into the template, which only
// shortens distances to the template's texels.  The cell's clearance compared
// with the primitive's requirement gext tells, warp-uniformly, that no pixel
// of the footprint can get a fragment (clearance grid), or that every pixel's
// mask is exactly 1 (solid grid, for a footprint whose texel box lies inside
// the template).
__device__ __forceinline__ int grid_cell(const Geom& g, const float4& g0, const float4& g1, float cx, float cy) {
  const float dx = cx - g0.x, dy = cy - g0.y;
  const float tx = fminf(fmaxf(fmaf(g1.x, dx, fmaf(g1.y, dy, g.hx)), 0.f), g.wm1);
  const float ty = fminf(fmaxf(fmaf(g1.z, dx, fmaf(g1.w, dy, g.hy)), 0.f), g.hm1);
  float unused;
  const int ix = floor_small(tx, &unused) >> g.gsx;
  const int iy = floor_small(ty, &unused) >> g.gsy;
  return iy * g.gGx + ix;
}

// Texel coordinates of one pixel.
struct Coord {
  float tx, ty;
  bool ok;    // pixel live, inside the cull square and inside [0,W-1]x[0,H-1]
};

// Texel coordinates of a thread's two pixels for an entry, and whether each
// can yield a fragment (live, inside the cull square, inside
// [0,W-1]x[0,H-1]).  The second pixel's come from the first's, since the inverse
// affine is linear (32-pixel tiles), or from its own offset (16-pixel tiles).
// FAST: the warp footprint lies inside the cull square and its texel-space
// box inside the template (with margin), so every pixel passes both tests.
template <class L, bool FAST>
__device__ __forceinline__ void entry_coords(const Geom& g, const float4& g0, const float4& g1, bool inside,
                                             const float (&pxf)[2], const float (&pyf)[2], const bool (&live)[2],
                                             Coord (&s)[2]) {
  const float dx0 = pxf[0] - g0.x, dy0 = pyf[0] - g0.y;
  const float tx0 = fmaf(g1.x, dx0, fmaf(g1.y, dy0, g.hx));
  const float ty0 = fmaf(g1.z, dx0, fmaf(g1.w, dy0, g.hy));
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float tx = tx0, ty = ty0;
    if (p == 1) {
      if (L::kDirect) {
        const float dy = pyf[1] - g0.y;
        tx = fmaf(g1.x, dx0, fmaf(g1.y, dy, g.hx));
        ty = fmaf(g1.z, dx0, fmaf(g1.w, dy, g.hy));
      } else {
        tx = fmaf((float)L::kStep, g1.y, tx);
        ty = fmaf((float)L::kStep, g1.w, ty);
      }
    }
    if (FAST) {
      s[p].ok = live[p];
    } else {
      bool cull_ok = inside;
      if (!inside) cull_ok = !(fabsf(pxf[p] - g0.x) > g0.z || fabsf(pyf[p] - g0.y) > g0.w);
      const bool in_rng = tx >= 0.f && tx <= g.wm1 && ty >= 0.f && ty <= g.hm1;
      s[p].ok = live[p] && cull_ok && in_rng;
    }
    s[p].tx = tx;
    s[p].ty = ty;
  }
}

// ---------------------------------------------------------------------------
// Pixel pairs.  With 2 pixels per thread the per-entry arithmetic of both
// pixels runs as one float2 (x: pixel 0, y: pixel 1) through the packed FP32x2
// instructions of sm_100, one instruction for both pixels.  Each packed
// operation rounds exactly like its scalar counterpart; constant operands come
// as pairs from the kernel parameters (Geom) or the staged record.  Packed
// operations issue to the FMA-heavy pipe only, while scalar FP32 operations
// may also use the FMA-lite pipe, so some steps stay scalar to keep both pipes
// busy (measured on B200: the forward's blend and colour accumulation, the
// backward's colour and per-primitive product terms).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
// b - a, as the exact FMA a * -1 + b
__device__ __forceinline__ float2 sub2(const Geom& g, float2 b, float2 a) { return __ffma2_rn(a, g.m1, b); }

// Texel coordinates, sampling weights and neighbours of a thread's two pixels.
struct PairSample {
  float2 tx, ty;             // texel coordinates (not redirected)
  float2 wx, wy;             // bilinear weights of the fetched texel
  float2 v00, d01, v10, d11;  // neighbours in difference form (Quad)
  bool ok0, ok1;             // pixel can yield a fragment (as Coord::ok)
};

// A pixel pair's sample with its texel loads issued but not yet consumed.
template <int KIND>
struct PairPre {
  float2 wx, wy;
  typename AtlasFetch<KIND>::Raw r0, r1;   // the two pixels' records as loaded
  bool ok0, ok1;
  float2 tx, ty;                           // texel coordinates (colour-map walks only)
};

// Coordinates, weights and texel loads of both pixels for one entry; tx, ty
// (optional) receive the texel coordinates.
template <class L, int KIND, bool FAST>
__device__ __forceinline__ void pair_prep(const Geom& g, const void* __restrict__ atlas, int toff,
                                          const float4& g0, const float4& g1, bool inside, const float (&pxf)[2],
                                          const float (&pyf)[2], const bool (&live)[2], PairPre<KIND>& s,
                                          float2* ptx = nullptr, float2* pty = nullptr) {
  Coord c[2];
  entry_coords<L, FAST>(g, g0, g1, inside, pxf, pyf, live, c);
  s.ok0 = c[0].ok;
  s.ok1 = c[1].ok;
  if (ptx) {
    *ptx = make_float2(c[0].tx, c[1].tx);
    *pty = make_float2(c[0].ty, c[1].ty);
  }
  // pixels without a fragment sample texel 0 of the template (in bounds)
  const float2 tx = make_float2((FAST || c[0].ok) ? c[0].tx : 0.f, (FAST || c[1].ok) ? c[1].tx : 0.f);
  const float2 ty = make_float2((FAST || c[0].ok) ? c[0].ty : 0.f, (FAST || c[1].ok) ? c[1].ty : 0.f);
  // floor as in floor_small: adding 2^23 rounding toward zero
  const float2 bx = __fadd2_rz(tx, g.k23), by = __fadd2_rz(ty, g.k23);
  const float2 fx = fma2(g.m1, g.k23, bx), fy = fma2(g.m1, g.k23, by);
  s.wx = sub2(g, tx, fx);
  s.wy = sub2(g, ty, fy);
  if constexpr (KIND == ATLAS_F32) {
    const int x0 = __float_as_int(bx.x) - 0x4B000000, y0 = __float_as_int(by.x) - 0x4B000000;
    const int x1 = __float_as_int(bx.y) - 0x4B000000, y1 = __float_as_int(by.y) - 0x4B000000;
    s.r0 = AtlasFetch<KIND>::get_raw(atlas, toff, g.Ht, g.Wt, x0, y0);
    s.r1 = AtlasFetch<KIND>::get_raw(atlas, toff, g.Ht, g.Wt, x1, y1);
  } else {
    // record index toff + y0 Wt + x0 straight from the biased bit patterns
    // (2^23 + x0, 2^23 + y0): the bias is one constant per entry, and the
    // unsigned arithmetic wraps back to the in-range index
    const unsigned c = (unsigned)toff - g.kbias;
    s.r0 = AtlasFetch<KIND>::load(atlas, __float_as_uint(by.x) * (unsigned)g.Wt + __float_as_uint(bx.x) + c, g.Wt);
    s.r1 = AtlasFetch<KIND>::load(atlas, __float_as_uint(by.y) * (unsigned)g.Wt + __float_as_uint(bx.y) + c, g.Wt);
  }
}

// Consumes the loads of pair_prep: weights and neighbours as pairs (the
// neighbours in difference form); tx, ty are not set.
template <int KIND>
__device__ __forceinline__ void pair_unpack(const Geom& g, const PairPre<KIND>& p, PairSample& s) {
  s.wx = p.wx;
  s.wy = p.wy;
  s.ok0 = p.ok0;
  s.ok1 = p.ok1;
  if constexpr (KIND == ATLAS_F32) {
    // reference layout: both pixels' differences as packed subtractions
    s.v00 = make_float2(p.r0.x, p.r1.x);
    s.v10 = make_float2(p.r0.z, p.r1.z);
    s.d01 = sub2(g, make_float2(p.r0.y, p.r1.y), s.v00);
    s.d11 = sub2(g, make_float2(p.r0.w, p.r1.w), s.v10);
  } else {
    const Quad q0 = AtlasFetch<KIND>::unpack(p.r0), q1 = AtlasFetch<KIND>::unpack(p.r1);
    s.v00 = make_float2(q0.v00, q1.v00);
    s.d01 = make_float2(q0.d01, q1.d01);
    s.v10 = make_float2(q0.v10, q1.v10);
    s.d11 = make_float2(q0.d11, q1.d11);
  }
}

// Both phases for one entry, with the texel coordinates.
template <class L, int KIND, bool FAST>
__device__ __forceinline__ void pair_sample(const Geom& g, const void* __restrict__ atlas, int toff,
                                            const float4& g0, const float4& g1, bool inside, const float (&pxf)[2],
                                            const float (&pyf)[2], const bool (&live)[2], PairSample& s) {
  PairPre<KIND> p;
  pair_prep<L, KIND, FAST>(g, atlas, toff, g0, g1, inside, pxf, pyf, live, p, &s.tx, &s.ty);
  pair_unpack<KIND>(g, p, s);
}

// Bilinear mask of both pixels and, with GRAD, its texel-space gradient.
// PACKED: as FP32x2 instructions; otherwise as scalar ones (same roundings).
// The reference clamps the mask to [0,1] (tile_forward.cu:271, NaN -> 1); only
// the upper clamp is applied here, since every caller discards masks failing
// the fragment test mask > 1e-6, which the lower clamp cannot change.
template <bool GRAD, bool PACKED = true>
__device__ __forceinline__ float2 pair_blend(const Geom& g, const PairSample& s, float2* gx, float2* gy) {
  if (!PACKED) {
    const float top0 = fmaf(s.wx.x, s.d01.x, s.v00.x), top1 = fmaf(s.wx.y, s.d01.y, s.v00.y);
    const float bot0 = fmaf(s.wx.x, s.d11.x, s.v10.x), bot1 = fmaf(s.wx.y, s.d11.y, s.v10.y);
    const float d0 = bot0 - top0, d1 = bot1 - top1;
    if (GRAD) {
      *gx = make_float2(fmaf(s.wy.x, s.d11.x - s.d01.x, s.d01.x), fmaf(s.wy.y, s.d11.y - s.d01.y, s.d01.y));
      *gy = make_float2(d0, d1);
    }
    return make_float2(fminf(1.f, fmaf(s.wy.x, d0, top0)), fminf(1.f, fmaf(s.wy.y, d1, top1)));
  }
  const float2 dt = s.d01, db = s.d11;
  const float2 top = fma2(s.wx, dt, s.v00);
  const float2 bot = fma2(s.wx, db, s.v10);
  const float2 d = sub2(g, bot, top);
  const float2 m = fma2(s.wy, d, top);
  if (GRAD) {
    *gx = fma2(s.wy, sub2(g, db, dt), dt);
    *gy = d;
  }
  return make_float2(fminf(1.f, m.x), fminf(1.f, m.y));
}

// Colour-map sample (tile_forward.cu:17-89): the texel coordinate is clamped
// into the map, neighbours past the last row / column repeat it, bilinear in
// the reference's operation order.  cm: the primitive's (Ht,Wt,3) map.
__device__ __forceinline__ float3 sample_cmap(const float* __restrict__ cm, int Ht, int Wt, float tx, float ty) {
  const float cx = fmaxf(0.f, fminf((float)(Wt - 1), tx));
  const float cy = fmaxf(0.f, fminf((float)(Ht - 1), ty));
  const int x0 = (int)cx, y0 = (int)cy;
  const int x1 = min(x0 + 1, Wt - 1), y1 = min(y0 + 1, Ht - 1);
  const float fx = cx - (float)x0, fy = cy - (float)y0;
  const float* p00 = cm + 3 * (y0 * Wt + x0);
  const float* p10 = cm + 3 * (y0 * Wt + x1);
  const float* p01 = cm + 3 * (y1 * Wt + x0);
  const float* p11 = cm + 3 * (y1 * Wt + x1);
  float r[3];
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float c0 = fmaf(__ldg(p00 + ch), 1.f - fx, __ldg(p10 + ch) * fx);
    const float c1 = fmaf(__ldg(p01 + ch), 1.f - fx, __ldg(p11 + ch) * fx);
    r[ch] = fmaf(c0, 1.f - fy, c1 * fy);
  }
  return make_float3(r[0], r[1], r[2]);
}

// ---------------------------------------------------------------------------
// A staged chunk: its n surviving entries sit at w[0..n-1] in list order; bit j
// of each mask belongs to entry w[j].
struct Chunk {
  int n;             // entries the warp composites
  unsigned todo;     // which of the chunk's 32 entries they are
  unsigned inside;   // footprint entirely inside the entry's cull square
  unsigned fast;     // ... and its texel-space box inside the template
  unsigned solid;    // ... and its mask exactly 1 everywhere (solid grid)
  unsigned clear;    // clearance grid shows no fragment (counting walk only: skipped otherwise)
  unsigned miss;     // list entries whose cull square the footprint misses (counting walk only)
};
constexpr unsigned kInside = 1u, kFast = 2u, kSolid = 4u, kClear = 8u;

// What a forward walk leaves for the backward walk of the same warp: the masks of
// its first kKeptChunks chunks (of a chunk's 32 entries: which survived; of the
// survivors: inside, fast, solid), so that the backward walk stages them without
// the tests.  The fused kernel keeps them in shared memory, with which chunk's
// records the buffer holds (2048x2048, N=20000, FP16 quads, where a walk stages 2.5
// chunks: 492 -> 466 us); a forward call can leave them in global memory for the
// backward call (2048x2048, N=20000, FP16 quads: backward call 339 -> 332 us;
// 1024x1024, N=5000, FP32: 163 -> 156; 4096x4096, N=100000: 2058 -> 2041).
constexpr int kKeptChunks = DBMP_KEPT_CHUNKS;
struct Kept {
  uint4 masks[kKeptChunks];
  int in_buffer;   // index of the last staged chunk (-1: none)
};

// Staged record: [0] (mx, my, hw, hh)  [1] A  [2] (op, r, g, b)
// [3] (toff, flags, position in the tile's list, primitive id).
using Rec = float4[4];

// a / b for 2^-126 <= b <= 1, as a times the approximate reciprocal.
__device__ __forceinline__ float div_unit(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return a * r;
}

// CB: fragment colours blend a per-primitive colour map (cmap, (N,Ht,Wt,3))
// with weight cblend, (1 - cblend) sigmoid(c) + cblend c_o (tile_forward.cu:316-330).
template <int TS, int KIND, bool CB = false>
struct TileWalker {
  static constexpr int NP = 2;      // pixels of a thread
  using L = Layout<TS>;
  // sets of per-primitive sums of a lane: one over both pixels (32-pixel tiles, FP32
  // sums over a footprint's 64 pixels), or one for each (16-pixel tiles, over 32)
  static constexpr int kSumPx = TS == 16 ? 2 : 1;
  static constexpr bool kGrid = KIND != ATLAS_F32;   // packed atlases carry a clearance grid
  static constexpr bool kQuad = KIND == ATLAS_F32_QUAD || KIND == ATLAS_F16_QUAD || KIND == ATLAS_BF16_QUAD;

  int warp, lw, lane, start, end;   // warp: index within the tile, lw: within the CTA
  const float* cmap = nullptr;
  float cblend = 0.f;
  float pxf[NP], pyf[NP];
  bool valid[NP];
  float fcx, fcy;   // centre of the warp footprint

  // Colours of the pixel pair for an entry (g2.yzw = sigmoid(c)); with CB, the
  // map is sampled at the texel coordinates of the pixels with a fragment.  The
  // roundings of the map's arithmetic are written out (here, in sample_cmap and in
  // the backward's sums): left to the compiler they moved with the code around it.
  __device__ __forceinline__ void pair_colour(const Geom& g, const float4& g2, int id, float2 tx, float2 ty, bool f0,
                                              bool f1, float2& r, float2& gr, float2& b) const {
    r = make_float2(g2.y, g2.y);
    gr = make_float2(g2.z, g2.z);
    b = make_float2(g2.w, g2.w);
    if constexpr (CB) {
      const float* cm = cmap + (size_t)id * g.Ht * g.Wt * 3;
      const float k = 1.f - cblend;
      auto mix = [&](float c, float co) {   // (16- and 32-pixel tiles differ in which product is rounded)
        return L::kDirect ? fmaf(k, c, cblend * co) : fmaf(cblend, co, k * c);
      };
      if (f0) {
        const float3 co = sample_cmap(cm, g.Ht, g.Wt, tx.x, ty.x);
        r.x = mix(g2.y, co.x);
        gr.x = mix(g2.z, co.y);
        b.x = mix(g2.w, co.z);
      }
      if (f1) {
        const float3 co = sample_cmap(cm, g.Ht, g.Wt, tx.y, ty.y);
        r.y = mix(g2.y, co.x);
        gr.y = mix(g2.z, co.y);
        b.y = mix(g2.w, co.z);
      }
    }
  }

  // tile: the CTA's tile; part: which group of warps of the tile the CTA runs
  // (a CTA holds cta_warps of the tile's NW warps).
  __device__ __forceinline__ void init(const Geom& g, int tile, int part, int cta_warps,
                                       const int* __restrict__ offs) {
    lw = threadIdx.x >> 5;
    warp = part * cta_warps + lw;
    lane = threadIdx.x & 31;
    const int tx = tile % g.tilesX, ty = tile / g.tilesX;
    start = __ldg(offs + tile);
    end = __ldg(offs + tile + 1);
    const int bx = px(tile, g), by = py(tile, g, 0);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      pxf[p] = (float)bx;
      pyf[p] = (float)(by + p * L::kStep);
      valid[p] = bx < g.W && by + p * L::kStep < g.H;
    }
    fcx = (float)(tx * TS + (warp % L::WPR) * L::FW) + 0.5f * (float)(L::FW - 1);
    fcy = (float)(ty * TS + (warp / L::WPR) * L::FH) + 0.5f * (float)(L::FH - 1);
  }

  // Pixel coordinates of pixel p of this thread.
  __device__ __forceinline__ int px(int tile, const Geom& g) const {
    return (tile % g.tilesX) * TS + (warp % L::WPR) * L::FW + (lane & 7);
  }
  __device__ __forceinline__ int py(int tile, const Geom& g, int p) const {
    return (tile / g.tilesX) * TS + (warp / L::WPR) * L::FH + (lane >> 3) + p * L::kStep;
  }

  // Stages list positions [base, min(base + 32, stop)) into the warp's buffer
  // w: lane i tests position base + i, and the survivors' records go to
  // w[0..n-1].  With KEEP_CLEAR, entries the clearance grid rules out stay (the
  // counting walk checks them).  Out-of-range primitive ids never yield a
  // fragment (tile_forward.cu:184-185).  Compacted records let the walks step
  // through the buffer by constant offsets instead of searching a bit mask
  // for each entry, and carry the entry's position and id (2048x2048, N=20000,
  // FP16 quads: backward walk 319 -> 288 M instructions, 365 -> 348 us, fused
  // kernel 551 -> 535).  The tests load a record's parts as they need them, and
  // the survivors' loads are repeated after the ballot: holding the record, or
  // the next chunk's ids, in registers spills the walk's state (fused 565 us).
  template <bool KEEP_CLEAR>
  __device__ __forceinline__ Chunk stage(const Geom& g, const PrimInfo* __restrict__ prims,
                                         const int* __restrict__ idx, const unsigned char* __restrict__ grid,
                                         int base, int stop, Rec* w) const {
    bool keep = false, miss = false;
    unsigned flags = 0u;
    int id = -1, toff = kNoFrag;
    const int pos = base + lane;
    if (pos < stop) {
      id = __ldg(idx + pos);
      if (id >= 0 && id < g.N) {
        const float4* r = reinterpret_cast<const float4*>(prims + id);
        const float4 g0 = __ldg(r);
        miss = footprint_miss(g0, fcx, fcy);
        if (!miss) {
          const float4 q = __ldg(r + 3);
          toff = __float_as_int(q.x);
          if (toff != kNoFrag) {
            const float4 g1 = __ldg(r + 1);
            bool clear = false, solid = false;
            if (kGrid) {
              const unsigned char* cell = grid + __float_as_int(q.y) + grid_cell(g, g0, g1, fcx, fcy);
              const int need = __float_as_int(q.z);
              clear = (int)__ldg(cell) >= need;
              if (g.solid_delta != 0) solid = (int)__ldg(cell + g.solid_delta) >= need;
            }
            keep = KEEP_CLEAR || !clear;
            if (keep) {
              if (footprint_inside(g0, fcx, fcy)) {
                // texel box of the footprint: centre +- |A| (half extents), plus
                // 0.05 texel for the rounding of the per-pixel coordinates
                const float dx = fcx - g0.x, dy = fcy - g0.y;
                const float cx = fmaf(g1.x, dx, fmaf(g1.y, dy, g.hx));
                const float cy = fmaf(g1.z, dx, fmaf(g1.w, dy, g.hy));
                const float ex = fmaf(fabsf(g1.x), g.fhx, fmaf(fabsf(g1.y), g.fhy, 0.05f));
                const float ey = fmaf(fabsf(g1.z), g.fhx, fmaf(fabsf(g1.w), g.fhy, 0.05f));
                const bool fast = cx - ex >= 0.f && cx + ex <= g.wm1 && cy - ey >= 0.f && cy + ey <= g.hm1;
                flags = kInside | (fast ? kFast | (solid ? kSolid : 0u) : 0u);
              }
              if (KEEP_CLEAR && clear) flags |= kClear;
            }
          }
        }
      }
    }
    const unsigned todo = __ballot_sync(kFull, keep);
    __syncwarp();   // every lane is done with the previous chunk's records
    if (keep) {
      // reads the record again (L1) rather than holding it across the ballot
      const float4* r = reinterpret_cast<const float4*>(prims + id);
      float4* d = w[__popc(todo & ((1u << lane) - 1u))];
      float4 g2 = __ldg(r + 2);
      if (half_record(KIND)) {   // FP16 (alpha0, r) and (g, b) pairs
        const float2 ar = h2f(__float_as_uint(g2.x)), gb = h2f(__float_as_uint(g2.y));
        g2 = make_float4(ar.x, ar.y, gb.x, gb.y);
      }
      d[0] = __ldg(r);
      d[1] = __ldg(r + 1);
      d[2] = g2;
      d[3] = make_float4(__int_as_float(toff), __uint_as_float(flags), __int_as_float(pos - start),
                         __int_as_float(id));
    }
    __syncwarp();   // the records are visible to every lane
    Chunk c;
    c.n = __popc(todo);
    c.todo = todo;
    const unsigned f = lane < c.n ? __float_as_uint(w[lane][3].y) : 0u;
    c.inside = __ballot_sync(kFull, f & kInside);
    c.fast = __ballot_sync(kFull, f & kFast);
    c.solid = __ballot_sync(kFull, f & kSolid);
    c.clear = KEEP_CLEAR ? __ballot_sync(kFull, f & kClear) : 0u;
    c.miss = KEEP_CLEAR ? __ballot_sync(kFull, miss) : 0u;
    return c;
  }

  // stage() for a chunk whose masks the forward walk kept: only the survivors
  // up to list position `last` (relative to the tile's) are needed, and no test.
  // in_buffer: their records are still in w.
  __device__ __forceinline__ Chunk restage(const PrimInfo* __restrict__ prims, int num_prims,
                                           const int* __restrict__ idx, int base, int last, const uint4& m,
                                           bool in_buffer, Rec* w) const {
    Chunk c;
    c.todo = m.x;
    if (last - base < kChunk - 1) c.todo &= (2u << (last - base)) - 1u;
    c.n = __popc(c.todo);
    c.inside = m.y;
    c.fast = m.z;
    c.solid = m.w;
    if (in_buffer) return c;
    __syncwarp();   // every lane is done with the previous chunk's records
    if ((c.todo >> lane) & 1u) {
      int id = __ldg(idx + start + base + lane);
      if ((unsigned)id >= (unsigned)num_prims) id = 0;   // (never in the forward's own list; keeps the record read in bounds)
      const float4* r = reinterpret_cast<const float4*>(prims + id);
      float4* d = w[__popc(c.todo & ((1u << lane) - 1u))];
      float4 g2 = __ldg(r + 2);
      if (half_record(KIND)) {   // FP16 (alpha0, r) and (g, b) pairs
        const float2 ar = h2f(__float_as_uint(g2.x)), gb = h2f(__float_as_uint(g2.y));
        g2 = make_float4(ar.x, ar.y, gb.x, gb.y);
      }
      d[0] = __ldg(r);
      d[1] = __ldg(r + 1);
      d[2] = g2;
      d[3] = make_float4(__ldg(r + 3).x, 0.f, __int_as_float(base + lane), __int_as_float(id));
    }
    __syncwarp();   // the records are visible to every lane
    return c;
  }

  // Sums of acc[0..K-1] (one set per lane) over the warp by recursive halving: 8 sums
  // over 32 lanes in 9 shuffles, 16 in 16.  Lane l returns the sum whose index has
  // the bits of l reversed (in log2 K bits); the lanes beyond K repeat the first K.
  template <int K>
  __device__ __forceinline__ float warp_sums(float (&acc)[K]) const {
    int bit = 1;
#pragma unroll
    for (int n = K / 2; n >= 1; n >>= 1, bit <<= 1) {
      const bool b = lane & bit;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        const float send = b ? acc[k] : acc[k + n];
        const float keep = b ? acc[k + n] : acc[k];
        acc[k] = keep + __shfl_xor_sync(kFull, send, bit);
      }
    }
#pragma unroll
    for (; bit < 32; bit <<= 1) acc[0] += __shfl_xor_sync(kFull, acc[0], bit);
    return acc[0];
  }

  // Adds the warp's K per-primitive sums to dst[0..K-1] in FP64.  PX = 1: each lane
  // gives the sums of its two pixels.  PX = 2: it gives pixel 0's and then pixel
  // 1's, and the two halves of the footprint (8x4 pixels each) meet in FP64.
  // Returns the index of the sum that this lane added (-1: none) and its value.
  template <int K, int PX>
  __device__ __forceinline__ int add_sums(float (&acc)[PX * K], double* __restrict__ dst, double* value) const {
    const float sum = warp_sums(acc);
    double d = (double)sum;
    int l = lane;
    if (PX == 2) {
      d += __shfl_xor_sync(kFull, d, 1);
      l = (lane & 1) ? 32 : lane >> 1;   // lane bit 0 told the pixels apart
    }
    *value = d;
    if (l >= K || d == 0.0) return -1;
    const int k = K == 8 ? 4 * (l & 1) + (l & 2) + ((l >> 2) & 1) : 2 * (l & 1) + ((l >> 1) & 1);
    atomicAdd(dst + k, d);
    return k;
  }

  __device__ __forceinline__ void warp_add(float (&acc)[8 * kSumPx], double* __restrict__ dst) const {
    double d;
    add_sums<8, kSumPx>(acc, dst, &d);
  }

  // warp_add for a solid entry: acc holds sums 4..7 (the mask-gradient sums
  // 0..3 are 0), reduced in the same order.  A sum that is not finite (an infinite
  // or NaN gradient or colour) makes 0..3 NaN, as the product of such a term with
  // the zero mask gradient does.
  __device__ __forceinline__ void warp_add4(float (&acc)[4 * kSumPx], double* __restrict__ dst) const {
    double d;
    if (add_sums<4, kSumPx>(acc, dst + 4, &d) == 3 && !(fabs(d) < INFINITY)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) atomicAdd(dst + j, (double)NAN);
    }
  }

  // Phase 1 of a forward entry: coordinates and texel loads of the pixel pair.
  __device__ __forceinline__ void pair_issue(const Geom& g, const void* __restrict__ atlas, const Rec& r, bool inside,
                                             bool fast, const bool (&live)[2], PairPre<KIND>& p) const {
    const int toff = __float_as_int(r[3].x);
    const float4 g0 = r[0];
    const float4 g1 = r[1];
    float2* tx = CB ? &p.tx : nullptr;
    float2* ty = CB ? &p.ty : nullptr;
    if (fast) pair_prep<L, KIND, true>(g, atlas, toff, g0, g1, inside, pxf, pyf, live, p, tx, ty);
    else pair_prep<L, KIND, false>(g, atlas, toff, g0, g1, inside, pxf, pyf, live, p, tx, ty);
  }

  // Forward state of a pixel pair.
  struct PairFwd {
    float2 cr, cg, cb, t, tl;
    int lp0, lp1;
    bool live[2];
  };

  // Composites masks m of a staged entry (fragments f0, f1; CB: texel
  // coordinates tx, ty) onto the pixel pair.  Returns true when every pixel of
  // the warp has stopped (if vote).
  __device__ __forceinline__ bool pair_over(const Geom& g, const Rec& r, float2 m, bool f0, bool f1, float2 tx,
                                            float2 ty, PairFwd& f, bool vote) const {
    const float4 g2 = r[2];
    const int pos = __float_as_int(r[3].z);
    float2 cr, cg, cb;
    pair_colour(g, g2, CB ? __float_as_int(r[3].w) : 0, tx, ty, f0, f1, cr, cg, cb);
    const float2 a = make_float2(f0 ? g2.x * m.x : 0.f, f1 ? g2.x * m.y : 0.f);
    const float2 wt = make_float2(f.t.x * a.x, f.t.y * a.y);
    f.cr = make_float2(fmaf(wt.x, cr.x, f.cr.x), fmaf(wt.y, cr.y, f.cr.y));
    f.cg = make_float2(fmaf(wt.x, cg.x, f.cg.x), fmaf(wt.y, cg.y, f.cg.y));
    f.cb = make_float2(fmaf(wt.x, cb.x, f.cb.x), fmaf(wt.y, cb.y, f.cb.y));
    f.tl.x = f0 ? f.t.x : f.tl.x;
    f.tl.y = f1 ? f.t.y : f.tl.y;
    f.lp0 = f0 ? pos : f.lp0;
    f.lp1 = f1 ? pos : f.lp1;
    // T (1 - a); 0 when a > 1 (alpha_max > 1).  a >= 0 (alpha_max >= 0), so
    // T stays <= 1 and saturating equals max(., 0), NaN included (per pixel:
    // saturation has no packed form).
    f.t.x = __saturatef(fmaf(-f.t.x, a.x, f.t.x));
    f.t.y = __saturatef(fmaf(-f.t.y, a.y, f.t.y));
    f.live[0] = f.live[0] && !(f.t.x < g.t_stop);
    f.live[1] = f.live[1] && !(f.t.y < g.t_stop);
    return vote && __all_sync(kFull, !f.live[0] && !f.live[1]);
  }

  // Phase 2 of a forward entry: blend the loaded texels and composite.
  __device__ __forceinline__ bool pair_composite(const Geom& g, const Rec& r, const PairPre<KIND>& p, PairFwd& f,
                                                 bool vote) const {
    PairSample s;
    pair_unpack<KIND>(g, p, s);
    const float2 m = pair_blend<false, false>(g, s, nullptr, nullptr);
    // a pixel may have stopped since the loads were issued
    const bool f0 = s.ok0 && f.live[0] && m.x > 1e-6f, f1 = s.ok1 && f.live[1] && m.y > 1e-6f;
    return pair_over(g, r, m, f0, f1, p.tx, p.ty, f, vote);
  }

  // Forward walk.  Two sampled entries in a row go together: the texel loads
  // of both are issued before either is composited, so their latencies
  // overlap (a lone one on its own path: issuing a copy of it as the second
  // took 221 against 204 us at 2048x2048, N=20000, FP16 quads; three or four
  // together spill, as do two in the backward walk).  Solid entries (mask 1 on the whole footprint) are composited
  // straight from their record: they need a third of the instructions of a
  // sampled one, and at 2048x2048, N=20000, 256x256 bitmaps with soft rims they
  // are 44 % of the entries (forward walk 244 -> 218 us, backward 432 -> 361,
  // fused kernel 637 -> 548).
  __device__ __forceinline__ void forward(const Geom& g, const PrimInfo* __restrict__ prims,
                                          const void* __restrict__ atlas, const int* __restrict__ idx, Rec* w,
                                          float (&C)[2][3], float (&T)[2], float (&Tl)[2], int (&lp)[2],
                                          uint4* masks, int* in_buffer) const {
    const unsigned char* grid = static_cast<const unsigned char*>(atlas) + g.grid_off;
    PairFwd f;
    f.cr = f.cg = f.cb = make_float2(0.f, 0.f);
    f.t = f.tl = make_float2(1.f, 1.f);
    f.lp0 = f.lp1 = -1;
    f.live[0] = valid[0];
    f.live[1] = valid[1];
    bool warp_done = __all_sync(kFull, !f.live[0] && !f.live[1]);
    for (int base = start; base < end && !warp_done; base += kChunk) {
      const Chunk c = stage<false>(g, prims, idx, grid, base, end, w);
      if (masks && lane == 0) {
        const int k = (base - start) / kChunk;
        if (in_buffer) *in_buffer = k;
        if (k < kKeptChunks) masks[k] = make_uint4(c.todo, c.inside, c.fast, c.solid);
      }
      for (int j = 0; j < c.n;) {
        if ((c.solid >> j) & 1u) {   // every live pixel of the warp has mask 1: nothing to sample
          float2 tx, ty;
          if constexpr (CB) pair_coords(g, w[j], tx, ty);
          if (pair_over(g, w[j], make_float2(1.f, 1.f), f.live[0], f.live[1], tx, ty, f, true)) {
            warp_done = true;
            break;
          }
          ++j;
          continue;
        }
        if (j + 1 < c.n && !((c.solid >> (j + 1)) & 1u)) {
          // one termination vote per pair: a pixel that stops at the first has live
          // false, so the second composites nothing for it
          PairPre<KIND> p1, p2;
          pair_issue(g, atlas, w[j], (c.inside >> j) & 1u, (c.fast >> j) & 1u, f.live, p1);
          pair_issue(g, atlas, w[j + 1], (c.inside >> (j + 1)) & 1u, (c.fast >> (j + 1)) & 1u, f.live, p2);
          pair_composite(g, w[j], p1, f, false);
          if (pair_composite(g, w[j + 1], p2, f, true)) { warp_done = true; break; }
          j += 2;
        } else {
          PairPre<KIND> p1;
          pair_issue(g, atlas, w[j], (c.inside >> j) & 1u, (c.fast >> j) & 1u, f.live, p1);
          if (pair_composite(g, w[j], p1, f, true)) { warp_done = true; break; }
          ++j;
        }
      }
    }
    C[0][0] = f.cr.x; C[0][1] = f.cg.x; C[0][2] = f.cb.x;
    C[1][0] = f.cr.y; C[1][1] = f.cg.y; C[1][2] = f.cb.y;
    T[0] = f.t.x; T[1] = f.t.y;
    Tl[0] = f.tl.x; Tl[1] = f.tl.y;
    lp[0] = f.lp0; lp[1] = f.lp1;
  }

  // Colour and opacity terms of a lane's pixels: their sum, or one set after the other.
  __device__ __forceinline__ void colour_sums(float (&acc)[4 * kSumPx], float2 gcr, float2 gcg, float2 gcb, float2 wt,
                                              float2 dlda, float2 a) const {
    if constexpr (kSumPx == 2) {
      acc[0] = gcr.x * wt.x; acc[1] = gcg.x * wt.x; acc[2] = gcb.x * wt.x; acc[3] = dlda.x * a.x;
      acc[4] = gcr.y * wt.y; acc[5] = gcg.y * wt.y; acc[6] = gcb.y * wt.y; acc[7] = dlda.y * a.y;
    } else {
      acc[0] = fmaf(gcr.y, wt.y, gcr.x * wt.x);
      acc[1] = fmaf(gcg.y, wt.y, gcg.x * wt.x);
      acc[2] = fmaf(gcb.y, wt.y, gcb.x * wt.x);
      acc[3] = fmaf(dlda.y, a.y, dlda.x * a.x);
    }
  }

  // Texel coordinates of the pixel pair alone (solid entries of a colour-map walk).
  __device__ __forceinline__ void pair_coords(const Geom& g, const Rec& r, float2& tx, float2& ty) const {
    const bool live[2] = {true, true};
    Coord s[2];
    entry_coords<L, true>(g, r[0], r[1], true, pxf, pyf, live, s);
    tx = make_float2(s[0].tx, s[1].tx);
    ty = make_float2(s[0].ty, s[1].ty);
  }

  // Reverse walk.  gC/gA: upstream gradients per pixel; Ts: T entering each
  // pixel's last contributor (lp).  H = gC . R and B = prod(1 - a) over the
  // fragments behind the current one, where R is their colour composited from
  // T = 1; both obey X_{k-1} = (1 - a_k) X_k + a_k x_k, so
  // dL/da_k = T_k (gC.c_k - H + gA B).  Per entry the warp reduces its
  // per-primitive partial sums (each lane's two pixels added first) and lanes
  // 0..7 add them to gacc (N,8) f64 (layout documented at finalize_kernel).
  __device__ __forceinline__ void backward(const Geom& g, const PrimInfo* __restrict__ prims,
                                           const void* __restrict__ atlas, const int* __restrict__ idx, Rec* w,
                                           const float (&gC)[2][3], const float (&gA)[2], const float (&Ts)[2],
                                           const int (&lp)[2], double* __restrict__ gacc,
                                           const Kept* kept) const {
    const int warp_max = __reduce_max_sync(kFull, max(lp[0], lp[1]));
    if (warp_max < 0) return;
    const unsigned char* grid = static_cast<const unsigned char*>(atlas) + g.grid_off;
    const float2 gcr = make_float2(gC[0][0], gC[1][0]), gcg = make_float2(gC[0][1], gC[1][1]),
                 gcb = make_float2(gC[0][2], gC[1][2]), ga = make_float2(gA[0], gA[1]);
    float2 h = make_float2(0.f, 0.f), bt = make_float2(1.f, 1.f), ts = make_float2(Ts[0], Ts[1]);
    for (int cb = (warp_max / kChunk) * kChunk; cb >= 0; cb -= kChunk) {
      Chunk c;
      const int k = cb / kChunk;
      if (kept && k < kKeptChunks) c = restage(prims, g.N, idx, cb, warp_max, kept->masks[k], k == kept->in_buffer, w);
      else c = stage<false>(g, prims, idx, grid, start + cb, start + warp_max + 1, w);
      for (int j = c.n - 1; j >= 0; --j) {
        const Rec& r = w[j];
        const float4 g2 = r[2];
        const float4 q = r[3];
        const int pos = __float_as_int(q.z);
        const int id = __float_as_int(q.w);
        const bool live[2] = {pos <= lp[0], pos <= lp[1]};
        float2 col_r, col_g, col_b;
        if ((c.solid >> j) & 1u) {
          // mask 1 with gradient 0 on the whole footprint: the operations below
          // with m = 1 and gx = gy = 0, which leave the colour and opacity sums
          float2 tx, ty;
          if constexpr (CB) pair_coords(g, r, tx, ty);
          pair_colour(g, g2, id, tx, ty, live[0], live[1], col_r, col_g, col_b);
          const float om1 = __saturatef(1.f - g2.x);
          const float2 a = make_float2(live[0] ? g2.x : 0.f, live[1] ? g2.x : 0.f);
          const float2 om = make_float2(live[0] ? om1 : 1.f, live[1] ? om1 : 1.f);
          const float2 td = make_float2(div_unit(ts.x, om1), div_unit(ts.y, om1));
          const float2 tk = make_float2(pos < lp[0] ? td.x : ts.x, pos < lp[1] ? td.y : ts.y);
          ts = tk;
          const float2 gcc = make_float2(fmaf(gcr.x, col_r.x, fmaf(gcg.x, col_g.x, gcb.x * col_b.x)),
                                         fmaf(gcr.y, col_r.y, fmaf(gcg.y, col_g.y, gcb.y * col_b.y)));
          float2 dlda;
          if (kQuad) dlda = make_float2(tk.x * fmaf(ga.x, bt.x, gcc.x - h.x), tk.y * fmaf(ga.y, bt.y, gcc.y - h.y));
          else dlda = mul2(tk, fma2(ga, bt, sub2(g, gcc, h)));
          const float2 wt = mul2(a, tk);
          float acc[4 * kSumPx];
          colour_sums(acc, gcr, gcg, gcb, wt, dlda, a);
          h = make_float2(fmaf(om.x, h.x, a.x * gcc.x), fmaf(om.y, h.y, a.y * gcc.y));
          bt = make_float2(bt.x * om.x, bt.y * om.y);
          warp_add4(acc, gacc + (size_t)id * 8);
          continue;
        }
        PairSample s;
        const bool inside = (c.inside >> j) & 1u;
        if ((c.fast >> j) & 1u)
          pair_sample<L, KIND, true>(g, atlas, __float_as_int(q.x), r[0], r[1], inside, pxf, pyf, live, s);
        else
          pair_sample<L, KIND, false>(g, atlas, __float_as_int(q.x), r[0], r[1], inside, pxf, pyf, live, s);
        float2 gx, gy;
        const float2 m = pair_blend<true>(g, s, &gx, &gy);
        const float2 tx = s.tx, ty = s.ty;
        const bool f0 = s.ok0 && m.x > 1e-6f, f1 = s.ok1 && m.y > 1e-6f;
        pair_colour(g, g2, id, tx, ty, f0, f1, col_r, col_g, col_b);
        const float2 a = make_float2(f0 ? g2.x * m.x : 0.f, f1 ? g2.x * m.y : 0.f);
        const float2 om = make_float2(__saturatef(1.f - a.x), __saturatef(1.f - a.y));   // max(1 - a, 0) for a >= 0
        // T entering this fragment: stored for the last contributor, else undo
        // the forward product (om >= t_stop > 0 for every earlier fragment, so the
        // approximate division is well conditioned; om = 1 leaves ts unchanged
        // where there is no fragment)
        const float2 tk = make_float2((pos == lp[0]) ? ts.x : div_unit(ts.x, om.x),
                                      (pos == lp[1]) ? ts.y : div_unit(ts.y, om.y));
        ts = tk;
        const float2 gcc = make_float2(fmaf(gcr.x, col_r.x, fmaf(gcg.x, col_g.x, gcb.x * col_b.x)),
                                       fmaf(gcr.y, col_r.y, fmaf(gcg.y, col_g.y, gcb.y * col_b.y)));
        // dL/da and the mask-gradient terms: scalar for the quad layouts, packed
        // for the others (each measured faster on B200).  A pixel without a
        // fragment contributes nothing: a = 0 zeroes its colour and opacity terms,
        // and its mask gradient (from a redirected texel, possibly NaN) is
        // replaced by 0 rather than multiplied by 0.
        float2 dlda, u, v;
        if (kQuad) {
          dlda = make_float2(tk.x * fmaf(ga.x, bt.x, gcc.x - h.x), tk.y * fmaf(ga.y, bt.y, gcc.y - h.y));
          u = make_float2(dlda.x * (f0 ? gx.x : 0.f), dlda.y * (f1 ? gx.y : 0.f));
          v = make_float2(dlda.x * (f0 ? gy.x : 0.f), dlda.y * (f1 ? gy.y : 0.f));
        } else {
          dlda = mul2(tk, fma2(ga, bt, sub2(g, gcc, h)));
          u = mul2(dlda, make_float2(f0 ? gx.x : 0.f, f1 ? gx.y : 0.f));
          v = mul2(dlda, make_float2(f0 ? gy.x : 0.f, f1 ? gy.y : 0.f));
        }
        const float2 ex = add2(tx, g.nhx), ey = add2(ty, g.nhy);
        const float2 wt = mul2(a, tk);
        float acc[8 * kSumPx];
        const float2 e2 = fma2(u, ex, mul2(v, ey)), e3 = fma2(mul2(u, g.rxy2), ey, mul2(mul2(v, g.nryx2), ex));
        if constexpr (kSumPx == 2) {
          acc[0] = u.x; acc[1] = v.x; acc[2] = e2.x; acc[3] = e3.x;
          acc[8] = u.y; acc[9] = v.y; acc[10] = e2.y; acc[11] = e3.y;
          float c[8];
          colour_sums(c, gcr, gcg, gcb, wt, dlda, a);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            acc[4 + k] = c[k];
            acc[12 + k] = c[4 + k];
          }
        } else {
          acc[0] = u.x + u.y;
          acc[1] = v.x + v.y;
          if constexpr (CB) {
            acc[2] = fmaf(u.y, ex.y, fmaf(v.y, ey.y, e2.x));
            acc[3] = fmaf(u.y * g.rxy, ey.y, fmaf(-v.y * g.ryx, ex.y, e3.x));
          } else {
            acc[2] = e2.x + e2.y;
            acc[3] = e3.x + e3.y;
          }
          float c[4];
          colour_sums(c, gcr, gcg, gcb, wt, dlda, a);
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[4 + k] = c[k];
        }
        h = make_float2(fmaf(om.x, h.x, a.x * gcc.x), fmaf(om.y, h.y, a.y * gcc.y));
        bt = make_float2(bt.x * om.x, bt.y * om.y);
        if (__any_sync(kFull, f0 || f1)) warp_add(acc, gacc + (size_t)id * 8);
      }
    }
  }

  // Counting walk (diagnostics): (pixel, primitive) pairs that pass the cull
  // and fragments composited, both before termination, plus walk statistics;
  // it evaluates the clearance-grid test without skipping and counts the
  // warp entries it would skip and, among them, those with a fragment (a
  // correct grid gives 0).
  __device__ __forceinline__ void count(const Geom& g, const PrimInfo* __restrict__ prims,
                                        const void* __restrict__ atlas, const int* __restrict__ idx, Rec* w,
                                        unsigned long long* cnt) const {
    const unsigned char* grid = static_cast<const unsigned char*>(atlas) + g.grid_off;
    unsigned long long n_cand = 0, n_frag = 0, n_went = 0, n_slots = 0, n_miss = 0, n_empty = 0, n_clear = 0,
                       n_bad = 0;
    unsigned n_depth[NP] = {0u, 0u};
    float T[NP] = {1.f, 1.f};
    bool live[NP] = {valid[0], valid[1]};
    bool warp_done = __all_sync(kFull, !live[0] && !live[1]);
    for (int base = start; base < end && !warp_done; base += kChunk) {
      const Chunk c = stage<true>(g, prims, idx, grid, base, end, w);
      n_miss += __popc(c.miss);
      for (int j = 0; j < c.n; ++j) {
        const float4 g0 = w[j][0];
        const float op = w[j][2].x;
        const bool clear = (c.clear >> j) & 1u;
        ++n_went;
        n_clear += clear;
#pragma unroll
        for (int p = 0; p < NP; ++p) n_slots += __popc(__ballot_sync(kFull, live[p]));
        PairPre<KIND> pre;
        PairSample s;
        pair_issue(g, atlas, w[j], (c.inside >> j) & 1u, (c.fast >> j) & 1u, live, pre);
        pair_unpack<KIND>(g, pre, s);
        const float2 m2 = pair_blend<false, false>(g, s, nullptr, nullptr);
        const float m[NP] = {m2.x, m2.y};
        const bool ok[NP] = {s.ok0, s.ok1};
        const bool anyf = __any_sync(kFull, (ok[0] && m[0] > 1e-6f) || (ok[1] && m[1] > 1e-6f));
        n_empty += !anyf;
        n_bad += clear && anyf;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          n_cand += live[p] && !(fabsf(pxf[p] - g0.x) > g0.z || fabsf(pyf[p] - g0.y) > g0.w);
          const bool frag = ok[p] && m[p] > 1e-6f;
          n_frag += frag;
          n_depth[p] += frag;
          const float a = frag ? op * m[p] : 0.f;
          T[p] = __saturatef(fmaf(-T[p], a, T[p]));
          live[p] = live[p] && !(T[p] < g.t_stop);
        }
        if (__all_sync(kFull, !live[0] && !live[1])) { warp_done = true; break; }
      }
    }
    atomicAdd(cnt + 0, n_cand);
    atomicAdd(cnt + 1, n_frag);
    const unsigned dmax = __reduce_max_sync(kFull, max(n_depth[0], n_depth[1]));
    if (lane == 0) {
      atomicAdd(cnt + 3, n_went);
      atomicAdd(cnt + 4, n_slots);
      atomicAdd(cnt + 5, n_miss);
      atomicMax(cnt + 6, (unsigned long long)dmax);
      atomicAdd(cnt + 7, n_empty);
      atomicAdd(cnt + 8, n_clear);
      atomicAdd(cnt + 9, n_bad);
    }
  }
};

// CTA shape of the walk kernels.  The warps of a tile walk independently, so a
// tile may be split over several CTAs, which lets an SM refill as soon as a few
// warps finish: kFwdWarps per CTA in the forward walk, one in the walks with a
// backward part, whose warps differ more in length (2048x2048, N=20000, FP16
// quads, one / four warps: backward 325 / 339 us, fused 498 / 503; forward 208 /
// 204).  Registers are bounded for a number of resident warps per SM, tuned on
// B200 per atlas kind: 36 (56 registers a thread) for the packed atlases' forward
// walk, which waits mostly on texel loads and gains from the extra warps; 32 (64
// registers) for the reference layout and the colour-map walks.  One-warp CTAs
// have 64 registers in any case: an SM holds 32 CTAs.  Forward and backward come
// with and without kept masks as kernels of their own: a pointer tested in the
// walk costs registers (2048x2048, N=20000, FP16 quads: forward 207 -> 204 us,
// backward without masks 354 -> 339; 4096x4096, N=100000: 2133 -> 2058).
#ifndef DBMP_CTA_WARPS
#define DBMP_CTA_WARPS 4
#endif
#ifndef DBMP_WARPS_PER_SM
#define DBMP_WARPS_PER_SM 36
#endif
#ifndef DBMP_WARPS_PER_SM_F32
#define DBMP_WARPS_PER_SM_F32 32
#endif
template <int TS> constexpr int kTileWarps() { return Layout<TS>::NW; }
template <int TS> constexpr int kFwdWarps() {
  return kTileWarps<TS>() < DBMP_CTA_WARPS ? kTileWarps<TS>() : DBMP_CTA_WARPS;
}
template <int TS> constexpr int kFwdParts() { return kTileWarps<TS>() / kFwdWarps<TS>(); }
template <int KIND, bool CB = false> constexpr int kBlocksPerSM(int cta_warps) {
  return ((KIND == ATLAS_F32 || CB) ? DBMP_WARPS_PER_SM_F32 : DBMP_WARPS_PER_SM) / cta_warps;
}

// True where a followed atlas's templates differ from the packed ones that this walk
// would read: its *_changed_kernel then walks the templates.
template <int KIND> __device__ __forceinline__ bool packed_is_stale(const Geom& g, int word) {
  return KIND == ATLAS_F32_QUAD && g.changed != nullptr && follow_changed(g.changed + word);
}

// ---------------------------------------------------------------------------
// One block of a forward launch: kFwdWarps warps of a tile.
template <int TS, int KIND, bool CB, bool MASKED>
__device__ __forceinline__ void forward_block(
    const Geom& g, int block, Rec (*s_pi)[kChunk], const PrimInfo* __restrict__ prims, const void* __restrict__ atlas,
    const int* __restrict__ offs, const int* __restrict__ idx, float* __restrict__ out_color,
    float* __restrict__ out_alpha, float* __restrict__ T_last, int* __restrict__ last_pos,
    const float* __restrict__ cmap, float cblend, long long idx_stride, long long cmap_stride,
    const int* __restrict__ flags, uint4* __restrict__ masks) {
  constexpr int NP = 2;
  using TW = TileWalker<TS, KIND, CB>;
  // a batch of candidates is one grid over all their tiles: candidate b's
  // records, lists and images follow candidate b-1's
  const int gt = block / kFwdParts<TS>(), part = block % kFwdParts<TS>();
  const int b = gt / g.T, tile = gt - b * g.T;
  // binning overflowed for a candidate: its lists do not exist, and the caller
  // bins again (flags: list length and overflow per candidate)
  if (flags != nullptr && flags[2 * b + 1] != 0) return;
  const size_t pix = (size_t)b * g.H * g.W;
  prims += (size_t)b * g.N;
  offs += (size_t)b * (g.T + 1);
  idx += (size_t)b * idx_stride;
  out_color += 3 * pix; out_alpha += pix; T_last += pix; last_pos += pix;
  TW tw;
  tw.cmap = CB ? cmap + (size_t)b * cmap_stride : cmap;
  tw.cblend = cblend;
  tw.init(g, tile, part, kFwdWarps<TS>(), offs);
  float C[NP][3], T[NP], Tl[NP];
  int lp[NP];
  uint4* kept = nullptr;   // MASKED: this warp's masks for the backward
  if (MASKED) kept = masks + ((size_t)gt * kTileWarps<TS>() + tw.warp) * kKeptChunks;
  tw.forward(g, prims, atlas, idx, s_pi[tw.lw], C, T, Tl, lp, kept, nullptr);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    if (!tw.valid[p]) continue;
    const size_t q = (size_t)tw.py(tile, g, p) * g.W + tw.px(tile, g);
    out_color[3 * q + 0] = C[p][0];
    out_color[3 * q + 1] = C[p][1];
    out_color[3 * q + 2] = C[p][2];
    out_alpha[q] = 1.f - T[p];
    T_last[q] = Tl[p];
    last_pos[q] = lp[p];
  }
}

template <int TS, int KIND, bool CB, bool MASKED>
__global__ void __launch_bounds__(kFwdWarps<TS>() * 32, kBlocksPerSM<KIND, CB>(kFwdWarps<TS>())) forward_kernel(
    Geom g, const PrimInfo* __restrict__ prims, const void* __restrict__ atlas, const int* __restrict__ offs,
    const int* __restrict__ idx, float* __restrict__ out_color, float* __restrict__ out_alpha,
    float* __restrict__ T_last, int* __restrict__ last_pos, const float* __restrict__ cmap, float cblend,
    long long idx_stride, long long cmap_stride, const int* __restrict__ flags, uint4* __restrict__ masks) {
  __shared__ Rec s_pi[kFwdWarps<TS>()][kChunk];
  grid_dependency();
  if (packed_is_stale<KIND>(g, 0)) return;
  forward_block<TS, KIND, CB, MASKED>(g, blockIdx.x, s_pi, prims, atlas, offs, idx, out_color, out_alpha, T_last,
                                      last_pos, cmap, cblend, idx_stride, cmap_stride, flags, masks);
}

// The walks of a followed atlas whose templates have changed, on the templates, behind
// those on its packed copy that return at once then: for forwards of given lists,
// backwards and fits.  (A render tells the host to call again, and small masked
// backwards read the templates themselves.)  They nearly always find nothing to do, so a
// grid of at most the resident blocks loops over the tiles, rather than a block per
// tile that starts only to return.
template <int TS, bool CB, bool MASKED>
__global__ void __launch_bounds__(kFwdWarps<TS>() * 32, kBlocksPerSM<ATLAS_F32, CB>(kFwdWarps<TS>()))
    forward_changed_kernel(Geom g, unsigned blocks, const PrimInfo* __restrict__ prims, const int* __restrict__ offs,
                           const int* __restrict__ idx, float* __restrict__ out_color, float* __restrict__ out_alpha,
                           float* __restrict__ T_last, int* __restrict__ last_pos, const float* __restrict__ cmap,
                           float cblend, long long idx_stride, long long cmap_stride, const int* __restrict__ flags,
                           uint4* __restrict__ masks) {
  __shared__ Rec s_pi[kFwdWarps<TS>()][kChunk];
  grid_dependency();
  if (!follow_changed(g.changed)) return;
  for (unsigned b = blockIdx.x; b < blocks; b += gridDim.x)
    forward_block<TS, ATLAS_F32, CB, MASKED>(g, (int)b, s_pi, prims, g.live, offs, idx, out_color, out_alpha, T_last,
                                             last_pos, cmap, cblend, idx_stride, cmap_stride, flags, masks);
}

// Counting pass (diagnostics / roofline accounting): same walk as the
// forward, no outputs except the counters.
template <int TS, int KIND>
__global__ void __launch_bounds__(kFwdWarps<TS>() * 32) count_kernel(Geom g, const PrimInfo* __restrict__ prims,
                                                                     const void* __restrict__ atlas,
                                                                     const int* __restrict__ offs,
                                                                     const int* __restrict__ idx,
                                                                     unsigned long long* __restrict__ cnt) {
  using TW = TileWalker<TS, KIND>;
  __shared__ Rec s_pi[kFwdWarps<TS>()][kChunk];
  TW tw;
  const int tile = blockIdx.x / kFwdParts<TS>(), part = blockIdx.x % kFwdParts<TS>();
  tw.init(g, tile, part, kFwdWarps<TS>(), offs);
  tw.count(g, prims, atlas, idx, s_pi[tw.lw], cnt);
  if (threadIdx.x == 0 && part == 0) atomicAdd(cnt + 2, (unsigned long long)(tw.end - tw.start));
}

// One block of a backward launch: a warp of a tile.  kept: null without masks.
template <int TS, int KIND, bool CB, bool MASKED>
__device__ __forceinline__ void backward_block(
    const Geom& g, int block, Rec* s_pi, Kept* s_kept, const PrimInfo* __restrict__ prims,
    const void* __restrict__ atlas, const int* __restrict__ offs, const int* __restrict__ idx,
    const float* __restrict__ T_last, const int* __restrict__ last_pos, const float* __restrict__ grad_color,
    const float* __restrict__ grad_alpha, double* __restrict__ gacc, const float* __restrict__ cmap, float cblend,
    long long idx_stride, long long cmap_stride, const uint4* __restrict__ masks) {
  constexpr int NP = 2;
  using TW = TileWalker<TS, KIND, CB>;
  const int gt = block / kTileWarps<TS>(), part = block % kTileWarps<TS>();
  const int b = gt / g.T, tile = gt - b * g.T;     // candidate and tile (see forward_kernel)
  const size_t pix = (size_t)b * g.H * g.W;
  prims += (size_t)b * g.N;
  offs += (size_t)b * (g.T + 1);
  idx += (size_t)b * idx_stride;
  T_last += pix; last_pos += pix; grad_color += 3 * pix;
  if (grad_alpha != nullptr) grad_alpha += pix;
  gacc += (size_t)b * g.N * 8;
  TW tw;
  tw.cmap = CB ? cmap + (size_t)b * cmap_stride : cmap;
  tw.cblend = cblend;
  tw.init(g, tile, part, 1, offs);
  float gC[NP][3], gA[NP], Ts[NP];
  int lp[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    if (tw.valid[p]) {
      const size_t q = (size_t)tw.py(tile, g, p) * g.W + tw.px(tile, g);
      gC[p][0] = grad_color[3 * q + 0];
      gC[p][1] = grad_color[3 * q + 1];
      gC[p][2] = grad_color[3 * q + 2];
      gA[p] = grad_alpha ? grad_alpha[q] : 0.f;
      Ts[p] = T_last[q];
      lp[p] = last_pos[q];
    } else {
      gC[p][0] = gC[p][1] = gC[p][2] = 0.f;
      gA[p] = 0.f; Ts[p] = 1.f; lp[p] = -1;
    }
  }
  if constexpr (MASKED) {
    const size_t at = ((size_t)gt * kTileWarps<TS>() + tw.warp) * kKeptChunks;
    if (tw.lane < kKeptChunks) s_kept->masks[tw.lane] = masks[at + tw.lane];   // (those never written are never used)
    if (tw.lane == 0) s_kept->in_buffer = -1;
    __syncwarp();
  }
  tw.backward(g, prims, atlas, idx, s_pi, gC, gA, Ts, lp, gacc, MASKED ? s_kept : nullptr);
}

// INNER: the masked walk on FP32 quads with the walk on a followed atlas's templates
// beside it, for small launches.  Behind it in a launch of its own, that one costs the
// host 5 us, which small calls wait for; inside, it costs the kernel's code 3 to 4 %
// (backward at 1024x1024, N=5000: 128.5 -> 132.5 us; 4096x4096, N=100000: 2369 ->
// 2455), bounded to the 72 registers that leave it its 28 warps per SM.  Forward and
// backward together, launched apart / inside: 512x512 (host-bound) 224 / 220 us,
// 1024x1024 243 / 243, 4096x4096 3370 / 3450.
constexpr long long kInnerWarps = 12288;   // walks of up to about 887x887 pixels

template <int TS, int KIND, bool CB, bool MASKED, bool INNER = false>
__global__ void __launch_bounds__(32, INNER && !CB ? 28 : kBlocksPerSM<KIND, CB>(1)) backward_kernel(
    Geom g, const PrimInfo* __restrict__ prims, const void* __restrict__ atlas, const int* __restrict__ offs,
    const int* __restrict__ idx, const float* __restrict__ T_last, const int* __restrict__ last_pos,
    const float* __restrict__ grad_color, const float* __restrict__ grad_alpha, double* __restrict__ gacc,
    const float* __restrict__ cmap, float cblend, long long idx_stride, long long cmap_stride,
    const uint4* __restrict__ masks) {
  __shared__ Rec s_pi[kChunk];
  __shared__ Kept s_kept;
  grid_dependency();
  if (packed_is_stale<KIND>(g, 1)) {
    if constexpr (INNER)   // (the masks belong to the packed templates)
      backward_block<TS, ATLAS_F32, CB, false>(g, blockIdx.x, s_pi, nullptr, prims, g.live, offs, idx, T_last, last_pos,
                                               grad_color, grad_alpha, gacc, cmap, cblend, idx_stride, cmap_stride,
                                               nullptr);
    return;
  }
  backward_block<TS, KIND, CB, MASKED>(g, blockIdx.x, s_pi, &s_kept, prims, atlas, offs, idx, T_last, last_pos,
                                       grad_color, grad_alpha, gacc, cmap, cblend, idx_stride, cmap_stride, masks);
}

// (see forward_changed_kernel; the forward's masks belong to the packed templates)
template <int TS, bool CB>
__global__ void __launch_bounds__(32, kBlocksPerSM<ATLAS_F32, CB>(1)) backward_changed_kernel(
    Geom g, unsigned blocks, const PrimInfo* __restrict__ prims, const int* __restrict__ offs,
    const int* __restrict__ idx, const float* __restrict__ T_last, const int* __restrict__ last_pos,
    const float* __restrict__ grad_color, const float* __restrict__ grad_alpha, double* __restrict__ gacc,
    const float* __restrict__ cmap, float cblend, long long idx_stride, long long cmap_stride) {
  __shared__ Rec s_pi[kChunk];
  grid_dependency();
  if (!follow_changed(g.changed + 1)) return;
  for (unsigned b = blockIdx.x; b < blocks; b += gridDim.x)
    backward_block<TS, ATLAS_F32, CB, false>(g, (int)b, s_pi, nullptr, prims, g.live, offs, idx, T_last, last_pos,
                                             grad_color, grad_alpha, gacc, cmap, cblend, idx_stride, cmap_stride,
                                             nullptr);
}

__device__ __forceinline__ double sigmoid_d(double x) {
  if (x >= 0.0) { const double z = exp(-x); return 1.0 / (1.0 + z); }
  const double z = exp(x);
  return z / (1.0 + z);
}

// Converts the accumulated per-primitive sums into the reference's gradient
// outputs (tile_backward.cu:255-343 chain rule, applied once per primitive).
// gacc[n] = { S dLda*gx, S dLda*gy, S dLda*(gx*ex + gy*ey),
//             S dLda*(gx*ey*hx/hy - gy*ex*hy/hx), S gC_r*a*T, S gC_g*a*T,
//             S gC_b*a*T, S dLda*a }  summed over the primitive's fragments,
// with (ex, ey) the texel coordinate minus (hx, hy) and gx, gy = d mask/d tex.
__global__ void finalize_kernel(Geom g, const float* __restrict__ radii, const float* __restrict__ rot,
                                const float* __restrict__ opac, const float* __restrict__ colors,
                                const double* __restrict__ gacc, float* __restrict__ g_means,
                                float* __restrict__ g_radii, float* __restrict__ g_rot, float* __restrict__ g_opac,
                                float* __restrict__ g_colors) {
  grid_dependency();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= g.N) return;
  const double* S = gacc + (size_t)n * 8;
  const float r = radii[n];
  const double rinv = (r > 1e-6f) ? 1.0 / (double)r : 1e6;
  double s, c;
  sincos((double)rot[n], &s, &c);
  const double sv = sigmoid_d((double)opac[n]);
  const double a0 = (double)g.alpha_max * sv;
  const double hx = g.hx, hy = g.hy;
  // A primitive without fragments has zero sums and zero gradients, also when
  // its rotation is not finite (the reference adds gradients per fragment): a
  // zero sum contributes 0 rather than NaN * 0.
  const double cx = S[0] != 0.0 ? c * hx * S[0] : 0.0, sx = S[0] != 0.0 ? s * hx * S[0] : 0.0;
  const double cy = S[1] != 0.0 ? c * hy * S[1] : 0.0, sy = S[1] != 0.0 ? s * hy * S[1] : 0.0;
  g_means[2 * n + 0] = (float)(a0 * rinv * (sy - cx));
  g_means[2 * n + 1] = (float)(a0 * rinv * (-sx - cy));
  g_radii[n] = (float)(-a0 * rinv * S[2]);
  g_rot[n] = (float)(a0 * S[3]);
  g_opac[n] = (float)((1.0 - sv) * S[7]);
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const double sc = sigmoid_d((double)colors[3 * n + ch]);
    g_colors[3 * n + ch] = (float)(sc * (1.0 - sc) * S[4 + ch]);
  }
}

// ---------------------------------------------------------------------------
// Fused forward + L2 loss + backward for image fitting.  The loss is the
// reference's mse_loss(rendered, target) (pydiffbmp/util/loss_functions.py:20-40)
// on rendered = C + (1 - A) * background (simple_tile_renderer.py:704-707):
//   dL/dC = 2 (rendered - target) / (3HW),  dL/dA = -sum_c dL/dC_c * bg_c.
// loss_out (f64, may be null) receives sum((rendered - target)^2) / (3HW),
// one add per warp.
template <int TS, int KIND>
__device__ __forceinline__ void fused_block(const Geom& g, int block, Rec* s_pi, Kept& s_kept,
                                            const PrimInfo* __restrict__ prims, const void* __restrict__ atlas,
                                            const int* __restrict__ offs, const int* __restrict__ idx,
                                            const float* __restrict__ target, const float* __restrict__ background,
                                            float* __restrict__ out_image, double* __restrict__ gacc,
                                            double* __restrict__ loss_out) {
  constexpr int NP = 2;
  using TW = TileWalker<TS, KIND>;
  TW tw;
  const int tile = block / kTileWarps<TS>(), part = block % kTileWarps<TS>();
  tw.init(g, tile, part, 1, offs);
  float C[NP][3], T[NP], Tl[NP], gC[NP][3], gA[NP];
  int lp[NP];
  tw.forward(g, prims, atlas, idx, s_pi, C, T, Tl, lp, s_kept.masks, &s_kept.in_buffer);
  const float inv = 1.f / (3.f * (float)g.H * (float)g.W);
  float lsum = 0.f;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    gA[p] = 0.f;
    gC[p][0] = gC[p][1] = gC[p][2] = 0.f;
    if (!tw.valid[p]) continue;
    const size_t q = (size_t)tw.py(tile, g, p) * g.W + tw.px(tile, g);
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      const float bg = background ? background[3 * q + ch] : 0.f;
      const float img = fmaf(T[p], bg, C[p][ch]);
      if (out_image) out_image[3 * q + ch] = img;
      const float d = img - target[3 * q + ch];
      lsum = fmaf(d, d, lsum);
      gC[p][ch] = 2.f * d * inv;
      gA[p] -= gC[p][ch] * bg;
    }
  }
  if (loss_out) {
    lsum += __shfl_xor_sync(kFull, lsum, 16);
    lsum += __shfl_xor_sync(kFull, lsum, 8);
    lsum += __shfl_xor_sync(kFull, lsum, 4);
    lsum += __shfl_xor_sync(kFull, lsum, 2);
    lsum += __shfl_xor_sync(kFull, lsum, 1);
    if (tw.lane == 0) atomicAdd(loss_out, (double)lsum * (double)inv);
  }
  __syncwarp();   // s_kept is visible to every lane
  tw.backward(g, prims, atlas, idx, s_pi, gC, gA, Tl, lp, gacc, &s_kept);
}

template <int TS, int KIND, bool INNER = false>   // INNER: see backward_kernel
__global__ void __launch_bounds__(32, INNER ? 28 : kBlocksPerSM<KIND>(1)) fused_kernel(
    Geom g, const PrimInfo* __restrict__ prims, const void* __restrict__ atlas, const int* __restrict__ offs,
    const int* __restrict__ idx, const float* __restrict__ target, const float* __restrict__ background,
    float* __restrict__ out_image, double* __restrict__ gacc, double* __restrict__ loss_out,
    const int* __restrict__ skip_flag) {
  __shared__ Rec s_pi[kChunk];
  __shared__ Kept s_kept;
  grid_dependency();
  if (skip_flag != nullptr && *skip_flag != 0) return;   // binning overflowed: leave all state untouched
  if (packed_is_stale<KIND>(g, 1)) {
    if constexpr (INNER)
      fused_block<TS, ATLAS_F32>(g, blockIdx.x, s_pi, s_kept, prims, g.live, offs, idx, target, background, out_image, gacc,
                                 loss_out);
    return;
  }
  fused_block<TS, KIND>(g, blockIdx.x, s_pi, s_kept, prims, atlas, offs, idx, target, background, out_image, gacc,
                        loss_out);
}

// (see forward_changed_kernel)
template <int TS>
__global__ void __launch_bounds__(32, kBlocksPerSM<ATLAS_F32>(1)) fused_changed_kernel(
    Geom g, unsigned blocks, const PrimInfo* __restrict__ prims, const int* __restrict__ offs,
    const int* __restrict__ idx, const float* __restrict__ target, const float* __restrict__ background,
    float* __restrict__ out_image, double* __restrict__ gacc, double* __restrict__ loss_out,
    const int* __restrict__ skip_flag) {
  __shared__ Rec s_pi[kChunk];
  __shared__ Kept s_kept;
  grid_dependency();
  if ((skip_flag != nullptr && *skip_flag != 0) || !follow_changed(g.changed + 1)) return;
  for (unsigned b = blockIdx.x; b < blocks; b += gridDim.x) {
    __syncwarp();   // every lane is done with the previous block's masks
    fused_block<TS, ATLAS_F32>(g, (int)b, s_pi, s_kept, prims, g.live, offs, idx, target, background, out_image, gacc,
                               loss_out);
  }
}

// The comparison alone, for forwards of given lists (renders compare beside the
// counting of their binning, backwards and fits beside the zeroing of their sums).
// Without a trigger: the walk's CTAs launch as these end.  Launched beside them, they
// crowd onto the SMs that are free first (fit step of 256x256, N=5000, 16 of 256x256:
// 125 us, 89 without, 90.5 without a comparison).
__global__ void __launch_bounds__(1024) follow_kernel(Follow f) {
  cudaGridDependencySynchronize();
  follow_compare(f, blockIdx.x);
}

// ---------------------------------------------------------------------------
#define DBMP_KIND_SWITCH(kind, ...)                                                   \
  switch (kind) {                                                                     \
    case ATLAS_F32: { constexpr int KD = ATLAS_F32; __VA_ARGS__; } break;             \
    case ATLAS_F32_QUAD: { constexpr int KD = ATLAS_F32_QUAD; __VA_ARGS__; } break;   \
    case ATLAS_F16_QUAD: { constexpr int KD = ATLAS_F16_QUAD; __VA_ARGS__; } break;   \
    case ATLAS_BF16_QUAD: { constexpr int KD = ATLAS_BF16_QUAD; __VA_ARGS__; } break; \
    case ATLAS_F16_PAIR: { constexpr int KD = ATLAS_F16_PAIR; __VA_ARGS__; } break;   \
    case ATLAS_BF16_PAIR: { constexpr int KD = ATLAS_BF16_PAIR; __VA_ARGS__; } break; \
    default: set_error("unknown atlas kind %d", kind); return DBMP_ERR_INVALID;       \
  }

#define DBMP_TS_SWITCH(ts, ...)                                      \
  if ((ts) == 32) { constexpr int TSV = 32; __VA_ARGS__; }           \
  else if ((ts) == 16) { constexpr int TSV = 16; __VA_ARGS__; }      \
  else { set_error("tile_size %d is not supported (16 or 32)", ts); return DBMP_ERR_INVALID; }

// batch > 1: `batch` candidates of the same canvas in one grid, candidate b's
// records at prims + b N, lists at offs + b (T+1) / idx + b idx_stride,
// images at b H W (x3 for colour), colour maps at cmap + b cmap_stride.
// Grid of a *_changed_kernel: at most what is resident at once.
static dim3 changed_grid(long long blocks, int per_sm) {
  return dim3((unsigned)(blocks < 148ll * per_sm ? blocks : 148ll * per_sm));
}

size_t walk_mask_bytes(const Geom& g, int batch) {
  const size_t warps = (size_t)batch * g.T * (g.TS == 32 ? kTileWarps<32>() : kTileWarps<16>());
  return warps * kKeptChunks * sizeof(uint4);
}

int launch_forward_blend(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                         const int* idx, float* color, float* alpha, float* T_last, int* last_pos, const float* cmap,
                         float cblend, cudaStream_t st, int batch, long long idx_stride, long long cmap_stride,
                         const int* flags, void* masks) {
  if (g.T == 0 || batch == 0) return DBMP_OK;
  const long long ctas = (long long)batch * g.T * kFwdParts<32>();
  if (ctas > 0x7fffffffll) { set_error("forward: %d candidates x %d tiles exceed one grid", batch, g.T); return DBMP_ERR_INVALID; }
  const bool blend = cmap != nullptr && cblend > 0.f;
  auto go = [&](auto kernel, int parts, int threads) {
    return launch_chained("forward_kernel", kernel, dim3((unsigned)(batch * g.T * parts)), threads, 0, st, g, prims,
                          atlas, offs, idx, color, alpha, T_last, last_pos, blend ? cmap : nullptr,
                          blend ? cblend : 0.f, idx_stride, blend ? cmap_stride : 0ll, flags, (uint4*)masks);
  };
  auto walk = [&]() -> int {
    DBMP_TS_SWITCH(g.TS, DBMP_KIND_SWITCH(kind, constexpr int parts = kFwdParts<TSV>(), threads = kFwdWarps<TSV>() * 32;
        if (blend) return masks ? go(forward_kernel<TSV, KD, true, true>, parts, threads)
                                : go(forward_kernel<TSV, KD, true, false>, parts, threads);
        return masks ? go(forward_kernel<TSV, KD, false, true>, parts, threads)
                     : go(forward_kernel<TSV, KD, false, false>, parts, threads)));
    return DBMP_OK;
  };
  // flags: behind a binning, which compared a followed atlas and told the host
  if (!g.live || flags != nullptr) return walk();
  const Follow f = make_follow(g, atlas, 0);
  int rc = launch_chained("follow_kernel", follow_kernel, dim3(f.blocks), 1024, 0, st, f);
  if (!rc) rc = walk();
  if (rc) return rc;
  auto again = [&](auto kernel, int parts, int threads) {
    const long long blocks = (long long)batch * g.T * parts;
    return launch_chained("forward_changed_kernel", kernel, changed_grid(blocks, DBMP_WARPS_PER_SM_F32 * 32 / threads),
                          threads, 0, st, g, (unsigned)blocks, prims, offs, idx, color, alpha, T_last, last_pos,
                          blend ? cmap : nullptr, blend ? cblend : 0.f, idx_stride, blend ? cmap_stride : 0ll, flags,
                          (uint4*)masks);
  };
  DBMP_TS_SWITCH(g.TS, constexpr int parts = kFwdParts<TSV>(), threads = kFwdWarps<TSV>() * 32;
      if (blend) return masks ? again(forward_changed_kernel<TSV, true, true>, parts, threads)
                              : again(forward_changed_kernel<TSV, true, false>, parts, threads);
      return masks ? again(forward_changed_kernel<TSV, false, true>, parts, threads)
                   : again(forward_changed_kernel<TSV, false, false>, parts, threads));
  return DBMP_OK;
}

int launch_forward(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                   const int* idx, float* color, float* alpha, float* T_last, int* last_pos, cudaStream_t st) {
  return launch_forward_blend(g, kind, prims, atlas, offs, idx, color, alpha, T_last, last_pos, nullptr, 0.f, st, 1,
                              0, 0, nullptr, nullptr);
}

int launch_count(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs, const int* idx,
                 unsigned long long* cnt, cudaStream_t st) {
  if (g.T == 0) return DBMP_OK;
  if (g.live) {   // counts what the reference layout's walk does
    kind = ATLAS_F32;
    atlas = g.live;
  }
  DBMP_TS_SWITCH(g.TS, DBMP_KIND_SWITCH(kind, (count_kernel<TSV, KD><<<g.T * kFwdParts<TSV>(), kFwdWarps<TSV>() * 32, 0, st>>>(
                                                   g, prims, atlas, offs, idx, cnt))));
  DBMP_CHECK_LAUNCH("count_kernel");
  return DBMP_OK;
}

int launch_backward_blend(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                          const int* idx, const float* T_last, const int* last_pos, const float* grad_color,
                          const float* grad_alpha, double* gacc, const float* cmap, float cblend, cudaStream_t st,
                          int batch, long long idx_stride, long long cmap_stride, const void* masks) {
  if (g.T == 0 || batch == 0) return DBMP_OK;
  const long long ctas = (long long)batch * g.T * kTileWarps<32>();
  if (ctas > 0x7fffffffll) { set_error("backward: %d candidates x %d tiles exceed one grid", batch, g.T); return DBMP_ERR_INVALID; }
  const bool blend = cmap != nullptr && cblend > 0.f;
  auto go = [&](auto kernel, int warps) {
    return launch_chained("backward_kernel", kernel, dim3((unsigned)(batch * g.T * warps)), 32, 0, st, g, prims, atlas,
                          offs, idx, T_last, last_pos, grad_color, grad_alpha, gacc, blend ? cmap : nullptr,
                          blend ? cblend : 0.f, idx_stride, blend ? cmap_stride : 0ll, (const uint4*)masks);
  };
  auto walk = [&]() -> int {
    DBMP_TS_SWITCH(g.TS, DBMP_KIND_SWITCH(kind,
        if (blend) return masks ? go(backward_kernel<TSV, KD, true, true>, kTileWarps<TSV>())
                                : go(backward_kernel<TSV, KD, true, false>, kTileWarps<TSV>());
        return masks ? go(backward_kernel<TSV, KD, false, true>, kTileWarps<TSV>())
                     : go(backward_kernel<TSV, KD, false, false>, kTileWarps<TSV>())));
    return DBMP_OK;
  };
  if (!g.live) return walk();
  // launch_zero has compared a followed atlas
  if (masks != nullptr && ctas <= kInnerWarps && kind == ATLAS_F32_QUAD) {
    DBMP_TS_SWITCH(g.TS, return blend ? go(backward_kernel<TSV, ATLAS_F32_QUAD, true, true, true>, kTileWarps<TSV>())
                                      : go(backward_kernel<TSV, ATLAS_F32_QUAD, false, true, true>, kTileWarps<TSV>()));
  }
  const int rc = walk();
  if (rc) return rc;
  auto again = [&](auto kernel, int warps) {
    const long long blocks = (long long)batch * g.T * warps;
    return launch_chained("backward_changed_kernel", kernel, changed_grid(blocks, DBMP_WARPS_PER_SM_F32), 32, 0, st, g,
                          (unsigned)blocks, prims, offs, idx, T_last, last_pos, grad_color, grad_alpha, gacc,
                          blend ? cmap : nullptr, blend ? cblend : 0.f, idx_stride, blend ? cmap_stride : 0ll);
  };
  DBMP_TS_SWITCH(g.TS, return blend ? again(backward_changed_kernel<TSV, true>, kTileWarps<TSV>())
                                    : again(backward_changed_kernel<TSV, false>, kTileWarps<TSV>()));
  return DBMP_OK;
}

int launch_backward(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                    const int* idx, const float* T_last, const int* last_pos, const float* grad_color,
                    const float* grad_alpha, double* gacc, cudaStream_t st) {
  return launch_backward_blend(g, kind, prims, atlas, offs, idx, T_last, last_pos, grad_color, grad_alpha, gacc,
                               nullptr, 0.f, st, 1, 0, 0, nullptr);
}

// Zeroes n doubles at a and, when given, one at b: a kernel rather than memsets, so
// that the launches around it stay chained.  Its first blocks also compare a followed
// atlas's templates for the walk behind.
__global__ void __launch_bounds__(1024) zero_kernel(double* __restrict__ a, long long n, double* __restrict__ b, Follow f) {
  cudaGridDependencySynchronize();
  if (f.live == nullptr) cudaTriggerProgrammaticLaunchCompletion();   // (see follow_kernel)
  else if (blockIdx.x < f.blocks) follow_compare(f, blockIdx.x);
  const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long i = i0; i < n; i += (long long)gridDim.x * blockDim.x) a[i] = 0.0;
  if (b != nullptr && i0 == 0) *b = 0.0;
}

int launch_zero(double* a, long long n, double* b, const Follow& f, cudaStream_t st) {
  if (n == 0 && b == nullptr && f.live == nullptr) return DBMP_OK;
  const unsigned threads = f.live ? 1024 : 256;
  long long ctas = (n + threads - 1) / threads;
  if (ctas < 1) ctas = 1;
  if (ctas < f.blocks) ctas = f.blocks;
  if (ctas > 1184) ctas = 1184;
  return launch_chained("zero_kernel", zero_kernel, dim3((unsigned)ctas), threads, 0, st, a, n, b, f);
}

int launch_finalize(const Geom& g, const float* radii, const float* rot, const float* opac, const float* colors,
                    const double* gacc, float* gm, float* gr, float* grot, float* go, float* gc, cudaStream_t st) {
  if (g.N == 0) return DBMP_OK;
  return launch_chained("finalize_kernel", finalize_kernel, dim3((g.N + 63) / 64), 64, 0, st, g, radii, rot, opac,
                        colors, gacc, gm, gr, grot, go, gc);
}

int launch_fused(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs, const int* idx,
                 const float* target, const float* background, float* out_image, double* gacc, double* loss,
                 const int* skip_flag, cudaStream_t st) {
  if (g.T == 0) return DBMP_OK;
  auto walk = [&]() -> int {
    DBMP_TS_SWITCH(g.TS, DBMP_KIND_SWITCH(kind, return launch_chained(
        "fused_kernel", fused_kernel<TSV, KD>, dim3((unsigned)(g.T * kTileWarps<TSV>())), 32, 0, st, g, prims, atlas,
        offs, idx, target, background, out_image, gacc, loss, skip_flag)));
    return DBMP_OK;
  };
  if (!g.live) return walk();
  // launch_zero has compared a followed atlas
  DBMP_TS_SWITCH(g.TS, if ((long long)g.T * kTileWarps<TSV>() <= kInnerWarps) return launch_chained(
      "fused_kernel", fused_kernel<TSV, ATLAS_F32_QUAD, true>, dim3((unsigned)(g.T * kTileWarps<TSV>())), 32, 0, st, g,
      prims, atlas, offs, idx, target, background, out_image, gacc, loss, skip_flag));
  const int rc = walk();
  if (rc) return rc;
  DBMP_TS_SWITCH(g.TS, const long long blocks = (long long)g.T * kTileWarps<TSV>(); return launch_chained(
      "fused_changed_kernel", fused_changed_kernel<TSV>, changed_grid(blocks, DBMP_WARPS_PER_SM_F32), 32, 0, st, g,
      (unsigned)blocks, prims, offs, idx, target, background, out_image, gacc, loss, skip_flag));
}

}  // namespace dbmp
