// Device binning: per-primitive preparation, primitive -> tile rectangles,
// then CSR tile lists built row by row without a sort: the tiles' entries are
// counted from difference arrays of rectangle corners, and for each tile row a
// group of CTAs takes the primitives in index order, compacts those whose
// rectangle touches the group's tiles, and each warp writes the entries of its
// own tiles.  Lists therefore come out in ascending primitive order per tile,
// as the reference's per-tile nonzero() gives them, with no host round trip.
//
// This translation unit is compiled WITHOUT fast-math: the world-space bbox
// must reproduce the reference's float32 torch element-wise arithmetic
// (pydiffbmp/core/renderer/vector_renderer.py:214-250: torch.cos/torch.sin,
// then one rounding per multiply / add, no FMA) bit for bit.
#include <cub/cub.cuh>

#include "dbmp_internal.cuh"

namespace dbmp {

// ---------------------------------------------------------------------------
// Template bboxes (simple_tile_renderer.py:130-171): min/max texel column and
// row over texels > 1e-6, mapped with u = (col/(W-1))*2-1 in float32.  The
// map is monotone, so min/max of the integer indices give min/max of u.
__global__ void template_bbox_kernel(const float* __restrict__ tmpl, int Ht, int Wt,
                                     float* __restrict__ out) {
  const int p = blockIdx.x;
  const float* t = tmpl + (size_t)p * Ht * Wt;
  int mnx = INT_MAX, mxx = -1, mny = INT_MAX, mxy = -1;
  for (int i = threadIdx.x; i < Ht * Wt; i += blockDim.x) {
    if (t[i] > 1e-6f) {
      const int y = i / Wt, x = i - y * Wt;
      mnx = min(mnx, x); mxx = max(mxx, x); mny = min(mny, y); mxy = max(mxy, y);
    }
  }
  typedef cub::BlockReduce<int, 256> BR;
  __shared__ typename BR::TempStorage tmp;
  const int a = BR(tmp).Reduce(mnx, cub::Min()); __syncthreads();
  const int b = BR(tmp).Reduce(mxx, cub::Max()); __syncthreads();
  const int c = BR(tmp).Reduce(mny, cub::Min()); __syncthreads();
  const int d = BR(tmp).Reduce(mxy, cub::Max());
  if (threadIdx.x == 0) {
    if (b < 0) {
      out[4 * p + 0] = -1.f; out[4 * p + 1] = 1.f; out[4 * p + 2] = -1.f; out[4 * p + 3] = 1.f;
    } else {
      const float dw = (float)(Wt - 1), dh = (float)(Ht - 1);
      out[4 * p + 0] = __fsub_rn(__fmul_rn(__fdiv_rn((float)a, dw), 2.f), 1.f);
      out[4 * p + 1] = __fsub_rn(__fmul_rn(__fdiv_rn((float)b, dw), 2.f), 1.f);
      out[4 * p + 2] = __fsub_rn(__fmul_rn(__fdiv_rn((float)c, dh), 2.f), 1.f);
      out[4 * p + 3] = __fsub_rn(__fmul_rn(__fdiv_rn((float)d, dh), 2.f), 1.f);
    }
  }
}

// ---------------------------------------------------------------------------
// Atlas repacking into bilinear quads / pairs (precision form).  Each record
// holds a texel and the difference to its right neighbour, the difference
// taken against the stored (rounded) texel, so that stored texel + stored
// difference is the neighbour up to one rounding of the difference.
template <typename OutT>
__device__ __forceinline__ OutT to_storage(float v);
template <> __device__ __forceinline__ float to_storage<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_storage<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 to_storage<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float from_storage(float v) { return v; }
__device__ __forceinline__ float from_storage(__half v) { return __half2float(v); }
__device__ __forceinline__ float from_storage(__nv_bfloat16 v) { return __bfloat162float(v); }

// Pair layout: (P, Ht+1, Wt) records of (t[y][x], t[y][x+1] - t[y][x]); row Ht is zero.
template <typename OutT>
__global__ void atlas_pair_kernel(const float* __restrict__ tmpl, int P, int Ht, int Wt, OutT* __restrict__ out) {
  const long long total = (long long)P * (Ht + 1) * Wt;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % Wt);
    const int y = (int)((i / Wt) % (Ht + 1));
    const long long p = i / ((long long)(Ht + 1) * Wt);
    const float* t = tmpl + (size_t)p * Ht * Wt;
    const float v0 = (y < Ht) ? t[(size_t)y * Wt + x] : 0.f;
    const float v1 = (y < Ht && x + 1 < Wt) ? t[(size_t)y * Wt + x + 1] : 0.f;
    const OutT s0 = to_storage<OutT>(v0);
    out[2 * i] = s0;
    out[2 * i + 1] = to_storage<OutT>(v1 - from_storage(s0));
  }
}

// Quad layout: (P, Ht, Wt) records of (t[y][x], t[y][x+1] - t[y][x], t[y+1][x],
// t[y+1][x+1] - t[y+1][x]); neighbours outside the template are 0.
template <typename OutT>
__global__ void atlas_pack_kernel(const float* __restrict__ tmpl, int P, int Ht, int Wt, OutT* __restrict__ out) {
  const long long total = (long long)P * Ht * Wt;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % Wt);
    const int y = (int)((i / Wt) % Ht);
    const float* t = tmpl + (i - (long long)y * Wt - x);
    const bool xr = x + 1 < Wt, yr = y + 1 < Ht;
    const float v00 = t[(size_t)y * Wt + x];
    const float v01 = xr ? t[(size_t)y * Wt + x + 1] : 0.f;
    const float v10 = yr ? t[(size_t)(y + 1) * Wt + x] : 0.f;
    const float v11 = (xr && yr) ? t[(size_t)(y + 1) * Wt + x + 1] : 0.f;
    OutT* o = out + 4 * i;
    const OutT s00 = to_storage<OutT>(v00), s10 = to_storage<OutT>(v10);
    o[0] = s00; o[1] = to_storage<OutT>(v01 - from_storage(s00));
    o[2] = s10; o[3] = to_storage<OutT>(v11 - from_storage(s10));
  }
}

// ---------------------------------------------------------------------------
// Per-primitive preparation.
__device__ __forceinline__ float nan_min(float a, float b) { return (isnan(a) || isnan(b)) ? __int_as_float(0x7fc00000) : fminf(a, b); }
__device__ __forceinline__ float nan_max(float a, float b) { return (isnan(a) || isnan(b)) ? __int_as_float(0x7fc00000) : fmaxf(a, b); }

// Tile columns hit by [bmin, bmax] under the reference's inclusive test
// !(bmax < tile_start || bmin > tile_end) with tile_end = min(start+ts, W)
// compared in float32 (vector_renderer.py:437-438).  NaN makes the test pass.
__device__ __forceinline__ int2 tile_span_content(float bmin, float bmax, int ts, int extent, int ntiles) {
  auto ts_start = [&](int t) { return (float)(t * ts); };
  auto ts_end = [&](int t) { return (float)min(t * ts + ts, extent); };
  int lo, hi;
  if (isnan(bmin)) lo = 0;
  else if (bmin > (float)extent) lo = ntiles;
  else if (bmin <= 0.f) lo = 0;
  else {
    lo = max(0, (int)floorf(bmin / (float)ts) - 2);
    while (lo < ntiles && bmin > ts_end(lo)) ++lo;
  }
  if (isnan(bmax)) hi = ntiles - 1;
  else if (bmax < 0.f) hi = -1;
  else if (bmax >= ts_start(ntiles - 1)) hi = ntiles - 1;
  else {
    hi = min(ntiles - 1, (int)floorf(bmax / (float)ts) + 2);
    while (hi >= 0 && bmax < ts_start(hi)) --hi;
  }
  return make_int2(lo, hi);
}

// Pixels p in [0, extent) that pass the kernel's square cull
// !(fabsf((float)p - m) > h) (tile_forward.cu:208), as a tile span.  The
// predicate is monotone in |p - m|, so the passing pixels form an interval.
__device__ __forceinline__ int2 tile_span_cull(float m, float h, int ts, int extent) {
  auto pass = [&](int p) { return !(fabsf((float)p - m) > h); };
  if (isnan(m) || isnan(h)) return make_int2(0, (extent - 1) / ts);
  if (h < 0.f) return make_int2(1, 0);
  const float lo_f = fminf(fmaxf(floorf(m - h) - 2.f, 0.f), (float)extent);
  const float hi_f = fminf(fmaxf(ceilf(m + h) + 2.f, -1.f), (float)(extent - 1));
  int a = (int)lo_f, b = (int)hi_f;
  while (a <= b && !pass(a)) ++a;
  while (b >= a && !pass(b)) --b;
  if (a > b) return make_int2(1, 0);
  return make_int2(a / ts, b / ts);
}

// blockIdx.y: the candidate of a batch, whose inputs and outputs follow those
// of the one before (sel: sel_stride apart).  row_total (tilesY per candidate)
// is zeroed for counts_kernel, and the flags of a followed atlas for the walks.
__global__ void prepare_kernel(Geom g, const float* __restrict__ means2D, const float* __restrict__ radii,
                               const float* __restrict__ rot, const float* __restrict__ opac,
                               const float* __restrict__ colors, const int* __restrict__ sel, long long sel_stride,
                               const float* __restrict__ tbbox, int bin_mode, PrimInfo* __restrict__ out,
                               int4* __restrict__ rects, unsigned long long* __restrict__ row_total) {
  grid_dependency();
  if (g.changed != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) g.changed[threadIdx.x] = 0;
  const size_t b = blockIdx.y, bn = b * g.N;
  means2D += 2 * bn; radii += bn; rot += bn; opac += bn; colors += 3 * bn;
  sel += b * sel_stride;
  out += bn;
  if (rects != nullptr) {
    rects += bn;
    if (blockIdx.x == 0)
      for (int i = threadIdx.x; i < g.tilesY; i += blockDim.x) row_total[b * g.tilesY + i] = 0ull;
  }
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= g.N) return;
  const float mx = means2D[2 * n], my = means2D[2 * n + 1];
  const float r = radii[n], th = rot[n];
  const int tid = sel[n];
  const bool valid = tid >= 0 && tid < g.P;

  PrimInfo pi;
  pi.mx = mx; pi.my = my;
  // square cull half extents, in the reference's operation order (tile_forward.cu:198-205)
  const float maxd = fmaxf((float)g.Wt, (float)g.Ht);
  const float scale = __fdiv_rn(r, __fmul_rn(maxd, 0.5f));
  pi.hw = __fmul_rn(__fmul_rn((float)g.Wt, 0.5f), scale);
  pi.hh = __fmul_rn(__fmul_rn((float)g.Ht, 0.5f), scale);
  // inverse affine in double, rounded once (tile_forward.cu:250-264)
  const double rinv = (r > 1e-6f) ? 1.0 / (double)r : 1e6;
  double s, c;
  sincos((double)th, &s, &c);
  pi.a00 = (float)(c * rinv * (double)g.hx);
  pi.a01 = (float)(s * rinv * (double)g.hx);
  pi.a10 = (float)(-s * rinv * (double)g.hy);
  pi.a11 = (float)(c * rinv * (double)g.hy);
  pi.alpha0 = g.alpha_max * sigmoid_precise(opac[n]);
  pi.cr = sigmoid_precise(colors[3 * n + 0]);
  pi.cg = sigmoid_precise(colors[3 * n + 1]);
  pi.cb = sigmoid_precise(colors[3 * n + 2]);
  if (half_record(g.kind)) {   // the precision form stores opacity and colours in FP16
    const __half2 ar = __floats2half2_rn(pi.alpha0, pi.cr), gb = __floats2half2_rn(pi.cg, pi.cb);
    pi.alpha0 = __uint_as_float(*reinterpret_cast<const unsigned*>(&ar));
    pi.cr = __uint_as_float(*reinterpret_cast<const unsigned*>(&gb));
    pi.cg = pi.cb = 0.f;
  }
  const bool nan_geom = isnan(pi.a00) || isnan(pi.a01) || isnan(pi.a10) || isnan(pi.a11) || isnan(mx) || isnan(my);
  pi.toff = (!valid || nan_geom) ? kNoFrag : tid * template_records(g.kind, g.Ht, g.Wt);
  // clearance a warp footprint needs before the walk may skip it: the
  // footprint's texel-space half extent, plus the bilinear reach of 1 texel,
  // plus slack for the rounding of the per-pixel texel coordinates
  const float ex = fabsf(pi.a00) * g.fhx + fabsf(pi.a01) * g.fhy;
  const float ey = fabsf(pi.a10) * g.fhx + fabsf(pi.a11) * g.fhy;
  const float need = fmaxf(ex, ey) + 1.05f;
  pi.goff = valid ? tid * g.gGx * g.gGy : 0;
  pi.gext = (atlas_has_grid(g.kind) && need < (float)kGridCap) ? (int)ceilf(need) : kGridCap + 1;
  pi.pad = 0;
  out[n] = pi;

  if (rects == nullptr) return;
  int2 sx, sy;
  if (bin_mode == DBMP_BIN_CONTENT || bin_mode == DBMP_BIN_CONTENT_REF) {
    // vector_renderer.py:221-250 with the bbox of this primitive's template,
    // or, in the reference-exact mode, of template (N-1-n) % P as the
    // reference always takes it (vector_renderer.py:220-226)
    const int q = (bin_mode == DBMP_BIN_CONTENT_REF) ? (g.N - 1 - n) % g.P : (valid ? tid : 0);
    const float c32 = cosf(th), s32 = sinf(th);
    const float cu[4] = {tbbox[4 * q + 0], tbbox[4 * q + 1], tbbox[4 * q + 0], tbbox[4 * q + 1]};
    const float cv[4] = {tbbox[4 * q + 2], tbbox[4 * q + 2], tbbox[4 * q + 3], tbbox[4 * q + 3]};
    float xmn = 0.f, xmx = 0.f, ymn = 0.f, ymx = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float wx = __fadd_rn(mx, __fmul_rn(r, __fsub_rn(__fmul_rn(cu[k], c32), __fmul_rn(cv[k], s32))));
      const float wy = __fadd_rn(my, __fmul_rn(r, __fadd_rn(__fmul_rn(cu[k], s32), __fmul_rn(cv[k], c32))));
      if (k == 0) { xmn = xmx = wx; ymn = ymx = wy; }
      else { xmn = nan_min(xmn, wx); xmx = nan_max(xmx, wx); ymn = nan_min(ymn, wy); ymx = nan_max(ymx, wy); }
    }
    sx = tile_span_content(xmn, xmx, g.TS, g.W, g.tilesX);
    sy = tile_span_content(ymn, ymx, g.TS, g.H, g.tilesY);
  } else {
    if (valid) {
      sx = tile_span_cull(mx, pi.hw, g.TS, g.W);
      sy = tile_span_cull(my, pi.hh, g.TS, g.H);
    } else {
      sx = make_int2(1, 0); sy = make_int2(1, 0);
    }
  }
  rects[n] = make_int4(sx.x, sx.y, sy.x, sy.y);
}

// Tile lists, four launches (prepare, counts, offsets, rows).  Counts: one CTA per
// primitive slice marks its rectangles' corners in a 2-D difference array in
// shared memory and prefix-sums it into counts[t * S + part], the number of
// the slice's rectangles covering tile t (S counting slices), and adds each tile row's sum to
// row_total.
// Write: one CTA per (tile row, group of kBinGroup tiles, primitive slice),
// kBinTPW tiles per warp (warp w: tiles w + k kBinWarps of the group).  The CTA
// walks the primitives of its slice in index order in chunks of
// kBinThreads, compacts those whose rectangle covers its row and overlaps its
// tile group, and each warp writes the ids of the compacted rectangles
// containing each of its tiles, so a tile's entries come out in ascending
// primitive order.  Two tiles per warp halve the per-tile share of the row
// filter, compaction and count scan (write pass 39.8 -> 29.4 us at 2048x2048,
// N=20000 on a B200).  The write pass also publishes tile_offsets, L and the
// overflow flag, and leaves the outputs untouched when L exceeds the capacity.
// The write loop is bound by its instructions: write positions are pointers and
// the compaction buffer is padded, so that it holds neither 64-bit index sums nor
// bounds tests.  Replayed from a graph: 16.5 -> 11.3 us at 256x256, N=512;
// 20.5 -> 14.1 at 1024x1024, N=5000 (against a memset, a difference array in global
// memory and a library scan of all counts, six launches); with the masks of
// use_masks 49.0 -> 34.2 at 2048x2048, N=20000 and 487 -> 268 at 4096x4096, N=100000.
constexpr int kBinThreads = 512;
constexpr int kBinWarps = kBinThreads / 32;
constexpr int kBinTPW = 2;                       // tiles per warp
constexpr int kBinGroup = kBinTPW * kBinWarps;   // tiles per CTA

struct BinGrid {
  int groups;   // tile groups per row
  int slices;   // primitive slices
  int span;     // primitives per slice (multiple of kBinThreads)
  int subs;     // counting slices per slice
  int cspan;    // primitives per counting slice
  int words;    // 32-bit words of a cell's primitive mask (0: lists written without masks)
  long long ctas;
};

constexpr size_t kCountsSmem = 200 * 1024;
// A masking CTA: its primitives, their words, and its words of shared memory
// (an odd stride, so that a cell's words lie in different banks).
constexpr int kMaskPrims = kBinThreads, kMaskWords = kMaskPrims / 32;
__host__ __device__ static inline size_t mask_stride(int cells) { return (size_t)cells | 1; }

// Whether lists are written from primitive masks of the cells (tile row, group of
// kBinGroup tiles).  Testing every rectangle in every cell costs cells x chunks,
// marking the masks about as much as the lists are long.  By cells x chunks, without
// and with masks (whole binning, us): 1280 (1024x1024, N=20000) 22.9 / 24.3; 1536
// (2048x2048, N=6000) 25.1 / 25.6; 1760 (1024x1024, N=28000) 28.7 / 27.7; 5120
// (2048x2048, N=20000) 45.1 / 36.6; 100352 (4096x4096, N=100000) 437 / 281.  With
// few chunks there is less to skip: 512 x 4 (4096x4096, N=2000) 33.3 / 35.3; 1128 x 4
// (6000x6000, N=2000) 58.8 / 50.1; 2538 x 1 (9000x9000, N=500) even.  The
// marks of a masking CTA have to fit its shared memory (cells up to 3200, canvases
// to about 10000x10000 at tile 32), and the masks 64 MB of workspace.
static inline bool use_masks(long long cells, int chunks) {
  return chunks >= 3 && cells * chunks >= (chunks < 8 ? 2560 : 1600) && cells * chunks <= (1ll << 20) &&
         cells <= INT_MAX && mask_stride((int)cells) * kMaskWords * sizeof(unsigned) <= kCountsSmem;
}

// Enough slices to give every SM several CTAs (with masks, where a CTA has little
// to do per primitive, half as many: 36.6 us against 39.1 at 2048x2048, N=20000),
// never a slice below one chunk.
static inline BinGrid bin_grid(int N, int tilesX, int tilesY) {
  BinGrid b;
  b.groups = (tilesX + kBinGroup - 1) / kBinGroup;
  const long long base = (long long)b.groups * tilesY;
  const int chunks = N > 0 ? (N + kBinThreads - 1) / kBinThreads : 1;
  b.words = use_masks(base, chunks) ? chunks * kMaskWords : 0;
  const long long want = (148 * (b.words ? 4 : 8) + base - 1) / base;
  b.slices = (int)(want < chunks ? want : chunks);
  if (b.slices < 1) b.slices = 1;
  const int per = (chunks + b.slices - 1) / b.slices;
  b.span = per * kBinThreads;
  b.slices = N > 0 ? (N + b.span - 1) / b.span : 1;
  // counted in up to 64 finer slices: a counting CTA's shared-memory adds run at
  // about one rectangle per 30 cycles (100,000 rectangles: 3 CTAs take 110 us, 49
  // take 9), but every writing CTA sums the counts left of its tiles
  int cspan = (N + 63) / 64 > kBinThreads ? (N + 63) / 64 : kBinThreads;
  if (cspan > b.span) cspan = b.span;
  b.subs = (b.span + cspan - 1) / cspan;
  b.cspan = (b.span + b.subs - 1) / b.subs;
  b.ctas = base * b.slices;
  return b;
}

// The part of the counting launch that marks, for each cell (tile row, group of
// kBinGroup tiles), which of kMaskPrims primitives touch it, and writes the cells'
// words of masks[cell][word].  Two threads per primitive, one for every other row
// of its rectangle, each lane of a warp starting at another row, so that lanes with
// tall rectangles rarely meet in a word.
__device__ __forceinline__ void mask_rects(const Geom& g, const BinGrid& bg, const int4* __restrict__ rects,
                                           unsigned* s, int block, unsigned* __restrict__ masks) {
  const int cells = bg.groups * g.tilesY;
  const int stride = (int)mask_stride(cells);
  for (int i = threadIdx.x; i < stride * kMaskWords; i += blockDim.x) s[i] = 0u;
  __syncthreads();
  const int own = threadIdx.x % kMaskPrims, n = block * kMaskPrims + own;
  if (n < g.N) {
    const int4 rc = rects[n];
    if (rc.x <= rc.y && rc.z <= rc.w) {
      const int g0 = rc.x / kBinGroup, g1 = rc.y / kBinGroup, h = rc.w - rc.z + 1;
      unsigned* mine = s + (own >> 5) * stride;
      const unsigned bit = 1u << (own & 31);
      int y = (own & 31) % h;
      for (int i = 0; i < h; ++i) {
        if ((i & 1) == threadIdx.x / kMaskPrims)
          for (int q = g0; q <= g1; ++q) atomicOr(mine + (rc.z + y) * bg.groups + q, bit);
        y = y + 1 == h ? 0 : y + 1;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cells * kMaskWords; i += blockDim.x) {
    const int cell = i / kMaskWords, w = i % kMaskWords;
    masks[(size_t)cell * bg.words + block * kMaskWords + w] = s[w * stride + cell];
  }
}

// One CTA per (counting slice, candidate); slice s has counting slices s subs to
// s subs + subs - 1.  The difference array of (tilesY+1) x
// (tilesX+1) counters sits in dynamic shared memory, or, for canvases beyond
// about 7500 x 7500 pixels at tile 32, in the slice's own part of scratch.
// Rows are scanned by whole warps (shuffle scans over 32-column chunks), then
// columns the same way.
__global__ void __launch_bounds__(1024) counts_kernel(Geom g, BinGrid bg, const int4* __restrict__ rects,
                                                      int* __restrict__ scratch, int* __restrict__ counts,
                                                      unsigned long long* __restrict__ row_total,
                                                      unsigned* __restrict__ masks, Follow follow) {
  extern __shared__ int s_diff[];
  grid_dependency();
  const int part = blockIdx.x, parts = bg.slices * bg.subs;   // counting slice
  const size_t b = blockIdx.y;
  if (part >= parts + bg.words / kMaskWords) {                // the CTAs behind the marking ones
    if (b == 0) follow_compare(follow, part - parts - bg.words / kMaskWords);
    return;
  }
  if (part >= parts) {
    mask_rects(g, bg, rects + b * g.N, (unsigned*)s_diff, part - parts,
               masks + b * ((size_t)bg.groups * g.tilesY * bg.words));
    return;
  }
  const int gw = g.tilesX + 1;
  const int cells = (g.tilesY + 1) * gw;
  int* d = scratch ? scratch + (b * parts + part) * cells : s_diff;
  rects += b * g.N;
  counts += b * g.T * parts;
  row_total += b * g.tilesY;
  for (int i = threadIdx.x; i < cells; i += blockDim.x) d[i] = 0;
  __syncthreads();
  // the rectangles' corners; the array's 2-D prefix sum is the number of
  // rectangles covering each tile
  const int slice = part / bg.subs, sub = part - slice * bg.subs;
  const int lo = slice * bg.span + sub * bg.cspan;
  const int hi = min(g.N, min(lo + bg.cspan, (slice + 1) * bg.span));
  for (int n = lo + threadIdx.x; n < hi; n += blockDim.x) {
    const int4 rc = rects[n];
    if (rc.x <= rc.y && rc.z <= rc.w) {
      atomicAdd(d + rc.z * gw + rc.x, 1);
      atomicAdd(d + rc.z * gw + rc.y + 1, -1);
      atomicAdd(d + (rc.w + 1) * gw + rc.x, -1);
      atomicAdd(d + (rc.w + 1) * gw + rc.y + 1, 1);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  auto scan = [&](int* p, int len, int stride) {   // inclusive prefix sum of p[0], p[stride], ... by one warp
    int carry = 0;
    for (int i0 = 0; i0 < len; i0 += 32) {
      const int i = i0 + lane;
      int v = i < len ? p[(size_t)i * stride] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      v += carry;
      if (i < len) p[(size_t)i * stride] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  };
  for (int y = warp; y < g.tilesY; y += nwarps) scan(d + y * gw, g.tilesX, 1);
  __syncthreads();
  for (int x = warp; x < g.tilesX; x += nwarps) scan(d + x, g.tilesY, gw);
  __syncthreads();
  for (int y = warp; y < g.tilesY; y += nwarps) {
    unsigned long long sum = 0;
    for (int x = lane; x < g.tilesX; x += 32) {
      const int v = d[y * gw + x];
      counts[((size_t)y * g.tilesX + x) * parts + part] = v;
      sum += (unsigned long long)v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && sum) atomicAdd(row_total + y, sum);
  }
}

// One CTA per (tile row, candidate): the list position of each (tile, writing
// slice) of the row, offs[t * S + slice] (tile-major, slice-minor over the
// canvas), from the totals of the rows above and a scan over the row's counts.
// The last row's CTA also writes offs[T * S] = L.
// PER counts per thread and round: as few as a round needs to take the whole row, up
// to eight (whole binning with 1 / 4 / 8: 14.1 / 14.7 / 15.3 us at 1024x1024, N=5000,
// 320 counts in a row; 36.5 / 34.9 / 34.1 at 2048x2048, N=20000, 2560 counts; 282 /
// 272 / 268 at 4096x4096, N=100000, 8192).
constexpr int kOffsThreads = 512;

template <int PER>
__global__ void __launch_bounds__(kOffsThreads) offsets_kernel(Geom g, BinGrid bg, const int* __restrict__ counts,
                                                               const unsigned long long* __restrict__ row_total,
                                                               long long* __restrict__ offs) {
  __shared__ long long s_base;
  __shared__ int s_warp[kOffsThreads / 32];
  grid_dependency();
  const int ty = blockIdx.x;
  const size_t cand = blockIdx.y;
  const int parts = bg.slices * bg.subs;
  counts += (cand * g.T + (size_t)ty * g.tilesX) * parts;
  row_total += cand * g.tilesY;
  offs += cand * ((size_t)g.T * bg.slices + 1) + (size_t)ty * g.tilesX * bg.slices;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    long long above = 0;
    for (int y = lane; y < ty; y += 32) above += (long long)row_total[y];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) above += __shfl_xor_sync(0xffffffffu, above, o);
    if (lane == 0) {
      s_base = above;
      if (ty == g.tilesY - 1) offs[(size_t)g.tilesX * bg.slices] = above + (long long)row_total[ty];
    }
  }
  const int len = g.tilesX * parts;
  long long carry = 0;
  for (int i0 = 0; i0 < len; i0 += kOffsThreads * PER) {
    const int first = i0 + threadIdx.x * PER;
    int own[PER], v = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      own[k] = first + k < len ? counts[first + k] : 0;
      v += own[k];
    }
    const int mine = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    int w = lane < kOffsThreads / 32 ? s_warp[lane] : 0;   // inclusive prefix of the warps' sums, one per lane
#pragma unroll
    for (int o = 1; o < kOffsThreads / 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    const int before = warp > 0 ? __shfl_sync(0xffffffffu, w, warp - 1) : 0;
    const int total = __shfl_sync(0xffffffffu, w, kOffsThreads / 32 - 1);
    long long at = s_base + carry + before + v - mine;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = first + k;
      if (i < len && i % bg.subs == 0) offs[i / bg.subs] = at;
      at += own[k];
    }
    carry += total;
    __syncthreads();   // s_warp is rewritten by the next round
  }
}

// What the writing kernels share.  A CTA's cell and slice, and of its warps' tiles
// gx0 + warp + k kBinWarps: the column a rectangle must reach (INT_MAX for a tile
// past the canvas, which no rectangle contains) and the next write position.
struct BinTiles {
  int slice, ty, gx0, gx1;
  int col[kBinTPW];
  int* cur[kBinTPW];

  // Publishes tile_offsets, L and the overflow flag; false when the lists do not fit.
  __device__ __forceinline__ bool open(const Geom& g, const BinGrid& bg, const long long* __restrict__ offs,
                                       long long cap, int* __restrict__ indices, long long index_stride,
                                       int* __restrict__ tile_offsets, int* __restrict__ total_out,
                                       int* __restrict__ overflow_out, long long flag_stride,
                                       volatile int* host_flags, const int* changed) {
    const size_t cand = blockIdx.y;   // candidate of a batch
    const long long nslots = (long long)g.T * bg.slices;
    offs += cand * (nslots + 1);
    indices += cand * index_stride;
    tile_offsets += cand * (g.T + 1);
    slice = blockIdx.x % bg.slices;
    const int rg = blockIdx.x / bg.slices;
    ty = rg / bg.groups;
    gx0 = (rg - ty * bg.groups) * kBinGroup;
    gx1 = min(gx0 + kBinGroup - 1, g.tilesX - 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long L = offs[nslots];
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (first) {
      if (total_out) total_out[cand * flag_stride] = (int)min(L, (long long)INT_MAX);
      if (overflow_out) overflow_out[cand * flag_stride] = (L > cap) ? 1 : 0;
      if (host_flags) {   // the host polls the second word
        host_flags[2 * cand] = (int)min(L, (long long)INT_MAX);
        __threadfence_system();
        // (bit 1: a followed atlas's templates have changed, and the host calls again)
        host_flags[2 * cand + 1] = (L > cap ? 1 : 0) | (changed != nullptr && follow_changed(changed) ? 2 : 0);
        __threadfence_system();
      }
    }
    if (L > cap) return false;   // uniform over the CTA
    if (first) tile_offsets[g.T] = (int)L;
#pragma unroll
    for (int k = 0; k < kBinTPW; ++k) {
      const int tx = gx0 + warp + k * kBinWarps;
      col[k] = INT_MAX;
      cur[k] = indices;
      if (tx <= gx1) {
        const int t = ty * g.tilesX + tx;
        const long long at = offs[(long long)t * bg.slices + slice];
        col[k] = tx;
        cur[k] = indices + at;
        if (lane == 0 && slice == 0) tile_offsets[t] = (int)at;
      }
    }
    return true;
  }

  // Appends the ids of those of the compacted rectangles (padded to a multiple of
  // 32 with empty ones) that contain each of the warp's tiles.
  __device__ __forceinline__ void append(const int* s_id, const int2* s_xr, int padded) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    for (int j = lane; j < padded; j += 32) {
      const int2 xr = s_xr[j];
      const int id = s_id[j];   // (not set in the padding, nor used there)
#pragma unroll
      for (int k = 0; k < kBinTPW; ++k) {
        const bool in = xr.x <= col[k] && col[k] <= xr.y;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) cur[k][__popc(m & lt)] = id;
        cur[k] += __popc(m);
      }
    }
  }
};

// The lists from the cells' primitive masks: a thread expands the bits of a word of
// its CTA's slice into the compaction buffer, so that a chunk is kBinThreads words,
// 16384 primitives, where testing every rectangle of the canvas in every cell takes
// a chunk per kBinThreads rectangles (4096x4096, N=100000, L=167e6: binning 437 ->
// 281 us, of which writing the lists takes 103 at the copy rate).  What is left is
// mostly the write loop's population counts.  Not faster: their sums as byte
// counters of four tiles in a shuffle scan (321 us), four tiles per warp (329).
constexpr int kMaskBuffer = 2048;

__global__ void __launch_bounds__(kBinThreads, 3) bin_masks_kernel(
    Geom g, BinGrid bg, const int4* __restrict__ rects, const unsigned* __restrict__ masks,
    const long long* __restrict__ offs, long long cap, int* __restrict__ indices, long long index_stride,
    int* __restrict__ tile_offsets, int* __restrict__ total_out, int* __restrict__ overflow_out, long long flag_stride,
    volatile int* host_flags, const int* changed) {
  __shared__ int s_id[kMaskBuffer];
  __shared__ int2 s_xr[kMaskBuffer];   // the rectangle's tile columns x0, x1
  __shared__ int s_wcnt[kBinWarps];
  grid_dependency();
  BinTiles bt;
  if (!bt.open(g, bg, offs, cap, indices, index_stride, tile_offsets, total_out, overflow_out, flag_stride, host_flags,
               changed))
    return;
  rects += (size_t)blockIdx.y * g.N;
  const int cell = blockIdx.x / bg.slices, cells = bg.groups * g.tilesY;
  masks += ((size_t)blockIdx.y * cells + cell) * bg.words;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lo = bt.slice * (bg.span / 32), hi = min(bg.words, lo + bg.span / 32);
  for (int w0 = lo; w0 < hi; w0 += kBinThreads) {
    const int w = w0 + (int)threadIdx.x;
    unsigned word = w < hi ? masks[w] : 0u;
    int inc = __popc(word);
    const int own = inc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) s_wcnt[warp] = inc;
    __syncthreads();
    int sum = lane < kBinWarps ? s_wcnt[lane] : 0;
#pragma unroll
    for (int o = 1; o < kBinWarps; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += u;
    }
    const int total = __shfl_sync(0xffffffffu, sum, kBinWarps - 1);
    int at = inc - own + (warp == 0 ? 0 : __shfl_sync(0xffffffffu, sum, warp - 1));   // this word's first entry
    for (int base = 0; base < total; base += kMaskBuffer) {
      const int count = min(kMaskBuffer, total - base), padded = (count + 31) & ~31;
      while (word != 0u && at < base + kMaskBuffer) {
        s_id[at++ - base] = (w << 5) + __ffs(word) - 1;
        word &= word - 1u;
      }
      __syncthreads();
      for (int j = threadIdx.x; j < padded; j += kBinThreads) {
        int2 xr = make_int2(1, 0);   // contains no column
        if (j < count) xr = *reinterpret_cast<const int2*>(rects + s_id[j]);
        s_xr[j] = xr;
      }
      __syncthreads();
      bt.append(s_id, s_xr, padded);
      __syncthreads();
    }
    __syncthreads();   // s_wcnt is rewritten by the next round
  }
}

__global__ void __launch_bounds__(kBinThreads, 3) bin_rows_kernel(Geom g, BinGrid bg,
                                                                  const int4* __restrict__ rects,
                                                                  const long long* __restrict__ offs, long long cap,
                                                                  int* __restrict__ indices, long long index_stride,
                                                                  int* __restrict__ tile_offsets,
                                                                  int* __restrict__ total_out,
                                                                  int* __restrict__ overflow_out,
                                                                  long long flag_stride,
                                                                  volatile int* host_flags,
                                                                  const int* changed) {
  // Two compaction buffers: chunk c is compacted into buffer c & 1 while the
  // warps may still read chunk c - 1 from the other one, so one barrier per
  // chunk orders everything (see the loop).
  __shared__ int s_id[2][kBinThreads];
  __shared__ int2 s_xr[2][kBinThreads];   // the rectangle's tile columns x0, x1
  __shared__ int s_wcnt[2][kBinWarps];
  grid_dependency();
  BinTiles bt;
  if (!bt.open(g, bg, offs, cap, indices, index_stride, tile_offsets, total_out, overflow_out, flag_stride, host_flags,
               changed))
    return;
  rects += (size_t)blockIdx.y * g.N;
  const int slice = bt.slice, ty = bt.ty, gx0 = bt.gx0, gx1 = bt.gx1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int lo = slice * bg.span, hi = min(g.N, lo + bg.span);
  const int4 none = make_int4(1, 0, 1, 0);
  // a rectangle survives the CTA's test when it covers row ty and overlaps the tile group
  auto covers = [&](const int4& rc) { return rc.x <= rc.y && rc.z <= ty && ty <= rc.w && rc.x <= gx1 && rc.y >= gx0; };
  // chunk lo: test, count; the rectangles of the next chunk are loaded one chunk ahead
  int n = lo + (int)threadIdx.x;
  int4 rc = n < hi ? rects[n] : none;
  int4 rn = n + kBinThreads < hi ? rects[n + kBinThreads] : none;
  bool f = n < hi && covers(rc);
  unsigned b = __ballot_sync(0xffffffffu, f);
  if (lane == 0) s_wcnt[0][warp] = __popc(b);
  __syncthreads();
  int buf = 0;
  for (int base = lo; base < hi; base += kBinThreads, buf ^= 1) {
    // (1) compact chunk base into buffer buf (its counts were published before
    // the last barrier): lane w < kBinWarps scans the counts of warps 0..w
    int inc = lane < kBinWarps ? s_wcnt[buf][lane] : 0;
#pragma unroll
    for (int o = 1; o < kBinWarps; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const int total = __shfl_sync(0xffffffffu, inc, kBinWarps - 1);
    const int wbase = warp == 0 ? 0 : __shfl_sync(0xffffffffu, inc, warp - 1);
    if (f) {
      const int p = wbase + __popc(b & lt);
      s_id[buf][p] = n;
      s_xr[buf][p] = make_int2(rc.x, rc.y);
    }
    // pad the last group of 32 with rectangles that contain no column
    const int padded = (total + 31) & ~31;
    if ((int)threadIdx.x >= total && (int)threadIdx.x < padded) s_xr[buf][threadIdx.x] = make_int2(1, 0);
    // (2) test and count the next chunk, and load the one after it
    n += kBinThreads;
    rc = rn;
    rn = n + kBinThreads < hi ? rects[n + kBinThreads] : none;
    f = n < hi && covers(rc);
    b = __ballot_sync(0xffffffffu, f);
    if (lane == 0) s_wcnt[buf ^ 1][warp] = __popc(b);
    // One barrier per chunk.  After it, buffer buf holds chunk base and
    // s_wcnt[buf ^ 1] the next chunk's counts.  The next iteration writes
    // buffer buf ^ 1, last read by this iteration's predecessor (before this
    // barrier), and s_wcnt[buf], last read in (1) above (before this barrier).
    __syncthreads();
    // (3) each warp writes the compacted rectangles that contain its tiles
    bt.append(s_id[buf], s_xr[buf], padded);
  }
}

// ---------------------------------------------------------------------------
struct BinWorkspace {
  int4* rects;                     // N tile rectangles (x0, x1, y0, y1) per candidate
  int* counts;                     // (tile, counting slice) entries per candidate
  long long* offs;                 // list positions per (tile, writing slice), and L, per candidate
  unsigned long long* row_total;   // tilesY list lengths of the tile rows per candidate
  unsigned* masks;                 // primitive masks of the cells per candidate (null without)
  int* scratch;                    // difference arrays that do not fit shared memory (null otherwise)
};

static inline size_t align_up(size_t v) { return (v + 255) & ~(size_t)255; }

static inline size_t diff_cells_bytes(int tilesX, int tilesY) {
  return sizeof(int) * (size_t)(tilesY + 1) * (tilesX + 1);
}

// Lays the workspace out from base and returns its size.
static size_t layout_ws(void* base, int batch, int N, int T, int tilesX, int tilesY, const BinGrid& bg,
                        BinWorkspace* w) {
  const size_t B = batch, parts = (size_t)bg.slices * bg.subs;
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += align_up(bytes); return o; };
  const size_t o_rects = take(sizeof(int4) * B * (N > 0 ? N : 1));
  const size_t o_counts = take(sizeof(int) * B * T * parts);
  const size_t o_offs = take(sizeof(long long) * B * ((size_t)T * bg.slices + 1));
  const size_t o_rows = take(sizeof(unsigned long long) * B * tilesY);
  const size_t mask_words = (size_t)bg.groups * tilesY * bg.words;
  const size_t o_masks = mask_words ? take(sizeof(unsigned) * B * mask_words) : 0;
  const size_t cells = diff_cells_bytes(tilesX, tilesY);
  const size_t o_scratch = cells > kCountsSmem ? take(cells * B * parts) : 0;
  if (w) {
    char* b = static_cast<char*>(base);
    w->rects = reinterpret_cast<int4*>(b + o_rects);
    w->counts = reinterpret_cast<int*>(b + o_counts);
    w->offs = reinterpret_cast<long long*>(b + o_offs);
    w->row_total = reinterpret_cast<unsigned long long*>(b + o_rows);
    w->masks = mask_words ? reinterpret_cast<unsigned*>(b + o_masks) : nullptr;
    w->scratch = cells > kCountsSmem ? reinterpret_cast<int*>(b + o_scratch) : nullptr;
  }
  return off;
}

size_t bin_workspace_bytes(int batch, int N, int T, int tilesX, int tilesY) {
  return layout_ws(nullptr, batch, N, T, tilesX, tilesY, bin_grid(N, tilesX, tilesY), nullptr);
}

int launch_template_bboxes(const float* tmpl, int P, int Ht, int Wt, float* out, cudaStream_t st) {
  if (P <= 0) return DBMP_OK;
  template_bbox_kernel<<<P, 256, 0, st>>>(tmpl, Ht, Wt, out);
  DBMP_CHECK_LAUNCH("template_bbox_kernel");
  return DBMP_OK;
}

size_t atlas_bytes(int P, int Ht, int Wt, int kind) {
  if (kind < ATLAS_F32 || kind > ATLAS_BF16_PAIR) return 0;
  if (!atlas_has_grid(kind)) return atlas_record_bytes(P, Ht, Wt, kind);
  int sx, sy, gx, gy;
  grid_shape(Wt, &sx, &gx);
  grid_shape(Ht, &sy, &gy);
  return atlas_grid_offset(P, Ht, Wt, kind) + (size_t)P * gx * gy;
}

// Clearance grid and, with SOLID, the solid grid of the same cells (layouts in
// dbmp_internal.cuh), one CTA per (template, strip of cell rows).
// Bounding texels are the support texels, respectively the texels other than
// exactly 1 (NaN counts as either).  First a warp takes each template row that
// can matter to the strip (up to kGridCap-1 rows beyond it): ballots turn the
// row into bit masks, and each cell column's distance to the row's nearest
// bounding texel comes from the 64-bit windows left and right of the cell.
// Then each cell takes the minimum over rows of max(row distance, y-distance),
// going outwards until the y-distance alone reaches its minimum.  1024 templates
// of 256x256 take 1.4 ms; scanning every texel within reach of a cell column for
// each row, as one CTA per (cell column, template), took 4.6 ms.  With few
// templates the kernel is latency-bound (8 of 128x128: 20 us).
constexpr int kGridThreads = 1024;   // latency-bound: a warp's rows and a thread's cells run in series

struct GridArgs {
  int Ht, Wt, gsx, gsy, Gx, Gy;
  int strip;   // cell rows of a CTA
  int words;   // 32-bit words of a row's mask: Wt bits, rounded up, and 5 zero words (2 before, 3 after)
  int rows;    // template rows of a strip at most
  unsigned char* grid;
  unsigned char* solid;
};

// Bits [pos, pos + 64) of a mask with two zero words before bit 0 (pos >= -64).
__device__ __forceinline__ unsigned long long mask_window(const unsigned* m, int pos) {
  const int q = pos + 64, w = q >> 5, s = q & 31;
  const unsigned a = __funnelshift_r(m[w], m[w + 1], s), b = __funnelshift_r(m[w + 1], m[w + 2], s);
  return ((unsigned long long)b << 32) | a;
}

// Distance of the cell range [lo, hi] to the nearest set bit, capped at kGridCap.
__device__ __forceinline__ int mask_distance(const unsigned* m, int lo, int hi) {
  for (int x = lo; x <= hi; x += 64) {
    unsigned long long v = mask_window(m, x);
    if (hi - x < 63) v &= (2ull << (hi - x)) - 1ull;
    if (v) return 0;
  }
  const unsigned long long l = mask_window(m, lo - 64), r = mask_window(m, hi + 1);
  const int dl = l ? __clzll((long long)l) + 1 : kGridCap, dr = r ? __ffsll((long long)r) : kGridCap;
  return min(min(dl, dr), kGridCap);
}

template <bool SOLID>
__global__ void __launch_bounds__(kGridThreads) atlas_grid_kernel(const float* __restrict__ tmpl, GridArgs a) {
  extern __shared__ unsigned s_mem[];
  constexpr int K = SOLID ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  unsigned* mask = s_mem + (size_t)warp * K * a.words;                             // this warp's row masks
  unsigned char* dist = reinterpret_cast<unsigned char*>(s_mem + (size_t)nwarps * K * a.words);   // K x rows x Gx
  const int strips = (a.Gy + a.strip - 1) / a.strip;
  const int p = blockIdx.x / strips;
  const float* t = tmpl + (size_t)p * a.Ht * a.Wt;
  const int c0 = (blockIdx.x - p * strips) * a.strip, c1 = min(c0 + a.strip, a.Gy);
  const int y0 = max(0, (c0 << a.gsy) - (kGridCap - 1)), y1 = min(a.Ht - 1, (c1 << a.gsy) + (kGridCap - 1));
  for (int i = lane; i < K * a.words; i += 32) mask[i] = 0u;
  __syncwarp();
  for (int y = y0 + warp; y <= y1; y += nwarps) {
    const float* row = t + (size_t)y * a.Wt;
#pragma unroll 4
    for (int x0 = 0; x0 < a.Wt; x0 += 32) {
      const bool in = x0 + lane < a.Wt;
      const float v = in ? row[x0 + lane] : 0.f;
      const unsigned b = __ballot_sync(0xffffffffu, in && !(v <= kGridSupport));
      const unsigned c = SOLID ? __ballot_sync(0xffffffffu, in && !(v == 1.f)) : 0u;
      if (lane == 0) {
        mask[2 + (x0 >> 5)] = b;
        if (SOLID) mask[a.words + 2 + (x0 >> 5)] = c;
      }
    }
    __syncwarp();
    for (int ix = lane; ix < a.Gx; ix += 32) {
      const int lo = ix << a.gsx, hi = min((ix + 1) << a.gsx, a.Wt - 1);
      dist[(size_t)(y - y0) * a.Gx + ix] = (unsigned char)mask_distance(mask, lo, hi);
      if (SOLID) dist[(size_t)(a.rows + y - y0) * a.Gx + ix] = (unsigned char)mask_distance(mask + a.words, lo, hi);
    }
    __syncwarp();   // the masks are rewritten for the next row
  }
  __syncthreads();
  for (int i = threadIdx.x; i < K * (c1 - c0) * a.Gx; i += blockDim.x) {
    const int k = i / ((c1 - c0) * a.Gx), j = i - k * (c1 - c0) * a.Gx;
    const int iy = c0 + j / a.Gx, ix = j % a.Gx;
    const int ylo = iy << a.gsy, yhi = min((iy + 1) << a.gsy, a.Ht - 1);
    const unsigned char* d = dist + (size_t)k * a.rows * a.Gx + ix;
    int best = kGridCap;
    for (int y = ylo; y <= yhi; ++y) best = min(best, (int)d[(size_t)(y - y0) * a.Gx]);
    for (int e = 1; e < best; ++e) {
      int m = kGridCap;
      if (ylo - e >= y0) m = d[(size_t)(ylo - e - y0) * a.Gx];
      if (yhi + e <= y1) m = min(m, (int)d[(size_t)(yhi + e - y0) * a.Gx]);
      best = min(best, max(m, e));
    }
    (k == 0 ? a.grid : a.solid)[((size_t)p * a.Gy + iy) * a.Gx + ix] = (unsigned char)best;
  }
}

// The grids of a packed atlas of kind `kind` at `out`; solid_off: the solid grid's byte offset there (0: none).
static int launch_grids(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, size_t solid_off,
                        cudaStream_t st) {
  GridArgs a;
  a.Ht = Ht;
  a.Wt = Wt;
  grid_shape(Wt, &a.gsx, &a.Gx);
  grid_shape(Ht, &a.gsy, &a.Gy);
  a.grid = static_cast<unsigned char*>(out) + atlas_grid_offset(P, Ht, Wt, kind);
  a.solid = solid_off ? static_cast<unsigned char*>(out) + solid_off : nullptr;
  a.words = (Wt + 31) / 32 + 5;
  const int k = a.solid ? 2 : 1;
  const size_t row_bytes = (size_t)k * a.words * 4;
  constexpr size_t kSmem = 224 * 1024;
  // strips of 32 cell rows, or fewer while the grid has less than two CTAs per
  // SM (a shorter strip scans more rows beyond it per row of its own) or the
  // row distances do not fit
  size_t smem = 0;
  int warps = kGridThreads / 32;
  for (a.strip = 32;; a.strip >>= 1) {
    const long long rows = ((long long)a.strip << a.gsy) + 2 * kGridCap;
    a.rows = (int)(rows < Ht ? rows : Ht);
    const size_t dist_bytes = (size_t)k * a.rows * a.Gx;
    smem = warps * row_bytes + dist_bytes;
    if (a.strip > 8 && (long long)((a.Gy + a.strip - 1) / a.strip) * P < 296) continue;
    if (smem <= kSmem || a.strip == 1) {
      while (warps > 1 && smem > kSmem) {
        warps >>= 1;
        smem = warps * row_bytes + dist_bytes;
      }
      break;
    }
  }
  if (smem > kSmem) {   // a side of tens of thousands of texels: distance 0 never skips
    cudaError_t e = cudaMemsetAsync(a.grid, 0, atlas_grid_bytes(P, Ht, Wt), st);
    if (e == cudaSuccess && a.solid) e = cudaMemsetAsync(a.solid, 0, atlas_grid_bytes(P, Ht, Wt), st);
    return e == cudaSuccess ? DBMP_OK : cuda_status(e, "cudaMemsetAsync(grid)");
  }
  // in one dimension: the others end at 65535
  const long long ctas = (long long)((a.Gy + a.strip - 1) / a.strip) * P;
  if (ctas > 0x7fffffffll) { set_error("dbmp_atlas_pack: %d templates of %dx%d exceed one grid", P, Ht, Wt); return DBMP_ERR_INVALID; }
  if (smem > 48 * 1024) {
    const cudaError_t e = a.solid ? cudaFuncSetAttribute(atlas_grid_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem)
                                  : cudaFuncSetAttribute(atlas_grid_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(atlas_grid_kernel)");
  }
  if (a.solid) atlas_grid_kernel<true><<<(unsigned)ctas, warps * 32, smem, st>>>(tmpl, a);
  else atlas_grid_kernel<false><<<(unsigned)ctas, warps * 32, smem, st>>>(tmpl, a);
  DBMP_CHECK_LAUNCH("atlas_grid_kernel");
  return DBMP_OK;
}

// Packs the records and grids of a packed kind; solid_off as in launch_grids.
static int pack_records(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, size_t solid_off,
                        cudaStream_t st) {
  const long long total = (long long)P * (Ht + 1) * Wt;
  if (total == 0) return DBMP_OK;
  const int blocks = (int)((total + 255) / 256 < 148 * 32 ? (total + 255) / 256 : 148 * 32);
  switch (kind) {
    case ATLAS_F16_PAIR: atlas_pair_kernel<__half><<<blocks, 256, 0, st>>>(tmpl, P, Ht, Wt, (__half*)out); break;
    case ATLAS_BF16_PAIR: atlas_pair_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(tmpl, P, Ht, Wt, (__nv_bfloat16*)out); break;
    case ATLAS_F32_QUAD: atlas_pack_kernel<float><<<blocks, 256, 0, st>>>(tmpl, P, Ht, Wt, (float*)out); break;
    case ATLAS_F16_QUAD: atlas_pack_kernel<__half><<<blocks, 256, 0, st>>>(tmpl, P, Ht, Wt, (__half*)out); break;
    case ATLAS_BF16_QUAD: atlas_pack_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(tmpl, P, Ht, Wt, (__nv_bfloat16*)out); break;
    default: set_error("dbmp_atlas_pack: kind %d is not a packed kind", kind); return DBMP_ERR_INVALID;
  }
  DBMP_CHECK_LAUNCH("atlas_pack_kernel");
  return launch_grids(tmpl, P, Ht, Wt, kind, out, solid_off, st);
}

int launch_atlas_pack(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, cudaStream_t st) {
  return pack_records(tmpl, P, Ht, Wt, kind, out, 0, st);
}

int launch_atlas_extended(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, cudaStream_t st) {
  if (P == 0) return DBMP_OK;
  const AtlasExt x = atlas_ext(P, Ht, Wt, kind);
  if (x.rec_off != 0) {   // DBMP_ATLAS_F32: the plain templates come first
    if (tmpl != out) {
      const cudaError_t e = cudaMemcpyAsync(out, tmpl, sizeof(float) * (size_t)P * Ht * Wt, cudaMemcpyDeviceToDevice, st);
      if (e != cudaSuccess) return cuda_status(e, "cudaMemcpyAsync(templates)");
    }
    tmpl = static_cast<const float*>(out);   // quads and grids are those of the copy, whatever happens to the original
  }
  return pack_records(tmpl, P, Ht, Wt, x.kind, static_cast<unsigned char*>(out) + x.rec_off, x.solid_off, st);
}

// Gaussian blur of the templates (pydiffbmp/util/utils.py:22-67,
// gaussian_blur, as vector_renderer.py:80-96 applies it to the atlas): a K x K
// kernel, K = 2 round(3 sigma) + 1, weights k[i] k[j] of the normalised 1-D
// Gaussian exp(-0.5 ((i - K/2) / sigma)^2), zero padding, same output size.
// One thread per output texel; the 1-D weights sit in shared memory.
__device__ __forceinline__ void blur_weights(float sigma, int K, float* s_k) {
  float sum = 0.f;
  for (int i = 0; i < K; ++i) {
    const float a = (float)(i - K / 2) / sigma;
    s_k[i] = expf(-0.5f * (a * a));
    sum += s_k[i];
  }
  for (int i = 0; i < K; ++i) s_k[i] /= sum;
}

__device__ __forceinline__ void blur_texels(const float* __restrict__ in, int P, int Ht, int Wt, int K,
                                            const float* s_k, float* __restrict__ out) {
  const long long total = (long long)P * Ht * Wt;
  const int h = K / 2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t % Wt), y = (int)((t / Wt) % Ht);
    const float* src = in + (t - (long long)y * Wt - x);
    float acc = 0.f;
    for (int i = 0; i < K; ++i) {
      const int yy = y + i - h;
      if (yy < 0 || yy >= Ht) continue;
      for (int j = 0; j < K; ++j) {
        const int xx = x + j - h;
        if (xx < 0 || xx >= Wt) continue;
        acc = fmaf(s_k[i] * s_k[j], src[(size_t)yy * Wt + xx], acc);
      }
    }
    out[t] = acc;
  }
}

__global__ void template_blur_kernel(const float* __restrict__ in, int P, int Ht, int Wt, int K, float sigma,
                                     float* __restrict__ out) {
  extern __shared__ float s_k[];
  if (threadIdx.x == 0) blur_weights(sigma, K, s_k);
  __syncthreads();
  blur_texels(in, P, Ht, Wt, K, s_k, out);
}

// Kernel size of a blur sigma: 2 round(3 sigma) + 1 with Python's round (ties
// to even, as rint does).
__host__ __device__ inline int blur_kernel_size(double sigma) { return (int)(2.0 * rint(3.0 * sigma) + 1.0); }

// The blur of one fit iteration it = *step_count under a schedule
// (simple_tile_renderer.py:1015-1021): sigma in double as the reference's
// Python computes it, the kernel size from that double, the weights in float
// (gaussian_blur's float32 tensor arithmetic); sigma <= 0 copies.  The weight
// buffer holds kmax entries, the largest kernel of the schedule.
__global__ void template_blur_sched_kernel(const float* __restrict__ in, int P, int Ht, int Wt,
                                           dbmp_blur_schedule sched, const int* __restrict__ step_count, int kmax,
                                           float* __restrict__ out) {
  extern __shared__ float s_k[];
  __shared__ int s_K;
  if (threadIdx.x == 0) {
    double sigma = 0.0;
    if (sched.mode == 1) {
      sigma = (double)sched.sigma;
    } else if (sched.mode == 2) {
      const double progress = (double)*step_count / (double)sched.num_iterations;
      sigma = (double)sched.sigma_start * (1.0 - progress) + (double)sched.sigma_end * progress;
    }
    int K = sigma > 0.0 ? blur_kernel_size(sigma) : 0;
    if (K > kmax) K = kmax;      // cannot happen for a linear schedule between its two ends
    if (K > 0) blur_weights((float)sigma, K, s_k);
    s_K = K;
  }
  __syncthreads();
  const int K = s_K;
  if (K > 0) {
    blur_texels(in, P, Ht, Wt, K, s_k, out);
    return;
  }
  const long long total = (long long)P * Ht * Wt;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x)
    out[t] = in[t];
}

int launch_template_blur(const float* in, int P, int Ht, int Wt, float sigma, float* out, cudaStream_t st) {
  const long long total = (long long)P * Ht * Wt;
  if (total == 0) return DBMP_OK;
  if (!(sigma > 0.f)) {   // sigma <= 0 leaves the templates unchanged (utils.py:37-38)
    if (in == out) return DBMP_OK;
    cudaError_t e = cudaMemcpyAsync(out, in, sizeof(float) * (size_t)total, cudaMemcpyDeviceToDevice, st);
    return e == cudaSuccess ? DBMP_OK : cuda_status(e, "cudaMemcpyAsync(templates)");
  }
  const int K = blur_kernel_size((double)sigma);
  if (K > 4097) { set_error("dbmp_template_blur: sigma %g gives a kernel of %d texels", (double)sigma, K); return DBMP_ERR_INVALID; }
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  template_blur_kernel<<<blocks, 256, sizeof(float) * K, st>>>(in, P, Ht, Wt, K, sigma, out);
  DBMP_CHECK_LAUNCH("template_blur_kernel");
  return DBMP_OK;
}

int launch_template_blur_sched(const float* in, int P, int Ht, int Wt, const dbmp_blur_schedule* sched,
                               const int* step_count, float* out, cudaStream_t st) {
  const long long total = (long long)P * Ht * Wt;
  if (total == 0) return DBMP_OK;
  // largest kernel over the schedule: sigma is constant or linear between its ends
  double smax = 0.0;
  if (sched->mode == 1) smax = sched->sigma;
  if (sched->mode == 2) smax = sched->sigma_start > sched->sigma_end ? sched->sigma_start : sched->sigma_end;
  const int kmax = smax > 0.0 ? blur_kernel_size(smax) : 1;
  if (kmax > 4097) {
    set_error("dbmp_template_blur_scheduled: sigma %g gives a kernel of %d texels", smax, kmax);
    return DBMP_ERR_INVALID;
  }
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  template_blur_sched_kernel<<<blocks, 256, sizeof(float) * kmax, st>>>(in, P, Ht, Wt, *sched, step_count, kmax,
                                                                         out);
  DBMP_CHECK_LAUNCH("template_blur_sched_kernel");
  return DBMP_OK;
}

// Threads per CTA of prepare_kernel: a primitive is one long chain of double
// and float functions, so few primitives are spread over many SMs.
constexpr int kPrepThreads = 64;

int launch_prepare(const Geom& g, const float* means2D, const float* radii, const float* rot, const float* opac,
                   const float* colors, const int* sel, PrimInfo* out, cudaStream_t st) {
  if (g.N == 0) return DBMP_OK;
  return launch_chained("prepare_kernel", prepare_kernel, dim3((g.N + kPrepThreads - 1) / kPrepThreads), kPrepThreads, 0,
                        st, g, means2D, radii, rot, opac, colors, sel, 0ll, (const float*)nullptr, 0, out,
                        (int4*)nullptr, (unsigned long long*)nullptr);
}

int launch_bin(const Geom& g, int batch, int bin_mode, const float* means2D, const float* radii, const float* rot,
               const float* opac, const float* colors, const int* sel, long long sel_stride, const float* tbbox,
               PrimInfo* prim_info, int* tile_offsets, int* tile_indices, long long index_stride, long long cap,
               int* total_out, int* overflow_out, long long flag_stride, int* host_flags, const Follow& follow, void* ws,
               size_t ws_bytes, cudaStream_t st) {
  const BinGrid bg = bin_grid(g.N, g.tilesX, g.tilesY);
  BinWorkspace w{};
  const size_t need = layout_ws(ws, batch, g.N, g.T, g.tilesX, g.tilesY, bg, &w);
  if (ws_bytes < need) {
    set_error("dbmp_bin: workspace of %zu bytes is smaller than the %zu bytes required", ws_bytes, need);
    return DBMP_ERR_CAPACITY;
  }
  if (bg.ctas > 0x7fffffffll || batch > 65535) {
    set_error("dbmp_bin: canvas, primitive count or batch too large");
    return DBMP_ERR_INVALID;
  }
  // prepare also runs with N = 0: it zeroes the row totals and the flags
  const dim3 prep(g.N > 0 ? (g.N + kPrepThreads - 1) / kPrepThreads : 1, batch);
  int rc = launch_chained("prepare_kernel", prepare_kernel, prep, kPrepThreads, 0, st, g, means2D, radii, rot, opac,
                          colors, sel, sel_stride, tbbox, bin_mode, prim_info, w.rects, w.row_total);
  if (rc) return rc;
  size_t smem = w.scratch ? 0 : diff_cells_bytes(g.tilesX, g.tilesY);
  if (bg.words) smem = std::max(smem, mask_stride(bg.groups * g.tilesY) * kMaskWords * sizeof(unsigned));
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(counts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCountsSmem);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(counts_kernel)");
  }
  rc = launch_chained("counts_kernel", counts_kernel,
                      dim3(bg.slices * bg.subs + bg.words / kMaskWords + follow.blocks, batch), 1024, smem, st, g, bg,
                      (const int4*)w.rects, w.scratch, w.counts, w.row_total, w.masks, follow);
  if (rc) return rc;
  const long long row = (long long)g.tilesX * bg.slices * bg.subs;   // counts of a tile row
  auto* offsets = row > 4 * kOffsThreads ? offsets_kernel<8> : row > kOffsThreads ? offsets_kernel<4> : offsets_kernel<1>;
  rc = launch_chained("offsets_kernel", offsets, dim3(g.tilesY, batch), kOffsThreads, 0, st, g, bg,
                      (const int*)w.counts, (const unsigned long long*)w.row_total, w.offs);
  if (rc) return rc;
  if (bg.words)
    return launch_chained("bin_masks_kernel", bin_masks_kernel, dim3((unsigned)bg.ctas, batch), kBinThreads, 0, st, g,
                          bg, (const int4*)w.rects, (const unsigned*)w.masks, (const long long*)w.offs, cap,
                          tile_indices, index_stride, tile_offsets, total_out, overflow_out, flag_stride,
                          (volatile int*)host_flags, (const int*)follow.changed);
  return launch_chained("bin_rows_kernel", bin_rows_kernel, dim3((unsigned)bg.ctas, batch), kBinThreads, 0, st, g, bg,
                        (const int4*)w.rects, (const long long*)w.offs, cap, tile_indices, index_stride, tile_offsets,
                        total_out, overflow_out, flag_stride, (volatile int*)host_flags, (const int*)follow.changed);
}

}  // namespace dbmp
