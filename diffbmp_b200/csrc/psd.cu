// PSD layer export: one cropped uint8 RGBA layer per primitive.
//
// Replaces cuda_tile_rasterizer/cuda_kernels/psd_export_kernels.cu.  The
// reference launches N x (all 16x16 canvas tiles) blocks and has each thread
// loop over a canvas tile for its primitive, O(N*H*W) work for O(sum of crop
// areas) output.  Here a layout pass prefix-sums each layer's byte size and
// 16x16 block count on the device, and a persistent grid walks only the
// blocks of the crops, one pixel per thread, writing one uchar4 per pixel.
//
// The per-pixel arithmetic must give the reference's bytes exactly, and the
// reference builds it with --use_fast_math (setup_psd_export.py:69), so this
// file is compiled with --use_fast_math too and keeps each expression in the
// reference's operation order (psd_export_common.h:55-121,
// psd_export_kernels.cu:26-55,96-195).
#include <cstdint>

#include <type_traits>

#include "dbmp_internal.cuh"

namespace dbmp {

constexpr int kPsdBlock = 16;

// Stage 1 (psd_export_kernels.cu:12-55): crop box [x0,x1) x [y0,y1) of each
// primitive's scaled square of half extent 1.5 r, clipped to the canvas; an
// empty box becomes (0,0,1,1).
__global__ void psd_bbox_kernel(const float* __restrict__ means2D, const float* __restrict__ radii, int N, int H,
                                int W, float scale, int* __restrict__ bbox, int* __restrict__ sizes) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float x = means2D[n * 2 + 0] * scale;
  const float y = means2D[n * 2 + 1] * scale;
  const float r = radii[n] * scale;
  const float half_extent = r * 1.5f;
  const int x0 = max(0, (int)floorf(x - half_extent));
  const int y0 = max(0, (int)floorf(y - half_extent));
  const int x1 = min(W, (int)ceilf(x + half_extent));
  const int y1 = min(H, (int)ceilf(y + half_extent));
  int4 b = (x1 <= x0 || y1 <= y0) ? make_int4(0, 0, 1, 1) : make_int4(x0, y0, x1, y1);
  reinterpret_cast<int4*>(bbox)[n] = b;
  sizes[2 * n + 0] = b.z - b.x;
  sizes[2 * n + 1] = b.w - b.y;
}

// Layout: exclusive prefix sums of layer bytes (w*h*4) and of 16x16 blocks,
// in one CTA (the reference does the byte sum on the host,
// psd_export_uint8.py:70-77).  blk has N+1 entries; total_bytes is written.
__global__ void psd_layout_kernel(const int* __restrict__ sizes, int N, long long* __restrict__ layer_offsets,
                                  long long* __restrict__ blk, long long* __restrict__ total_bytes) {
  __shared__ long long s_b[1024], s_k[1024];
  const int t = threadIdx.x, nt = blockDim.x;
  const int per = (N + nt - 1) / nt;
  const int lo = min(N, t * per), hi = min(N, lo + per);
  long long sb = 0, sk = 0;
  for (int n = lo; n < hi; ++n) {
    const long long w = sizes[2 * n], h = sizes[2 * n + 1];
    sb += w * h * 4;
    sk += ((w + kPsdBlock - 1) / kPsdBlock) * ((h + kPsdBlock - 1) / kPsdBlock);
  }
  s_b[t] = sb; s_k[t] = sk;
  __syncthreads();
  for (int d = 1; d < nt; d <<= 1) {   // Hillis-Steele inclusive scan
    const long long vb = t >= d ? s_b[t - d] : 0, vk = t >= d ? s_k[t - d] : 0;
    __syncthreads();
    s_b[t] += vb; s_k[t] += vk;
    __syncthreads();
  }
  long long ob = s_b[t] - sb, ok = s_k[t] - sk;
  for (int n = lo; n < hi; ++n) {
    const long long w = sizes[2 * n], h = sizes[2 * n + 1];
    layer_offsets[n] = ob;
    blk[n] = ok;
    ob += w * h * 4;
    ok += ((w + kPsdBlock - 1) / kPsdBlock) * ((h + kPsdBlock - 1) / kPsdBlock);
  }
  if (t == nt - 1) {
    blk[N] = s_k[t];
    *total_bytes = s_b[t];
  }
}

// Template value at canvas pixel (px,py): psd_export_common.h:55-103, with
// each floating-point operation in the reference's order (the layers must be
// byte-identical under --use_fast_math).  The texel coordinate (sx, sy) comes
// from (px - x) / r rotated by theta; outside [0, W-1) x [0, H-1) the value is
// a hard zero.  After that test the cell (ix, iy) = floor(sx, sy) lies in
// [0, W-2] x [0, H-2] (a NaN coordinate converts to cell 0), so it needs no
// clamp, and the weights take the floors as floats, which equal the cell
// indices exactly.
__device__ __forceinline__ float psd_template_value(const float* __restrict__ tmpl, int t_idx, int P, int Ht, int Wt,
                                                    int px, int py, float x, float y, float r, float cos_t,
                                                    float sin_t) {
  const float qx = ((float)px - x) / (r);
  const float qy = ((float)py - y) / (r);
  const float ex = cos_t * qx + sin_t * qy;
  const float ey = -sin_t * qx + cos_t * qy;
  const float sx = (ex + 1.0f) * 0.5f * (Wt - 1);
  const float sy = (ey + 1.0f) * 0.5f * (Ht - 1);
  if (sx < 0.0f || sx >= Wt - 1 || sy < 0.0f || sy >= Ht - 1) return 0.0f;
  if (t_idx < 0 || t_idx >= P) return 0.0f;   // the reference reads out of bounds here
  const float flx = floorf(sx), fly = floorf(sy);
  const int ix = (int)flx, iy = (int)fly;
  const float fx = sx - flx;
  const float fy = sy - fly;
  const float gx = 1.0f - fx;
  const float gy = 1.0f - fy;
  const float* row = tmpl + (size_t)t_idx * Ht * Wt + iy * Wt + ix;
  const float s00 = row[0], s01 = row[1], s10 = row[Wt], s11 = row[Wt + 1];
  return gx * gy * s00 + fx * gy * s01 + gx * fy * s10 + fx * fy * s11;
}

// Clamped bilinear of a per-primitive RGB map (psd_export_common.h:124-196,
// operations in its order), used only with c_blend > 0: the coordinate is
// clamped into the map and the neighbours past the last row / column repeat it.
__device__ __forceinline__ float3 psd_color_map(const float* __restrict__ cm, int map_h, int map_w, float x, float y,
                                                float radius, float rotation) {
  const float inv = radius > 1e-6f ? (1.0f / radius) : 1e6f;
  const float qx = x * inv;
  const float qy = y * inv;
  const float ct = cosf(rotation);
  const float st = sinf(rotation);
  const float ex = ct * qx + st * qy;
  const float ey = -st * qx + ct * qy;
  float sx = (ex + 1.0f) * 0.5f * (map_w - 1);
  float sy = (ey + 1.0f) * 0.5f * (map_h - 1);
  sx = fmaxf(0.0f, fminf(map_w - 1, sx));
  sy = fmaxf(0.0f, fminf(map_h - 1, sy));
  const int ix = (int)sx, iy = (int)sy;
  const int jx = min(ix + 1, map_w - 1), jy = min(iy + 1, map_h - 1);
  const float fx = sx - ix;
  const float fy = sy - iy;
  float3 out;
  float* o = &out.x;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float a0 = cm[3 * (iy * map_w + ix) + ch], b0 = cm[3 * (jy * map_w + ix) + ch];
    const float a1 = cm[3 * (iy * map_w + jx) + ch], b1 = cm[3 * (jy * map_w + jx) + ch];
    const float top = a0 * (1.0f - fx) + a1 * fx;
    const float bot = b0 * (1.0f - fx) + b1 * fx;
    o[ch] = top * (1.0f - fy) + bot * fy;
  }
  return out;
}

__device__ __forceinline__ uint8_t to_u8(float v) { return (uint8_t)fmaxf(0.0f, fminf(255.0f, v * 255.0f)); }

struct PsdArgs {
  int N, P, Ht, Wt;
  float scale, alpha_max, c_blend;
};

// Stage 2 (psd_export_kernels.cu:61-198): the 16x16 blocks of all crops, block
// b of layer n for blk[n] <= b < blk[n+1].  Each warp takes a contiguous range
// of blocks and walks them in order, a whole block at a time: lane l owns
// column l % 16 and rows l / 16, l / 16 + 2, ... of the block (eight pixels;
// each half-warp stores 64 contiguous bytes of a row).  Lane 0 follows the
// layer index forward from block to block (a binary search only for the
// range's first block) and loads the layer's box, centre, radius, rotation
// with its cosine and sine, opacity and colour once per layer, broadcast to
// the lanes.  Each thread then computes its pixels with the reference's
// per-pixel operations on the same values, so the bytes are the ones a
// per-pixel evaluation gives.  Bound by its instructions: without a colour map the
// colour bytes of a layer are converted once, since a pixel's mask factor is 1
// wherever its template value is above 0, and stores step a pointer.  Many short
// ranges (96 CTAs of four warps per SM) keep the SMs filled to the end, where ranges
// of cheap outside blocks finish early.  1024x1024, N=1500: 289 -> 212 us (ranges
// alone 258, one kernel with and without colour map 219); N=5000 913 -> 642;
// 2048x2048, N=20000: 11.7 -> 9.7 ms.
template <bool MAPPED>
__global__ void __launch_bounds__(128, 8) psd_layers_kernel(PsdArgs a, const float* __restrict__ means2D,
                                                         const float* __restrict__ radii,
                                                         const float* __restrict__ rot,
                                                         const float* __restrict__ colors,
                                                         const float* __restrict__ vis,
                                                         const float* __restrict__ tmpl, const int* __restrict__ sel,
                                                         const int* __restrict__ bbox,
                                                         const long long* __restrict__ layer_offsets,
                                                         const long long* __restrict__ blk,
                                                         const float* __restrict__ colors_orig,
                                                         uint8_t* __restrict__ out) {
  const long long nblk = blk[a.N];
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long per = (nblk + nwarps - 1) / nwarps;
  const long long b0 = gw * per, b1 = min(b0 + per, nblk);
  const int lx = lane & (kPsdBlock - 1), ly0 = lane >> 4;   // this thread's column and first row in a block
  int n = -1;                      // the current layer (lane 0's bookkeeping, broadcast below)
  long long next = 0;              // blk[n + 1]
  int4 bb = make_int4(0, 0, 0, 0);
  float x = 0.f, y = 0.f, r = 0.f, theta = 0.f, cos_t = 0.f, sin_t = 0.f, vs = 0.f, cr = 0.f, cg = 0.f, cb = 0.f;
  unsigned rgb8 = 0u;              // the layer's colour bytes
  int t_idx = 0, bx_n = 1;
  long long off = 0, first = 0;    // the layer's byte offset and first block
  int bx = 0, by = 0;              // the current block's first pixel within the crop
  for (long long b = b0; b < b1; ++b) {
    bool changed = false;
    if (lane == 0 && (n < 0 || b >= next)) {
      if (n < 0) {   // largest n with blk[n] <= b
        int lo = 0, hi = a.N;
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (blk[mid] <= b) lo = mid; else hi = mid;
        }
        n = lo;
      } else {
        while (blk[n + 1] <= b) ++n;   // empty crops have no blocks
      }
      next = blk[n + 1];
      changed = true;
    }
    if (__shfl_sync(0xffffffffu, changed, 0)) {
      if (lane == 0) {
        bb = reinterpret_cast<const int4*>(bbox)[n];
        x = means2D[n * 2 + 0] * a.scale;
        y = means2D[n * 2 + 1] * a.scale;
        r = radii[n] * a.scale;
        theta = rot[n];
        cos_t = cosf(theta);
        sin_t = sinf(theta);
        vs = vis[n];
        cr = colors[n * 3 + 0]; cg = colors[n * 3 + 1]; cb = colors[n * 3 + 2];
        t_idx = sel[n];
        off = layer_offsets[n];
        first = blk[n];
        bx_n = (bb.z - bb.x + kPsdBlock - 1) / kPsdBlock;
      }
      n = __shfl_sync(0xffffffffu, n, 0);
      bb.x = __shfl_sync(0xffffffffu, bb.x, 0); bb.y = __shfl_sync(0xffffffffu, bb.y, 0);
      bb.z = __shfl_sync(0xffffffffu, bb.z, 0); bb.w = __shfl_sync(0xffffffffu, bb.w, 0);
      x = __shfl_sync(0xffffffffu, x, 0); y = __shfl_sync(0xffffffffu, y, 0); r = __shfl_sync(0xffffffffu, r, 0);
      theta = __shfl_sync(0xffffffffu, theta, 0);
      cos_t = __shfl_sync(0xffffffffu, cos_t, 0); sin_t = __shfl_sync(0xffffffffu, sin_t, 0);
      vs = __shfl_sync(0xffffffffu, vs, 0);
      cr = __shfl_sync(0xffffffffu, cr, 0); cg = __shfl_sync(0xffffffffu, cg, 0); cb = __shfl_sync(0xffffffffu, cb, 0);
      rgb8 = to_u8(cr) | to_u8(cg) << 8 | to_u8(cb) << 16;
      t_idx = __shfl_sync(0xffffffffu, t_idx, 0);
      off = __shfl_sync(0xffffffffu, off, 0);
      first = __shfl_sync(0xffffffffu, first, 0);
      bx_n = __shfl_sync(0xffffffffu, bx_n, 0);
      const int k = (int)(b - first);   // block within the crop (a crop has < 2^31 blocks)
      bx = (k % bx_n) * kPsdBlock;
      by = (k / bx_n) * kPsdBlock;
    } else {                            // the next block of the same crop, row-major
      bx += kPsdBlock;
      if (bx >= bb.z - bb.x) { bx = 0; by += kPsdBlock; }
    }
    const int bw = bb.z - bb.x, bh = bb.w - bb.y;
    // Warp-uniform: true when the whole block maps outside the template
    // square [-1, 1) x [-1, 1) of the normalised frame (rotated (p - c) / r)
    // by a margin of 1e-3, far above the rounding of the per-pixel
    // coordinates; each of its pixels then takes the hard zero, and its bytes
    // are stored as zeros without the per-pixel arithmetic.  The map is affine,
    // so the block's four corner pixels bound it.  Only for finite inputs with
    // r > 1e-3: a non-finite coordinate or opacity can give nonzero bytes.
    bool outside = false;
    if (r > 1e-3f && isfinite(r) && isfinite(x) && isfinite(y) && isfinite(cos_t) && isfinite(sin_t) &&
        isfinite(vs) && isfinite(a.alpha_max)) {
      const float inv = 1.0f / r;
      const float qx0 = ((float)(bb.x + bx) - x) * inv, qx1 = ((float)(bb.x + bx + kPsdBlock - 1) - x) * inv;
      const float qy0 = ((float)(bb.y + by) - y) * inv, qy1 = ((float)(bb.y + by + kPsdBlock - 1) - y) * inv;
      const float ex00 = cos_t * qx0 + sin_t * qy0, ex10 = cos_t * qx1 + sin_t * qy0;
      const float ex01 = cos_t * qx0 + sin_t * qy1, ex11 = cos_t * qx1 + sin_t * qy1;
      const float ey00 = cos_t * qy0 - sin_t * qx0, ey10 = cos_t * qy0 - sin_t * qx1;
      const float ey01 = cos_t * qy1 - sin_t * qx0, ey11 = cos_t * qy1 - sin_t * qx1;
      const float m = 1e-3f;
      outside = fmaxf(fmaxf(ex00, ex10), fmaxf(ex01, ex11)) < -1.0f - m ||
                fminf(fminf(ex00, ex10), fminf(ex01, ex11)) > 1.0f + m ||
                fmaxf(fmaxf(ey00, ey10), fmaxf(ey01, ey11)) < -1.0f - m ||
                fminf(fminf(ey00, ey10), fminf(ey01, ey11)) > 1.0f + m;
    }
    const int lpx = bx + lx;
    if (lpx >= bw) continue;
    const int px = bb.x + lpx;
    const int rows = min(kPsdBlock, bh - by);   // rows of this block inside the crop
    uint8_t* dst = out + off + ((long long)(by + ly0) * bw + lpx) * 4;   // this thread's pixel of the row
    const long long step = (long long)bw * 8;
    if (outside) {
      for (int ly = ly0; ly < rows; ly += 2, dst += step) *reinterpret_cast<uchar4*>(dst) = make_uchar4(0, 0, 0, 0);
      continue;
    }
    for (int ly = ly0; ly < rows; ly += 2, dst += step) {
      const int py = bb.y + by + ly;
      // The column is hidden from the optimiser in every row, so no part of
      // the pixel's expression is hoisted out of the loop: a hoisted cos*u
      // lets the compiler fuse the other product instead, which changes the
      // fast-math rounding and, rarely, a byte against the reference kernel.
      int pxr = px;
      asm volatile("" : "+r"(pxr));
      const float tv = psd_template_value(tmpl, t_idx, a.P, a.Ht, a.Wt, pxr, py, x, y, r, cos_t, sin_t);
      const float alpha_val = tv * vs * a.alpha_max;
      unsigned px4 = 0u;
      if (!(alpha_val < 0.001f)) {
        if (!MAPPED && tv > 0.0f) {
          px4 = rgb8 | (unsigned)to_u8(alpha_val) << 24;
        } else {
          float rgb_r = cr, rgb_g = cg, rgb_b = cb;
          if constexpr (MAPPED) {
            const float* cm = colors_orig + (size_t)n * a.Ht * a.Wt * 3;
            const float ux = x / a.scale, uy = y / a.scale;
            const float upx = (float)pxr / a.scale, upy = (float)py / a.scale;
            const float ur = r / a.scale;
            const float3 co = psd_color_map(cm, a.Ht, a.Wt, upx - ux, upy - uy, ur, theta);
            rgb_r = (1.0f - a.c_blend) * rgb_r + a.c_blend * co.x;
            rgb_g = (1.0f - a.c_blend) * rgb_g + a.c_blend * co.y;
            rgb_b = (1.0f - a.c_blend) * rgb_b + a.c_blend * co.z;
          }
          const float mask = tv > 0.0f ? 1.0f : 0.0f;
          px4 = to_u8(mask * rgb_r) | to_u8(mask * rgb_g) << 8 | to_u8(mask * rgb_b) << 16 |
                (unsigned)to_u8(alpha_val) << 24;
        }
      }
      *reinterpret_cast<unsigned*>(dst) = px4;
    }
  }
}

// ---------------------------------------------------------------------------
// PSD file assembly: PackBits (RLE) channel data.
//
// The reference hands each cropped layer to psd-tools (PixelLayer.frompil,
// then PSDImage.save; psd_export_uint8.py:153-186, psd_exporter.py:468-501),
// which splits it into planes and RLE-compresses them row by row on the host.
// Here every (layer, channel, row) is encoded on the device.  Rows are taken
// 32 at a time, one warp per group of 32 rows of a layer, in chunks of 32 columns.
// The warp first looks at the chunk four rows at a time, four pixels per lane:
// ballots of "differs from its left neighbour" give each channel's run starts as
// bit masks.  Then each lane takes one row and visits only the set bits of its
// four masks, so equal pixels, nearly all of a layer, cost a dozen instructions per
// 128 of them.  (Encoders that looked at every pixel of their row took, at
// 1024x1024, N=5000, 388 M and 510 M instructions for the two passes.)
//
// Encoding rule (a valid PackBits stream; a packet never crosses a row):
//   - a maximal run of L >= 3 equal bytes becomes replicate packets
//     [1-k, v] of k = min(remaining, 128) bytes each; a one-byte remainder
//     becomes the literal packet [0, v];
//   - maximal runs of one or two bytes are gathered into literal segments,
//     written as packets [k-1, k bytes] of 128 bytes and a last shorter one.
// The count pass writes each row's encoded size (at most w + ceil(w/128)
// bytes, so 16 bits suffice for w <= 30000, the PSD width limit that the C
// ABI enforces on width_limit) and each
// group's per-channel totals; the host plans where every channel block goes;
// the write pass re-encodes and stores.  Each store is checked against the
// planned extent of its row and the output size, so a plan that does not
// match the data can write wrong bytes but never out of bounds.
// ---------------------------------------------------------------------------

constexpr int kRleWarps = 4;      // warps per CTA
// Words per staged row: three unused, the pixel left of the chunk, the chunk's
// 32.  Pixels start at a multiple of 16 bytes, and eight lanes' 16-byte reads of
// a row, as the lanes' 4-byte reads of their own rows, cover distinct banks.
constexpr int kRlePitch = 36;
constexpr int kRleFirst = 4;      // word of the chunk's first pixel

struct RleArgs {
  const uint8_t* layers;        // packed RGBA crops, row-major per layer
  const int* sizes;             // (N,2) w, h
  const long long* layer_off;   // (N) byte offset of each crop
  const long long* group_base;  // (N+1) exclusive prefix of ceil(h/32)
  long long G;                  // number of row groups
  int N;
  unsigned order;               // byte index (0..3) of channel slot s in bits 8s..8s+1
  int width_limit;
  unsigned short* row_bytes;    // (G*32, 4) encoded size of each row's four channels
  int* group_tot;               // (G, 4) per-group totals (count pass)
  int* alpha_any;               // (N) 1 if a layer has a nonzero byte 3 (count pass; may be null)
  const long long* chan_off;    // (N, 4) channel block offsets in out, < 0 skips (write pass)
  const long long* group_dst;   // (G, 4) output offset of the group's first row (write pass)
  uint8_t* out;                 // (write pass)
  long long out_bytes;
};

// A PackBits encoder of one channel of one row, fed with its runs in order:
// counting output bytes only (count pass).  A literal segment's headers are
// added when the segment closes, or when 128 bytes are in.
struct RleCount {
  int pos = 0, lit = 0;

  __device__ __forceinline__ void run(int L, unsigned) {
    if (L >= 3) {
      if (lit > 0) pos += 1 + lit;
      lit = 0;
      pos += 2 * ((L + 127) >> 7);
    } else {
      lit += L;
      if (lit >= 128) {
        pos += 129;
        lit -= 128;
      }
    }
  }
  __device__ __forceinline__ void finish() {
    if (lit > 0) pos += 1 + lit;
  }
};

// The encoder that stores its bytes (write pass); positions are byte offsets
// within the row's output.  A literal byte is stored as soon as its run closes
// (a run of one or two bytes), at its final place: a literal packet's header
// position is reserved when the packet opens and written when it closes (127
// when 128 bytes are in, the count minus one at the end of the segment).
struct RleWrite {
  int pos = 0, lit = 0, hdr = 0, lim = 0;
  uint8_t* dst = nullptr;   // the row's first output byte

  __device__ __forceinline__ void store(int p, unsigned v) {
    if (p < lim) dst[p] = (uint8_t)v;
  }
  __device__ __forceinline__ void put(unsigned v) {
    store(pos, v);
    ++pos;
  }
  // Appends one byte to the open literal segment.
  __device__ __forceinline__ void lit_byte(unsigned v) {
    if ((lit & 127) == 0) hdr = pos++;
    put(v);
    if ((++lit & 127) == 0) store(hdr, 127u);
  }
  __device__ __forceinline__ void end_literal() {
    if (lit & 127) store(hdr, (unsigned)((lit & 127) - 1));
    lit = 0;
  }
  // A run of L bytes v.
  __device__ __forceinline__ void run(int L, unsigned v) {
    if (L >= 3) {
      end_literal();
      for (int rem = L; rem > 0; rem -= 128) {
        const int k = min(rem, 128);
        put(k >= 2 ? (unsigned)(1 - k) & 0xFFu : 0u);
        put(v);
      }
    } else {
      if (L >= 1) lit_byte(v);
      if (L >= 2) lit_byte(v);
    }
  }
  __device__ __forceinline__ void finish() { end_literal(); }
};

// One 4-byte asynchronous copy from global to shared memory (cp.async).
__device__ __forceinline__ void cp_async_word(uint32_t* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Largest i < n with base[i] <= g (base[0] <= g), by a whole warp: 32 probes a step.
__device__ __forceinline__ int warp_search(const long long* __restrict__ base, int n, long long g, int lane) {
  int lo = 0, len = n;
  while (len > 1) {
    const int step = (len + 31) >> 5;
    const int at = lo + lane * step;
    const unsigned le = __ballot_sync(0xffffffffu, lane * step < len && base[at] <= g);
    const int k = 31 - __clz(le);   // bit 0 is set: base[lo] <= g
    lo += k * step;
    len = min(step, len - k * step);
  }
  return lo;
}

// Planes of a row's run starts (see psd_rle_kernel) to one bit per column, in
// order: a transpose in three masked exchanges.
__device__ __forceinline__ unsigned planes_to_columns(unsigned v) {
  unsigned t = (v ^ (v >> 12)) & 0x0000F0F0u;
  v ^= t ^ (t << 12);
  t = (v ^ (v >> 6)) & 0x00CC00CCu;
  v ^= t ^ (t << 6);
  t = (v ^ (v >> 3)) & 0x0A0A0A0Au;
  v ^= t ^ (t << 3);
  return v;
}

// The registers are bounded for 36 resident warps per SM in the count pass and 28
// in the write pass.
template <bool WRITE>
__global__ void __launch_bounds__(kRleWarps * 32, WRITE ? 7 : 9) psd_rle_kernel(RleArgs a) {
  // Per warp one buffer of 32 rows x (1 + 32) pixels, filled asynchronously: the
  // count pass refills it as soon as the masks are taken.  Many warps with one
  // buffer hide the copies better than 24 warps with two (count / write pass at
  // 1024x1024, N=5000: 538 / 658 us with two buffers, 442 / 504 with one, 356 /
  // 450 with one group per warp as well; 597 / 871 for encoders that look at
  // every pixel.  At 2048x2048, N=20000, 15.8 GB: 6.2 / 8.0 -> 4.0 / 4.5 ms, 0.61
  // and 0.55 of the copy bandwidth.)  What bounds them now is the visits to the
  // run starts, with 28 of 32 lanes active and two fifths of the issue slots used.
  __shared__ __align__(16) uint32_t stage[kRleWarps][32 * kRlePitch];
  const int lane = threadIdx.x & 31;
  uint32_t* buf = stage[threadIdx.x >> 5];
  const long long nwarps = (long long)gridDim.x * kRleWarps;
  for (long long g = (long long)blockIdx.x * kRleWarps + (threadIdx.x >> 5); g < a.G; g += nwarps) {
    const int i = warp_search(a.group_base, a.N, g, lane);   // the group's layer
    const int w = a.sizes[2 * i], h = a.sizes[2 * i + 1];
    const long long off = a.layer_off[i];
    const bool ok = w >= 1 && w <= a.width_limit && h >= 1 && off >= 0 && (off & 3) == 0;
    const long long y0 = (g - a.group_base[i]) * 32;
    const int y = (int)y0 + lane;
    const bool active = ok && y0 + lane < h;
    const uint8_t* base = a.layers + (ok ? off : 0);

    std::conditional_t<WRITE, RleWrite, RleCount> e[4];
    unsigned short planned[4] = {0, 0, 0, 0};
    bool skip = !ok;
    if constexpr (WRITE) {
#pragma unroll
      for (int s = 0; s < 4; ++s) e[s].dst = a.out;
      if (ok && active) {
        const ushort4 rb = reinterpret_cast<const ushort4*>(a.row_bytes)[g * 32 + lane];
        planned[0] = rb.x; planned[1] = rb.y; planned[2] = rb.z; planned[3] = rb.w;
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        int pre = planned[s];   // exclusive prefix over the group's rows
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, pre, d);
          if (lane >= d) pre += t;
        }
        pre -= planned[s];
        const long long co = ok ? a.chan_off[4 * i + s] : -1;
        const long long gd = ok ? a.group_dst[4 * g + s] : -1;
        if (co >= 0 && gd >= 0) {   // otherwise every store of this slot is dropped
          const long long start = gd + pre;
          e[s].dst = a.out + start;
          e[s].lim = (int)max(0ll, min((long long)planned[s], a.out_bytes - start));
          if (active) {   // row byte count, big-endian, in the block's table; block header on row 0
            const long long t = co + 2 + 2ll * y;
            if (t + 1 < a.out_bytes) { a.out[t] = (uint8_t)(planned[s] >> 8); a.out[t + 1] = (uint8_t)planned[s]; }
            if (y == 0 && co + 1 < a.out_bytes) { a.out[co] = 0; a.out[co + 1] = 1; }
          }
        }
      }
      skip = skip || (a.chan_off[4 * i] < 0 && a.chan_off[4 * i + 1] < 0 && a.chan_off[4 * i + 2] < 0 &&
                      a.chan_off[4 * i + 3] < 0);
    }

    uint32_t any_alpha = 0;
    if (!skip) {   // warp-uniform: skip depends on the layer only
      int from[4] = {0, 0, 0, 0};       // first column of the channel's open run
      unsigned val[4] = {0, 0, 0, 0};   // its byte (write pass)
      const int rows = (int)min(32ll, h - y0);
      unsigned byte_of[4];              // channel slot -> mask of its byte in a pixel
#pragma unroll
      for (int s = 0; s < 4; ++s) byte_of[s] = 0xFFu << (8 * ((a.order >> (8 * s)) & 3));
      const uint32_t* row0 = reinterpret_cast<const uint32_t*>(base) + y0 * w;
      // columns x0 - 1 .. x0 + 31 of the group's rows (column -1 and the columns
      // past the layer are not copied, and not looked at)
      auto stage_chunk = [&](int x0) {
        if (x0 > 0 && lane < rows) cp_async_word(buf + lane * kRlePitch + kRleFirst - 1, row0 + (long long)lane * w + x0 - 1);
        if (x0 + lane < w) {
          const uint32_t* q = row0 + x0 + lane;
          uint32_t* d = buf + kRleFirst + lane;
#pragma unroll 8
          for (int r = 0; r < rows; ++r, q += w, d += kRlePitch) cp_async_word(d, q);
        }
      };
      __syncwarp();   // every lane is done with the buffer (previous group)
      stage_chunk(0);
      for (int x0 = 0; x0 < w; x0 += 32) {
        cp_async_wait_all();
        __syncwarp();   // the lanes' copies of this chunk are visible to the whole warp
        // Run starts of this lane's row per channel slot, in planes of eight bits:
        // bit l of plane 0, 1, 2, 3 is pixel 4 l + 0, 2, 1, 3 of the chunk.
        unsigned m[4] = {0, 0, 0, 0};
        const int l = lane & 7, left_cols = w - x0 - 4 * l;   // columns of the layer from this lane's first on
        const uint32_t* q = buf + (lane >> 3) * kRlePitch + kRleFirst + 4 * l;
        const unsigned pick = (unsigned)(lane & 3);           // byte of a ballot that holds this lane's row
        for (int k = 0; 4 * k < rows; ++k, q += 4 * kRlePitch) {
          const bool row_in = 4 * k + (lane >> 3) < rows;
          const uint4 p = *reinterpret_cast<const uint4*>(q);
          uint32_t prev = __shfl_up_sync(0xffffffffu, p.w, 1);
          if (l == 0) prev = x0 > 0 ? q[-1] : p.x;
          uint32_t d[4] = {p.x ^ prev, p.y ^ p.x, p.z ^ p.y, p.w ^ p.z};
          if (left_cols < 4 || !row_in) {   // columns or rows past the layer hold leftovers
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j >= left_cols || !row_in) d[j] = 0u;
          }
          if (!WRITE && row_in) {
            if (left_cols > 0) any_alpha |= p.x & 0xFF000000u;
            if (left_cols > 1) any_alpha |= p.y & 0xFF000000u;
            if (left_cols > 2) any_alpha |= p.z & 0xFF000000u;
            if (left_cols > 3) any_alpha |= p.w & 0xFF000000u;
          }
          const uint32_t any = d[0] | d[1] | d[2] | d[3];
          if (__any_sync(0xffffffffu, any != 0u)) {
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              if (!__any_sync(0xffffffffu, any & byte_of[s])) continue;
              unsigned b[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) b[j] = __ballot_sync(0xffffffffu, d[j] & byte_of[s]);
              const unsigned lo = __byte_perm(b[0], b[2], pick | (pick + 4) << 4);
              const unsigned hi = __byte_perm(b[1], b[3], pick | (pick + 4) << 4);
              if ((lane >> 2) == k) m[s] = __byte_perm(lo, hi, 0x5410);
            }
          }
        }
        if (!WRITE) {
          __syncwarp();   // every lane is done with the buffer
          if (x0 + 32 < w) stage_chunk(x0 + 32);
        }
        if (WRITE && x0 == 0) {
          const uint32_t p = buf[lane * kRlePitch + kRleFirst];
#pragma unroll
          for (int s = 0; s < 4; ++s) val[s] = (p >> (8 * ((a.order >> (8 * s)) & 3))) & 0xFFu;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          unsigned k = planes_to_columns(m[s]);
          while (k) {
            const int j = __ffs(k) - 1;
            k &= k - 1;
            const int x = x0 + j;
            e[s].run(x - from[s], val[s]);
            from[s] = x;
            if (WRITE) val[s] = (buf[lane * kRlePitch + kRleFirst + j] >> (8 * ((a.order >> (8 * s)) & 3))) & 0xFFu;
          }
        }
        if (WRITE) {
          __syncwarp();   // every lane is done with the buffer
          if (x0 + 32 < w) stage_chunk(x0 + 32);
        }
      }
      if (active) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          e[s].run(w - from[s], val[s]);
          e[s].finish();
        }
      }
    }
    if constexpr (!WRITE) {
      int c[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) c[s] = active && !skip ? e[s].pos : 0;
      reinterpret_cast<ushort4*>(a.row_bytes)[g * 32 + lane] =
          make_ushort4((unsigned short)c[0], (unsigned short)c[1], (unsigned short)c[2], (unsigned short)c[3]);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) c[s] += __shfl_xor_sync(0xffffffffu, c[s], d);
      }
      if (lane == 0) reinterpret_cast<int4*>(a.group_tot)[g] = make_int4(c[0], c[1], c[2], c[3]);
      if (__any_sync(0xffffffffu, any_alpha != 0) && lane == 0 && a.alpha_any) a.alpha_any[i] = 1;
    }
  }
}

int launch_psd_rle(bool write, const uint8_t* layers, const int* sizes, const long long* layer_off,
                   const long long* group_base, int N, long long G, unsigned order, int width_limit,
                   unsigned short* row_bytes, int* group_tot, int* alpha_any, const long long* chan_off,
                   const long long* group_dst, uint8_t* out, long long out_bytes, cudaStream_t st) {
  if (G == 0 || N == 0) return DBMP_OK;
  const RleArgs a{layers, sizes, layer_off, group_base, G, N, order, width_limit, row_bytes, group_tot,
                  alpha_any, chan_off, group_dst, out, out_bytes};
  // One group per warp, so that the SMs refill as groups of uneven width finish
  // (a persistent grid-stride loop left them a third empty on average); the loop
  // only serves counts beyond a grid's limit.
  long long ctas = (G + kRleWarps - 1) / kRleWarps;
  if (ctas > 0x7fffffffll) ctas = 0x7fffffffll;
  if (write) psd_rle_kernel<true><<<(int)ctas, kRleWarps * 32, 0, st>>>(a);
  else psd_rle_kernel<false><<<(int)ctas, kRleWarps * 32, 0, st>>>(a);
  DBMP_CHECK_LAUNCH("psd_rle_kernel");
  return DBMP_OK;
}

int launch_psd_bboxes(const float* means2D, const float* radii, int N, int H, int W, float scale, int* bbox,
                      int* sizes, cudaStream_t st) {
  if (N == 0) return DBMP_OK;
  psd_bbox_kernel<<<(N + 255) / 256, 256, 0, st>>>(means2D, radii, N, H, W, scale, bbox, sizes);
  DBMP_CHECK_LAUNCH("psd_bbox_kernel");
  return DBMP_OK;
}

int launch_psd_layout(const int* sizes, int N, long long* layer_offsets, long long* blk, long long* total,
                      cudaStream_t st) {
  psd_layout_kernel<<<1, 1024, 0, st>>>(sizes, N, layer_offsets, blk, total);
  DBMP_CHECK_LAUNCH("psd_layout_kernel");
  return DBMP_OK;
}

int launch_psd_layers(int N, int P, int Ht, int Wt, float scale, float alpha_max, float c_blend,
                      const float* means2D, const float* radii, const float* rot, const float* colors,
                      const float* vis, const float* tmpl, const int* sel, const int* bbox,
                      const long long* layer_offsets, const long long* blk, const float* colors_orig, uint8_t* out,
                      cudaStream_t st) {
  if (N == 0) return DBMP_OK;
  PsdArgs a{N, P, Ht, Wt, scale, alpha_max, c_blend};
  const bool mapped = colors_orig != nullptr && c_blend > 0.0f;
  auto* kernel = mapped ? psd_layers_kernel<true> : psd_layers_kernel<false>;
  kernel<<<148 * 96, 128, 0, st>>>(a, means2D, radii, rot, colors, vis, tmpl, sel, bbox, layer_offsets, blk,
                                        colors_orig, out);
  DBMP_CHECK_LAUNCH("psd_layers_kernel");
  return DBMP_OK;
}

}  // namespace dbmp
