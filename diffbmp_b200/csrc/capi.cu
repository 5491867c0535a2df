// C ABI of libdbmp.so (declarations and contracts in include/dbmp.h).
#include <atomic>
#include <chrono>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <thread>

#include "dbmp_internal.cuh"

namespace dbmp {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int cuda_status(cudaError_t e, const char* what) {
  set_error("%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
  (void)cudaGetLastError();   // reported here, not by the next call's check of its launches
  return DBMP_ERR_CUDA;
}

// launchers (binning.cu, raster.cu)
size_t bin_workspace_bytes(int batch, int N, int T, int tilesX, int tilesY);
size_t atlas_bytes(int P, int Ht, int Wt, int kind);
int launch_template_bboxes(const float* tmpl, int P, int Ht, int Wt, float* out, cudaStream_t st);
int launch_template_blur(const float* in, int P, int Ht, int Wt, float sigma, float* out, cudaStream_t st);
int launch_atlas_pack(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, cudaStream_t st);
int launch_atlas_extended(const float* tmpl, int P, int Ht, int Wt, int kind, void* out, cudaStream_t st);
int launch_convert(int n, const void* const* src, void* const* dst, const long long* counts, bool to_half,
                   cudaStream_t st);
int launch_zero(double* a, long long n, double* b, const Follow& f, cudaStream_t st);
int launch_prepare(const Geom& g, const float* means2D, const float* radii, const float* rot, const float* opac,
                   const float* colors, const int* sel, PrimInfo* out, cudaStream_t st);
int launch_bin(const Geom& g, int batch, int bin_mode, const float* means2D, const float* radii, const float* rot,
               const float* opac, const float* colors, const int* sel, long long sel_stride, const float* tbbox,
               PrimInfo* prim_info, int* tile_offsets, int* tile_indices, long long index_stride, long long cap,
               int* total_out, int* overflow_out, long long flag_stride, int* host_flags, const Follow& follow, void* ws,
               size_t ws_bytes, cudaStream_t st);
int launch_forward(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                   const int* idx, float* color, float* alpha, float* T_last, int* last_pos, cudaStream_t st);
int launch_forward_blend(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                         const int* idx, float* color, float* alpha, float* T_last, int* last_pos, const float* cmap,
                         float cblend, cudaStream_t st, int batch, long long idx_stride, long long cmap_stride,
                         const int* flags, void* masks);
int launch_backward_blend(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                          const int* idx, const float* T_last, const int* last_pos, const float* grad_color,
                          const float* grad_alpha, double* gacc, const float* cmap, float cblend, cudaStream_t st,
                          int batch, long long idx_stride, long long cmap_stride,
                          const void* masks);
size_t walk_mask_bytes(const Geom& g, int batch);
int launch_count(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs, const int* idx,
                 unsigned long long* cnt, cudaStream_t st);
int launch_backward(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs,
                    const int* idx, const float* T_last, const int* last_pos, const float* grad_color,
                    const float* grad_alpha, double* gacc, cudaStream_t st);
int launch_finalize(const Geom& g, const float* radii, const float* rot, const float* opac, const float* colors,
                    const double* gacc, float* gm, float* gr, float* grot, float* go, float* gc, cudaStream_t st);
int launch_fused(const Geom& g, int kind, const PrimInfo* prims, const void* atlas, const int* offs, const int* idx,
                 const float* target, const float* background, float* out_image, double* gacc, double* loss,
                 const int* skip_flag, cudaStream_t st);
int launch_prune(const Geom& g, const PruneArgs& a, const int* step_count, const float* pool, int* state,
                 float* means2D, float* radii, float* rot, float* opac, float* colors, const int* skip_flag,
                 cudaStream_t st);
int launch_template_blur_sched(const float* in, int P, int Ht, int Wt, const dbmp_blur_schedule* sched,
                               const int* step_count, float* out, cudaStream_t st);
int launch_adam(const Geom& g, const AdamArgs& a, const double* gacc, float* means2D, float* radii, float* rot,
                float* opac, float* colors, float* m1, float* m2, int* step_count, const int* skip_flag,
                cudaStream_t st);

int launch_psd_bboxes(const float* means2D, const float* radii, int N, int H, int W, float scale, int* bbox,
                      int* sizes, cudaStream_t st);
int launch_psd_layout(const int* sizes, int N, long long* layer_offsets, long long* blk, long long* total,
                      cudaStream_t st);
int launch_psd_layers(int N, int P, int Ht, int Wt, float scale, float alpha_max, float c_blend,
                      const float* means2D, const float* radii, const float* rot, const float* colors,
                      const float* vis, const float* tmpl, const int* sel, const int* bbox,
                      const long long* layer_offsets, const long long* blk, const float* colors_orig, uint8_t* out,
                      cudaStream_t st);
int launch_psd_rle(bool write, const uint8_t* layers, const int* sizes, const long long* layer_off,
                   const long long* group_base, int N, long long G, unsigned order, int width_limit,
                   unsigned short* row_bytes, int* group_tot, int* alpha_any, const long long* chan_off,
                   const long long* group_dst, uint8_t* out, long long out_bytes, cudaStream_t st);

// Validates a canvas description and derives the launch geometry.
int make_geom(const dbmp_canvas* cv, Geom* g, const char* who) {
  if (!cv) { set_error("%s: canvas is null", who); return DBMP_ERR_INVALID; }
  if (cv->height <= 0 || cv->width <= 0) { set_error("%s: canvas %dx%d is empty", who, cv->height, cv->width); return DBMP_ERR_INVALID; }
  if (cv->tile_size != 16 && cv->tile_size != 32) { set_error("%s: tile_size %d is not supported (16 or 32)", who, cv->tile_size); return DBMP_ERR_INVALID; }
  if (cv->num_prims < 0) { set_error("%s: num_prims %d < 0", who, cv->num_prims); return DBMP_ERR_INVALID; }
  if (cv->num_templates <= 0 || cv->tmpl_h < 2 || cv->tmpl_w < 2) {
    set_error("%s: template atlas %dx%dx%d is invalid (need P>=1, Ht,Wt>=2)", who, cv->num_templates, cv->tmpl_h, cv->tmpl_w);
    return DBMP_ERR_INVALID;
  }
  if (cv->atlas_kind < DBMP_ATLAS_F32 || cv->atlas_kind > DBMP_ATLAS_BF16_PAIR) { set_error("%s: atlas_kind %d unknown", who, cv->atlas_kind); return DBMP_ERR_INVALID; }
  if (!(cv->alpha_max >= 0.f && cv->alpha_max < INFINITY)) { set_error("%s: alpha_max %g is not a finite value >= 0", who, (double)cv->alpha_max); return DBMP_ERR_INVALID; }
  if (half_record(cv->atlas_kind) && !(cv->alpha_max <= 65504.f)) {
    set_error("%s: alpha_max %g exceeds the FP16 range of the half / bfloat16 atlas kinds", who, (double)cv->alpha_max);
    return DBMP_ERR_INVALID;
  }
  if (!(cv->t_stop >= 1e-30f && cv->t_stop < 1.f)) { set_error("%s: t_stop %g outside [1e-30, 1)", who, (double)cv->t_stop); return DBMP_ERR_INVALID; }
  if ((long long)cv->height * cv->width > (1ll << 31) / 4) { set_error("%s: canvas too large", who); return DBMP_ERR_INVALID; }
  g->H = cv->height; g->W = cv->width; g->TS = cv->tile_size;
  g->tilesX = (cv->width + cv->tile_size - 1) / cv->tile_size;
  g->tilesY = (cv->height + cv->tile_size - 1) / cv->tile_size;
  g->T = g->tilesX * g->tilesY;
  g->N = cv->num_prims; g->P = cv->num_templates; g->Ht = cv->tmpl_h; g->Wt = cv->tmpl_w;
  g->hx = 0.5f * (float)(cv->tmpl_w - 1);
  g->hy = 0.5f * (float)(cv->tmpl_h - 1);
  g->rxy = g->hx / g->hy;
  g->ryx = g->hy / g->hx;
  g->k23 = make_float2(8388608.f, 8388608.f);
  g->m1 = make_float2(-1.f, -1.f);
  g->nhx = make_float2(-g->hx, -g->hx);
  g->nhy = make_float2(-g->hy, -g->hy);
  g->rxy2 = make_float2(g->rxy, g->rxy);
  g->nryx2 = make_float2(-g->ryx, -g->ryx);
  g->kbias = 0x4B000000u * (unsigned)(cv->tmpl_w + 1);
  g->wm1 = (float)(cv->tmpl_w - 1);
  g->hm1 = (float)(cv->tmpl_h - 1);
  g->kind = cv->atlas_kind;
  g->alpha_max = cv->alpha_max;
  g->t_stop = cv->t_stop;
  g->fhx = 0.5f * (float)(Layout<32>::FW - 1);   // both tile sizes have the same footprint
  g->fhy = 0.5f * (float)(Layout<32>::FH - 1);
  grid_shape(cv->tmpl_w, &g->gsx, &g->gGx);
  grid_shape(cv->tmpl_h, &g->gsy, &g->gGy);
  g->solid_delta = 0;
  g->rec_off = 0;
  g->live = nullptr;
  g->changed = nullptr;
  if (cv->reserved == DBMP_CANVAS_FOLLOWED_ATLAS) {
    const dbmp_followed_canvas* f = reinterpret_cast<const dbmp_followed_canvas*>(cv);
    if (cv->atlas_kind != DBMP_ATLAS_F32 || !f->templates || !f->changed) {
      set_error("%s: a followed atlas is DBMP_ATLAS_F32 and comes with its templates and two flags", who);
      return DBMP_ERR_INVALID;
    }
    g->live = f->templates;
    g->changed = f->changed;
  }
  if (cv->reserved == DBMP_CANVAS_EXTENDED_ATLAS || g->live) {
    const AtlasExt x = atlas_ext(g->P, g->Ht, g->Wt, g->kind);
    g->kind = x.kind;
    g->rec_off = (long long)x.rec_off;
    g->solid_delta = (int)(x.solid_off - atlas_grid_offset(g->P, g->Ht, g->Wt, x.kind));
  }
  g->grid_off = (long long)atlas_grid_offset(g->P, g->Ht, g->Wt, g->kind);
  return DBMP_OK;
}

#define REQUIRE(cond, ...) \
  do { if (!(cond)) { set_error(__VA_ARGS__); return DBMP_ERR_INVALID; } } while (0)

}  // namespace dbmp

using namespace dbmp;

extern "C" {

const char* dbmp_last_error(void) { return g_err; }
int dbmp_version(void) { return 1; }

int dbmp_num_tiles(const dbmp_canvas* cv) {
  Geom g;
  if (make_geom(cv, &g, "dbmp_num_tiles") != DBMP_OK) return -1;
  return g.T;
}

size_t dbmp_prim_info_bytes(int num_prims) { return sizeof(PrimInfo) * (size_t)(num_prims > 0 ? num_prims : 0); }

int dbmp_template_bboxes(const float* templates, int P, int Ht, int Wt, float* out_bbox, void* stream) {
  REQUIRE(P >= 0 && Ht >= 2 && Wt >= 2, "dbmp_template_bboxes: bad atlas shape %dx%dx%d", P, Ht, Wt);
  REQUIRE(P == 0 || (templates && out_bbox), "dbmp_template_bboxes: null pointer");
  return launch_template_bboxes(templates, P, Ht, Wt, out_bbox, (cudaStream_t)stream);
}

int dbmp_template_blur(const float* templates, int P, int Ht, int Wt, float sigma, float* out, void* stream) {
  REQUIRE(P >= 0 && Ht >= 1 && Wt >= 1, "dbmp_template_blur: bad atlas shape %dx%dx%d", P, Ht, Wt);
  REQUIRE(P == 0 || (templates && out), "dbmp_template_blur: null pointer");
  REQUIRE(templates != out || !(sigma > 0.f), "dbmp_template_blur: in-place blur is not supported");
  return launch_template_blur(templates, P, Ht, Wt, sigma, out, (cudaStream_t)stream);
}

int dbmp_atlas_pack(const float* templates, int P, int Ht, int Wt, int kind, void* out, void* stream) {
  REQUIRE(P >= 0 && Ht >= 1 && Wt >= 1, "dbmp_atlas_pack: bad atlas shape %dx%dx%d", P, Ht, Wt);
  REQUIRE(P == 0 || (templates && out), "dbmp_atlas_pack: null pointer");
  return launch_atlas_pack(templates, P, Ht, Wt, kind, out, (cudaStream_t)stream);
}

size_t dbmp_atlas_bytes(int P, int Ht, int Wt, int kind) {
  if (P < 0 || Ht < 1 || Wt < 1) return 0;
  return atlas_bytes(P, Ht, Wt, kind);
}

size_t dbmp_atlas_extended_bytes(int P, int Ht, int Wt, int kind) {
  if (P < 0 || Ht < 1 || Wt < 1 || kind < DBMP_ATLAS_F32 || kind > DBMP_ATLAS_BF16_PAIR) return 0;
  return atlas_ext(P, Ht, Wt, kind).total;
}

int dbmp_atlas_pack_extended(const float* templates, int P, int Ht, int Wt, int kind, void* out, void* stream) {
  REQUIRE(P >= 0 && Ht >= 1 && Wt >= 1, "dbmp_atlas_pack_extended: bad atlas shape %dx%dx%d", P, Ht, Wt);
  REQUIRE(kind >= DBMP_ATLAS_F32 && kind <= DBMP_ATLAS_BF16_PAIR, "dbmp_atlas_pack_extended: kind %d unknown", kind);
  REQUIRE(P == 0 || (templates && out), "dbmp_atlas_pack_extended: null pointer");
  REQUIRE(((uintptr_t)out & 255) == 0, "dbmp_atlas_pack_extended: out must be 256-byte aligned");
  return launch_atlas_extended(templates, P, Ht, Wt, kind, out, (cudaStream_t)stream);
}

size_t dbmp_bin_workspace_bytes(const dbmp_canvas* cv, long long capacity) {
  Geom g;
  if (make_geom(cv, &g, "dbmp_bin_workspace_bytes") != DBMP_OK) return 0;
  (void)capacity;   // the row binning needs no scratch per list entry
  return bin_workspace_bytes(1, g.N, g.T, g.tilesX, g.tilesY);
}

size_t dbmp_bin_batch_workspace_bytes(const dbmp_canvas* cv, int batch) {
  Geom g;
  if (make_geom(cv, &g, "dbmp_bin_batch_workspace_bytes") != DBMP_OK || batch < 0) return 0;
  return bin_workspace_bytes(batch, g.N, g.T, g.tilesX, g.tilesY);
}

int dbmp_prepare(const dbmp_canvas* cv, const float* means2D, const float* radii, const float* rotations,
                 const float* opacities, const float* colors, const int32_t* sel, void* prim_info, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_prepare");
  if (rc) return rc;
  REQUIRE(g.N == 0 || (means2D && radii && rotations && opacities && colors && sel && prim_info),
          "dbmp_prepare: null pointer");
  REQUIRE(((uintptr_t)prim_info & 15) == 0, "dbmp_prepare: prim_info must be 16-byte aligned");
  return launch_prepare(g, means2D, radii, rotations, opacities, colors, sel, (PrimInfo*)prim_info,
                        (cudaStream_t)stream);
}

int dbmp_bin(const dbmp_canvas* cv, const float* means2D, const float* radii, const float* rotations,
             const float* opacities, const float* colors, const int32_t* sel, const float* tmpl_bbox,
             void* prim_info, int32_t* tile_offsets, int32_t* tile_indices, long long capacity,
             int32_t* total_out, int32_t* overflow_out, void* workspace, size_t workspace_bytes, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_bin");
  if (rc) return rc;
  REQUIRE(cv->bin_mode == DBMP_BIN_CONTENT || cv->bin_mode == DBMP_BIN_CULL || cv->bin_mode == DBMP_BIN_CONTENT_REF,
          "dbmp_bin: bin_mode %d unknown", cv->bin_mode);
  REQUIRE(g.N == 0 || (means2D && radii && rotations && opacities && colors && sel && prim_info),
          "dbmp_bin: null pointer");
  REQUIRE(cv->bin_mode == DBMP_BIN_CULL || tmpl_bbox, "dbmp_bin: tmpl_bbox is required in the DBMP_BIN_CONTENT modes");
  REQUIRE(tile_offsets && total_out && workspace, "dbmp_bin: null output or workspace");
  REQUIRE(capacity >= 0 && capacity <= 0x7fffffffll, "dbmp_bin: capacity %lld outside [0, 2^31)", capacity);
  REQUIRE(capacity == 0 || tile_indices, "dbmp_bin: tile_indices is null");
  REQUIRE(((uintptr_t)prim_info & 15) == 0 && ((uintptr_t)workspace & 255) == 0,
          "dbmp_bin: prim_info must be 16-byte and workspace 256-byte aligned");
  return launch_bin(g, 1, cv->bin_mode, means2D, radii, rotations, opacities, colors, sel, 0, tmpl_bbox,
                    (PrimInfo*)prim_info, tile_offsets, tile_indices, 0, capacity, total_out, overflow_out, 0,
                    nullptr, Follow{}, workspace, workspace_bytes, (cudaStream_t)stream);
}

static int bin_checked(const Geom& g, const char* who, const dbmp_canvas* cv, int batch, const float* means2D,
                       const float* radii, const float* rotations, const float* opacities, const float* colors,
                       const int32_t* sel, long long sel_stride, const float* tmpl_bbox, void* prim_info,
                       int32_t* tile_offsets, int32_t* tile_indices, long long index_stride, long long capacity,
                       int32_t* total_and_overflow, int32_t* host_flags, const Follow& follow, void* workspace,
                       size_t workspace_bytes, cudaStream_t st) {
  REQUIRE(batch >= 0, "%s: batch %d < 0", who, batch);
  if (batch == 0) return DBMP_OK;
  REQUIRE(cv->bin_mode == DBMP_BIN_CONTENT || cv->bin_mode == DBMP_BIN_CULL || cv->bin_mode == DBMP_BIN_CONTENT_REF,
          "%s: bin_mode %d unknown", who, cv->bin_mode);
  REQUIRE(g.N == 0 || (means2D && radii && rotations && opacities && colors && sel && prim_info), "%s: null pointer",
          who);
  REQUIRE(cv->bin_mode == DBMP_BIN_CULL || tmpl_bbox, "%s: tmpl_bbox is required in the DBMP_BIN_CONTENT modes", who);
  REQUIRE(tile_offsets && total_and_overflow && workspace, "%s: null output or workspace", who);
  REQUIRE(capacity >= 0 && capacity <= 0x7fffffffll, "%s: capacity %lld outside [0, 2^31)", who, capacity);
  REQUIRE(capacity <= index_stride || batch == 1, "%s: index_stride %lld below the capacity %lld", who, index_stride,
          capacity);
  REQUIRE(capacity == 0 || tile_indices, "%s: tile_indices is null", who);
  REQUIRE(sel_stride == 0 || sel_stride >= g.N, "%s: sel_stride %lld", who, sel_stride);
  REQUIRE(((uintptr_t)prim_info & 15) == 0 && ((uintptr_t)workspace & 255) == 0,
          "%s: prim_info must be 16-byte and workspace 256-byte aligned", who);
  return launch_bin(g, batch, cv->bin_mode, means2D, radii, rotations, opacities, colors, sel, sel_stride, tmpl_bbox,
                    (PrimInfo*)prim_info, tile_offsets, tile_indices, index_stride, capacity, total_and_overflow,
                    total_and_overflow + 1, 2, host_flags, follow, workspace, workspace_bytes, st);
}

int dbmp_bin_batch(const dbmp_canvas* cv, int batch, const float* means2D, const float* radii,
                   const float* rotations, const float* opacities, const float* colors, const int32_t* sel,
                   long long sel_stride, const float* tmpl_bbox, void* prim_info, int32_t* tile_offsets,
                   int32_t* tile_indices, long long index_stride, long long capacity, int32_t* total_and_overflow,
                   void* workspace, size_t workspace_bytes, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_bin_batch");
  if (rc) return rc;
  return bin_checked(g, "dbmp_bin_batch", cv, batch, means2D, radii, rotations, opacities, colors, sel, sel_stride,
                     tmpl_bbox, prim_info, tile_offsets, tile_indices, index_stride, capacity, total_and_overflow,
                     nullptr, Follow{}, workspace, workspace_bytes, (cudaStream_t)stream);
}

int dbmp_render(const dbmp_canvas* cv, int batch, const float* means2D, const float* radii, const float* rotations,
                const float* opacities, const float* colors, const int32_t* sel, long long sel_stride,
                const float* tmpl_bbox, const void* atlas, void* prim_info, int32_t* tile_offsets,
                int32_t* tile_indices, long long index_stride, long long capacity, int32_t* total_and_overflow,
                int32_t* host_flags, const float* colors_orig, long long colors_orig_stride, float c_blend,
                float* out_color, float* out_alpha, float* T_last, int32_t* last_pos, void* walk_masks,
                void* workspace, size_t workspace_bytes, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_render");
  if (rc) return rc;
  if (batch == 0) return DBMP_OK;
  REQUIRE(atlas && out_color && out_alpha && T_last && last_pos && host_flags, "dbmp_render: null pointer");
  REQUIRE(colors_orig_stride >= 0, "dbmp_render: negative stride");
  REQUIRE(((uintptr_t)walk_masks & 15) == 0, "dbmp_render: walk_masks must be 16-byte aligned");
  REQUIRE(c_blend >= 0.f && c_blend <= 1.f, "dbmp_render: c_blend %g outside [0, 1]", (double)c_blend);
  REQUIRE(c_blend == 0.f || g.N == 0 || colors_orig, "dbmp_render: colors_orig is null with c_blend > 0");
  REQUIRE((long long)batch * g.T * 4 <= 0x7fffffffll, "dbmp_render: %d candidates x %d tiles exceed one grid", batch, g.T);
  // the host waits for the flags, which a captured launch would never write
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing((cudaStream_t)stream, &cap);
  if (e != cudaSuccess) return cuda_status(e, "dbmp_render: cudaStreamIsCapturing");
  REQUIRE(cap == cudaStreamCaptureStatusNone, "dbmp_render: cannot be captured in a CUDA graph (the list length is "
          "read on the host)");
  for (int b = 0; b < batch; ++b) host_flags[2 * b + 1] = -1;
  rc = bin_checked(g, "dbmp_render", cv, batch, means2D, radii, rotations, opacities, colors, sel, sel_stride,
                   tmpl_bbox, prim_info, tile_offsets, tile_indices, index_stride, capacity, total_and_overflow,
                   host_flags, make_follow(g, g.records(atlas), 0), workspace, workspace_bytes, (cudaStream_t)stream);
  if (rc) return rc;
  // the forward runs behind the binning without waiting for the host; a
  // candidate whose lists overflowed renders nothing, and none does when the
  // templates of a followed atlas have changed
  return launch_forward_blend(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices,
                              out_color, out_alpha, T_last, last_pos, colors_orig, c_blend, (cudaStream_t)stream,
                              batch, index_stride, colors_orig_stride, total_and_overflow, walk_masks);
}

int dbmp_convert_half(int n, const void* const* src, void* const* dst, const long long* counts, int to_half,
                      void* stream) {
  REQUIRE(n >= 0 && n <= 8, "dbmp_convert_half: %d arrays outside [0, 8]", n);
  REQUIRE(n == 0 || (src && dst && counts), "dbmp_convert_half: null pointer");
  for (int k = 0; k < n; ++k) {
    REQUIRE(counts[k] >= 0, "dbmp_convert_half: negative count");
    REQUIRE(counts[k] == 0 || (src[k] && dst[k]), "dbmp_convert_half: null array");
  }
  return launch_convert(n, src, dst, counts, to_half != 0, (cudaStream_t)stream);
}

int dbmp_render_wait(const int32_t* host_flags, int batch, void* stream) {
  REQUIRE(host_flags && batch >= 0, "dbmp_render_wait: null pointer");
  const volatile int32_t* f = host_flags;
  const auto t0 = std::chrono::steady_clock::now();
  for (int b = 0; b < batch; ++b) {
    for (unsigned spin = 1; f[2 * b + 1] < 0; ++spin) {
      if (spin % 4096 != 0) continue;
      // the binning of an idle stream reports within 0.3 ms (4096x4096, N=100000);
      // behind a longer queue a core is not held: 50 us more are little there
      auto waited = std::chrono::steady_clock::now() - t0;
      while (f[2 * b + 1] < 0 && waited >= std::chrono::milliseconds(1) && waited < std::chrono::seconds(2)) {
        std::this_thread::sleep_for(std::chrono::microseconds(50));
        waited = std::chrono::steady_clock::now() - t0;
      }
      // a launch that failed, or a stream busy for long: wait for it as usual
      if (f[2 * b + 1] >= 0 || waited < std::chrono::seconds(2)) continue;
      const cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
      if (e != cudaSuccess) return cuda_status(e, "dbmp_render_wait: cudaStreamSynchronize");
      REQUIRE(f[2 * b + 1] >= 0, "dbmp_render_wait: the binning did not report");
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return DBMP_OK;
}

int dbmp_forward(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                 const int32_t* tile_indices, float* out_color, float* out_alpha, float* T_last, int32_t* last_pos,
                 void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_forward");
  if (rc) return rc;
  REQUIRE(atlas && tile_offsets && tile_indices && out_color && out_alpha && T_last && last_pos,
          "dbmp_forward: null pointer");
  REQUIRE(g.N == 0 || prim_info, "dbmp_forward: prim_info is null");
  return launch_forward(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices, out_color,
                        out_alpha, T_last, last_pos, (cudaStream_t)stream);
}

int dbmp_backward(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                  const int32_t* tile_indices, const float* T_last, const int32_t* last_pos, const float* grad_color,
                  const float* grad_alpha, const float* radii, const float* rotations, const float* opacities,
                  const float* colors, double* grad_accum, float* grad_means2D, float* grad_radii,
                  float* grad_rotations, float* grad_opacities, float* grad_colors, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_backward");
  if (rc) return rc;
  REQUIRE(atlas && tile_offsets && tile_indices && T_last && last_pos && grad_color, "dbmp_backward: null input");
  REQUIRE(g.N == 0 || (prim_info && radii && rotations && opacities && colors), "dbmp_backward: null parameter");
  REQUIRE(g.N == 0 || (grad_accum && grad_means2D && grad_radii && grad_rotations && grad_opacities && grad_colors),
          "dbmp_backward: null output");
  cudaStream_t st = (cudaStream_t)stream;
  rc = launch_zero(grad_accum, 8ll * g.N, nullptr, make_follow(g, g.records(atlas), 1), st);
  if (rc) return rc;
  rc = launch_backward(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices, T_last,
                       last_pos, grad_color, grad_alpha, grad_accum, st);
  if (rc) return rc;
  return launch_finalize(g, radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii,
                         grad_rotations, grad_opacities, grad_colors, st);
}

int dbmp_grads_from_accum(const dbmp_canvas* cv, const double* grad_accum, const float* radii,
                          const float* rotations, const float* opacities, const float* colors, float* grad_means2D,
                          float* grad_radii, float* grad_rotations, float* grad_opacities, float* grad_colors,
                          void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_grads_from_accum");
  if (rc) return rc;
  REQUIRE(g.N == 0 || (grad_accum && radii && rotations && opacities && colors), "dbmp_grads_from_accum: null input");
  REQUIRE(g.N == 0 || (grad_means2D && grad_radii && grad_rotations && grad_opacities && grad_colors),
          "dbmp_grads_from_accum: null output");
  return launch_finalize(g, radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii,
                         grad_rotations, grad_opacities, grad_colors, (cudaStream_t)stream);
}

int dbmp_forward_blend(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                       const int32_t* tile_indices, const float* colors_orig, float c_blend, float* out_color,
                       float* out_alpha, float* T_last, int32_t* last_pos, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_forward_blend");
  if (rc) return rc;
  REQUIRE(atlas && tile_offsets && tile_indices && out_color && out_alpha && T_last && last_pos,
          "dbmp_forward_blend: null pointer");
  REQUIRE(g.N == 0 || prim_info, "dbmp_forward_blend: prim_info is null");
  REQUIRE(c_blend >= 0.f && c_blend <= 1.f, "dbmp_forward_blend: c_blend %g outside [0, 1]", (double)c_blend);
  REQUIRE(c_blend == 0.f || g.N == 0 || colors_orig, "dbmp_forward_blend: colors_orig is null with c_blend > 0");
  return launch_forward_blend(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices,
                              out_color, out_alpha, T_last, last_pos, colors_orig, c_blend, (cudaStream_t)stream, 1,
                              0, 0, nullptr, nullptr);
}

int dbmp_backward_blend(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                        const int32_t* tile_indices, const float* colors_orig, float c_blend, const float* T_last,
                        const int32_t* last_pos, const float* grad_color, const float* grad_alpha,
                        const float* radii, const float* rotations, const float* opacities, const float* colors,
                        double* grad_accum, float* grad_means2D, float* grad_radii, float* grad_rotations,
                        float* grad_opacities, float* grad_colors, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_backward_blend");
  if (rc) return rc;
  REQUIRE(atlas && tile_offsets && tile_indices && T_last && last_pos && grad_color,
          "dbmp_backward_blend: null input");
  REQUIRE(g.N == 0 || (prim_info && radii && rotations && opacities && colors), "dbmp_backward_blend: null parameter");
  REQUIRE(g.N == 0 || (grad_accum && grad_means2D && grad_radii && grad_rotations && grad_opacities && grad_colors),
          "dbmp_backward_blend: null output");
  REQUIRE(c_blend >= 0.f && c_blend <= 1.f, "dbmp_backward_blend: c_blend %g outside [0, 1]", (double)c_blend);
  REQUIRE(c_blend == 0.f || g.N == 0 || colors_orig, "dbmp_backward_blend: colors_orig is null with c_blend > 0");
  cudaStream_t st = (cudaStream_t)stream;
  rc = launch_zero(grad_accum, 8ll * g.N, nullptr, make_follow(g, g.records(atlas), 1), st);
  if (rc) return rc;
  rc = launch_backward_blend(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices,
                             T_last, last_pos, grad_color, grad_alpha, grad_accum, colors_orig, c_blend, st, 1, 0, 0,
                             nullptr);
  if (rc) return rc;
  return launch_finalize(g, radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii,
                         grad_rotations, grad_opacities, grad_colors, st);
}

int dbmp_forward_batch(const dbmp_canvas* cv, int batch, const void* prim_info, const void* atlas,
                       const int32_t* tile_offsets, const int32_t* tile_indices, long long index_stride,
                       const float* colors_orig, long long colors_orig_stride, float c_blend, float* out_color,
                       float* out_alpha, float* T_last, int32_t* last_pos, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_forward_batch");
  if (rc) return rc;
  REQUIRE(batch >= 0, "dbmp_forward_batch: batch %d < 0", batch);
  REQUIRE(index_stride >= 0 && colors_orig_stride >= 0, "dbmp_forward_batch: negative stride");
  REQUIRE(batch == 0 || (atlas && tile_offsets && tile_indices && out_color && out_alpha && T_last && last_pos),
          "dbmp_forward_batch: null pointer");
  REQUIRE(batch == 0 || g.N == 0 || prim_info, "dbmp_forward_batch: prim_info is null");
  REQUIRE(c_blend >= 0.f && c_blend <= 1.f, "dbmp_forward_batch: c_blend %g outside [0, 1]", (double)c_blend);
  REQUIRE(c_blend == 0.f || g.N == 0 || colors_orig, "dbmp_forward_batch: colors_orig is null with c_blend > 0");
  REQUIRE(((uintptr_t)prim_info & 15) == 0, "dbmp_forward_batch: prim_info must be 16-byte aligned");
  return launch_forward_blend(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices,
                              out_color, out_alpha, T_last, last_pos, colors_orig, c_blend, (cudaStream_t)stream,
                              batch, index_stride, colors_orig_stride, nullptr, nullptr);
}

static int backward_batch(const char* who, const void* walk_masks, const dbmp_canvas* cv, int batch,
                          const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                          const int32_t* tile_indices, long long index_stride, const float* colors_orig,
                          long long colors_orig_stride, float c_blend, const float* T_last, const int32_t* last_pos,
                          const float* grad_color, const float* grad_alpha, const float* radii,
                          const float* rotations, const float* opacities, const float* colors, double* grad_accum,
                          float* grad_means2D, float* grad_radii, float* grad_rotations, float* grad_opacities,
                          float* grad_colors, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, who);
  if (rc) return rc;
  REQUIRE(batch >= 0, "%s: batch %d < 0", who, batch);
  REQUIRE(index_stride >= 0 && colors_orig_stride >= 0, "%s: negative stride", who);
  REQUIRE(batch == 0 || (atlas && tile_offsets && tile_indices && T_last && last_pos && grad_color),
          "%s: null input", who);
  const bool work = batch > 0 && g.N > 0;
  REQUIRE(!work || (prim_info && radii && rotations && opacities && colors), "%s: null parameter", who);
  REQUIRE(!work || (grad_accum && grad_means2D && grad_radii && grad_rotations && grad_opacities && grad_colors),
          "%s: null output", who);
  REQUIRE(c_blend >= 0.f && c_blend <= 1.f, "%s: c_blend %g outside [0, 1]", who, (double)c_blend);
  REQUIRE(c_blend == 0.f || g.N == 0 || colors_orig, "%s: colors_orig is null with c_blend > 0", who);
  if (!work) return DBMP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  rc = launch_zero(grad_accum, 8ll * g.N * batch, nullptr, make_follow(g, g.records(atlas), 1), st);
  if (rc) return rc;
  rc = launch_backward_blend(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices,
                             T_last, last_pos, grad_color, grad_alpha, grad_accum, colors_orig, c_blend, st, batch,
                             index_stride, colors_orig_stride, walk_masks);
  if (rc) return rc;
  // the chain rule is per primitive: the batch's (B, N) primitives are one flat array
  Geom gb = g;
  gb.N = g.N * batch;
  return launch_finalize(gb, radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii,
                         grad_rotations, grad_opacities, grad_colors, st);
}

int dbmp_backward_batch(const dbmp_canvas* cv, int batch, const void* prim_info, const void* atlas,
                        const int32_t* tile_offsets, const int32_t* tile_indices, long long index_stride,
                        const float* colors_orig, long long colors_orig_stride, float c_blend, const float* T_last,
                        const int32_t* last_pos, const float* grad_color, const float* grad_alpha,
                        const float* radii, const float* rotations, const float* opacities, const float* colors,
                        double* grad_accum, float* grad_means2D, float* grad_radii, float* grad_rotations,
                        float* grad_opacities, float* grad_colors, void* stream) {
  return backward_batch("dbmp_backward_batch", nullptr, cv, batch, prim_info, atlas, tile_offsets, tile_indices,
                        index_stride, colors_orig, colors_orig_stride, c_blend, T_last, last_pos, grad_color, grad_alpha,
                        radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii, grad_rotations,
                        grad_opacities, grad_colors, stream);
}

int dbmp_backward_masked(const dbmp_canvas* cv, int batch, const void* walk_masks, const void* prim_info,
                         const void* atlas, const int32_t* tile_offsets, const int32_t* tile_indices,
                         long long index_stride, const float* colors_orig, long long colors_orig_stride,
                         float c_blend, const float* T_last, const int32_t* last_pos, const float* grad_color,
                         const float* grad_alpha, const float* radii, const float* rotations, const float* opacities,
                         const float* colors, double* grad_accum, float* grad_means2D, float* grad_radii,
                         float* grad_rotations, float* grad_opacities, float* grad_colors, void* stream) {
  REQUIRE(((uintptr_t)walk_masks & 15) == 0, "dbmp_backward_masked: walk_masks must be 16-byte aligned");
  return backward_batch("dbmp_backward_masked", walk_masks, cv, batch, prim_info, atlas, tile_offsets, tile_indices,
                        index_stride, colors_orig, colors_orig_stride, c_blend, T_last, last_pos, grad_color, grad_alpha,
                        radii, rotations, opacities, colors, grad_accum, grad_means2D, grad_radii, grad_rotations,
                        grad_opacities, grad_colors, stream);
}

size_t dbmp_walk_mask_bytes(const dbmp_canvas* cv, int batch) {
  Geom g;
  if (make_geom(cv, &g, "dbmp_walk_mask_bytes") != DBMP_OK || batch < 0) return 0;
  return walk_mask_bytes(g, batch);
}

int dbmp_count(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
               const int32_t* tile_indices, unsigned long long* counts, void* stream) {
  Geom g;
  // t_stop = 0 is allowed here: counting without termination (every fragment)
  dbmp_canvas c2 = cv ? *cv : dbmp_canvas{};
  const bool no_stop = cv && cv->t_stop == 0.f;
  if (no_stop) c2.t_stop = 0.5f;
  int rc = make_geom(cv ? &c2 : nullptr, &g, "dbmp_count");
  if (rc) return rc;
  if (no_stop) g.t_stop = 0.f;
  REQUIRE(atlas && tile_offsets && tile_indices && counts, "dbmp_count: null pointer");
  REQUIRE(g.N == 0 || prim_info, "dbmp_count: prim_info is null");
  cudaError_t e = cudaMemsetAsync(counts, 0, 10 * sizeof(unsigned long long), (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_status(e, "cudaMemsetAsync(counts)");
  return launch_count(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices, counts,
                      (cudaStream_t)stream);
}

int dbmp_fused_fwd_bwd(const dbmp_canvas* cv, const void* prim_info, const void* atlas, const int32_t* tile_offsets,
                       const int32_t* tile_indices, const float* target, const float* background, float* out_image,
                       double* grad_accum, double* loss_out, const int32_t* skip_flag, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_fused_fwd_bwd");
  if (rc) return rc;
  REQUIRE(atlas && tile_offsets && tile_indices && target && loss_out, "dbmp_fused_fwd_bwd: null input");
  REQUIRE(g.N == 0 || (prim_info && grad_accum), "dbmp_fused_fwd_bwd: null prim_info / grad_accum");
  cudaStream_t st = (cudaStream_t)stream;
  rc = launch_zero(grad_accum, 8ll * g.N, loss_out, make_follow(g, g.records(atlas), 1), st);
  if (rc) return rc;
  return launch_fused(g, g.kind, (const PrimInfo*)prim_info, g.records(atlas), tile_offsets, tile_indices, target,
                      background, out_image, grad_accum, loss_out, skip_flag, st);
}

int dbmp_adam_step(const dbmp_canvas* cv, const dbmp_adam_cfg* cfg, const double* grad_accum, float* means2D,
                   float* radii, float* rotations, float* opacities, float* colors, float* adam_m, float* adam_v,
                   int32_t* step_count, const int32_t* skip_flag, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_adam_step");
  if (rc) return rc;
  REQUIRE(cfg && step_count, "dbmp_adam_step: null cfg / step_count");
  REQUIRE(g.N == 0 || (grad_accum && means2D && radii && rotations && opacities && colors && adam_m && adam_v),
          "dbmp_adam_step: null pointer");
  REQUIRE(cfg->beta1 >= 0.f && cfg->beta1 < 1.f && cfg->beta2 >= 0.f && cfg->beta2 < 1.f && cfg->eps > 0.f,
          "dbmp_adam_step: betas must be in [0,1) and eps > 0");
  AdamArgs a;
  for (int k = 0; k < 8; ++k) a.lr[k] = cfg->lr[k];
  a.beta1 = cfg->beta1; a.beta2 = cfg->beta2; a.eps = cfg->eps;
  a.x_max = cfg->x_max; a.y_max = cfg->y_max; a.r_min = cfg->r_min; a.r_max = cfg->r_max;
  a.clamp = cfg->clamp;
  a.gamma = (cfg->lr_gamma == 0.f) ? 1.f : cfg->lr_gamma;
  REQUIRE(a.gamma > 0.f && a.gamma <= 1e6f, "dbmp_adam_step: lr_gamma %g must be positive", (double)cfg->lr_gamma);
  return launch_adam(g, a, grad_accum, means2D, radii, rotations, opacities, colors, adam_m, adam_v, step_count,
                     skip_flag, (cudaStream_t)stream);
}

int dbmp_prune(const dbmp_canvas* cv, const dbmp_prune_cfg* cfg, const int32_t* step_count, const float* pool,
               int32_t* state, float* means2D, float* radii, float* rotations, float* opacities, float* colors,
               const int32_t* skip_flag, void* stream) {
  Geom g;
  int rc = make_geom(cv, &g, "dbmp_prune");
  if (rc) return rc;
  REQUIRE(cfg && step_count && state, "dbmp_prune: null cfg / step_count / state");
  REQUIRE(cfg->every >= 1 && cfg->pool_rows >= 1, "dbmp_prune: every (%d) and pool_rows (%d) must be >= 1",
          cfg->every, cfg->pool_rows);
  REQUIRE(g.N == 0 || (pool && means2D && radii && rotations && opacities && colors), "dbmp_prune: null pointer");
  PruneArgs a{cfg->every, cfg->num_iterations, cfg->no_prune_last, cfg->warmup, cfg->threshold, cfg->pool_rows};
  return launch_prune(g, a, step_count, pool, state, means2D, radii, rotations, opacities, colors, skip_flag,
                      (cudaStream_t)stream);
}

int dbmp_template_blur_scheduled(const float* templates, int P, int Ht, int Wt, const dbmp_blur_schedule* sched,
                                 const int32_t* step_count, float* out, void* stream) {
  REQUIRE(P >= 0 && Ht >= 1 && Wt >= 1, "dbmp_template_blur_scheduled: bad atlas shape %dx%dx%d", P, Ht, Wt);
  REQUIRE(sched && step_count, "dbmp_template_blur_scheduled: null schedule / step_count");
  REQUIRE(P == 0 || (templates && out && templates != out), "dbmp_template_blur_scheduled: null or in-place buffers");
  REQUIRE(sched->mode >= 0 && sched->mode <= 2, "dbmp_template_blur_scheduled: mode %d unknown", sched->mode);
  REQUIRE(sched->mode != 2 || sched->num_iterations >= 1, "dbmp_template_blur_scheduled: num_iterations must be >= 1");
  return launch_template_blur_sched(templates, P, Ht, Wt, sched, step_count, out, (cudaStream_t)stream);
}

int dbmp_psd_bboxes(const float* means2D, const float* radii, int N, int H, int W, float scale, int32_t* out_bbox,
                    int32_t* out_sizes, void* stream) {
  REQUIRE(N >= 0 && H > 0 && W > 0, "dbmp_psd_bboxes: bad sizes N=%d H=%d W=%d", N, H, W);
  REQUIRE(N == 0 || (means2D && radii && out_bbox && out_sizes), "dbmp_psd_bboxes: null pointer");
  REQUIRE(((uintptr_t)out_bbox & 15) == 0, "dbmp_psd_bboxes: out_bbox must be 16-byte aligned");
  return launch_psd_bboxes(means2D, radii, N, H, W, scale, out_bbox, out_sizes, (cudaStream_t)stream);
}

int dbmp_psd_layout(const int32_t* sizes, int N, int64_t* layer_offsets, int64_t* block_offsets,
                    int64_t* total_bytes, void* stream) {
  REQUIRE(N >= 0, "dbmp_psd_layout: N=%d", N);
  REQUIRE(block_offsets && total_bytes && (N == 0 || (sizes && layer_offsets)), "dbmp_psd_layout: null pointer");
  return launch_psd_layout(sizes, N, (long long*)layer_offsets, (long long*)block_offsets, (long long*)total_bytes,
                           (cudaStream_t)stream);
}

int dbmp_psd_layers(const float* means2D, const float* radii, const float* rotations, const float* colors,
                    const float* visibility, const float* templates, int P, int Ht, int Wt, const int32_t* sel,
                    const int32_t* bbox, const int64_t* layer_offsets, const int64_t* block_offsets, int N,
                    float scale, float alpha_max, float c_blend, const float* colors_orig, uint8_t* out,
                    void* stream) {
  REQUIRE(N >= 0 && P > 0 && Ht >= 2 && Wt >= 2, "dbmp_psd_layers: bad sizes N=%d P=%d Ht=%d Wt=%d", N, P, Ht, Wt);
  REQUIRE(N == 0 || (means2D && radii && rotations && colors && visibility && templates && sel && bbox &&
                     layer_offsets && block_offsets && out), "dbmp_psd_layers: null pointer");
  REQUIRE(((uintptr_t)bbox & 15) == 0 && ((uintptr_t)out & 3) == 0,
          "dbmp_psd_layers: bbox must be 16-byte and out 4-byte aligned");
  return launch_psd_layers(N, P, Ht, Wt, scale, alpha_max, c_blend, means2D, radii, rotations, colors, visibility,
                           templates, sel, bbox, (const long long*)layer_offsets, (const long long*)block_offsets,
                           colors_orig, out, (cudaStream_t)stream);
}

static int check_psd_rle(const char* who, const uint8_t* layers, const int32_t* sizes, const int64_t* layer_offsets,
                         const int64_t* group_base, int N, long long num_groups, int channel_order,
                         int width_limit, const uint16_t* row_bytes) {
  REQUIRE(N >= 0 && num_groups >= 0, "%s: N=%d num_groups=%lld", who, N, num_groups);
  REQUIRE(width_limit >= 1 && width_limit <= 30000, "%s: width_limit %d outside [1, 30000] (PSD limit)", who,
          width_limit);
  REQUIRE(((unsigned)channel_order & ~0x03030303u) == 0, "%s: channel_order 0x%08x: each byte must be 0..3", who,
          (unsigned)channel_order);
  if (N == 0 || num_groups == 0) return DBMP_OK;
  REQUIRE(layers && sizes && layer_offsets && group_base && row_bytes, "%s: null pointer", who);
  REQUIRE(((uintptr_t)layers & 3) == 0 && ((uintptr_t)sizes & 3) == 0 && ((uintptr_t)row_bytes & 7) == 0,
          "%s: layers and sizes must be 4-byte and row_bytes 8-byte aligned", who);
  return DBMP_OK;
}

int dbmp_psd_rle_count(const uint8_t* layers, const int32_t* sizes, const int64_t* layer_offsets,
                       const int64_t* group_base, int N, long long num_groups, int channel_order, int width_limit,
                       uint16_t* row_bytes, int32_t* group_totals, int32_t* alpha_any, void* stream) {
  int rc = check_psd_rle("dbmp_psd_rle_count", layers, sizes, layer_offsets, group_base, N, num_groups,
                         channel_order, width_limit, row_bytes);
  if (rc != DBMP_OK) return rc;
  if (N == 0 || num_groups == 0) return DBMP_OK;
  REQUIRE(group_totals && ((uintptr_t)group_totals & 15) == 0,
          "dbmp_psd_rle_count: group_totals must be non-null and 16-byte aligned");
  return launch_psd_rle(false, layers, sizes, (const long long*)layer_offsets, (const long long*)group_base, N,
                        num_groups, (unsigned)channel_order, width_limit, (unsigned short*)row_bytes, group_totals,
                        alpha_any, nullptr, nullptr, nullptr, 0, (cudaStream_t)stream);
}

int dbmp_psd_rle_write(const uint8_t* layers, const int32_t* sizes, const int64_t* layer_offsets,
                       const int64_t* group_base, int N, long long num_groups, int channel_order, int width_limit,
                       const uint16_t* row_bytes, const int64_t* channel_offsets, const int64_t* group_offsets,
                       uint8_t* out, long long out_bytes, void* stream) {
  int rc = check_psd_rle("dbmp_psd_rle_write", layers, sizes, layer_offsets, group_base, N, num_groups,
                         channel_order, width_limit, row_bytes);
  if (rc != DBMP_OK) return rc;
  REQUIRE(out_bytes >= 0, "dbmp_psd_rle_write: out_bytes %lld < 0", out_bytes);
  if (N == 0 || num_groups == 0) return DBMP_OK;
  REQUIRE(channel_offsets && group_offsets && (out || out_bytes == 0), "dbmp_psd_rle_write: null pointer");
  return launch_psd_rle(true, layers, sizes, (const long long*)layer_offsets, (const long long*)group_base, N,
                        num_groups, (unsigned)channel_order, width_limit, (unsigned short*)row_bytes, nullptr,
                        nullptr, (const long long*)channel_offsets, (const long long*)group_offsets, out, out_bytes,
                        (cudaStream_t)stream);
}

}  // extern "C"
