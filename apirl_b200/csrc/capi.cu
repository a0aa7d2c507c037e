// The C ABI declared in include/apirl_b200.h: projector objects, argument
// checks, error reporting, and the MLEM / OSEM drivers.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>
#include <climits>

#include "internal.h"
#include "../../include/apirl_b200.h"

using apirl::HostTables;
using apirl::ImgGeom;
using apirl::LorTable;
using apirl::SubsetSel;

namespace {

thread_local std::string g_err;

}  // namespace

apirl_status apirl_internal_fail(apirl_status code, const char* msg) {
  g_err = msg;
  return code;
}

// A CUDA error left pending by an earlier launch (this library's or the
// caller's) is reported by the next entry point instead of being discarded:
// that call returns APIRL_ERR_CUDA naming the error and does no work.
// Reading the error resets a non-sticky one, as cudaGetLastError() does for
// any caller, so the call after it runs normally.
apirl_status apirl_internal_pending(void) {
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return APIRL_OK;
  char buf[384];
  snprintf(buf, sizeof buf, "a CUDA error was pending before this call (left by an earlier launch): %s: %s",
           cudaGetErrorName(e), cudaGetErrorString(e));
  g_err = buf;
  return e == cudaErrorMemoryAllocation ? APIRL_ERR_OOM : APIRL_ERR_CUDA;
}

namespace {

apirl_status fail(apirl_status code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

apirl_status cuda_fail(cudaError_t e, const char* what) {
  if (e == cudaErrorMemoryAllocation) return fail(APIRL_ERR_OOM, "%s: %s", what, cudaGetErrorString(e));
  return fail(APIRL_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define CK(call)                                                  \
  do {                                                            \
    cudaError_t e_ = (call);                                      \
    if (e_ != cudaSuccess) return cuda_fail(e_, #call);           \
  } while (0)

// Makes `dev` current for the scope and restores the caller's device after.
struct DeviceScope {
  int prev = -1;
  cudaError_t err = cudaSuccess;
  explicit DeviceScope(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) err = cudaSetDevice(dev);
  }
  ~DeviceScope() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

// Also refuses to run over an error pending from an earlier launch
// (apirl_internal_pending), so that the cudaGetLastError() after each of our
// launches reports that launch only.
#define DEVICE_SCOPE(dev)                                                       \
  DeviceScope scope_(dev);                                                      \
  if (scope_.err != cudaSuccess) return cuda_fail(scope_.err, "cudaSetDevice"); \
  if (apirl_status pend_ = apirl_internal_pending()) return pend_
#define NO_PENDING()                                         \
  do {                                                       \
    if (apirl_status pend_ = apirl_internal_pending()) return pend_; \
  } while (0)

// The accumulation form set on a projector applies to its padded passes; a
// projector that no longer takes them (FP64 walk, sampling, dual layout off)
// refuses to backproject with another form than plain atomics.
apirl_status check_acc(const apirl_projector* p) {
  const bool dual = p->is3d && p->dual_layout && !p->pg.enabled && p->pad.pA && !p->t.lor_s;
  if (p->pad.acc != APIRL_ACC_ATOMIC && !dual)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the accumulation form needs the padded 3D layouts");
  return APIRL_OK;
}

bool use_dual(const apirl_projector* p) {
  return p->is3d && p->dual_layout && !p->pg.enabled && p->pad.pA && !p->t.lor_s;
}

// The column walk serves the padded 3D passes with plain atomics.
bool use_cols(const apirl_projector* p) {
  return use_dual(p) && p->cols.half && p->pad.acc == APIRL_ACC_ATOMIC && !p->pad.window &&
         p->t.n_sinos >= apirl::kColMinSinos;
}

// The fused passes with several rays a bin: on their own column layout where
// set_sampling made it, from the sinograms on that pay in the plain passes.  A
// block holds a list a radial sample, so wide images and many samples leave
// few rays in flight on an SM (the blocks that their lists leave room for
// times the sinograms): over more than 2000 LORs the columns want 224 of them.
// Us bin by bin -> columns, by rays in flight, 5 % and 90 % bins with counts:
// 96 (16 sinograms, 64 x 64, 12 samples) 412 -> 887, 758 -> 981; 192 (24, 96 x
// 96, 6 samples) 732 -> 941, dense 0.88 of the time; 240 (40, 64 x 64, 12) 811
// -> 968, 0.71; 320 (40, 96 x 96, 6) 0.91 and 0.62; 861 LORs of the first job
// 0.71 and 0.67.
bool use_ray_cols(const apirl_projector* p, SubsetSel ss) {
  if (!(p->t.lor_s && p->dual_layout && !p->pg.enabled && p->ray_cols.half && p->pad.acc == APIRL_ACC_ATOMIC &&
        p->t.n_sinos >= apirl::kColMinSinos))
    return false;
  const size_t smem = p->t.n_rs * apirl::col_list_bytes(p->g) + 1536;  // the block's own and the reserved, too
  const int64_t blocks = std::min<int64_t>(32, 227 * 1024 / smem);
  return (int64_t)ss.nk * p->t.n_r <= 2000 || blocks * p->t.n_sinos >= 224;
}

// A slot for work queued on s until slot_done, which the lock covers: the one
// s used last, else the one unused the longest; s waits for its last use.
// (No event is queried: a query in one thread breaks a global-mode capture in
// another.)
template <int N>
apirl_status slot_take(apirl_projector::ColSlot (&slots)[N], cudaStream_t s, apirl_projector::ColSlot** out) {
  apirl_projector::ColSlot* pick = &slots[0];
  unsigned long long last = 0;
  for (auto& c : slots) {
    if (c.use < pick->use) pick = &c;
    if (c.use > last) last = c.use;
  }
  for (auto& c : slots)
    if (c.use && c.last == s) pick = &c;
  CK(cudaStreamWaitEvent(s, pick->done, 0));
  pick->last = s;
  pick->use = last + 1;
  *out = pick;
  return APIRL_OK;
}
apirl_status slot_done(apirl_projector::ColSlot* c, cudaStream_t s) {
  CK(cudaEventRecord(c->done, s));
  return APIRL_OK;
}
// Whether s is being captured: a captured call keeps to the kernels without
// slots (a graph may be replayed beside any other work).
apirl_status capturing(cudaStream_t s, bool* is) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(s, &cs));
  *is = cs != cudaStreamCaptureStatusNone;
  return APIRL_OK;
}

// Whether a projection takes the column walk.  Its block lists a LOR's
// crossings (about 2600 warp instructions) and its warps walk the sinograms 32
// at a time (250 each, 17 a step); the direct kernel sets every ray up (300 a
// warp) and takes 26 a step on bins finer than the voxels, up to 60 where they
// are as wide as the voxels and its lanes' voxels lie apart.  Measured, direct
// -> column walk in us, the smaller estimate last: 128 x 128 image, 166 x 166
// bins, 19 sinograms 153 -> 123 (columns), 91 sinograms 616 -> 247 (columns);
// 134 x 134 image, 344 bins, 34 sinograms 285 -> 373 (direct); 82 x 82, 344
// bins, 47 sinograms 83 -> 92 (direct); 58 x 58, 344 bins, 139 sinograms 175 ->
// 169 (columns).  With one warp a block, the lists of images wider than 160 x
// 160 leave fewer blocks on an SM than there is room for warps: measured over
// the estimate 0.98 at 160 x 160, 1.16 at 192 x 192, 1.40 at 224 x 224, 1.57 at
// 256 x 256 (16 sinograms, all angles, 765 -> 925 us; two warps a block 1.01).
// Below 1e7 bins times voxels of a row and a column, the copy's
// launch costs more than the walk gains (48 x 48 image, 57 K bins: 16.5 -> 18.6).
bool project_cols(const apirl_projector* p, SubsetSel ss) {
  const double side = (double)p->g.nx + p->g.ny;
  if ((double)p->t.n_sinos * ss.nk * p->t.n_r * side < 1e7) return false;
  const double pitch = 2.0 * p->r_fov / p->t.n_r / p->g.dx, steps = 0.65 * side;
  const double crowded = p->t.n_sinos <= 32 ? std::max(1.0, side / 323) : 1;
  const double cols = crowded * (2600 + (p->t.n_sinos + 31) / 32 * (250 + 17 * steps));
  const double direct = p->t.n_sinos / 32.0 * (300 + steps * (26 + 34 * (pitch < 1 ? pitch : 1)));
  return cols <= direct;
}

// Whether a DivideAndBackproject takes the column walk: not where its two
// launches take longer than the direct kernel's one (32 x 32 image: 9.2 K bins
// 13.3 -> 14.3 us, 60 K bins 27.6 -> 16.0; 64 x 64, 14 K bins 21.5 -> 16.3).
bool divide_cols(const apirl_projector* p, SubsetSel ss) {
  return (double)p->t.n_sinos * ss.nk * p->t.n_r * ((double)p->g.nx + p->g.ny) >= 1.5e6;
}

// Forward projection of the subset into d_sino.
apirl_status project(apirl_projector* p, SubsetSel ss, const float* d_image, float* d_sino, cudaStream_t s) {
  if (use_cols(p) && p->col_img[0].buf && project_cols(p, ss)) {
    bool captured = false;
    apirl_status st = capturing(s, &captured);
    if (st) return st;
    if (!captured) {
      std::lock_guard<std::mutex> lock(p->col_mu);
      apirl_projector::ColSlot* c = nullptr;
      if ((st = slot_take(p->col_img, s, &c))) return st;
      CK(apirl::launch_col_copy(p->g, p->cols, d_image, c->buf, s));
      CK(apirl::launch_project_cols(p->g, p->cols, p->t, ss, c->buf, d_sino, s));
      return slot_done(c, s);
    }
  }
  CK(apirl::launch_project(p->g, p->t, ss, d_image, d_sino, s, p->pg));
  return APIRL_OK;
}

bool valid_img(const apirl_image_geom* g) {
  return g && g->nx > 0 && g->ny > 0 && g->nz > 0 && g->dx > 0 && g->dy > 0 && g->dz > 0 &&
         (int64_t)g->nx * g->ny * g->nz < (int64_t)1 << 31;
}

// Bounds the length of every Siddon walk: a LOR spans at most the scanner
// diameter, so it records at most about 2 R / d segments per axis.  Geometries
// that would give walks of more than ~1e5 segments per axis are rejected.
bool walk_bounded(const apirl_image_geom* g, float r_scanner, float axial) {
  const float d = fminf(g->dx, fminf(g->dy, g->dz));
  const float span = fmaxf(2.f * r_scanner, axial);
  return span / d < 1.0e5f && (float)g->nx * g->dx < 1.0e6f && (float)g->nz * g->dz < 1.0e6f;
}

SubsetSel make_subset(const apirl_projector* p, int subset, int nsub) {
  SubsetSel s;
  s.subset = subset < 0 ? -1 : subset;
  s.nsub = subset < 0 ? 1 : nsub;
  s.nk = apirl::subset_nproj(p->t.n_proj, s.subset, s.nsub);
  return s;
}

apirl_status check_subset(const apirl_projector* p, int subset, int nsub) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  if (subset >= 0 && (nsub <= 0 || subset >= nsub || nsub > p->t.n_proj))
    return fail(APIRL_ERR_INVALID, "subset %d of %d is out of range (%d angles)", subset, nsub, p->t.n_proj);
  return APIRL_OK;
}

// Waits for the tables and zeros written on the legacy stream: a memset, or a
// copy from pageable memory, may return before the device has it, and a
// projector's first pass may run on a stream that does not wait for that one.
apirl_status settled() {
  CK(cudaStreamSynchronize(nullptr));
  return APIRL_OK;
}

// Places in a device block that is sized before it is taken: a fresh mapping
// costs about 0.35 ms (0.28 ms to free), whatever its size, so a projector's
// buffers share one.
struct Places {
  size_t bytes = 0;
  size_t add(size_t n) {
    const size_t at = bytes;
    bytes += (n + 511) / 512 * 512;
    return at;
  }
};

// The block of places() with the layouts that fit: those asked for, else
// fewer.  *out stays null where not even the last does (APIRL_ERR_OOM).
template <class F>
apirl_status take_block(apirl::Layouts& layouts, char** out, F&& places) {
  for (;;) {
    const cudaError_t e = cudaMalloc((void**)out, places(layouts).bytes);
    if (e == cudaSuccess) return APIRL_OK;
    *out = nullptr;
    if (e != cudaErrorMemoryAllocation || layouts == apirl::Layouts::kPair) return cuda_fail(e, "projector buffers");
    (void)cudaGetLastError();  // handled: not left for the next call
    layouts = layouts == apirl::Layouts::kCalls ? apirl::Layouts::kPasses : apirl::Layouts::kPair;
  }
}

// The projector's device block: tables and scratch; in 3D the padded
// two-layout buffers of the fused pass (volumes whose padded size does not fit
// a 32-bit index keep the single unpadded layout), with kPasses the column
// layout's image copy, sums and queue, with kCalls the slots'
// (apirl_projector::ColSlot) too; in 2D the padded slices.  All are made here,
// so that no later call allocates (passes may be captured into CUDA graphs).
apirl_status finish_create(apirl_projector* p, apirl_projector** out) {
  SubsetSel all = make_subset(p, -1, 1);
  p->n_partials = apirl::em_pass_blocks(p->t, all);
  const int64_t cp = apirl::col_partials(p->t, all) + apirl::col_dots(p->g);
  if (cp > p->n_partials) p->n_partials = cp;
  const int64_t lb = apirl::likelihood_blocks((int64_t)p->t.n_sinos * p->t.n_proj * p->t.n_r);
  if (lb > p->n_partials) p->n_partials = lb;
  const int64_t pv64 = (int64_t)(p->g.nx + 2 * apirl::kPad) * (p->g.ny + 2 * apirl::kPad) * (p->g.nz + 2 * apirl::kPad);
  const size_t pv = p->is3d && pv64 <= INT_MAX ? (size_t)pv64 : 0;
  apirl::ColBuffers c;
  if (p->is3d && p->host.n_sinos >= apirl::kColMinSinos)
    c = apirl::col_layout(p->g, p->host.z.data(), (int)p->host.z.size());
  const size_t n = c.half ? (size_t)c.floats : 0, lors = (size_t)p->t.n_proj * p->t.n_r;
  // (Images of several slices, of which a 2D pass projects the first and updates
  // all, keep to the unpadded pass.)
  const size_t lim = !p->is3d && p->g.nz == 1 && (int64_t)lors <= INT_MAX - 31 ? apirl::planar_lim(p->g) : 0;
  constexpr size_t copies = apirl::kPlanarCopies;
  size_t at_lor, at_z, at_ok, at_partials, at_minmax, at_scalars, at_chunk, at_item, at_list, at_bins, at_zeros, at_pad, at_col, at_planar;
  auto places = [&](apirl::Layouts l) {
    const bool more = l != apirl::Layouts::kPair;
    Places b;
    at_lor = b.add(p->host.lor.size() * sizeof(float));
    at_z = b.add(p->host.z.size() * sizeof(float));
    at_ok = b.add(p->host.ok.size());
    at_partials = b.add(p->n_partials * sizeof(double));
    at_minmax = b.add(2 * sizeof(unsigned));
    at_scalars = b.add(8 * sizeof(double));
    at_chunk = b.add(sizeof(unsigned long long) + 2 * sizeof(unsigned));  // and the queue's numbers
    const bool queue = more && n;
    const size_t line = (size_t)apirl::col_direct_lors(p->g), deferred = std::min(lors, line);
    at_item = b.add(queue ? deferred * sizeof(uint2) : 0);
    at_list = b.add(queue ? deferred * apirl::kColFew * sizeof(uint16_t) : 0);
    const size_t direct = apirl::col_direct_room(p->host.n_sinos);
    at_bins = b.add(queue && lors > line ? lors * direct * sizeof(unsigned) : 0);
    at_zeros = b.bytes;
    at_pad = b.add(4 * pv * sizeof(float));
    at_col = b.add((l == apirl::Layouts::kCalls ? 7 : more ? 3 : 0) * n * sizeof(float));
    at_planar = b.add(more ? 2 * (1 + copies) * lim * sizeof(float) : 0);
    return b;
  };
  if (apirl_status st = take_block(p->layouts, &p->block, places)) return st;
  char* const b = p->block;
  const size_t zeros = places(p->layouts).bytes - at_zeros;
  p->d_lor = (float4*)(b + at_lor);
  CK(cudaMemcpy(p->d_lor, p->host.lor.data(), p->host.lor.size() * sizeof(float), cudaMemcpyHostToDevice));
  p->d_z = (float2*)(b + at_z);
  CK(cudaMemcpy(p->d_z, p->host.z.data(), p->host.z.size() * sizeof(float), cudaMemcpyHostToDevice));
  p->d_ok = (uint8_t*)(b + at_ok);
  CK(cudaMemcpy(p->d_ok, p->host.ok.data(), p->host.ok.size(), cudaMemcpyHostToDevice));
  p->t.lor = p->d_lor;
  p->t.z = p->d_z;
  p->t.ok = p->d_ok;
  p->d_partials = (double*)(b + at_partials);
  p->d_minmax = (unsigned*)(b + at_minmax);
  p->d_scalars = (double*)(b + at_scalars);
  p->d_chunk = (unsigned long long*)(b + at_chunk);
  if (zeros) CK(cudaMemset(b + at_zeros, 0, zeros));
  if (p->is3d) CK(apirl::prepare_em_kernels(p->em_block));
  if (pv) {
    // The four images side by side: an L2 access policy window can cover them
    // all (APIRL_OPT_L2_PERSIST).
    p->pad.pA = (float*)(b + at_pad);
    p->pad.pT = p->pad.pA + pv;
    p->pad.bA = p->pad.pA + 2 * pv;
    p->pad.bT = p->pad.pA + 3 * pv;
    p->pad.lim = (unsigned)pv;
  }
  if (n && p->layouts != apirl::Layouts::kPair) {
    c.img = (float*)(b + at_col);
    c.acc = c.img + n;
    p->cols = c;
    p->queue.n = (unsigned*)(p->d_chunk + 1);
    p->queue.item = (uint2*)(b + at_item);
    p->queue.list = (uint16_t*)(b + at_list);
    p->queue.bins = (unsigned*)(b + at_bins);
  }
  if (n && p->layouts == apirl::Layouts::kCalls) {
    p->col_sum[0].buf = c.img + 3 * n;
    CK(cudaEventCreateWithFlags(&p->col_sum[0].done, cudaEventDisableTiming));
    for (int k = 0; k < 2; k++) {
      p->col_img[k].buf = c.img + (5 + k) * n;
      CK(cudaEventCreateWithFlags(&p->col_img[k].done, cudaEventDisableTiming));
    }
  }
  if (lim && p->layouts != apirl::Layouts::kPair) {
    apirl::PlanarBuffers& pl = p->planar;
    pl.img = (float*)(b + at_planar);
    pl.imgT = pl.img + lim;
    pl.sum = pl.imgT + lim;
    pl.sumT = pl.sum + copies * lim;
    pl.lim = (unsigned)lim;
  }
  if (apirl_status st = settled()) return st;
  *out = p;
  return APIRL_OK;
}

}  // namespace

namespace apirl {
// The host half of a 3D projector: checks the image and sinogram geometry
// (cylindrical or Siemens mMR) and builds the LOR and end-point tables into p
// (g, host, t's sizes, the geometry as given), touching no device.
apirl_status setup_3d(const apirl_image_geom* img, const apirl_sino3d_geom* sino, apirl_projector* p) {
  if (!sino) return fail(APIRL_ERR_INVALID, "invalid 3D sinogram geometry");
  if (sino->scanner != APIRL_SCANNER_CYLINDRICAL && sino->scanner != APIRL_SCANNER_MMR)
    return fail(APIRL_ERR_INVALID, "unknown scanner %d", sino->scanner);
  const bool mmr = sino->scanner == APIRL_SCANNER_MMR;
  if (!valid_img(img)) return fail(APIRL_ERR_INVALID, "invalid image geometry");
  if (mmr) {
    if (sino->n_proj < 2 || sino->n_r <= 0 || sino->n_rings <= 0 || sino->n_segments <= 0 || !sino->min_ring_diff ||
        !sino->max_ring_diff)
      return fail(APIRL_ERR_INVALID, "invalid mMR sinogram geometry (need n_proj >= 2, n_r, n_rings, segments)");
    if (!walk_bounded(img, apirl::kMmrRadius + apirl::kMmrDoi, apirl::kMmrAxialFov))
      return fail(APIRL_ERR_INVALID, "voxels too small for the scanner size (walks above 1e5 segments)");
  } else {
    if (sino->n_proj <= 0 || sino->n_r <= 0 || sino->n_rings <= 0 || sino->n_segments <= 0 ||
        !sino->min_ring_diff || !sino->max_ring_diff || !(sino->r_fov > 0) || !(sino->axial_fov > 0) ||
        !(sino->r_scanner > sino->r_fov))
      return fail(APIRL_ERR_INVALID, "invalid 3D sinogram geometry");
    if (!walk_bounded(img, sino->r_scanner, sino->axial_fov))
      return fail(APIRL_ERR_INVALID, "voxels too small for the scanner size (walks above 1e5 segments)");
  }
  for (int i = 0; i < sino->n_segments; i++)
    if (sino->min_ring_diff[i] > sino->max_ring_diff[i])
      return fail(APIRL_ERR_INVALID, "segment %d: minimum ring difference above maximum", i);
  p->is3d = 1;
  p->scanner = sino->scanner;
  p->g = make_img_geom(img->nx, img->ny, img->nz, img->dx, img->dy, img->dz);
  const bool built = mmr ? build_tables_mmr(sino->n_proj, sino->n_r, sino->n_rings, sino->n_segments,
                                            sino->min_ring_diff, sino->max_ring_diff, p->host)
                         : build_tables_3d(sino->n_proj, sino->n_r, sino->n_rings, sino->r_fov, sino->axial_fov,
                                           sino->r_scanner, sino->n_segments, sino->min_ring_diff,
                                           sino->max_ring_diff, p->host);
  if (!built) return fail(APIRL_ERR_INVALID, "segment table yields no sinograms");
  p->t.n_proj = sino->n_proj;
  p->t.n_r = sino->n_r;
  p->t.n_sinos = p->host.n_sinos;
  p->t.is3d = 1;
  p->n_rings = sino->n_rings;
  p->r_fov = mmr ? kMmrRFov : sino->r_fov;
  p->axial_fov = mmr ? kMmrAxialFov : sino->axial_fov;
  p->r_scanner = mmr ? kMmrRadius : sino->r_scanner;
  p->min_rd.assign(sino->min_ring_diff, sino->min_ring_diff + sino->n_segments);
  p->max_rd.assign(sino->max_ring_diff, sino->max_ring_diff + sino->n_segments);
  if ((int64_t)p->t.n_sinos * p->t.n_proj * p->t.n_r >= ((int64_t)1 << 40))
    return fail(APIRL_ERR_INVALID, "sinogram too large");
  return APIRL_OK;
}
}  // namespace apirl

namespace apirl {
apirl_status create_2d(const apirl_image_geom* img, const apirl_sino2d_geom* sino, int device, Layouts layouts,
                       apirl_projector** out) {
  if (!out) return fail(APIRL_ERR_INVALID, "null output pointer");
  *out = nullptr;
  if (!valid_img(img)) return fail(APIRL_ERR_INVALID, "invalid image geometry");
  if (!sino || sino->n_proj <= 0 || sino->n_r <= 0 || !(sino->r_fov > 0) || !(sino->r_scanner > sino->r_fov))
    return fail(APIRL_ERR_INVALID, "invalid 2D sinogram geometry (need n_proj, n_r > 0 and 0 < r_fov < r_scanner)");
  if (!walk_bounded(img, sino->r_scanner, 0.f))
    return fail(APIRL_ERR_INVALID, "voxels too small for the scanner radius (walks above 1e5 segments)");
  DEVICE_SCOPE(device);
  apirl_projector* p = new apirl_projector;
  p->device = device;
  p->layouts = layouts;
  p->is3d = 0;
  p->g = make_img_geom(img->nx, img->ny, img->nz, img->dx, img->dy, img->dz);
  build_tables_2d(sino->n_proj, sino->n_r, sino->r_fov, sino->r_scanner, p->host);
  p->t.n_proj = sino->n_proj;
  p->t.n_r = sino->n_r;
  p->t.n_sinos = 1;
  p->t.is3d = 0;
  apirl_status st = finish_create(p, out);
  if (st != APIRL_OK) { std::string m = g_err; apirl_projector_destroy(p); g_err = m; }
  return st;
}

apirl_status create_3d(const apirl_image_geom* img, const apirl_sino3d_geom* sino, int device, Layouts layouts,
                       apirl_projector** out) {
  if (!out) return fail(APIRL_ERR_INVALID, "null output pointer");
  *out = nullptr;
  apirl_projector* p = new apirl_projector;
  apirl_status st = setup_3d(img, sino, p);
  if (st != APIRL_OK) {
    delete p;
    return st;
  }
  {
    DEVICE_SCOPE(device);
    p->device = device;
    p->layouts = layouts;
    st = finish_create(p, out);
  }
  if (st != APIRL_OK) { std::string m = g_err; apirl_projector_destroy(p); g_err = m; }
  return st;
}
}  // namespace apirl

extern "C" {

const char* apirl_last_error(void) { return g_err.c_str(); }
const char* apirl_version(void) { return "apirl_b200 0.1 (sm_100a)"; }

apirl_status apirl_lor_table(int n_proj, int n_r, float r_fov, float r_scanner, float* h_lor) {
  if (n_proj <= 0 || n_r <= 0 || !h_lor || !(r_scanner > r_fov)) return fail(APIRL_ERR_INVALID, "bad arguments");
  HostTables t;
  apirl::build_tables_2d(n_proj, n_r, r_fov, r_scanner, t);
  memcpy(h_lor, t.lor.data(), t.lor.size() * sizeof(float));
  return APIRL_OK;
}

int apirl_sino3d_ring_z(const apirl_sino3d_geom* sino, float* h_z) {
  if (!sino || sino->n_rings <= 0 || sino->n_segments <= 0 || !sino->min_ring_diff || !sino->max_ring_diff) {
    fail(APIRL_ERR_INVALID, "invalid 3D sinogram geometry");
    return -1;
  }
  HostTables t;
  const float afov = sino->scanner == APIRL_SCANNER_MMR ? apirl::kMmrAxialFov : sino->axial_fov;
  if (!apirl::build_tables_3d(1, 1, sino->n_rings, 1.f, afov, 2.f, sino->n_segments,
                              sino->min_ring_diff, sino->max_ring_diff, t))
    return 0;
  if (h_z) memcpy(h_z, t.z.data(), t.z.size() * sizeof(float));
  return t.n_sinos;
}

apirl_status apirl_projector_create_2d(const apirl_image_geom* img, const apirl_sino2d_geom* sino, int device,
                                       apirl_projector** out) {
  return apirl::create_2d(img, sino, device, apirl::Layouts::kCalls, out);
}

apirl_status apirl_mmr_lor_table(int n_proj, int n_r, float* h_lor) {
  if (n_proj < 2 || n_r <= 0 || !h_lor) return fail(APIRL_ERR_INVALID, "bad arguments");
  std::vector<float> lor;
  apirl::mmr_lor_table(n_proj, n_r, lor);
  memcpy(h_lor, lor.data(), lor.size() * sizeof(float));
  return APIRL_OK;
}

apirl_status apirl_projector_create_3d_mmr(const apirl_image_geom* img, int n_proj, int n_r, int n_rings,
                                           int n_segments, const int* min_ring_diff, const int* max_ring_diff,
                                           int device, apirl_projector** out) {
  apirl_sino3d_geom sino;
  memset(&sino, 0, sizeof sino);
  sino.n_proj = n_proj;
  sino.n_r = n_r;
  sino.n_rings = n_rings;
  sino.n_segments = n_segments;
  sino.min_ring_diff = min_ring_diff;
  sino.max_ring_diff = max_ring_diff;
  sino.scanner = APIRL_SCANNER_MMR;
  return apirl_projector_create_3d(img, &sino, device, out);
}

apirl_status apirl_projector_create_3d(const apirl_image_geom* img, const apirl_sino3d_geom* sino, int device,
                                       apirl_projector** out) {
  return apirl::create_3d(img, sino, device, apirl::Layouts::kCalls, out);
}

void apirl_projector_destroy(apirl_projector* p) {
  if (!p) return;
  DeviceScope scope(p->device);
  if (p->l2_limit_set) cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, p->l2_limit_prev);
  cudaFree(p->block);
  cudaFree(p->ray_block);
  cudaFree(p->pad2.bA);
  cudaFree(p->pad2.bT);
  cudaFree(p->nz.list);
  cudaFree(p->nz.tiles);
  cudaFree(p->nz.n_list);
  cudaFree(p->d_lor64);
  cudaFree(p->d_z64);
  for (auto& c : p->col_img)
    if (c.done) cudaEventDestroy(c.done);
  for (auto& c : p->col_sum)
    if (c.done) cudaEventDestroy(c.done);
  cudaFree(p->pad.eA);
  cudaFree(p->pad.eT);
  if (p->ev0) cudaEventDestroy(p->ev0);
  if (p->ev1) cudaEventDestroy(p->ev1);
  if (p->copy_ready) cudaEventDestroy(p->copy_ready);
  for (auto& e : p->staged)
    if (e.done) cudaEventDestroy(e.done);
  if (p->copy_stream) cudaStreamDestroy(p->copy_stream);
  delete p;
}

int64_t apirl_projector_num_bins(const apirl_projector* p, int subset, int nsubsets) {
  if (!p || (subset >= 0 && (nsubsets <= 0 || subset >= nsubsets))) return -1;
  SubsetSel s = make_subset(p, subset, nsubsets);
  return (int64_t)p->t.n_sinos * s.nk * p->t.n_r;
}

int apirl_projector_num_sinograms(const apirl_projector* p) { return p ? p->host.n_sinos : -1; }

apirl_status apirl_projector_tables(const apirl_projector* p, float* h_lor, float* h_z) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  if (h_lor) memcpy(h_lor, p->host.lor.data(), p->host.lor.size() * sizeof(float));
  if (h_z && p->is3d) memcpy(h_z, p->host.z.data(), p->host.z.size() * sizeof(float));
  return APIRL_OK;
}

apirl_status apirl_projector_set_alpha_precision(apirl_projector* p, int mode) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  if (mode != APIRL_ALPHA_F32 && mode != APIRL_ALPHA_F64) return fail(APIRL_ERR_INVALID, "unknown alpha mode %d", mode);
  if (mode == APIRL_ALPHA_F64 && !p->is3d)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the FP64-alpha walk is implemented for 3D projectors");
  if (mode == APIRL_ALPHA_F64 && p->scanner != APIRL_SCANNER_CYLINDRICAL)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the FP64-alpha tables are built for the cylindrical scanner");
  if (mode == APIRL_ALPHA_F64 && p->t.lor_s)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the FP64-alpha walk takes one ray per bin (sampling is set)");
  DEVICE_SCOPE(p->device);
  if (mode == APIRL_ALPHA_F64 && !p->d_lor64) {
    std::vector<double> lor, z;
    apirl::build_tables_3d_f64(p->t.n_proj, p->t.n_r, p->n_rings, p->r_fov, p->axial_fov, p->r_scanner,
                               (int)p->min_rd.size(), p->min_rd.data(), p->max_rd.data(), lor, z);
    CK(cudaMalloc(&p->d_lor64, lor.size() * sizeof(double)));
    CK(cudaMemcpy(p->d_lor64, lor.data(), lor.size() * sizeof(double), cudaMemcpyHostToDevice));
    CK(cudaMalloc(&p->d_z64, z.size() * sizeof(double)));
    CK(cudaMemcpy(p->d_z64, z.data(), z.size() * sizeof(double), cudaMemcpyHostToDevice));
    p->pg.lor = p->d_lor64;
    p->pg.z = p->d_z64;
    p->pg.nx = p->g.nx; p->pg.ny = p->g.ny; p->pg.nz = p->g.nz;
    p->pg.dx = p->g.dx; p->pg.dy = p->g.dy; p->pg.dz = p->g.dz;
    p->pg.rfov = ((double)p->g.dx * p->g.nx) / 2;
    p->pg.offz = (double)p->g.dz / 2;
    if (apirl_status st = settled()) return st;
  }
  p->alpha_mode = mode;
  p->pg.enabled = mode == APIRL_ALPHA_F64;
  return APIRL_OK;
}

apirl_status apirl_projector_set_sampling(apirl_projector* p, int n_samples, int n_axial_samples,
                                         int multiple_lors_per_bin) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  if (n_samples < 1 || n_axial_samples < 1 || n_samples > APIRL_MAX_SAMPLES || n_axial_samples > APIRL_MAX_SAMPLES)
    return fail(APIRL_ERR_INVALID, "samples per bin must be 1..%d (got %d radial, %d axial)", APIRL_MAX_SAMPLES,
                n_samples, n_axial_samples);
  const bool plain = n_samples == 1 && n_axial_samples == 1 && !multiple_lors_per_bin;
  if (!p->is3d && !plain)
    return fail(APIRL_ERR_NOT_SUPPORTED, "2D projectors take one ray per bin (the reference's 2D loops ignore "
                                         "the sample counts)");
  if (p->scanner != APIRL_SCANNER_CYLINDRICAL && !plain)
    return fail(APIRL_ERR_NOT_SUPPORTED, "sampled rays are built for the cylindrical scanner");
  if (!plain && p->alpha_mode == APIRL_ALPHA_F64)
    return fail(APIRL_ERR_NOT_SUPPORTED, "sampling is not combined with the FP64-alpha walk");
  if (!plain && p->t.n_r < 2 && (n_samples > 1 || n_axial_samples > 1))
    return fail(APIRL_ERR_INVALID, "oversampling needs at least 2 radial bins (getDeltaR)");
  DEVICE_SCOPE(p->device);
  // Drop any previous sampled tables.
  cudaFree(p->ray_block);
  p->ray_block = nullptr;
  p->ray_cols = apirl::ColBuffers();
  p->t.lor_s = nullptr; p->t.zs = nullptr; p->t.zoff = nullptr; p->t.n_rs = 1; p->t.n_as = 1;
  p->t_dab = p->t;
  p->n_samples = 1; p->n_axial_samples = 1; p->multi_lors = 0;
  if (plain) return APIRL_OK;
  LorTable* dst[2] = {&p->t, &p->t_dab};
  apirl::RayTables rt[2];
  for (int k = 0; k < 2; k++) {
    if (!apirl::build_rays_3d(p->t.n_proj, p->t.n_r, p->n_rings, p->r_fov, p->axial_fov, p->r_scanner,
                              (int)p->min_rd.size(), p->min_rd.data(), p->max_rd.data(), n_samples, n_axial_samples,
                              multiple_lors_per_bin != 0, k == 1, rt[k]))
      return fail(APIRL_ERR_INVALID, "a sampled ray end point is not finite (sample outside the scanner radius)");
    if ((int)rt[k].zoff.size() != p->t.n_sinos + 1) return fail(APIRL_ERR_INVALID, "ring-pair table mismatch");
  }
  // One block: the tables, and the column layout of the passes (image copy and
  // two sums), whose end points lie up to half a ring beyond the rings'.
  // Without room for it, or for so many lists, the passes walk bin by bin.
  apirl::ColBuffers c;
  if (p->host.n_sinos >= apirl::kColMinSinos && apirl::col_rays_fit(p->g, n_samples))
    c = apirl::col_layout(p->g, rt[0].zs.data(), (int)rt[0].zs.size());
  apirl::Layouts layouts = p->layouts == apirl::Layouts::kPair || !c.half ? apirl::Layouts::kPair : apirl::Layouts::kPasses;
  size_t at_lor[2], at_zs[2], at_zoff[2], at_col;
  if (apirl_status st = take_block(layouts, &p->ray_block, [&](apirl::Layouts l) {
        Places b;
        for (int k = 0; k < 2; k++) {
          at_lor[k] = b.add(rt[k].lor.size() * sizeof(float));
          at_zs[k] = b.add(rt[k].zs.size() * sizeof(float));
          at_zoff[k] = b.add(rt[k].zoff.size() * sizeof(int));
        }
        at_col = b.add(l == apirl::Layouts::kPair ? 0 : 3 * (size_t)c.floats * sizeof(float));
        return b;
      }))
    return st;
  for (int k = 0; k < 2; k++) {
    char* const b = p->ray_block;
    CK(cudaMemcpy(b + at_lor[k], rt[k].lor.data(), rt[k].lor.size() * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(b + at_zs[k], rt[k].zs.data(), rt[k].zs.size() * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(b + at_zoff[k], rt[k].zoff.data(), rt[k].zoff.size() * sizeof(int), cudaMemcpyHostToDevice));
  }
  if (layouts != apirl::Layouts::kPair) {
    c.img = (float*)(p->ray_block + at_col);
    c.acc = c.img + c.floats;
    CK(cudaMemset(c.img, 0, 3 * (size_t)c.floats * sizeof(float)));
    p->ray_cols = c;
  }
  if (apirl_status st = settled()) return st;
  for (int k = 0; k < 2; k++) {
    dst[k]->lor_s = (const float4*)(p->ray_block + at_lor[k]);
    dst[k]->zs = (const float2*)(p->ray_block + at_zs[k]);
    dst[k]->zoff = (const int*)(p->ray_block + at_zoff[k]);
    dst[k]->n_rs = n_samples;
    dst[k]->n_as = n_axial_samples;
  }
  p->n_samples = n_samples;
  p->n_axial_samples = n_axial_samples;
  p->multi_lors = multiple_lors_per_bin != 0;
  return APIRL_OK;
}

apirl_status apirl_projector_set_shard(apirl_projector* p, int first_sinogram, int n_sinograms) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  const int total = p->host.n_sinos;
  if (first_sinogram < 0 || n_sinograms < 1 || first_sinogram + n_sinograms > total)
    return fail(APIRL_ERR_INVALID, "shard %d + %d outside the %d sinograms", first_sinogram, n_sinograms, total);
  p->t.g0 = first_sinogram;
  p->t.n_sinos = n_sinograms;
  p->t_dab.g0 = first_sinogram;
  p->t_dab.n_sinos = n_sinograms;
  return APIRL_OK;
}

apirl_status apirl_count_steps(apirl_projector* p, int subset, int nsubsets, int32_t* d_steps, void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_steps) return fail(APIRL_ERR_INVALID, "null output");
  DEVICE_SCOPE(p->device);
  CK(apirl::launch_count_steps(p->g, p->t, make_subset(p, subset, nsubsets), d_steps, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_project(apirl_projector* p, const float* d_image, float* d_sino, int subset, int nsubsets,
                           void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_image || !d_sino) return fail(APIRL_ERR_INVALID, "null image or sinogram");
  DEVICE_SCOPE(p->device);
  return project(p, make_subset(p, subset, nsubsets), d_image, d_sino, (cudaStream_t)stream);
}

apirl_status apirl_backproject(apirl_projector* p, const float* d_sino, float* d_image, int subset, int nsubsets,
                               void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if ((st = check_acc(p))) return st;
  if (!d_image || !d_sino) return fail(APIRL_ERR_INVALID, "null image or sinogram");
  DEVICE_SCOPE(p->device);
  CK(apirl::backproject_sino(p, make_subset(p, subset, nsubsets), d_sino, 0, d_image, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_backproject_ones(apirl_projector* p, float* d_image, int subset, int nsubsets, void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if ((st = check_acc(p))) return st;
  if (!d_image) return fail(APIRL_ERR_INVALID, "null image");
  DEVICE_SCOPE(p->device);
  CK(apirl::backproject_sino(p, make_subset(p, subset, nsubsets), nullptr, 2, d_image, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_backproject_and_ones(apirl_projector* p, const float* d_sino, float* d_image, float* d_ones_image,
                                        int subset, int nsubsets, void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_image || !d_sino || !d_ones_image) return fail(APIRL_ERR_INVALID, "null image or sinogram");
  if (d_image == d_ones_image) return fail(APIRL_ERR_INVALID, "the two images must differ");
  DEVICE_SCOPE(p->device);
  return apirl::backproject_sino_and_ones(p, make_subset(p, subset, nsubsets), d_sino, 0, d_image, d_ones_image,
                                          (cudaStream_t)stream);
}

apirl_status apirl_divide_and_backproject(apirl_projector* p, const float* d_meas, const float* d_est,
                                          float* d_image, int subset, int nsubsets, void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_image || !d_meas || !d_est) return fail(APIRL_ERR_INVALID, "null image or sinogram");
  DEVICE_SCOPE(p->device);
  if (use_cols(p) && p->col_sum[0].buf && !p->t_dab.lor_s && divide_cols(p, make_subset(p, subset, nsubsets))) {
    cudaStream_t s = (cudaStream_t)stream;
    bool captured = false;
    if ((st = capturing(s, &captured))) return st;
    if (!captured) {
      std::lock_guard<std::mutex> lock(p->col_mu);
      apirl_projector::ColSlot* c = nullptr;
      if ((st = slot_take(p->col_sum, s, &c))) return st;
      CK(apirl::launch_scatter_cols(p->g, p->cols, p->t, make_subset(p, subset, nsubsets), d_meas, d_est, c->buf, s));
      CK(apirl::launch_col_reduce(p->g, p->cols, c->buf, 1, nullptr, d_image, nullptr, nullptr, 0.f, 0, s));
      return slot_done(c, s);
    }
  }
  CK(apirl::launch_backproject(p->g, p->t_dab.lor_s ? p->t_dab : p->t, make_subset(p, subset, nsubsets), d_meas, 0,
                               d_est, 1, d_image, (cudaStream_t)stream, p->pg));
  return APIRL_OK;
}

apirl_status apirl_generate_acf(apirl_projector* p, const float* d_mu, float* d_acf, int subset, int nsubsets,
                                void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_mu || !d_acf) return fail(APIRL_ERR_INVALID, "null image or sinogram");
  DEVICE_SCOPE(p->device);
  SubsetSel ss = make_subset(p, subset, nsubsets);
  const int64_t nb = (int64_t)p->t.n_sinos * ss.nk * p->t.n_r;
  if (!p->is3d) CK(cudaMemsetAsync(d_acf, 0, nb * sizeof(float), (cudaStream_t)stream));
  if ((st = project(p, ss, d_mu, d_acf, (cudaStream_t)stream))) return st;
  CK(apirl::launch_exp_nonzero(nb, d_acf, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_inverse_divide(int64_t n, const float* d_meas, float* d_est, void* stream) {
  if (n < 0 || (n > 0 && (!d_meas || !d_est))) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  CK(apirl::launch_inverse_divide(n, d_meas, d_est, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_add_bins(int64_t n, const float* d_add, float* d_est, void* stream) {
  if (n < 0 || (n > 0 && (!d_add || !d_est))) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  CK(apirl::launch_add_bins(n, d_add, d_est, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_likelihood(int64_t n, const float* d_est, const float* d_meas, int gt0, double* d_out,
                              void* stream) {
  if (n <= 0 || !d_est || !d_meas || !d_out) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  // The per-block partials live in a small allocation owned by this call path.
  const int64_t nb = apirl::likelihood_blocks(n);
  double* part = nullptr;
  CK(cudaMallocAsync(&part, nb * sizeof(double), (cudaStream_t)stream));
  cudaError_t e = apirl::launch_likelihood(n, d_est, d_meas, gt0, part, nb, d_out, (cudaStream_t)stream);
  cudaFreeAsync(part, (cudaStream_t)stream);
  CK(e);
  return APIRL_OK;
}

apirl_status apirl_mlem_threshold(int64_t n, const float* d_sens, float* d_thr, void* stream) {
  if (n <= 0 || !d_sens || !d_thr) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  unsigned* mm = nullptr;
  CK(cudaMallocAsync(&mm, 2 * sizeof(unsigned), (cudaStream_t)stream));
  cudaError_t e = apirl::launch_threshold(n, d_sens, mm, d_thr, (cudaStream_t)stream);
  cudaFreeAsync(mm, (cudaStream_t)stream);
  CK(e);
  return APIRL_OK;
}

apirl_status apirl_update_pixels(int64_t n, float* d_x, float* d_bp, const float* d_sens, const float* d_thr,
                                 float thr_value, int ge, int zero_bp, void* stream) {
  if (n < 0 || (n > 0 && (!d_x || !d_bp || !d_sens))) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  CK(apirl::launch_update(n, d_x, d_bp, d_sens, d_thr, thr_value, ge, zero_bp, (cudaStream_t)stream));
  return APIRL_OK;
}

apirl_status apirl_force_positive(int64_t n, float* d_x, void* stream) {
  if (n < 0 || (n > 0 && !d_x)) return fail(APIRL_ERR_INVALID, "bad arguments");
  NO_PENDING();
  CK(apirl::launch_force_positive(n, d_x, (cudaStream_t)stream));
  return APIRL_OK;
}

namespace {

// The padded pass on the column layout.  It has one launch form: the options
// of the padded pair's launch (persistent, block size, gather segments) do not
// change it, an ordered list keeps to the pair.
// A pass over every bin of few sinograms on a wide image pays for lists that
// serve half a warp and leave few blocks on an SM.  Us on the pair -> columns
// at 1 %, 20 %, 95 % bins with counts: 320 x 320 image, 16 sinograms 224 -> 355,
// 284 -> 430, 360 -> 433; 24 sinograms 298 -> 392, 384 -> 461, 481 -> 464; 256 x
// 256, 18 sinograms 162 -> 187, 196 -> 220, 224 -> 221; 160 x 160, 16 sinograms
// 197 -> 246, 261 -> 306, 333 -> 310.  The line lies where full data take the
// same time; in long passes, where neither layout's launches count, at more
// sinograms (230 x 230, 19 sinograms: 89 K LORs 642 -> 913 us at 5 %, 931 ->
// 1044 full, 11 K LORs 149 -> 161, 188 -> 180).
bool wide_pass(const apirl_projector* p, SubsetSel ss) {
  return p->g.nx + p->g.ny > ((int64_t)ss.nk * p->t.n_r > 20000 ? 20 : 27) * p->t.n_sinos;
}
bool pass_cols(const apirl_projector* p, SubsetSel ss, bool listed) {
  return (use_cols(p) && (listed ? !p->nz.order : !wide_pass(p, ss))) || use_ray_cols(p, ss);
}
// Whether the fused pass has one launch form only, which the block size and the
// gather segments do not change: on the columns, and on the padded 2D layouts.
bool one_shape(const apirl_projector* p, SubsetSel ss, bool listed) {
  return p->planar.lim || ((use_dual(p) || p->t.lor_s) && pass_cols(p, ss, listed));
}
const apirl::ColBuffers& pass_layout(const apirl_projector* p) { return p->t.lor_s ? p->ray_cols : p->cols; }

// Before the padded pass: the image into its copy.  After it: the update of x
// (mode 0), or bp += the backprojection (mode 1).  On the column layout they
// carry the likelihood's dot product and sum too.
apirl_status pass_begin(apirl_projector* p, SubsetSel ss, const float* d_x, const float* d_zimg, double* d_lik,
                        cudaStream_t s) {
  if (pass_cols(p, ss, d_zimg != nullptr))
    CK(apirl::launch_col_copy(p->g, pass_layout(p), d_x, pass_layout(p).img, s, d_lik ? d_zimg : nullptr,
                              p->d_partials + apirl::col_partials(p->t, ss), d_zimg ? p->queue.n : nullptr));
  else
    CK(apirl::launch_pad_copy(p->g, d_x, p->pad, s));
  return APIRL_OK;
}
apirl_status pass_end(apirl_projector* p, SubsetSel ss, int mode, float* d_x, float* d_bp, const float* d_sens,
                      const float* d_thr, float thr_value, int ge, const float* d_zimg, const double* d_zero_add,
                      double* d_lik, cudaStream_t s) {
  if (pass_cols(p, ss, d_zimg != nullptr)) {
    const int64_t lors = (int64_t)ss.nk * p->t.n_r;  // no LORs: no partials written
    const int64_t n = lors ? apirl::col_partials(p->t, ss) + (d_zimg ? apirl::col_dots(p->g) : 0) : 0;
    CK(apirl::launch_col_reduce(p->g, pass_layout(p), pass_layout(p).acc, mode, d_x, d_bp, d_sens, d_thr, thr_value, ge, s,
                                p->d_partials, n, d_zimg ? d_zero_add : nullptr, lors ? d_lik : nullptr));
  } else {
    CK(apirl::launch_pad_reduce(p->g, p->pad, mode, d_x, d_bp, d_sens, d_thr, thr_value, ge, s));
  }
  return APIRL_OK;
}

// The fused kernel, bracketed by timing events when enabled.
apirl_status fused(apirl_projector* p, SubsetSel ss, const void* d_counts, int dtype, int packed, const float* d_add,
                   const float* d_x, float* d_bp, bool dual, double* d_lik, cudaStream_t s,
                   const float* d_zimg = nullptr, const double* d_zero_add = nullptr) {
  if (p->pad.acc != APIRL_ACC_ATOMIC && !(dual && p->persistent))
    return fail(APIRL_ERR_NOT_SUPPORTED, "the accumulation form needs the persistent pass over the padded layouts");
  if (p->timing) {
    if (!p->ev0) {
      CK(cudaEventCreate(&p->ev0));
      CK(cudaEventCreate(&p->ev1));
    }
    CK(cudaEventRecord(p->ev0, s));
  }
  if (dual && p->t.lor_s) {
    CK(apirl::launch_em_cols_rays(p->g, p->ray_cols, p->t, ss, d_counts, dtype, packed, d_add, 1, p->d_partials, s));
  } else if (dual && pass_cols(p, ss, d_zimg != nullptr)) {
    CK(apirl::launch_em_cols(p->g, p->cols, p->t, ss, d_counts, dtype, packed, d_add, 1, p->d_partials,
                             d_zimg ? (p->sparse_image ? 2 : 1) : 0, p->queue, s));
  } else if (p->planar.lim) {
    CK(apirl::launch_planar_pass(p->g, p->t, ss, d_counts, dtype, packed, d_add, d_x, p->planar, 1, 1, p->d_partials, s));
  } else {
    CK(apirl::launch_em_pass(p->g, p->t, ss, d_counts, dtype, packed, d_add, d_x, d_bp, 1, p->is3d ? 0 : 1,
                             p->d_partials, d_lik, s, p->pg, dual ? p->pad : apirl::PadBuffers(), p->em_block,
                             d_zimg, d_zero_add, p->persistent ? p->d_chunk : nullptr, p->sparse_image, p->nz));
  }
  if (p->timing) {
    CK(cudaEventRecord(p->ev1, s));
    p->timed = 1;
  }
  return APIRL_OK;
}

apirl_status check_em(apirl_projector* p, const void* d_counts, int dtype, const float* d_x, const float* d_bp,
                      int subset, int nsubsets) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_counts || !d_x || !d_bp) return fail(APIRL_ERR_INVALID, "null buffer");
  if (dtype != APIRL_F32 && dtype != APIRL_U32 && dtype != APIRL_U16)
    return fail(APIRL_ERR_INVALID, "unknown counts dtype %d", dtype);
  return APIRL_OK;
}

}  // namespace

apirl_status apirl_em_pass(apirl_projector* p, const void* d_counts, int counts_dtype, int counts_packed,
                           const float* d_add, float* d_x, float* d_bp, const float* d_sens, const float* d_thr,
                           float thr_value, int ge, int subset, int nsubsets, double* d_lik, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_bp, subset, nsubsets);
  if (st) return st;
  if (!d_sens) return fail(APIRL_ERR_INVALID, "null sensitivity");
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  SubsetSel ss = make_subset(p, subset, nsubsets);
  const int64_t nv = (int64_t)p->g.nx * p->g.ny * p->g.nz;
  if (use_dual(p) || use_ray_cols(p, ss)) {
    if ((st = pass_begin(p, ss, d_x, nullptr, d_lik, s))) return st;
    st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, true, d_lik, s);
    if (st) return st;
    return pass_end(p, ss, 0, d_x, nullptr, d_sens, d_thr, thr_value, ge, nullptr, nullptr, d_lik, s);
  }
  st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, false, d_lik, s);
  if (st) return st;
  if (p->planar.lim)
    CK(apirl::launch_planar_update(p->g, p->planar, 0, d_x, nullptr, d_sens, d_thr, thr_value, ge, p->d_partials,
                                   ((int64_t)ss.nk * p->t.n_r + 31) / 32, d_lik, s));
  else
    CK(apirl::launch_update(nv, d_x, d_bp, d_sens, d_thr, thr_value, ge, 1, s));
  return APIRL_OK;
}

apirl_status apirl_zero_count_image(apirl_projector* p, const void* d_counts, int counts_dtype, int counts_packed,
                                    const float* d_add, float* d_zimg, double* d_zero_add, int subset, int nsubsets,
                                    void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!d_counts || !d_zimg) return fail(APIRL_ERR_INVALID, "null buffer");
  if (counts_dtype != APIRL_F32 && counts_dtype != APIRL_U32 && counts_dtype != APIRL_U16)
    return fail(APIRL_ERR_INVALID, "unknown counts dtype %d", counts_dtype);
  if (!p->is3d || p->t.lor_s)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the sparse pass needs a 3D projector with one ray per bin");
  DEVICE_SCOPE(p->device);
  CK(apirl::launch_zero_bins(p->g, p->t, make_subset(p, subset, nsubsets), d_counts, counts_dtype, counts_packed,
                             d_add, d_zimg, p->d_partials, d_zero_add, (cudaStream_t)stream,
                             use_dual(p) ? p->pad : apirl::PadBuffers()));
  return APIRL_OK;
}

apirl_status apirl_em_pass_sparse(apirl_projector* p, const void* d_counts, int counts_dtype, int counts_packed,
                                  const float* d_add, float* d_x, float* d_bp, const float* d_sens,
                                  const float* d_zimg, const double* d_zero_add, const float* d_thr, float thr_value,
                                  int ge, int subset, int nsubsets, double* d_lik, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_bp, subset, nsubsets);
  if (st) return st;
  if (!d_sens || !d_zimg) return fail(APIRL_ERR_INVALID, "null sensitivity or zero-count image");
  if (!p->is3d || p->t.lor_s || p->pg.enabled)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the sparse pass needs a 3D projector with one float ray per bin");
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  SubsetSel ss = make_subset(p, subset, nsubsets);
  const int64_t nv = (int64_t)p->g.nx * p->g.ny * p->g.nz;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(s, &cs));
  if (cs == cudaStreamCaptureStatusNone) {
    st = apirl::prepare_nz_list(p, apirl_projector_num_bins(p, subset, nsubsets));
    if (st) return st;
  }
  if (use_dual(p)) {
    if ((st = pass_begin(p, ss, d_x, d_zimg, d_lik, s))) return st;
    st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, true, d_lik, s, d_zimg, d_zero_add);
    if (st) return st;
    return pass_end(p, ss, 0, d_x, nullptr, d_sens, d_thr, thr_value, ge, d_zimg, d_zero_add, d_lik, s);
  }
  st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, false, d_lik, s, d_zimg, d_zero_add);
  if (st) return st;
  CK(apirl::launch_update(nv, d_x, d_bp, d_sens, d_thr, thr_value, ge, 1, s));
  return APIRL_OK;
}

apirl_status apirl_em_project_backproject_sparse(apirl_projector* p, const void* d_counts, int counts_dtype,
                                                 int counts_packed, const float* d_add, const float* d_x, float* d_bp,
                                                 const float* d_zimg, const double* d_zero_add, int subset,
                                                 int nsubsets, double* d_lik, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_bp, subset, nsubsets);
  if (st) return st;
  if (!d_zimg) return fail(APIRL_ERR_INVALID, "null zero-count or geometry image");
  if (!p->is3d || p->t.lor_s || p->pg.enabled)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the sparse pass needs a 3D projector with one float ray per bin");
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  SubsetSel ss = make_subset(p, subset, nsubsets);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(s, &cs));
  if (cs == cudaStreamCaptureStatusNone) {
    st = apirl::prepare_nz_list(p, apirl_projector_num_bins(p, subset, nsubsets));
    if (st) return st;
  }
  if (use_dual(p)) {
    if ((st = pass_begin(p, ss, d_x, d_zimg, d_lik, s))) return st;
    st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, true, d_lik, s, d_zimg, d_zero_add);
    if (st) return st;
    return pass_end(p, ss, 1, nullptr, d_bp, nullptr, nullptr, 0.f, 0, d_zimg, d_zero_add, d_lik, s);
  }
  return fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, false, d_lik, s, d_zimg, d_zero_add);
}

apirl_status apirl_em_project_backproject(apirl_projector* p, const void* d_counts, int counts_dtype,
                                          int counts_packed, const float* d_add, const float* d_x, float* d_bp,
                                          int subset, int nsubsets, double* d_lik, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_bp, subset, nsubsets);
  if (st) return st;
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  SubsetSel ss = make_subset(p, subset, nsubsets);
  if (use_dual(p) || use_ray_cols(p, ss)) {
    if ((st = pass_begin(p, ss, d_x, nullptr, d_lik, s))) return st;
    st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, true, d_lik, s);
    if (st) return st;
    return pass_end(p, ss, 1, nullptr, d_bp, nullptr, nullptr, 0.f, 0, nullptr, nullptr, d_lik, s);
  }
  st = fused(p, ss, d_counts, counts_dtype, counts_packed, d_add, d_x, d_bp, false, d_lik, s);
  if (st) return st;
  if (p->planar.lim)
    CK(apirl::launch_planar_update(p->g, p->planar, 1, nullptr, d_bp, nullptr, nullptr, 0.f, 0, p->d_partials,
                                   ((int64_t)ss.nk * p->t.n_r + 31) / 32, d_lik, s));
  return APIRL_OK;
}

apirl_status apirl_projector_set_option(apirl_projector* p, int option, int value) {
  if (!p) return fail(APIRL_ERR_INVALID, "null projector");
  switch (option) {
    case APIRL_OPT_DUAL_LAYOUT: p->dual_layout = value != 0; return APIRL_OK;
    case APIRL_OPT_KERNEL_TIMING: p->timing = value != 0; p->timed = 0; return APIRL_OK;
    case APIRL_OPT_PERSISTENT: p->persistent = value != 0; return APIRL_OK;
    case APIRL_OPT_SPARSE_IMAGE:
      if (value != APIRL_SPARSE_ZERO_COUNT && value != APIRL_SPARSE_GEOMETRY)
        return fail(APIRL_ERR_INVALID, "unknown sparse image kind %d", value);
      p->sparse_image = value;
      return APIRL_OK;
    case APIRL_OPT_L2_PERSIST: {
      if (value && !use_dual(p))
        return fail(APIRL_ERR_NOT_SUPPORTED, "the L2 window covers the padded 3D layouts");
      DEVICE_SCOPE(p->device);
      p->pad.window = 0;
      p->pad.hit_ratio = 0.f;
      if (p->l2_limit_set) {
        CK(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, p->l2_limit_prev));
        p->l2_limit_set = false;
      }
      if (value) {
        int max_window = 0, max_persist = 0;
        CK(cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, p->device));
        CK(cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, p->device));
        const size_t want = (size_t)4 * p->pad.lim * sizeof(float);
        const size_t win = want < (size_t)max_window ? want : (size_t)max_window;
        const size_t aside = win < (size_t)max_persist ? win : (size_t)max_persist;
        if (win == 0 || aside == 0) return fail(APIRL_ERR_NOT_SUPPORTED, "this device has no persisting L2");
        // The set-aside is a limit of this process's context on the device.
        CK(cudaDeviceGetLimit(&p->l2_limit_prev, cudaLimitPersistingL2CacheSize));
        CK(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, aside));
        p->l2_limit_set = true;
        p->pad.window = win;
        p->pad.hit_ratio = (float)((double)aside / (double)win);
      }
      return APIRL_OK;
    }
    case APIRL_OPT_GATHER_UNROLL:
      if (value != 0 && value != 4 && value != 6 && value != 8)
        return fail(APIRL_ERR_INVALID, "gather segments in flight: 0, 4, 6 or 8");
      p->pad.unroll = value;
      return APIRL_OK;
    case APIRL_OPT_LIST_ORDER:
      if (value != 0 && (value < 32 || value > apirl::kNzTile || (value & (value - 1))))
        return fail(APIRL_ERR_INVALID, "list order: 0, or a power of two from 32 to %d", apirl::kNzTile);
      p->nz.order = value;
      return APIRL_OK;
    case APIRL_OPT_ACCUMULATE: {
      if (value != APIRL_ACC_ATOMIC && value != APIRL_ACC_WARP && value != APIRL_ACC_COMPENSATED)
        return fail(APIRL_ERR_INVALID, "unknown accumulation form %d", value);
      if (value != APIRL_ACC_ATOMIC && !use_dual(p))  // use_dual: the padded layouts are taken
        return fail(APIRL_ERR_NOT_SUPPORTED, "accumulation forms need the padded 3D layouts (3D, float walk, one ray "
                                             "per bin, dual layout)");
      if (value == APIRL_ACC_COMPENSATED && !p->pad.eA) {
        DEVICE_SCOPE(p->device);
        const size_t pv = (size_t)p->pad.lim;
        CK(cudaMalloc(&p->pad.eA, pv * sizeof(float)));
        CK(cudaMalloc(&p->pad.eT, pv * sizeof(float)));
        CK(cudaMemset(p->pad.eA, 0, pv * sizeof(float)));
        CK(cudaMemset(p->pad.eT, 0, pv * sizeof(float)));
        if (apirl_status st = settled()) return st;
      }
      p->pad.acc = value;
      return APIRL_OK;
    }
    case APIRL_OPT_EM_BLOCK:
      if (value < 32 || value > 256 || value % 32) return fail(APIRL_ERR_INVALID, "block size must be 32..256, x32");
      p->em_block = value;
      if (p->is3d) {
        DEVICE_SCOPE(p->device);
        CK(apirl::prepare_em_kernels(value));
      }
      return APIRL_OK;
    default: return fail(APIRL_ERR_INVALID, "unknown option %d", option);
  }
}

apirl_status apirl_projector_autotune(apirl_projector* p, const void* d_counts, int counts_dtype, const float* d_x,
                                     int subset, int nsubsets, int repeats, int* best_block, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_x, subset, nsubsets);
  if (st) return st;
  if (repeats < 1) repeats = 1;
  if (one_shape(p, make_subset(p, subset, nsubsets), false)) {  // nothing to choose from
    if (best_block) *best_block = p->em_block;
    return APIRL_OK;
  }
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nv = (int64_t)p->g.nx * p->g.ny * p->g.nz;
  float* bp = nullptr;
  CK(cudaMalloc(&bp, nv * sizeof(float)));
  cudaEvent_t a = nullptr, b = nullptr;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int cands[] = {64, 96, 128, 192, 256};
  const int saved_timing = p->timing;
  p->timing = 0;
  float best = 1e30f;
  int best_b = p->em_block;
  for (int c : cands) {
    p->em_block = c;
    CK(cudaMemsetAsync(bp, 0, nv * sizeof(float), s));
    st = apirl_em_project_backproject(p, d_counts, counts_dtype, 0, nullptr, d_x, bp, subset, nsubsets, nullptr, s);
    if (st) break;
    cudaEventRecord(a, s);
    for (int r = 0; r < repeats && !st; r++)
      st = apirl_em_project_backproject(p, d_counts, counts_dtype, 0, nullptr, d_x, bp, subset, nsubsets, nullptr, s);
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    if (ms < best) { best = ms; best_b = c; }
  }
  p->timing = saved_timing;
  p->em_block = best_b;
  if (!st) {
    cudaError_t pe = apirl::prepare_em_kernels(best_b);
    if (pe != cudaSuccess) st = fail(APIRL_ERR_CUDA, "prepare_em_kernels: %s", cudaGetErrorString(pe));
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(bp);
  if (st) return st;
  if (best_block) *best_block = best_b;
  return APIRL_OK;
}

apirl_status apirl_projector_autotune_ex(apirl_projector* p, const void* d_counts, int counts_dtype,
                                        const float* d_x, const float* d_zimg, int subset, int nsubsets, int repeats,
                                        apirl_tune* out, void* stream) {
  apirl_status st = check_em(p, d_counts, counts_dtype, d_x, d_x, subset, nsubsets);
  if (st) return st;
  if (!use_dual(p) || !p->persistent || p->pad.acc != APIRL_ACC_ATOMIC)
    return fail(APIRL_ERR_NOT_SUPPORTED, "the launch shape is tuned for the persistent pass over the padded layouts "
                                         "with plain atomics");
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nv = (int64_t)p->g.nx * p->g.ny * p->g.nz;
  float* bp = nullptr;
  CK(cudaMalloc(&bp, nv * sizeof(float)));
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t ce = cudaEventCreate(&a);
  if (ce == cudaSuccess) ce = cudaEventCreate(&b);
  std::vector<int> blocks{64, 96, 128, 192, 256}, unrolls{4, 6, 8};
  if (one_shape(p, make_subset(p, subset, nsubsets), d_zimg != nullptr)) {  // the one there is, timed
    blocks = {p->em_block};
    unrolls = {p->pad.unroll};
  }
  const int saved_timing = p->timing, saved_block = p->em_block, saved_unroll = p->pad.unroll;
  p->timing = 0;
  float best = 1e30f;
  int best_b = p->em_block, best_u = p->pad.unroll;
  if (repeats < 1) repeats = 1;
  auto pass = [&]() {
    return d_zimg ? apirl_em_project_backproject_sparse(p, d_counts, counts_dtype, 0, nullptr, d_x, bp, d_zimg,
                                                        nullptr, subset, nsubsets, nullptr, s)
                  : apirl_em_project_backproject(p, d_counts, counts_dtype, 0, nullptr, d_x, bp, subset, nsubsets,
                                                 nullptr, s);
  };
  for (int blk : blocks) {
    if (ce != cudaSuccess) break;
    p->em_block = blk;
    if ((ce = apirl::prepare_em_kernels(blk)) != cudaSuccess) break;
    for (int u : unrolls) {
      p->pad.unroll = u;
      if ((ce = cudaMemsetAsync(bp, 0, nv * sizeof(float), s)) != cudaSuccess) break;
      if ((st = pass())) break;  // warm-up (and the list, for the sparse pass)
      if ((ce = cudaEventRecord(a, s)) != cudaSuccess) break;
      for (int r = 0; r < repeats && !st; r++) st = pass();
      if (st) break;
      if ((ce = cudaEventRecord(b, s)) != cudaSuccess || (ce = cudaEventSynchronize(b)) != cudaSuccess) break;
      float ms = 0;
      if ((ce = cudaEventElapsedTime(&ms, a, b)) != cudaSuccess) break;
      if (ms < best) { best = ms; best_b = blk; best_u = u; }
    }
    if (st) break;
  }
  p->timing = saved_timing;
  if (!st && ce == cudaSuccess) {
    p->em_block = best_b;
    p->pad.unroll = best_u;
    ce = apirl::prepare_em_kernels(best_b);
  } else {
    p->em_block = saved_block;
    p->pad.unroll = saved_unroll;
  }
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  cudaFree(bp);
  if (st) return st;
  if (ce != cudaSuccess) return cuda_fail(ce, "autotune");
  if (out) {
    out->block = best_b;
    out->unroll = best_u ? best_u : d_zimg ? 6 : 4;  // 0: the pass kind's default
    out->ms = best / repeats;
  }
  return APIRL_OK;
}

apirl_status apirl_projector_kernel_ms(apirl_projector* p, double* ms) {
  if (!p || !ms) return fail(APIRL_ERR_INVALID, "bad arguments");
  if (!p->timed) return fail(APIRL_ERR_INVALID, "no timed pass recorded (enable APIRL_OPT_KERNEL_TIMING)");
  DEVICE_SCOPE(p->device);
  CK(cudaEventSynchronize(p->ev1));
  float f = 0.f;
  CK(cudaEventElapsedTime(&f, p->ev0, p->ev1));
  *ms = f;
  return APIRL_OK;
}

apirl_status apirl_stage_counts(apirl_projector* p, const void* h_counts_subset, int counts_dtype, void* d_counts_stage,
                                int subset, int nsubsets, void* stream) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!h_counts_subset || !d_counts_stage) return fail(APIRL_ERR_INVALID, "null buffer");
  if (counts_dtype != APIRL_F32 && counts_dtype != APIRL_U32 && counts_dtype != APIRL_U16)
    return fail(APIRL_ERR_INVALID, "unknown counts dtype %d", counts_dtype);
  const int64_t nb = apirl_projector_num_bins(p, subset, nsubsets);
  const size_t esz = counts_dtype == APIRL_U16 ? 2 : 4;
  DEVICE_SCOPE(p->device);
  if (!p->copy_stream) {
    CK(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&p->copy_ready, cudaEventDisableTiming));
    for (auto& e : p->staged) CK(cudaEventCreateWithFlags(&e.done, cudaEventDisableTiming));
  }
  // A free slot, or the one staging the same device buffer (restaged).
  apirl_projector::Staged* slot = nullptr;
  for (auto& e : p->staged)
    if (e.dev == d_counts_stage) slot = &e;
  for (auto& e : p->staged)
    if (!slot && !e.dev) slot = &e;
  if (!slot) return fail(APIRL_ERR_INVALID, "more than 4 staged copies outstanding");
  // The copy starts after the caller's stream's earlier work (which may still
  // read d_counts_stage) and runs beside its later work.
  CK(cudaEventRecord(p->copy_ready, (cudaStream_t)stream));
  CK(cudaStreamWaitEvent(p->copy_stream, p->copy_ready, 0));
  CK(cudaMemcpyAsync(d_counts_stage, h_counts_subset, nb * esz, cudaMemcpyHostToDevice, p->copy_stream));
  CK(cudaEventRecord(slot->done, p->copy_stream));
  slot->host = h_counts_subset;
  slot->dev = d_counts_stage;
  return APIRL_OK;
}

}  // extern "C"

namespace {
// apirl_em_pass_host and apirl_em_pass_host_async; `wait`: synchronise the
// stream before returning.
apirl_status em_pass_host(apirl_projector* p, const void* h_counts_subset, int counts_dtype, void* d_counts_stage,
                          float* d_x, float* d_bp, const float* d_sens, const float* d_zimg,
                          const double* d_zero_add, float thr_value, int ge, int subset, int nsubsets,
                          float* h_x_out, double* h_lik, void* stream, bool wait) {
  apirl_status st = check_subset(p, subset, nsubsets);
  if (st) return st;
  if (!h_counts_subset || !d_counts_stage) return fail(APIRL_ERR_INVALID, "null buffer");
  const int64_t nb = apirl_projector_num_bins(p, subset, nsubsets);
  const size_t esz = counts_dtype == APIRL_U16 ? 2 : 4;
  DEVICE_SCOPE(p->device);
  cudaStream_t s = (cudaStream_t)stream;
  apirl_projector::Staged* slot = nullptr;
  for (auto& e : p->staged)
    if (e.dev == d_counts_stage && e.host == h_counts_subset) slot = &e;
  if (slot) {
    CK(cudaStreamWaitEvent(s, slot->done, 0));  // staged ahead by apirl_stage_counts
    slot->dev = nullptr;
    slot->host = nullptr;
  } else {
    CK(cudaMemcpyAsync(d_counts_stage, h_counts_subset, nb * esz, cudaMemcpyHostToDevice, s));
  }
  double* d_lik = p->d_scalars;
  if (d_zimg)
    st = apirl_em_pass_sparse(p, d_counts_stage, counts_dtype, 1, nullptr, d_x, d_bp, d_sens, d_zimg, d_zero_add,
                              nullptr, thr_value, ge, subset, nsubsets, h_lik ? d_lik : nullptr, stream);
  else
    st = apirl_em_pass(p, d_counts_stage, counts_dtype, 1, nullptr, d_x, d_bp, d_sens, nullptr, thr_value, ge,
                       subset, nsubsets, h_lik ? d_lik : nullptr, stream);
  if (st) return st;
  const int64_t nv = (int64_t)p->g.nx * p->g.ny * p->g.nz;
  if (h_x_out) CK(cudaMemcpyAsync(h_x_out, d_x, nv * sizeof(float), cudaMemcpyDeviceToHost, s));
  if (h_lik) CK(cudaMemcpyAsync(h_lik, d_lik, sizeof(double), cudaMemcpyDeviceToHost, s));
  if (wait) CK(cudaStreamSynchronize(s));
  return APIRL_OK;
}
}  // namespace

extern "C" {

apirl_status apirl_em_pass_host(apirl_projector* p, const void* h_counts_subset, int counts_dtype,
                                void* d_counts_stage, float* d_x, float* d_bp, const float* d_sens,
                                const float* d_zimg, const double* d_zero_add, float thr_value, int ge, int subset,
                                int nsubsets, float* h_x_out, double* h_lik, void* stream) {
  return em_pass_host(p, h_counts_subset, counts_dtype, d_counts_stage, d_x, d_bp, d_sens, d_zimg, d_zero_add,
                      thr_value, ge, subset, nsubsets, h_x_out, h_lik, stream, true);
}

apirl_status apirl_em_pass_host_async(apirl_projector* p, const void* h_counts_subset, int counts_dtype,
                                      void* d_counts_stage, float* d_x, float* d_bp, const float* d_sens,
                                      const float* d_zimg, const double* d_zero_add, float thr_value, int ge,
                                      int subset, int nsubsets, float* h_x_out, double* h_lik, void* stream) {
  return em_pass_host(p, h_counts_subset, counts_dtype, d_counts_stage, d_x, d_bp, d_sens, d_zimg, d_zero_add,
                      thr_value, ge, subset, nsubsets, h_x_out, h_lik, stream, false);
}

}  // extern "C"

namespace apirl {
apirl_status prepare_nz_list(apirl_projector* p, int64_t total) {
  if (total <= p->nz.cap || !p->is3d || (use_cols(p) && !p->nz.order)) return APIRL_OK;
  DEVICE_SCOPE(p->device);
  cudaFree(p->nz.list);
  cudaFree(p->nz.tiles);
  p->nz.list = nullptr;
  p->nz.tiles = nullptr;
  p->nz.cap = 0;
  if (!p->nz.n_list) CK(cudaMalloc(&p->nz.n_list, sizeof(int)));
  const int64_t n_tiles = (total + apirl::kNzTile - 1) / apirl::kNzTile;
  CK(cudaMalloc(&p->nz.list, (size_t)total * sizeof(int)));
  CK(cudaMalloc(&p->nz.tiles, (size_t)n_tiles * sizeof(int)));
  p->nz.cap = total;
  return APIRL_OK;
}
}  // namespace apirl

namespace apirl {
cudaError_t backproject_sino(apirl_projector* p, SubsetSel ss, const float* vin, int vin_mode, float* img,
                             cudaStream_t st) {
  // Sensitivities and geometry images (factors, ones) stay on the padded pair:
  // the lengths of one angle's rays are nearly equal, and added LOR by LOR
  // their rounding errors in a voxel's sum go the same way.  Made on the
  // columns they moved the likelihood of the 256 x 256 x 81 job, which holds
  // x . G_s, by 5.6e-8 (one sum) or 1e-8 (two) of its value; the pair's, made
  // once per geometry, by 6e-9.
  if (use_cols(p) && vin_mode == 0) {
    const cudaError_t e = launch_scatter_cols(p->g, p->cols, p->t, ss, vin, nullptr, p->cols.acc, st, p->queue);
    if (e != cudaSuccess) return e;
    return launch_col_reduce(p->g, p->cols, p->cols.acc, 1, nullptr, img, nullptr, nullptr, 0.f, 0, st);
  }
  if (use_dual(p)) return launch_backproject_pad(p->g, p->t, ss, vin, vin_mode, img, p->pad, p->d_chunk, st);
  return launch_backproject(p->g, p->t, ss, vin, vin_mode, nullptr, 0, img, st, p->pg);
}
}  // namespace apirl

namespace apirl {
apirl_status backproject_sino_and_ones(apirl_projector* p, SubsetSel ss, const float* vin, int vin_mode, float* img,
                                       float* gimg, cudaStream_t st) {
  if (!use_dual(p)) {
    CK(backproject_sino(p, ss, vin, vin_mode, img, st));
    CK(backproject_sino(p, ss, nullptr, 2, gimg, st));
    return APIRL_OK;
  }
  if (!p->pad2.bA) {
    const size_t pv = (size_t)p->pad.lim;
    CK(cudaMalloc(&p->pad2.bA, pv * sizeof(float)));
    CK(cudaMalloc(&p->pad2.bT, pv * sizeof(float)));
    CK(cudaMemsetAsync(p->pad2.bA, 0, pv * sizeof(float), st));
    CK(cudaMemsetAsync(p->pad2.bT, 0, pv * sizeof(float), st));
    p->pad2.lim = p->pad.lim;
  }
  CK(launch_backproject_pad(p->g, p->t, ss, vin, vin_mode, img, p->pad, p->d_chunk, st, gimg, p->pad2));
  return APIRL_OK;
}
}  // namespace apirl

