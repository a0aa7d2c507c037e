// The column walk: Siddon walks of many sinograms along one (angle, r).
//
// The x and y crossings of a ray (its crossing parameters, hence the columns
// it passes and their order) come from its LOR's end points in the plane alone
// (recon/src/Siddon.cpp:48-140, :240-300), so they are the same floats for
// every sinogram: only the z crossings, the length factor and the voxels'
// slices differ.  A block takes one (angle, r): it lists the x/y crossings
// once in shared memory (col_list), then its warps walk 32 sinograms at a time
// along the list (col_walk).  The lanes pass the same columns in step, a step
// without a z crossing costs a length, an address, the access and its sum, and
// with the image stored column by column, z innermost, the lanes' voxels lie
// side by side.
//
// Column layout: [y][x][z'], z' = z + z0, the slices of one column split by
// parity, even z' first: consecutive rings lie two slices apart (dz is half
// the ring pitch in the scanners' images), so that the 32 lanes of a span-1
// segment touch 32 consecutive floats.  A column holds every slice that a ray
// of the scanner can enter, inside the image or not, and kColSpare beyond: walks
// need no test of z.
#pragma once
#include <cuda_runtime.h>
#include <cfloat>
#include <cstdint>
#include "siddon.cuh"

namespace apirl {

constexpr int kColBatch = 4;  // steps of the list taken together

// Slices that a column holds beyond those its rays can enter: kPad, and the
// z crossings that the walk may record between two looks at their number.
constexpr int kColSpare = kPad + kColBatch;

// Sizes of a column image: kPad border in x and y; z0 (even) slices before
// the image's first; half = floats of one parity, a multiple of 8 (one sector).
struct ColDims {
  int nx, ny, nz, z0, half;
  __host__ __device__ int px() const { return nx + 2 * kPad; }
  __host__ __device__ int py() const { return ny + 2 * kPad; }
  __host__ __device__ int stride() const { return 2 * half; }
  __host__ __device__ int64_t floats() const { return (int64_t)px() * py() * stride(); }
};

// Offset of slice z in its column.  From one slice to the next up it changes
// by half and 1 - half in turn, down by half - 1 and -half: each change is the
// direction less the one before it.
__device__ __forceinline__ int col_slice(const ColDims& d, int z) {
  const int zz = z + d.z0;
  return (zz & 1) * d.half + (zz >> 1);
}

// The x/y half of a walk (siddon3_setup's values, the same operations).
struct ColWalk {
  float ax, ay, axu, ayu, amin, amax, len2;
  int n;            // |di| + |dj|: crossings on the list
  int nx, ny;       // |di|, |dj|
  int col, sx, sy;  // entry column's first float, and its steps
  int listed;       // 0: the walk is not on the list (col_walk_checked serves it)
  int xmain;        // the ray runs mostly along x
  unsigned last;    // a border column: the memory guard of column indexes
};

// The block's list of the x/y crossings, in shared memory behind a ColWalk:
// records of kColBatch = 4 steps, three float4 each: the lengths an[j] -
// an[j - 1], the columns (int bits) and the crossing parameters an[j].  One
// address register reads a whole record.  Behind them lie the x and y chains
// that the list is merged from, and in their place then (an[j], column) step
// by step.  A block may keep several lists: `at`, here and below, is the first
// float4 of one.
extern __shared__ __align__(16) float4 col_smem4[];
constexpr int kColHead = (sizeof(ColWalk) + 15) / 16;  // float4s before the list
// Steps a list can need on this image (guarded walks: at most nx + 2 and
// ny + 2 crossings, two spare entries a chain), in whole records.
__host__ __device__ inline int col_cap(int nx, int ny) { return (nx + ny + 8 + kColBatch - 1) / kColBatch * kColBatch; }
__host__ __device__ inline size_t col_smem(int nx, int ny) {
  return (size_t)kColHead * 16 + (size_t)col_cap(nx, ny) * 20;  // whole float4s
}
__device__ __forceinline__ ColWalk& col_head(int at = 0) { return *reinterpret_cast<ColWalk*>(col_smem4 + at); }
// Float offset of what lies behind the records.
__device__ __forceinline__ int col_behind(const ColDims& d) { return kColHead * 4 + col_cap(d.nx, d.ny) * 3; }
// Step j's field f (0 length, 1 column, 2 crossing parameter).
__device__ __forceinline__ float& col_field(int j, int f, int at) {
  return reinterpret_cast<float*>(col_smem4 + at)[kColHead * 4 + (j >> 2) * 12 + f * 4 + (j & 3)];
}

__device__ __forceinline__ void col_setup_xy(const float4 P, const ImgGeom& g, const ColDims& d, ColWalk& w) {
  const float p0x = P.x, p0y = P.y, vx = A_SUB(P.z, P.x), vy = A_SUB(P.w, P.y);
  const float rFov = g.rfov;
  float amin, amax;
  if (vx == 0.f) {
    const float a1 = A_DIV(A_SUB(-rFov, p0y), vy), a2 = A_DIV(A_SUB(rFov, p0y), vy);
    if (a1 < a2) { amin = a1; amax = a2; } else { amin = a2; amax = a1; }
  } else if (vy == 0.f) {
    const float a1 = A_DIV(A_SUB(-rFov, p0x), vx), a2 = A_DIV(A_SUB(rFov, p0x), vx);
    if (a1 < a2) { amin = a1; amax = a2; } else { amin = a2; amax = a1; }
  } else {
    const float ax1 = A_DIV(A_SUB(-rFov, p0x), vx), ay1 = A_DIV(A_SUB(-rFov, p0y), vy);
    const float ax2 = A_DIV(A_SUB(rFov, p0x), vx), ay2 = A_DIV(A_SUB(rFov, p0y), vy);
    amin = fmax_ref(fmin_ref(ax1, ax2), fmin_ref(ay1, ay2));
    amax = fmin_ref(fmax_ref(ax1, ax2), fmax_ref(ay1, ay2));
  }
  if (amin < 0.f || amin > 1.f) amin = 0.f;
  if (amax > 1.f || amax < 0.f) amax = 1.f;
  const float x1 = A_ADD(p0x, A_MUL(vx, amin)), y1 = A_ADD(p0y, A_MUL(vy, amin));
  const float x2 = A_ADD(p0x, A_MUL(vx, amax)), y2 = A_ADD(p0y, A_MUL(vy, amax));
  const int imin = (int)floorf(A_DIV(A_ADD(x1, rFov), g.dx)), jmin = (int)floorf(A_DIV(A_ADD(y1, rFov), g.dy));
  const int imax = (int)floorf(A_DIV(A_ADD(x2, rFov), g.dx)), jmax = (int)floorf(A_DIV(A_ADD(y2, rFov), g.dy));
  w.nx = abs(imax - imin);
  w.ny = abs(jmax - jmin);
  w.n = w.nx + w.ny;
  w.listed = (min(imin, imax) >= -1) & (max(imin, imax) <= g.nx) & (min(jmin, jmax) >= -1) & (max(jmin, jmax) <= g.ny);
  const int iinc = vx > 0.f ? 1 : (vx < 0.f ? -1 : 0), jinc = vy > 0.f ? 1 : (vy < 0.f ? -1 : 0);
  const float ex = A_SUB(A_ADD(p0x, vx), p0x), ey = A_SUB(A_ADD(p0y, vy), p0y);
  w.len2 = A_ADD(A_MUL(ex, ex), A_MUL(ey, ey));
  w.axu = fabsf(A_DIV(g.dx, vx));
  w.ayu = fabsf(A_DIV(g.dy, vy));
  w.ax = vx > 0.f ? A_DIV(A_SUB(A_ADD(-rFov, A_MUL((float)(imin + iinc), g.dx)), p0x), vx)
       : (vx < 0.f ? A_DIV(A_SUB(A_ADD(-rFov, A_MUL((float)imin, g.dx)), p0x), vx) : FLT_MAX);
  w.ay = vy > 0.f ? A_DIV(A_SUB(A_ADD(-rFov, A_MUL((float)(jmin + jinc), g.dy)), p0y), vy)
       : (vy < 0.f ? A_DIV(A_SUB(A_ADD(-rFov, A_MUL((float)jmin, g.dy)), p0y), vy) : FLT_MAX);
  w.amin = amin;
  w.amax = amax;
  w.sx = iinc * d.stride();
  w.sy = jinc * d.px() * d.stride();
  w.col = ((jmin + kPad) * d.px() + imin + kPad) * d.stride();
  w.xmain = fabsf(vx) >= fabsf(vy);
  w.last = (unsigned)(d.floats() - d.stride());
}

// Makes the block's list of one LOR; every thread calls it, and finds it made
// on return.  The crossing parameters are the reference's running sums: two
// threads add the x and the y chain up, then every thread places entries at
// their rank among both (x before y on ties, Siddon.cpp:317-339).
__device__ __forceinline__ void col_list(const float4 P, const ImgGeom& g, const ColDims& d, int at = 0) {
  const int tid = threadIdx.x;
  ColWalk& h = col_head(at);
  float* const chain = reinterpret_cast<float*>(col_smem4 + at) + col_behind(d);
  if (tid < 32) {
    ColWalk w;
    col_setup_xy(P, g, d, w);
    if (tid < 2 && w.listed) {
      const int n = (tid ? w.ny : w.nx) + 2;
      float* ch = chain + (tid ? w.nx + 2 : 0);
      float v = tid ? w.ay : w.ax;
      const float u = tid ? w.ayu : w.axu;
      for (int i = 0; i < n; i++) {
        ch[i] = v;
        v = A_ADD(v, u);
      }
    }
    if (tid == 0) h = w;
  }
  __syncthreads();
  const bool listed = h.listed;
  if (listed) {
    const int nx = h.nx + 2, ny = h.ny + 2, n = h.n;
    const int col = h.col, sx = h.sx, sy = h.sy;
    const unsigned last = h.last;
    for (int e = tid; e < nx + ny; e += blockDim.x) {
      const bool isx = e < nx;
      const int i = isx ? e : e - nx;
      const float v = chain[e];
      const float* other = isx ? chain + nx : chain;
      int lo = 0, hi = isx ? ny : nx;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (isx ? other[mid] < v : other[mid] <= v) lo = mid + 1;
        else hi = mid;
      }
      const int p = i + lo;
      if (p < n) {
        col_field(p, 2, at) = v;
        col_field(p, 1, at) = __int_as_float((int)min((unsigned)(col + (isx ? i * sx + lo * sy : lo * sx + i * sy)), last));
        // The chain's last spare entry taken: the chain may be too short.
        if (i == (isx ? nx : ny) - 1) h.listed = 0;
      }
    }
  }
  __syncthreads();
  if (listed) {
    float2* const by_step = reinterpret_cast<float2*>(reinterpret_cast<float*>(col_smem4 + at) + col_behind(d));
    for (int p = tid; p < h.n; p += blockDim.x) {
      const float an = col_field(p, 2, at);
      col_field(p, 0, at) = A_SUB(an, p ? col_field(p - 1, 2, at) : h.amin);
      by_step[p] = make_float2(an, col_field(p, 1, at));
    }
  }
  __syncthreads();
}

// The z half of one ray.  rem: z crossings still to record, |dk| at first (a
// walk records |di| + |dj| + |dk| crossings in all, Siddon.cpp:220, which
// rounding can split otherwise than |di| + |dj| and |dk|: then rem ends above
// or below zero, by one, and kPad bounds it).  at, step: the slice's offset in
// the column and the next change of it; up: the z direction.
struct WalkZ {
  float az, azu, len;
  int at, step, up, rem;
};

// A ray that records nothing (length 0 on the border).
__device__ __forceinline__ WalkZ col_no_ray() { return WalkZ{FLT_MAX, 0.f, 0.f, 0, 0, 0, 0}; }

__device__ __forceinline__ WalkZ col_setup_z(const float2 e, const ColWalk& w, const ImgGeom& g, const ColDims& d) {
  WalkZ r;
  const float vz = A_SUB(e.y, e.x);
  const float z1 = A_ADD(e.x, A_MUL(vz, w.amin)), z2 = A_ADD(e.x, A_MUL(vz, w.amax));
  const int kmin = (int)floorf(A_DIV(A_SUB(z1, g.offz), g.dz)), kmax = (int)floorf(A_DIV(A_SUB(z2, g.offz), g.dz));
  r.up = vz > 0.f ? 1 : (vz < 0.f ? -1 : 0);
  const float ez = A_SUB(A_ADD(e.x, vz), e.x);
  r.len = __fsqrt_rn(A_ADD(w.len2, A_MUL(ez, ez)));
  r.azu = fabsf(A_DIV(g.dz, vz));
  r.az = vz > 0.f ? A_DIV(A_SUB(A_ADD(g.offz, A_MUL((float)(kmin + r.up), g.dz)), e.x), vz)
       : (vz < 0.f ? A_DIV(A_SUB(A_ADD(g.offz, A_MUL((float)kmin, g.dz)), e.x), vz) : FLT_MAX);
  r.at = col_slice(d, kmin);
  const bool odd = (kmin + d.z0) & 1;
  r.step = r.up > 0 ? (odd ? 1 - d.half : d.half) : (odd ? -d.half : d.half - 1);
  r.rem = abs(kmax - kmin);
  return r;
}

// Walks the lanes' rays along the block's list: visit(p, length) for every
// segment of a ray in its order (Siddon.cpp:310-340: record, then advance, x
// before y before z on ties), p the voxel's place in `base`.  All 32 lanes
// call it.  The list's steps are taken kColBatch at a time; where some lane's
// ray crosses in z within the batch, the crossing goes in among the batch's.
// Warps with a ray whose z crossings lie so close that a batch could hold two
// merge z crossings and list segment by segment, each lane at its own step.
template <class T, class V>
__device__ __forceinline__ void col_walk(WalkZ r, const ColDims& d, T* base, V&& visit, int list_at = 0) {
  const int n = col_head(list_at).n;
  T* p = base + r.at;
  // One z crossing of the lane's ray, from lo, in the column at `col`.
  auto cross = [&](int col, float& lo) {
    visit(p + col, A_MUL(A_SUB(r.az, lo), r.len));
    lo = r.az;
    r.at += r.step;
    p = base + r.at;
    r.step = r.up - r.step;
    r.az = A_ADD(r.az, r.azu);
    r.rem--;
  };
  float before = col_head(list_at).amin;  // the crossing before the batch
  // rem >= -kPad: up to the list's last kPad steps no walk has recorded all
  // its crossings, so only the steps after this loop ask.
  const int batches = (n - kPad) / kColBatch;
  // Four steps span at most four gaps of the denser of the x and y crossings:
  // where every lane's z crossings lie further apart, a batch holds one at most.
  const bool single = !__any_sync(0xffffffffu, r.azu != 0.f && r.azu < 4.01f * fminf(col_head(list_at).axu, col_head(list_at).ayu));
  if (!single && batches > 0) {
    const float2* const list = reinterpret_cast<const float2*>(reinterpret_cast<float*>(col_smem4 + list_at) + col_behind(d));
    const float2* at = list;
    const float2* const stop = list + batches * kColBatch;
    float2 next = *at;
    auto segment = [&]() {
      const bool z = r.az < next.x;
      const float an = fminf(r.az, next.x);
      visit(base + (r.at + __float_as_int(next.y)), A_MUL(A_SUB(an, before), r.len));
      before = an;
      r.at = z ? r.at + r.step : r.at;
      r.step = z ? r.up - r.step : r.step;
      r.az = z ? A_ADD(r.az, r.azu) : r.az;
      r.rem -= z;
      at += !z;
      next = *at;
    };
    // Every lane has as many segments as steps, and its z crossings more.
    #pragma unroll 1
    for (int b = 0; b < batches; b++) {
      #pragma unroll
      for (int u = 0; u < kColBatch; u++) segment();
      if (r.rem <= -kPad) r.az = FLT_MAX;
    }
    while (at < stop) {
      segment();
      if (r.rem <= -kPad) r.az = FLT_MAX;
    }
    __syncwarp();
    p = base + r.at;
    before = list[batches * kColBatch - 1].x;
  }
  unsigned rec = (unsigned)__cvta_generic_to_shared(col_smem4 + list_at + kColHead);
  const unsigned stop = rec + (single ? max(batches, 0) * 48u : 0u);
  #pragma unroll 1
  for (; rec != stop; rec += 48) {
    float4 dt;
    int4 col;
    float end;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(dt.x), "=f"(dt.y), "=f"(dt.z), "=f"(dt.w) : "r"(rec));
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4 + 16];" : "=r"(col.x), "=r"(col.y), "=r"(col.z), "=r"(col.w) : "r"(rec));
    asm volatile("ld.shared.f32 %0, [%1 + 44];" : "=f"(end) : "r"(rec));
    if (!__any_sync(0xffffffffu, r.az < end)) {
      visit.steps(p, col, dt, r.len);
    } else {
      float4 an;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4 + 32];" : "=f"(an.x), "=f"(an.y), "=f"(an.z), "=f"(an.w) : "r"(rec));
      // At most one z crossing a lane: its crossing goes in among the x/y
      // ones, five segments of which a lane without one skips the last.
      const float az = r.rem > -kPad ? r.az : FLT_MAX;
      const bool c0 = az < an.x, c1 = az < an.y, c2 = az < an.z, c3 = az < an.w;
      const int up = r.at + r.step;
      const float b0 = fminf(az, an.x), b1 = fmaxf(an.x, fminf(az, an.y)), b2 = fmaxf(an.y, fminf(az, an.z)),
                  b3 = fmaxf(an.z, fminf(az, an.w));
      const float4 ln = make_float4(A_SUB(b0, before), A_SUB(b1, b0), A_SUB(b2, b1), A_SUB(b3, b2));
      const int4 to = make_int4(r.at + col.x, c0 ? up + col.x : r.at + col.y, c1 ? up + col.y : r.at + col.z,
                                c2 ? up + col.z : r.at + col.w);
      visit.split(base, to, ln, r.len, c3, up + col.w, A_SUB(an.w, b3));
      r.at = c3 ? up : r.at;
      r.step = c3 ? r.up - r.step : r.step;
      r.az = c3 ? A_ADD(r.az, r.azu) : r.az;
      r.rem -= c3;
      p = base + r.at;
    }
    before = end;
  }
  #pragma unroll 1
  for (int j = max(batches, 0) * kColBatch; j < n; j++) {
    const float an = col_field(j, 2, list_at);
    const int col = __float_as_int(col_field(j, 1, list_at)), left = n - j;
    float lo = before;
    while (r.az < an && r.rem + left > 0 && r.rem > -kPad) cross(col, lo);
    if (r.rem + left > 0) visit(p + col, A_MUL(A_SUB(an, lo), r.len));
    before = an;
  }
  // z crossings still to record after the list, with the x and y ones that
  // come before them: the x/y chains are added up again to the list's end.
  if (r.rem > 0) {
    const ColWalk& h = col_head(list_at);
    float ax = h.ax, ay = h.ay, lo = h.amin;
    int col = h.col;
    auto next_xy = [&]() {
      if (ax <= ay) { lo = ax; col += h.sx; ax = A_ADD(ax, h.axu); }
      else { lo = ay; col += h.sy; ay = A_ADD(ay, h.ayu); }
    };
    for (int m = 0; m < n; m++) next_xy();
    while (r.rem > 0) {
      const int at = (int)min((unsigned)col, h.last);
      const float an = fminf(ax, ay);
      if (r.az < an) {
        cross(at, lo);
      } else {
        visit(p + at, A_MUL(A_SUB(an, lo), r.len));
        r.rem--;
        next_xy();
      }
    }
  }
}

__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b) {  // two rounded products in one instruction
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// Visitors: the gather's running sum and the scatter of length * v.  steps(): a batch in one slice, the gather's loads
// all in flight before its sums (which keep the walk's order); split(): a
// batch with a z crossing, the fifth segment only where `last`.
struct ColGather {
  float acc = 0.f;
  __device__ __forceinline__ void operator()(const float* p, float seg) { acc = A_ADD(acc, A_MUL(seg, __ldg(p))); }
  __device__ __forceinline__ void steps(const float* p, int4 col, float4 dt, float len) {
    const float v0 = __ldg(p + col.x), v1 = __ldg(p + col.y), v2 = __ldg(p + col.z), v3 = __ldg(p + col.w);
    const float2 l = make_float2(len, len);
    const float2 m = mul2_rn(mul2_rn(make_float2(dt.x, dt.y), l), make_float2(v0, v1));
    const float2 n = mul2_rn(mul2_rn(make_float2(dt.z, dt.w), l), make_float2(v2, v3));
    acc = A_ADD(A_ADD(A_ADD(A_ADD(acc, m.x), m.y), n.x), n.y);
  }
  __device__ __forceinline__ void split(const float* base, int4 to, float4 ln, float len, bool last, int to4, float ln4) {
    const float v0 = __ldg(base + to.x), v1 = __ldg(base + to.y), v2 = __ldg(base + to.z), v3 = __ldg(base + to.w);
    const float v4 = __ldg(base + to4);  // a voxel of the column for every lane
    acc = A_ADD(acc, A_MUL(A_MUL(ln.x, len), v0));
    acc = A_ADD(acc, A_MUL(A_MUL(ln.y, len), v1));
    acc = A_ADD(acc, A_MUL(A_MUL(ln.z, len), v2));
    acc = A_ADD(acc, A_MUL(A_MUL(ln.w, len), v3));
    const float with = A_ADD(acc, A_MUL(A_MUL(ln4, len), v4));
    acc = last ? with : acc;
  }
};
struct ColScatter {
  float v;  // 0: the lane adds nothing
  __device__ __forceinline__ void operator()(float* p, float seg) const {
    if (v != 0.f) red_add_global(p, A_MUL(seg, v));
  }
  __device__ __forceinline__ void steps(float* p, int4 col, float4 dt, float len) const {
    if (v == 0.f) return;
    const float2 l = make_float2(len, len), f = make_float2(v, v);
    const float2 m = mul2_rn(mul2_rn(make_float2(dt.x, dt.y), l), f);
    const float2 n = mul2_rn(mul2_rn(make_float2(dt.z, dt.w), l), f);
    red_add_global(p + col.x, m.x);
    red_add_global(p + col.y, m.y);
    red_add_global(p + col.z, n.x);
    red_add_global(p + col.w, n.y);
  }
  __device__ __forceinline__ void split(float* base, int4 to, float4 ln, float len, bool last, int to4, float ln4) const {
    if (v == 0.f) return;
    red_add_global(base + to.x, A_MUL(A_MUL(ln.x, len), v));
    red_add_global(base + to.y, A_MUL(A_MUL(ln.y, len), v));
    red_add_global(base + to.z, A_MUL(A_MUL(ln.z, len), v));
    red_add_global(base + to.w, A_MUL(A_MUL(ln.w, len), v));
    if (last) red_add_global(base + to4, A_MUL(A_MUL(ln4, len), v));
  }
};

// A lane's own walk over the column layout, for rays of LORs with too few to
// list the crossings for: the reference's steps (next_crossing), the voxel's
// place moving by a column or, in z, by the slice changes of WalkZ.  The LOR
// is one that could be listed: its walk stays within the border in x and y and
// the columns hold every slice that it can enter; the clamp of the place to
// the layout is a memory-safety net.  A step selects among all three axes' next
// crossings: few such rays are under way, and a pass over them waits for this
// chain (k_em_cols_direct).
struct ColRay {
  float ax, ay, az, axu, ayu, azu, ac, len;
  int at, sx, sy, step, up, n;
  __device__ __forceinline__ ColRay(const ColWalk& w, const WalkZ& r)
      : ax(w.ax), ay(w.ay), az(r.az), axu(w.axu), ayu(w.ayu), azu(r.azu), ac(w.amin), len(r.len), at(w.col + r.at),
        sx(w.sx), sy(w.sy), step(r.step), up(r.up), n(w.n + r.rem) {}
  __device__ __forceinline__ void next(int& place, float& seg) {
    const float an = fminf(fminf(ax, ay), az);
    const bool cx = ax == an, cy = !cx & (ay == an), cz = !(cx | cy);
    seg = A_MUL(A_SUB(an, ac), len);
    place = at;
    ac = an;
    at += cx ? sx : (cy ? sy : step);
    step = cz ? up - step : step;
    const float nx = A_ADD(ax, axu), ny = A_ADD(ay, ayu), nz = A_ADD(az, azu);
    ax = cx ? nx : ax;
    ay = cy ? ny : ay;
    az = cz ? nz : az;
  }
};
template <int U>
__device__ __forceinline__ float col_ray_gather(ColRay r, unsigned last, const float* __restrict__ img) {
  float acc = 0.f;
  int m = 0;
  for (; m + U <= r.n; m += U) {  // a batch's loads all in flight before its sums
    int place[U];
    float seg[U], v[U];
    #pragma unroll
    for (int u = 0; u < U; u++) r.next(place[u], seg[u]);
    #pragma unroll
    for (int u = 0; u < U; u++) v[u] = __ldg(img + min((unsigned)place[u], last));
    #pragma unroll
    for (int u = 0; u < U; u++) acc = A_ADD(acc, A_MUL(seg[u], v[u]));
  }
  for (; m < r.n; m++) {
    int place;
    float seg;
    r.next(place, seg);
    acc = A_ADD(acc, A_MUL(seg, __ldg(img + min((unsigned)place, last))));
  }
  return acc;
}
__device__ __forceinline__ void col_ray_scatter(ColRay r, unsigned last, float v, float* __restrict__ acc) {
  for (int m = 0; m < r.n; m++) {
    int place;
    float seg;
    r.next(place, seg);
    red_add_global(acc + min((unsigned)place, last), A_MUL(seg, v));
  }
}

// One ray with the reference's six-sided bounds test, for LORs that are not
// on the list: visit(place, length) for its segments in the image.
template <class T, class V>
__device__ __noinline__ void col_walk_checked(const float4 P, const float2 e, const ImgGeom& g, const ColDims& d,
                                              T* base, V& visit) {
  Walk3 w;
  siddon3_setup(P.x, P.y, e.x, A_SUB(P.z, P.x), A_SUB(P.w, P.y), A_SUB(e.y, e.x), g, w);
  if (walk_misses(w, g)) return;
  for (int m = 0; m < w.n; m++) {
    bool cx, cy;
    const float an = next_crossing(w, cx, cy);
    const float seg = A_MUL(A_SUB(an, w.ac), w.L);
    if (((unsigned)w.i < (unsigned)g.nx) & ((unsigned)w.j < (unsigned)g.ny) & ((unsigned)w.k < (unsigned)g.nz))
      visit(base + ((w.j + kPad) * d.px() + w.i + kPad) * d.stride() + col_slice(d, w.k), seg);
    w.ac = an;
    if (cx) { w.i += w.iinc; w.ax = A_ADD(w.ax, w.axu); }
    else if (cy) { w.j += w.jinc; w.ay = A_ADD(w.ay, w.ayu); }
    else { w.k += w.kinc; w.az = A_ADD(w.az, w.azu); }
  }
}

}  // namespace apirl
