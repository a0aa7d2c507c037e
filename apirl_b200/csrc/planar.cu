// The fused EM pass of 2D sinograms: project, add, likelihood term, ratio,
// backproject, on two padded layouts of the slice and two copies of each
// backprojection sum.
//
// Rays that run mostly along x walk the transposed layout, as in 3D: the 32
// neighbouring rays of a warp then touch neighbouring floats, where along a
// column of [y][x] every lane would touch a sector of its own.  Blocks add
// into copy blockIdx % kPlanarCopies, as the slice has few sectors for its
// adds (2048 for 7 M adds at 128 x 128), and the update sums the copies.
// Measured, one [y][x] sum and no copies -> this, the whole pass: 128 x 128
// image, 192 x 192 bins 55 -> 31 us; 256 x 256, 384 x 307 bins 157 -> 80 us;
// 48 x 48, 72 x 57 bins 20.6 -> 19.6 us (one copy of the sums: 33, 86, 19.6;
// sixteen: the update's reads cost more than the spread adds gain).
#include <cuda_runtime.h>
#include <cstdint>
#include "bins.cuh"
#include "internal.h"
#include "siddon.cuh"

namespace apirl {

namespace {

// A 2D walk under way over a padded layout: the next crossings, the last one,
// the voxel's index.
struct PlanarAt {
  float ax, ay, ac;
  int idx;
};

// The constants of a guarded walk, which stays inside the border, whose voxels
// read zero and whose sums nobody reads; the index is clamped to the padded
// slice (as siddon3_gather_pad's).
struct PlanarRay {
  float axu, ayu, L;
  int sx, sy;
  unsigned lim;
  // U segments from `at`: their places and lengths.
  template <int U>
  __device__ __forceinline__ void step(PlanarAt& at, unsigned (&place)[U], float (&seg)[U]) const {
    #pragma unroll
    for (int u = 0; u < U; u++) {
      const bool cx = at.ax <= at.ay;
      const float an = fminf(at.ax, at.ay);
      seg[u] = A_MUL(A_SUB(an, at.ac), L);
      place[u] = min((unsigned)at.idx, lim - 1u);
      at.ac = an;
      at.idx += cx ? sx : sy;
      const float nx = A_ADD(at.ax, axu), ny = A_ADD(at.ay, ayu);
      at.ax = cx ? nx : at.ax;
      at.ay = cx ? at.ay : ny;
    }
  }
};

// A ray that is not guarded, with the reference's bounds test: visit(index, length).
template <class V>
__device__ __forceinline__ void planar_checked(Walk2 w, const ImgGeom& g, int ux, int uy, V&& visit) {
  const int sx = w.iinc * ux, sy = w.jinc * uy;
  int idx = (w.j + kPad) * uy + (w.i + kPad) * ux;
  for (int m = 0; m < w.n; m++) {
    const bool cx = w.ax <= w.ay;
    const float an = cx ? w.ax : w.ay;
    if (((unsigned)w.i < (unsigned)g.nx) & ((unsigned)w.j < (unsigned)g.ny))
      visit((unsigned)idx, A_MUL(A_SUB(an, w.ac), w.L));
    w.ac = an;
    if (cx) { w.i += w.iinc; idx += sx; w.ax = A_ADD(w.ax, w.axu); }
    else { w.j += w.jinc; idx += sy; w.ay = A_ADD(w.ay, w.ayu); }
  }
}

// The fused pass.  Blocks of one warp: the pass is a few warps an SM whose
// rays differ in length, and small blocks even the SMs out (128 x 128, 192 x
// 192 bins, the whole pass: 31 us, 35 us with 64 threads, 39 us with 128).  It
// waits for the walks' chains of additions and for loads; four warps a 32 rays,
// a half of the forward walk and a quarter of the scatter each, took the same
// time there and 98 against 80 us on 256 x 256.  The likelihood partials are
// one per 32 bins.
constexpr int kPlanarU = 8;
template <typename CT>
__global__ void __launch_bounds__(32) k_planar_pass(ImgGeom g, LorTable t, SubsetSel s, const CT* __restrict__ counts,
                                                    int counts_packed, const float* __restrict__ add, PlanarBuffers pl,
                                                    int back, int lik_mode, double* __restrict__ partials, int total) {
  const int b = blockIdx.x * 32 + threadIdx.x;
  Walk2 w;
  w.n = 0;
  w.guarded = 1;
  bool ray = false, tr = false;
  int at0 = 0;
  if (b < total) {
    const int k = b / t.n_r, l = b - k * t.n_r;
    const int full = (s.subset < 0 ? k : s.subset + s.nsub * k) * t.n_r + l;
    at0 = counts_packed ? b : full;
    ray = __ldg(t.ok + l) != 0;
    const float4 L = __ldg(t.lor + full);
    const float vx = A_SUB(L.z, L.x), vy = A_SUB(L.w, L.y);
    tr = fabsf(vx) >= fabsf(vy);
    if (ray) siddon2_setup(L.x, L.y, vx, vy, g, w);
  }
  const int ux = tr ? g.ny + 2 * kPad : 1, uy = tr ? 1 : g.nx + 2 * kPad;
  const float* __restrict__ img = tr ? pl.imgT : pl.img;
  const PlanarRay p{w.axu, w.ayu, w.L, w.iinc * ux, w.jinc * uy, pl.lim};
  PlanarAt at{w.ax, w.ay, w.ac, (w.j + kPad) * uy + (w.i + kPad) * ux};
  const int batches = w.guarded ? w.n / kPlanarU : 0, rest = w.guarded ? w.n - batches * kPlanarU : 0;
  unsigned place[kPlanarU], place1[1];
  float seg[kPlanarU], seg1[1], e = 0.f;
  for (int i = 0; i < batches; i++) {  // a batch's loads all in flight before its sums
    p.step(at, place, seg);
    float v[kPlanarU];
    #pragma unroll
    for (int u = 0; u < kPlanarU; u++) v[u] = __ldg(img + place[u]);
    #pragma unroll
    for (int u = 0; u < kPlanarU; u++) e = A_ADD(e, A_MUL(seg[u], v[u]));
  }
  for (int i = 0; i < rest; i++) {
    p.step(at, place1, seg1);
    e = A_ADD(e, A_MUL(seg1[0], __ldg(img + place1[0])));
  }
  if (w.n > 0 && !w.guarded)
    planar_checked(w, g, ux, uy, [&](unsigned k, float len) { e = A_ADD(e, A_MUL(len, __ldg(img + k))); });
  double term = 0.0;
  float r = 0.f;
  if (b < total) {
    const float m = load_count<CT>(counts, at0);
    if (add) e = A_ADD(e, __ldg(add + at0));
    r = (m != 0.f && e != 0.f) ? A_DIV(m, e) : 0.f;
    if (lik_mode == 2) { if (r > 0.f) term = (double)m * log((double)r) - (double)r; }
    else if (lik_mode == 1 ? (e > 0.f) : (e != 0.f)) term = (double)m * log((double)e) - (double)e;
  }
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) term += __shfl_down_sync(0xffffffffu, term, o);
  if (threadIdx.x == 0) partials[blockIdx.x] = term;
  if (!back || r == 0.f || w.n == 0) return;
  float* __restrict__ sum = (tr ? pl.sumT : pl.sum) + (size_t)(blockIdx.x % (unsigned)kPlanarCopies) * pl.lim;
  if (!w.guarded) {
    planar_checked(w, g, ux, uy, [&](unsigned k, float len) { red_add_global(sum + k, A_MUL(len, r)); });
    return;
  }
  at = PlanarAt{w.ax, w.ay, w.ac, (w.j + kPad) * uy + (w.i + kPad) * ux};
  for (int i = 0; i < batches; i++) {
    p.step(at, place, seg);
    #pragma unroll
    for (int u = 0; u < kPlanarU; u++) red_add_global(sum + place[u], A_MUL(seg[u], r));
  }
  for (int i = 0; i < rest; i++) {
    p.step(at, place1, seg1);
    red_add_global(sum + place1[0], A_MUL(seg1[0], r));
  }
}

// img and imgT's interiors <- x ([y][x]); 32 x 8 voxels a block.
__global__ void __launch_bounds__(256) k_planar_copy(int nx, int ny, const float* __restrict__ x, PlanarBuffers pl) {
  __shared__ float tile[8][33];
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 8, lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  const int px = nx + 2 * kPad, py = ny + 2 * kPad;
  if (x0 + lx < nx && y0 + ly < ny) {
    const float v = x[(int64_t)(y0 + ly) * nx + x0 + lx];
    pl.img[(int64_t)(y0 + ly + kPad) * px + x0 + lx + kPad] = v;
    tile[ly][lx] = v;
  }
  __syncthreads();
  const int ty = threadIdx.x & 7, tx = threadIdx.x >> 3;
  if (x0 + tx < nx && y0 + ty < ny) pl.imgT[(int64_t)(x0 + tx + kPad) * py + y0 + ty + kPad] = tile[ty][tx];
}

// mode 0: EM update of x from the sum of the copies (threshold rule); mode 1:
// bp += that sum.  The copies are cleared.  With lik, the first row of blocks
// (y = 0) sums the n partials in a fixed order instead.
__global__ void __launch_bounds__(256) k_planar_update(int nx, int ny, PlanarBuffers pl, int mode,
                                                       float* __restrict__ x, float* __restrict__ bp,
                                                       const float* __restrict__ sens,
                                                       const float* __restrict__ thr_ptr, float thr_value, int ge,
                                                       const double* __restrict__ partials, int64_t n,
                                                       double* __restrict__ lik) {
  __shared__ double part[8];
  __shared__ float tile[8][33];
  if (lik && blockIdx.y == 0) {
    if (blockIdx.x) return;
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += 256) s += partials[i];
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      s = 0.0;
      for (int w = 0; w < 8; w++) s += part[w];
      *lik = s;
    }
    return;
  }
  const int x0 = blockIdx.x * 32, y0 = (blockIdx.y - (lik ? 1 : 0)) * 8, lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  const int ty = threadIdx.x & 7, tx = threadIdx.x >> 3;
  const int px = nx + 2 * kPad, py = ny + 2 * kPad;
  const bool inA = x0 + lx < nx && y0 + ly < ny, inT = x0 + tx < nx && y0 + ty < ny;
  float* const pA = pl.sum + (int64_t)(y0 + ly + kPad) * px + x0 + lx + kPad;
  float* const pT = pl.sumT + (int64_t)(x0 + tx + kPad) * py + y0 + ty + kPad;
  float a = 0.f, c = 0.f;
  #pragma unroll
  for (int r = 0; r < kPlanarCopies; r++) {
    a = A_ADD(a, inA ? pA[(size_t)r * pl.lim] : 0.f);
    c = A_ADD(c, inT ? pT[(size_t)r * pl.lim] : 0.f);
  }
  const int64_t i = (int64_t)(y0 + ly) * nx + x0 + lx;
  const float old = inA ? (mode == 0 ? x[i] : bp[i]) : 0.f, sv = inA && mode == 0 ? sens[i] : 0.f;
  const float thr = (mode == 0 && thr_ptr) ? *thr_ptr : thr_value;
  tile[ty][tx] = c;
  __syncthreads();
  #pragma unroll
  for (int r = 0; r < kPlanarCopies; r++) {
    if (inA) pA[(size_t)r * pl.lim] = 0.f;
    if (inT) pT[(size_t)r * pl.lim] = 0.f;
  }
  if (!inA) return;
  const float s = A_ADD(a, tile[ly][lx]);
  if (mode == 0) x[i] = (ge ? (sv >= thr) : (sv > thr)) ? A_DIV(A_MUL(old, s), sv) : 0.f;
  else bp[i] = A_ADD(old, s);
}

}  // namespace

unsigned planar_lim(const ImgGeom& g) {
  const int64_t n = (int64_t)(g.nx + 2 * kPad) * (g.ny + 2 * kPad);
  // (grids of at most 65535 rows, one of them the likelihood's)
  return n <= ((int64_t)1 << 25) && g.ny <= 65534 * 8 ? (unsigned)n : 0u;
}

cudaError_t launch_planar_pass(const ImgGeom& g, const LorTable& t, SubsetSel s, const void* counts, int counts_dtype,
                               int counts_packed, const float* add, const float* x, const PlanarBuffers& pl, int back, int lik_mode,
                               double* partials, cudaStream_t st) {
  const int total = s.nk * t.n_r;
  if (total == 0) return cudaSuccess;
  const dim3 grid((g.nx + 31) / 32, (g.ny + 7) / 8);
  k_planar_copy<<<grid, 256, 0, st>>>(g.nx, g.ny, x, pl);
  const unsigned blocks = (unsigned)((total + 31) / 32);
  switch (counts_dtype) {
    case APIRL_F32:
      k_planar_pass<float><<<blocks, 32, 0, st>>>(g, t, s, (const float*)counts, counts_packed, add, pl, back, lik_mode,
                                                           partials, total);
      break;
    case APIRL_U32:
      k_planar_pass<uint32_t><<<blocks, 32, 0, st>>>(g, t, s, (const uint32_t*)counts, counts_packed, add, pl, back, lik_mode,
                                                              partials, total);
      break;
    case APIRL_U16:
      k_planar_pass<uint16_t><<<blocks, 32, 0, st>>>(g, t, s, (const uint16_t*)counts, counts_packed, add, pl, back, lik_mode,
                                                              partials, total);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_planar_update(const ImgGeom& g, const PlanarBuffers& pl, int mode, float* x, float* bp,
                                 const float* sens, const float* thr_ptr, float thr_value, int ge,
                                 const double* partials, int64_t n, double* lik, cudaStream_t st) {
  const dim3 grid((g.nx + 31) / 32, (g.ny + 7) / 8 + (lik ? 1 : 0));
  k_planar_update<<<grid, 256, 0, st>>>(g.nx, g.ny, pl, mode, x, bp, sens, thr_ptr, thr_value, ge, partials, n, lik);
  return cudaGetLastError();
}

}  // namespace apirl
