// The parts of the column walk's kernels that the single and the batched passes
// share: a LOR's place in a subset, the fused pass of a warp's 32 rays, a
// block's list of sinograms with counts, and the tiles of the copies between
// images and the column layout.
#pragma once
#include "bins.cuh"
#include "columns.cuh"

namespace apirl {

struct ColLor {
  int k, l, a;  // subset angle, r, full angle
};

// LOR `at` of the subset, r first.
__device__ __forceinline__ ColLor col_lor(const LorTable& t, const SubsetSel& s, unsigned at) {
  ColLor c;
  c.k = (int)(at / (unsigned)t.n_r);
  c.l = (int)(at - (unsigned)c.k * (unsigned)t.n_r);
  c.a = s.subset < 0 ? c.k : s.subset + s.nsub * c.k;
  return c;
}

// The fused pass (k_em_pass_persist's steps, kernels.cu) of the warp's 32
// rays: forward walk, additive term, likelihood term, ratio, and the ratio
// scattered along the walk.  Returns the lane's likelihood term.
// gl: the lane's sinogram (within the shard), m its counts, ci the place of its
// additive term.
__device__ __forceinline__ double em_rays(const ImgGeom& g, const ColDims& d, const LorTable& t, const float4 P, int gl,
                                          bool in, float m, int64_t ci, const float* __restrict__ add,
                                          const float* __restrict__ img, float* __restrict__ acc, int back,
                                          int skip_zero) {
  const ColWalk& w = col_head();
  acc += w.xmain ? d.floats() : 0;
  const float2 ez = in ? __ldg(t.z + t.g0 + gl) : make_float2(0.f, 0.f);
  ColGather sum;
  WalkZ r = col_no_ray();
  if (w.listed) {
    if (in) r = col_setup_z(ez, w, g, d);
    col_walk(r, d, img, sum);
  } else if (in) {
    col_walk_checked(P, ez, g, d, img, sum);
  }
  double term = 0.0;
  float q = 0.f;
  if (in) {
    float e = sum.acc;
    if (add) e = A_ADD(e, __ldg(add + ci));
    if (e != 0.f) term = lik_term(m, e, skip_zero);
    q = (m != 0.f && e != 0.f && back) ? A_DIV(m, e) : 0.f;
  }
  if (__any_sync(0xffffffffu, q != 0.f)) {
    ColScatter out{q};
    if (w.listed) col_walk(q != 0.f ? r : col_no_ray(), d, acc, out);
    else if (q != 0.f) col_walk_checked(P, ez, g, d, acc, out);
  }
  return term;
}

// The block's list of a LOR's sinograms with counts, among kColWindow from
// g0: list[0 .. n) in order, n returned to every thread.
struct ColActive {
  unsigned mask[kColWindow / 32];
  int first[kColWindow / 32];
  int n;
  uint16_t list[kColWindow];
};
// count(i): the counts of sinogram g0 + i.
template <class C>
__device__ __forceinline__ int col_active(int n_sinos, int g0, C&& count, ColActive& act) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int left = min(n_sinos - g0, kColWindow), groups = (left + 31) >> 5;
  const int warps = blockDim.x >> 5;
  for (int q = warp; q < groups; q += 4 * warps) {  // four groups' counts in flight
    float m[4];
    #pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = (q + u * warps) * 32 + lane;
      m[u] = i < left ? count(i) : 0.f;
    }
    #pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned mask = __ballot_sync(0xffffffffu, m[u] != 0.f);
      if (lane == 0 && q + u * warps < groups) act.mask[q + u * warps] = mask;
    }
  }
  __syncthreads();
  if (warp == 0) {
    static_assert(kColWindow / 32 == 64, "two groups a lane");
    const int a = 2 * lane < groups ? __popc(act.mask[2 * lane]) : 0;
    const int b = 2 * lane + 1 < groups ? __popc(act.mask[2 * lane + 1]) : 0;
    int incl = a + b;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    act.first[2 * lane] = incl - a - b;
    act.first[2 * lane + 1] = incl - b;
    if (lane == 31) act.n = incl;
  }
  __syncthreads();
  for (int q = warp; q < groups; q += warps) {
    const unsigned m = act.mask[q];
    if (m >> lane & 1u) act.list[act.first[q] + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(q * 32 + lane);
  }
  __syncthreads();
  return act.n;
}

// Copies between images ([z][y][x]) and columns: a block of 256 threads (lx of
// 32, ly of 8) works 32 x of one row y and 32 slices z0 .. z0 + 31;
// tile[par * 16 + z / 2][x]: the slices in the order the columns store them.

// img's interior <- x.  With gimg: returns the thread's sum of x . gimg over
// its voxels where gimg != 0 (k_neg_dot's rule, kernels.cu), FP64.
__device__ __forceinline__ double col_copy_tile(const ColDims& d, const float* __restrict__ x,
                                                float* __restrict__ img, const float* __restrict__ gimg, int x0, int y,
                                                int z0, int lx, int ly, float (*tile)[33]) {
  float v[4], gv[4];
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int z = z0 + ly + 8 * q;
    const bool in = x0 + lx < d.nx && z < d.nz;
    const int64_t i = ((int64_t)z * d.ny + y) * d.nx + x0 + lx;
    v[q] = in ? x[i] : 0.f;
    gv[q] = gimg && in ? gimg[i] : 0.f;
  }
  double s = 0.0;
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int z = ly + 8 * q;
    tile[(z & 1) * 16 + (z >> 1)][lx] = v[q];
    if (gv[q] != 0.f) s += (double)v[q] * (double)gv[q];
  }
  __syncthreads();
  const int par = lx >> 4, z = z0 + 2 * (lx & 15) + par;
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int xx = ly + 8 * q;
    if (x0 + xx < d.nx && z < d.nz)
      img[((int64_t)(y + kPad) * d.px() + x0 + xx + kPad) * d.stride() + par * d.half + ((z + d.z0) >> 1)] =
          tile[lx][xx];
  }
  return s;
}

// mode 0: EM update of x from the two column sums acc (rule ge / gt, as
// k_update); mode 1: bp += their sum.  Their interiors are cleared, after the
// block's loads.
__device__ __forceinline__ void col_reduce_tile(const ColDims& d, float* __restrict__ acc, int mode,
                                                float* __restrict__ x, float* __restrict__ bp,
                                                const float* __restrict__ sens, float thr, int ge, int x0, int y,
                                                int z0, int lx, int ly, float (*tile)[33]) {
  const int par = lx >> 4, zc = z0 + 2 * (lx & 15) + par;
  float* out = mode == 0 ? x : bp;
  float xv[4], sv[4];
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int xx = ly + 8 * q;
    if (x0 + xx < d.nx && zc < d.nz) {
      const float* a = acc + ((int64_t)(y + kPad) * d.px() + x0 + xx + kPad) * d.stride() + par * d.half +
                       ((zc + d.z0) >> 1);
      tile[lx][xx] = A_ADD(a[0], a[d.floats()]);
    }
  }
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int z = z0 + ly + 8 * q;
    xv[q] = sv[q] = 0.f;
    if (x0 + lx < d.nx && z < d.nz) {
      const int64_t i = ((int64_t)z * d.ny + y) * d.nx + x0 + lx;
      xv[q] = out[i];
      if (mode == 0) sv[q] = sens[i];
    }
  }
  __syncthreads();
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int xx = ly + 8 * q;
    if (x0 + xx < d.nx && zc < d.nz) {
      float* a = acc + ((int64_t)(y + kPad) * d.px() + x0 + xx + kPad) * d.stride() + par * d.half + ((zc + d.z0) >> 1);
      a[0] = a[d.floats()] = 0.f;
    }
  }
  #pragma unroll
  for (int q = 0; q < 4; q++) {
    const int zl = ly + 8 * q, z = z0 + zl;
    if (x0 + lx >= d.nx || z >= d.nz) continue;
    const int64_t i = ((int64_t)z * d.ny + y) * d.nx + x0 + lx;
    const float b = tile[(zl & 1) * 16 + (zl >> 1)][lx];
    if (mode == 0) {
      const bool okv = ge ? (sv[q] >= thr) : (sv[q] > thr);
      out[i] = okv ? A_DIV(A_MUL(xv[q], b), sv[q]) : 0.f;
    } else {
      out[i] = A_ADD(xv[q], b);
    }
  }
}

}  // namespace apirl
