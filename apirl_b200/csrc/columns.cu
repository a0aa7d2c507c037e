// Kernels of the column walk (columns.cuh): projection, backprojection and the
// fused EM pass of 3D sinograms with one float ray per bin, and the copies
// between images and the column layout.
//
// A block takes one (angle, r) of the subset and all the sinograms of the
// shard, 32 to a warp at a time.  Blocks run r first, then angle: neighbours
// in r share columns in L1 and L2 (the listed pass of the 256 x 256 x 81 job
// 1.19 ms, angle first 1.28 ms).
//
// Measured on that job's subset 0 of 21 (6.78 M bins, 2.14e9 segments forward,
// 0.94e9 back, B200), the padded pair's kernels -> these: projection 3.59 ->
// 1.15 ms, backprojection 4.07 -> 1.86, full pass 2.68 -> 1.77, listed pass
// 1.76 -> 1.22.  The gathers are bound by instruction issue (70 % of the
// slots; 8 warp instructions a step without z crossings, 22 in a batch with
// one), the scatters by the SM-to-L2 path: 5.1 sectors a reduction of 32 lanes
// (the pair's rays along r: 10.3), 217 G sectors/s.
#include <cuda_runtime.h>
#include <climits>
#include <cmath>
#include <cstdint>
#include "columns_em.cuh"
#include "internal.h"

namespace apirl {

namespace {

// Eight warps, so that a list serves many sinograms, at 5 blocks an SM (48
// registers): the full pass of that job 1.71 ms, against 1.80 / 1.79 / 1.77 /
// 2.03 ms with 128 / 192 / 320 / 512 threads and 1.82 ms at 4 blocks (64
// registers, without the 56 bytes that k_em_cols spills here).
constexpr int kColBlock = 256;
constexpr int kColBlocks = 5;
// With several rays a bin and as many lists to make, blocks of up to 16 warps:
// 271 sinograms of a 46 x 46 x 37 job, 6 rays a bin 120 -> 92 us against 8, 784
// of 36 x 36 x 64 159 -> 113, 1141 of 80 x 80 x 78 548 -> 494.
constexpr int kRaysBlock = 512;
constexpr int kRaysBlocks = 2;
constexpr int kMaxWarps = kRaysBlock / 32;
// Blocks of the LORs with few counts.
constexpr int kColFewBlock = 64;
constexpr int kColFewBlocks = 20;
// Blocks of the bins walked one a lane (small, to spread few of them), and
// their loads in flight.
constexpr int kColDirectBlock = 64;
constexpr int kColDirectBlocks = 16;
constexpr int kColDirectU = 8;
constexpr int kColDirectBack = 8;  // values of a LOR that a backprojection walks so
// Blocks of the batched pass, whose LORs have from a few to hundreds of
// counts: ten mixed jobs of 64 - 128 x 1 - 41 slices in 16.7 ms, against 18.0 /
// 17.6 / 17.8 / 20.4 ms with 64 / 96 / 160 / 256 threads and 18.1 ms at 8 blocks
// (64 registers).
constexpr int kMultiColBlock = 128;
constexpr int kMultiColBlocks = 10;

__global__ void __launch_bounds__(kColBlock, kColBlocks) k_project_cols(ImgGeom g, ColDims d, LorTable t, SubsetSel s,
                                                            const float* __restrict__ img, float* __restrict__ out) {
  const ColLor lor = col_lor(t, s, blockIdx.x);
  const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
  col_list(P, g, d);
  const ColWalk& w = col_head();
  for (int g0 = threadIdx.x & ~31; g0 < t.n_sinos; g0 += blockDim.x) {
    const int gl = g0 + (threadIdx.x & 31);
    const bool in = gl < t.n_sinos;
    const float2 e = in ? __ldg(t.z + t.g0 + gl) : make_float2(0.f, 0.f);
    ColGather sum;
    if (w.listed) col_walk(in ? col_setup_z(e, w, g, d) : col_no_ray(), d, img, sum);
    else if (in) col_walk_checked(P, e, g, d, img, sum);
    if (in) out[((int64_t)gl * s.nk + lor.k) * t.n_r + lor.l] = sum.acc;
  }
}

// A ray's adds where v / e would leave the float range: (seg * v) / e.
struct ColScatterDivide {
  float v, e;
  __device__ __forceinline__ void operator()(float* p, float seg) const {
    red_add_global(p, A_DIV(A_MUL(seg, v), e));
  }
};

// acc += A_s^T v in the column layout: Backproject's rule (SiddonProjector.cpp:496,
// bins with v == 0 add nothing) and, with vest, DivideAndBackproject's
// (:669-683: (seg * v) / e where e != 0, else seg * v).  The ratio v / e is
// formed once per bin where v and the ratio are far from the ends of the
// float range, and per segment elsewhere.  LOOK (a thread a sinogram): a LOR
// without values is left before its crossings are listed, and the bins of one
// with at most `few` go to the queue (k_scatter_cols_direct).
template <bool LOOK>
__global__ void __launch_bounds__(kColBlock, kColBlocks) k_scatter_cols(ImgGeom g, ColDims d, LorTable t, SubsetSel s,
                                                                        const float* __restrict__ vin,
                                                                        const float* __restrict__ vest,
                                                                        float* __restrict__ acc, int few,
                                                                        ColQueue queue) {
  const ColLor lor = col_lor(t, s, blockIdx.x);
  if (LOOK) {
    const int gl = threadIdx.x;
    const bool any = gl < t.n_sinos && __ldg(vin + ((int64_t)gl * s.nk + lor.k) * t.n_r + lor.l) != 0.f;
    const int n = __syncthreads_count(any);
    if (n == 0) return;
    if (n <= few) {
      const unsigned mask = __ballot_sync(0xffffffffu, any), lane = threadIdx.x & 31;
      unsigned slot = 0;
      if (lane == 0 && mask) slot = atomicAdd(queue.n + 1, (unsigned)__popc(mask));
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (any) queue.bins[slot + __popc(mask & ((1u << lane) - 1u))] = blockIdx.x * (unsigned)t.n_sinos + gl;
      return;
    }
  }
  const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
  col_list(P, g, d);
  const ColWalk& w = col_head();
  acc += w.xmain ? d.floats() : 0;
  for (int g0 = threadIdx.x & ~31; g0 < t.n_sinos; g0 += blockDim.x) {
    const int gl = g0 + (threadIdx.x & 31);
    bool in = gl < t.n_sinos;
    const int64_t b = ((int64_t)gl * s.nk + lor.k) * t.n_r + lor.l;
    float v = 0.f, ends = 0.f;
    if (in) {
      v = __ldg(vin + b);
      in = v != 0.f;
      const float est = vest ? __ldg(vest + b) : 0.f;
      if (in && est != 0.f) {
        const float q = A_DIV(v, est), av = fabsf(v), aq = fabsf(q);
        if (av >= 1e-30f && av <= 1e30f && aq >= 1e-30f && aq <= 1e30f) v = q;
        else ends = est;
      }
    }
    const float2 e = in ? __ldg(t.z + t.g0 + gl) : make_float2(0.f, 0.f);
    if (ends != 0.f) {
      ColScatterDivide add{v, ends};
      col_walk_checked(P, e, g, d, acc, add);
      in = false;
    }
    if (!__any_sync(0xffffffffu, in)) continue;
    ColScatter add{in ? v : 0.f};
    if (w.listed) col_walk(in ? col_setup_z(e, w, g, d) : col_no_ray(), d, acc, add);
    else if (in) col_walk_checked(P, e, g, d, acc, add);
  }
}

// A backprojection's queued bins, a lane each.
__global__ void __launch_bounds__(kColDirectBlock, kColDirectBlocks) k_scatter_cols_direct(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const float* __restrict__ vin, float* __restrict__ acc,
    ColQueue queue) {
  const unsigned bins = queue.n[1], last = (unsigned)d.floats() - 1u;
  for (unsigned b = blockIdx.x * blockDim.x + threadIdx.x; b < bins; b += gridDim.x * blockDim.x) {
    const unsigned bin = queue.bins[b], at = bin / (unsigned)t.n_sinos;
    const ColLor lor = col_lor(t, s, at);
    const int gl = (int)(bin - at * (unsigned)t.n_sinos);
    const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
    const float2 ez = __ldg(t.z + t.g0 + gl);
    const float v = __ldg(vin + ((int64_t)gl * s.nk + lor.k) * t.n_r + lor.l);
    ColWalk w;
    col_setup_xy(P, g, d, w);
    float* const sums = acc + (w.xmain ? d.floats() : 0);
    ColScatter add{v};
    if (w.listed) col_ray_scatter(ColRay(w, col_setup_z(ez, w, g, d)), last, v, sums);
    else col_walk_checked(P, ez, g, d, sums, add);
  }
}

// Place of a bin (sinogram gl of the shard) in the counts / additive layout.
__device__ __forceinline__ int64_t bin_of(const LorTable& t, const SubsetSel& s, const ColLor& lor, int gl, int packed) {
  return (packed ? (int64_t)gl * s.nk + lor.k : (int64_t)(t.g0 + gl) * t.n_proj + lor.a) * t.n_r + lor.l;
}

// The LOR's likelihood partial: the sum of the block's terms, warps in order.
__device__ __forceinline__ void em_partial(double term, unsigned lor, double* __restrict__ partials) {
  __shared__ double part[kMaxWarps];
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) term += __shfl_down_sync(0xffffffffu, term, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = term;
  __syncthreads();
  if (threadIdx.x == 0) {
    term = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) term += part[w];
    partials[lor] = term;
  }
}

// The fused pass over every bin of the subset.
template <typename CT>
__global__ void __launch_bounds__(kColBlock, kColBlocks) k_em_cols(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const CT* __restrict__ counts, int counts_packed,
    const float* __restrict__ add, const float* __restrict__ img, float* __restrict__ acc, int back,
    double* __restrict__ partials) {
  const ColLor lor = col_lor(t, s, blockIdx.x);
  const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
  col_list(P, g, d);
  double term = 0.0;
  for (int g0 = threadIdx.x & ~31; g0 < t.n_sinos; g0 += blockDim.x) {
    const int gl = g0 + (threadIdx.x & 31);
    const bool in = gl < t.n_sinos;
    const int64_t ci = bin_of(t, s, lor, gl, counts_packed);
    term += em_rays(g, d, t, P, gl, in, in ? load_count<CT>(counts, ci) : 0.f, ci, add, img, acc, back, 0);
  }
  em_partial(term, blockIdx.x, partials);
}

// The fused pass with several rays a bin (for_rays' order, kernels.cu: ring
// pair, radial sample, axial sample; one running sum): a block keeps one list
// a radial sample, its lanes take their sinograms' ring pairs in step.  Bound
// by latency on small images, whose LORs are few: a 64 x 64 x 21 job's subset
// of 8 with 3 x 2 rays a bin (862 LORs, 91 sinograms) 246 us bin by bin, 100 us
// here.
template <typename CT>
__global__ void __launch_bounds__(kRaysBlock, kRaysBlocks) k_em_cols_rays(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const CT* __restrict__ counts, int counts_packed,
    const float* __restrict__ add, const float* __restrict__ img, float* __restrict__ acc, int back,
    double* __restrict__ partials) {
  const ColLor lor = col_lor(t, s, blockIdx.x);
  const float4* const L = t.lor_s + ((int64_t)lor.a * t.n_r + lor.l) * t.n_rs;
  const int one = (int)(col_smem(g.nx, g.ny) / 16);
  for (int o = 0; o < t.n_rs; o++) col_list(__ldg(L + o), g, d, o * one);
  double term = 0.0;
  for (int g0 = threadIdx.x & ~31; g0 < t.n_sinos; g0 += blockDim.x) {
    const int gl = g0 + (threadIdx.x & 31);
    const bool in = gl < t.n_sinos;
    const int first = in ? __ldg(t.zoff + t.g0 + gl) : 0, n = in ? __ldg(t.zoff + t.g0 + gl + 1) - first : 0;
    const int most = __reduce_max_sync(0xffffffffu, n);
    auto rays = [&](float* base, auto& visit, bool live) {
      for (int m = 0; m < most; m += t.n_as)
        for (int o = 0; o < t.n_rs; o++) {
          const ColWalk& w = col_head(o * one);
          for (int q = 0; q < t.n_as; q++) {
            const bool ray = live && m < n;
            const float2 e = ray ? __ldg(t.zs + first + m + q) : make_float2(0.f, 0.f);
            float* const sums = base + (base == acc && w.xmain ? d.floats() : 0);
            if (w.listed) col_walk(ray ? col_setup_z(e, w, g, d) : col_no_ray(), d, sums, visit, o * one);
            else if (ray) col_walk_checked(__ldg(L + o), e, g, d, sums, visit);
          }
        }
    };
    ColGather sum;
    rays(const_cast<float*>(img), sum, in);
    float q = 0.f;
    if (in) {
      const int64_t ci = bin_of(t, s, lor, gl, counts_packed);
      const float m = load_count<CT>(counts, ci);
      float e = sum.acc;
      if (add) e = A_ADD(e, __ldg(add + ci));
      if (e != 0.f) term += lik_term(m, e, 0);
      q = (m != 0.f && e != 0.f && back) ? A_DIV(m, e) : 0.f;
    }
    if (__any_sync(0xffffffffu, q != 0.f)) {
      ColScatter out{q};
      rays(acc, out, q != 0.f);
    }
  }
  em_partial(term, blockIdx.x, partials);
}

// The fused pass over the bins with counts: a block lists its LOR's
// sinograms with counts and its warps take 32 of them at a time.  skip_zero
// as lik_term.  A LOR with at most `few` (<= kColFew) counts would leave most
// of the block's warps idle: it goes to the queue with its list, for the small
// blocks of k_em_cols_few; or with at most `direct` its bins go there, for
// k_em_cols_direct.
template <typename CT>
__global__ void __launch_bounds__(kColBlock, kColBlocks) k_em_cols_listed(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const CT* __restrict__ counts, int counts_packed,
    const float* __restrict__ add, const float* __restrict__ img, float* __restrict__ acc, int back,
    double* __restrict__ partials, int skip_zero, int few, int direct, ColQueue queue) {
  __shared__ ColActive act;
  __shared__ unsigned slot;
  const ColLor lor = col_lor(t, s, blockIdx.x);
  const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
  const int64_t step = (int64_t)(counts_packed ? s.nk : t.n_proj) * t.n_r;  // from a sinogram to the next
  bool listed = false;
  double term = 0.0;
  for (int g0 = 0; g0 < t.n_sinos; g0 += kColWindow) {
    const int64_t first = bin_of(t, s, lor, g0, counts_packed);
    const int n = col_active(t.n_sinos, g0, [&](int i) { return load_count<CT>(counts, first + i * step); }, act);
    if ((n <= few || n <= direct) && t.n_sinos <= kColWindow) {
      if (n == 0) {
        if (threadIdx.x == 0) partials[blockIdx.x] = 0.0;
        return;
      }
      if (n <= direct) {
        if (threadIdx.x == 0) {
          slot = atomicAdd(queue.n + 1, (unsigned)n);
          partials[blockIdx.x] = 0.0;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) queue.bins[slot + i] = blockIdx.x * (unsigned)t.n_sinos + act.list[i];
        return;
      }
      if (threadIdx.x == 0) {
        slot = atomicAdd(queue.n, 1u);
        queue.item[slot] = make_uint2(blockIdx.x, (unsigned)n);
      }
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) queue.list[(int64_t)slot * kColFew + i] = act.list[i];
      return;
    }
    if (n > 0 && !listed) {
      col_list(P, g, d);
      listed = true;
    }
    for (int i0 = threadIdx.x & ~31; i0 < n; i0 += blockDim.x) {
      const int i = i0 + (threadIdx.x & 31);
      const bool in = i < n;
      const int gl = in ? g0 + act.list[i] : 0;
      const int64_t ci = bin_of(t, s, lor, gl, counts_packed);
      term += em_rays(g, d, t, P, gl, in, in ? load_count<CT>(counts, ci) : 0.f, ci, add, img, acc, back, skip_zero);
    }
    __syncthreads();
  }
  em_partial(term, blockIdx.x, partials);
}

template <typename CT>
__global__ void __launch_bounds__(kColFewBlock, kColFewBlocks) k_em_cols_few(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const CT* __restrict__ counts, int counts_packed,
    const float* __restrict__ add, const float* __restrict__ img, float* __restrict__ acc, int back,
    double* __restrict__ partials, int skip_zero, ColQueue queue) {
  const unsigned items = *queue.n;
  for (unsigned q = blockIdx.x; q < items; q += gridDim.x) {
    const uint2 item = queue.item[q];
    const int n = (int)item.y;
    const ColLor lor = col_lor(t, s, item.x);
    const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
    col_list(P, g, d);
    double term = 0.0;
    for (int i0 = threadIdx.x & ~31; i0 < n; i0 += blockDim.x) {
      const int i = i0 + (threadIdx.x & 31);
      const bool in = i < n;
      const int gl = in ? queue.list[(int64_t)q * kColFew + i] : 0;
      const int64_t ci = bin_of(t, s, lor, gl, counts_packed);
      term += em_rays(g, d, t, P, gl, in, in ? load_count<CT>(counts, ci) : 0.f, ci, add, img, acc, back, skip_zero);
    }
    em_partial(term, item.x, partials);
    __syncthreads();
  }
}

// The bins of LORs with too few counts to list the crossings for, a lane each,
// whose terms are added to their LOR's partial.  Bound by the latency of a step
// (select and eight loads in flight against branch and four: 16 sinograms of a
// 256 x 256 image at 0.2 % bins with counts, the pass 141 -> 94 us) where the
// bins are few, by instruction issue and scattered sectors where they are many.
template <typename CT>
__global__ void __launch_bounds__(kColDirectBlock, kColDirectBlocks) k_em_cols_direct(
    ImgGeom g, ColDims d, LorTable t, SubsetSel s, const CT* __restrict__ counts, int counts_packed,
    const float* __restrict__ add, const float* __restrict__ img, float* __restrict__ acc, int back,
    double* __restrict__ partials, int skip_zero, ColQueue queue) {
  const unsigned bins = queue.n[1], last = (unsigned)d.floats() - 1u;
  for (unsigned b = blockIdx.x * blockDim.x + threadIdx.x; b < bins; b += gridDim.x * blockDim.x) {
    const unsigned bin = queue.bins[b], at = bin / (unsigned)t.n_sinos;
    const ColLor lor = col_lor(t, s, at);
    const int gl = (int)(bin - at * (unsigned)t.n_sinos);
    const float4 P = __ldg(t.lor + (int64_t)lor.a * t.n_r + lor.l);
    const float2 ez = __ldg(t.z + t.g0 + gl);
    const int64_t ci = bin_of(t, s, lor, gl, counts_packed);
    const float m = load_count<CT>(counts, ci);
    ColWalk w;
    col_setup_xy(P, g, d, w);
    const ColRay ray(w, col_setup_z(ez, w, g, d));
    ColGather sum;
    if (w.listed) sum.acc = col_ray_gather<kColDirectU>(ray, last, img);
    else col_walk_checked(P, ez, g, d, img, sum);
    float e = sum.acc;
    if (add) e = A_ADD(e, __ldg(add + ci));
    if (e != 0.f) atomicAdd(partials + at, lik_term(m, e, skip_zero));
    const float q = (m != 0.f && e != 0.f && back) ? A_DIV(m, e) : 0.f;
    if (q == 0.f) continue;
    float* const sums = acc + (w.xmain ? d.floats() : 0);
    ColScatter out{q};
    if (w.listed) col_ray_scatter(ray, last, q, sums);
    else col_walk_checked(P, ez, g, d, sums, out);
  }
}

// The listed pass of many jobs (geometry form of the likelihood): LORs
// lor_begin .. of the segments, a block each, whose descriptor stays in shared
// memory.  Bound by the gathers' latency and the issue slots, as the single
// pass.  Ten mixed jobs of two iterations (single-slice ones on lists): walks
// 11.2 -> 8.5 + 1.0 ms, bin lists 2.1 -> 0.4 ms, the whole 20.6 -> 17.1 ms.
__global__ void __launch_bounds__(kMultiColBlock, kMultiColBlocks) k_em_multi_cols(const MultiCols* __restrict__ segs,
                                                                                  int nseg,
                                                                                  double* __restrict__ partials) {
  __shared__ ColActive act;
  static_assert(sizeof(MultiCols) % 8 == 0, "segment copy");
  __shared__ __align__(16) int seg_raw[sizeof(MultiCols) / 4];
  __shared__ int sk;
  const MultiCols& S = *reinterpret_cast<const MultiCols*>(seg_raw);
  if (threadIdx.x == 0) sk = find_entry(segs, nseg, blockIdx.x, [](const MultiCols& e) { return e.lor_begin; });
  __syncthreads();
  for (int i = threadIdx.x; i < (int)(sizeof(MultiCols) / 4); i += blockDim.x)
    seg_raw[i] = __ldg(reinterpret_cast<const int*>(segs + sk) + i);
  __syncthreads();
  const ColLor lor = col_lor(S.t, S.s, blockIdx.x - (unsigned)S.lor_begin);
  const ColDims d{S.g.nx, S.g.ny, S.g.nz, S.cols.z0, S.cols.half};
  const float4 P = __ldg(S.t.lor + (int64_t)lor.a * S.t.n_r + lor.l);
  const int64_t step = (int64_t)S.t.n_proj * S.t.n_r;
  bool listed = false;
  double term = 0.0;
  for (int g0 = 0; g0 < S.t.n_sinos; g0 += kColWindow) {
    const int64_t first = bin_of(S.t, S.s, lor, g0, 0);
    const int n = col_active(S.t.n_sinos, g0, [&](int i) {
      return load_count_any(S.counts, S.counts_dtype, first + i * step); }, act);
    if (n > 0 && !listed) {
      col_list(P, S.g, d);
      listed = true;
    }
    for (int i0 = threadIdx.x & ~31; i0 < n; i0 += blockDim.x) {
      const int i = i0 + (threadIdx.x & 31);
      const bool in = i < n;
      const int gl = in ? g0 + act.list[i] : 0;
      const int64_t ci = bin_of(S.t, S.s, lor, gl, 0);
      term += em_rays(S.g, d, S.t, P, gl, in, in ? load_count_any(S.counts, S.counts_dtype, ci) : 0.f, ci, S.add,
                      S.cols.img, S.cols.acc, S.back, 2);
    }
    __syncthreads();
  }
  em_partial(term, blockIdx.x, partials);
}

// ---- images to and from the column layout -----------------------------------
// img's interior <- x; with gimg: dots[block] = - (x . gimg) over the block's
// voxels.  queue_n (may be null) is set to 0.
__global__ void __launch_bounds__(256) k_col_copy(ColDims d, const float* __restrict__ x, float* __restrict__ img,
                                                  const float* __restrict__ gimg, double* __restrict__ dots,
                                                  unsigned* __restrict__ queue_n) {
  __shared__ float tile[32][33];
  __shared__ double part[8];
  const int lx = threadIdx.x, ly = threadIdx.y;
  if (queue_n && (blockIdx.x | blockIdx.y | blockIdx.z) == 0 && (lx | ly) == 0) queue_n[0] = queue_n[1] = 0;
  double s = col_copy_tile(d, x, img, gimg, blockIdx.x * 32, blockIdx.y, blockIdx.z * 32, lx, ly, tile);
  if (!gimg) return;
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lx == 0) part[ly] = s;
  __syncthreads();
  if (lx == 0 && ly == 0) {
    s = 0.0;
    for (int i = 0; i < 8; i++) s += part[i];
    dots[((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = -s;
  }
}

// The update of x (mode 0) or bp (mode 1) from the column sums.  With lik: one
// more layer of blocks (z = 0), whose first sums the n likelihood partials in a
// fixed order, less *less (may be null), beside the others' work.
__global__ void __launch_bounds__(256) k_col_reduce(ColDims d, float* __restrict__ acc, int mode,
                                                    float* __restrict__ x, float* __restrict__ bp,
                                                    const float* __restrict__ sens,
                                                    const float* __restrict__ thr_ptr, float thr_value, int ge,
                                                    const double* __restrict__ partials, int64_t n,
                                                    const double* __restrict__ less, double* __restrict__ lik) {
  __shared__ float tile[32][33];
  if (lik && blockIdx.z == 0) {
    if (blockIdx.x | blockIdx.y) return;
    double* const part = reinterpret_cast<double*>(tile);
    const int tid = threadIdx.y * 32 + threadIdx.x;
    double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int64_t i = tid;
    for (; i + 7 * 256 < n; i += 8 * 256) {
      #pragma unroll
      for (int u = 0; u < 8; u++) v[u] += partials[i + u * 256];
    }
    for (; i < n; i += 256) v[0] += partials[i];
    double s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) part[threadIdx.y] = s;
    __syncthreads();
    if (tid == 0) {
      s = 0.0;
      for (int w = 0; w < 8; w++) s += part[w];
      *lik = s - (less ? *less : 0.0);
    }
    return;
  }
  const float thr = (mode == 0 && thr_ptr) ? *thr_ptr : thr_value;
  col_reduce_tile(d, acc, mode, x, bp, sens, thr, ge, blockIdx.x * 32, blockIdx.y,
                  (lik ? blockIdx.z - 1 : blockIdx.z) * 32, threadIdx.x, threadIdx.y, tile);
}

// The list's shared memory: with the kernels' own (the listed pass's 4.7 KB)
// below the 48 KB that a block may take without asking for more.
constexpr size_t kColMaxSmem = 40 * 1024;

ColDims dims_of(const ImgGeom& g, const ColBuffers& c) { return ColDims{g.nx, g.ny, g.nz, c.z0, c.half}; }

dim3 voxel_grid(const ImgGeom& g) { return dim3((g.nx + 31) / 32, g.ny, (g.nz + 31) / 32); }

// Threads of a block: up to `most`, as few as give the same number of rounds over
// the sinograms.
int block_of(const LorTable& t, int most = kColBlock) {
  const int groups = (t.n_sinos + 31) / 32, rounds = (groups + most / 32 - 1) / (most / 32);
  return (groups + rounds - 1) / rounds * 32;
}

int64_t lors_of(const LorTable& t, const SubsetSel& s) { return (int64_t)s.nk * t.n_r; }

}  // namespace

ColBuffers col_layout(const ImgGeom& g, const float* z_ends, int n_ends) {
  // Slices that a ray between these end points can enter, and the spare ones.
  float lo = z_ends[0], hi = z_ends[0];
  for (int i = 1; i < n_ends; i++) {
    lo = fminf(lo, z_ends[i]);
    hi = fmaxf(hi, z_ends[i]);
  }
  ColBuffers c;
  const double first = floor(((double)lo - g.offz) / g.dz) - 1 - kColSpare, end = floor(((double)hi - g.offz) / g.dz) + 2 + kColSpare;
  const double z0 = ceil(fmax((double)kColSpare, -first) / 2) * 2, slices = fmax((double)g.nz + kColSpare, end) + z0;
  const double floats = (double)(g.nx + 2 * kPad) * (g.ny + 2 * kPad) * (slices + 16);
  // Bounded in bytes and against the image (a long scanner around a short
  // image), in grid sizes (a layer more for the likelihood) and in the list's
  // shared memory.
  if (!(floats < (double)(1 << 30)) || floats > 4.0 * g.nx * g.ny * g.nz + (1 << 22) || g.ny > 65535 ||
      g.nz > 65534 * 32 || col_smem(g.nx, g.ny) > kColMaxSmem)
    return c;
  c.z0 = (int)z0;
  c.half = (((int)slices + 1) / 2 + 7) / 8 * 8;
  c.floats = ColDims{g.nx, g.ny, g.nz, c.z0, c.half}.floats();
  return c;
}

bool col_rays_fit(const ImgGeom& g, int n_rs) { return n_rs * col_smem(g.nx, g.ny) <= kColMaxSmem; }

template <typename CT>
static cudaError_t em_cols_rays(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s, const CT* counts,
                                int counts_packed, const float* add, int back, double* partials, cudaStream_t st) {
  if (lors_of(t, s) == 0) return cudaSuccess;
  k_em_cols_rays<CT><<<(unsigned)lors_of(t, s), block_of(t, kRaysBlock), t.n_rs * col_smem(g.nx, g.ny), st>>>(
      g, dims_of(g, c), t, s, counts, counts_packed, add, c.img, c.acc, back, partials);
  return cudaGetLastError();
}

cudaError_t launch_em_cols_rays(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s,
                                const void* counts, int counts_dtype, int counts_packed, const float* add, int back,
                                double* partials, cudaStream_t st) {
  switch (counts_dtype) {
    case APIRL_F32: return em_cols_rays(g, c, t, s, (const float*)counts, counts_packed, add, back, partials, st);
    case APIRL_U32: return em_cols_rays(g, c, t, s, (const uint32_t*)counts, counts_packed, add, back, partials, st);
    case APIRL_U16: return em_cols_rays(g, c, t, s, (const uint16_t*)counts, counts_packed, add, back, partials, st);
    default: return cudaErrorInvalidValue;
  }
}

size_t col_list_bytes(const ImgGeom& g) { return col_smem(g.nx, g.ny); }

cudaError_t launch_multi_cols(const MultiStep& m, cudaStream_t st) {
  if (m.total_lors == 0) return cudaSuccess;
  k_em_multi_cols<<<(unsigned)m.total_lors, kMultiColBlock, m.col_smem, st>>>(m.cols, m.n_cols,
                                                                             m.partials + m.total_chunks);
  return cudaGetLastError();
}

cudaError_t load_multi_cols() {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, k_em_multi_cols);
}

int64_t col_partials(const LorTable& t, SubsetSel s) { return lors_of(t, s); }

int64_t col_dots(const ImgGeom& g) {
  const dim3 v = voxel_grid(g);
  return (int64_t)v.x * v.y * v.z;
}

cudaError_t launch_col_copy(const ImgGeom& g, const ColBuffers& c, const float* x, float* img, cudaStream_t st,
                            const float* gimg, double* dots, unsigned* queue_n) {
  k_col_copy<<<voxel_grid(g), dim3(32, 8), 0, st>>>(dims_of(g, c), x, img, gimg, dots, queue_n);
  return cudaGetLastError();
}

cudaError_t launch_col_reduce(const ImgGeom& g, const ColBuffers& c, float* acc, int mode, float* x, float* bp,
                              const float* sens, const float* thr_ptr, float thr_value, int ge, cudaStream_t st,
                              const double* partials, int64_t n, const double* less, double* lik) {
  dim3 grid = voxel_grid(g);
  if (lik) grid.z++;
  k_col_reduce<<<grid, dim3(32, 8), 0, st>>>(dims_of(g, c), acc, mode, x, bp, sens, thr_ptr, thr_value, ge, partials, n,
                                             less, lik);
  return cudaGetLastError();
}

cudaError_t launch_project_cols(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s,
                                const float* img, float* out, cudaStream_t st) {
  if (lors_of(t, s) == 0) return cudaSuccess;
  k_project_cols<<<(unsigned)lors_of(t, s), block_of(t), col_smem(g.nx, g.ny), st>>>(g, dims_of(g, c), t, s, img, out);
  return cudaGetLastError();
}

cudaError_t launch_scatter_cols(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s,
                                const float* vin, const float* vest, float* acc, cudaStream_t st,
                                const ColQueue& queue) {
  const int64_t lors = lors_of(t, s);
  if (lors == 0) return cudaSuccess;
  // Looking costs 1.6 us where every LOR has values and many are walked, 2 us
  // of 25 in short calls.  Backprojections of 27,556 LORs of a 128 x 128 image,
  // us on the padded pair / without / with, bins with values 0.2 %, 1 %, 5 %,
  // 20 %, all: 16 sinograms 33, 43, 62, 78, 178 / 60, 66, 84, 97, 99 / 36, 42, 71,
  // 97, 101; 34 sinograms 42, 55, 99, 130, 318 / 82, 102, 141, 157, 184 / 39, 67,
  // 134, 158, 186; 146 sinograms 110, 148, 344, 478, 1296 / 126, 179, 278, 344,
  // 605 / 87, 175, 288, 355, 612.  More sinograms have values in most LORs.
  const bool look = lors > col_direct_lors(g) && t.n_sinos <= kColBlock;
  // The queue, for LORs with up to 8 values (the list serves one walk, whose
  // reductions cost more lane by lane), costs 6 us more: there it gave 50, 89 and
  // 79, 141 us at 5 %, 20 % of 16 and 34 sinograms.  It is for long calls, from
  // 1e7 LORs times voxels of a row and a column on: 89,401 LORs of 19 sinograms,
  // 230 x 230, 5 % and all: pair 250, 913, without 359, 581, with 173, 588.
  const bool queued = look && !vest && queue.bins && (double)lors * (g.nx + g.ny) >= 1e7 && lors * t.n_sinos <= INT_MAX;
  cudaError_t e;
  if (queued && (e = cudaMemsetAsync(queue.n + 1, 0, sizeof(unsigned), st)) != cudaSuccess) return e;
  auto kernel = look ? k_scatter_cols<true> : k_scatter_cols<false>;
  kernel<<<(unsigned)lors, block_of(t), col_smem(g.nx, g.ny), st>>>(g, dims_of(g, c), t, s, vin, vest, acc,
                                                                   queued ? kColDirectBack : 0, queue);
  if ((e = cudaGetLastError()) != cudaSuccess || !queued) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  k_scatter_cols_direct<<<(unsigned)(sms * kColDirectBlocks), kColDirectBlock, 0, st>>>(g, dims_of(g, c), t, s, vin, acc,
                                                                                      queue);
  return cudaGetLastError();
}

template <typename CT>
static cudaError_t em_cols(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s, const CT* counts,
                           int counts_packed, const float* add, int back, double* partials, int skip_zero,
                           const ColQueue& queue, cudaStream_t st) {
  const ColDims d = dims_of(g, c);
  const unsigned grid = (unsigned)lors_of(t, s);
  const size_t smem = col_smem(g.nx, g.ny);
  if (!skip_zero) {
    k_em_cols<CT><<<grid, block_of(t), smem, st>>>(g, d, t, s, counts, counts_packed, add, c.img, c.acc, back,
                                                   partials);
    return cudaGetLastError();
  }
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  // Up to two waves of blocks the idle warps cost nothing, and a second
  // kernel's latency would follow the first's (747 LORs of a 64 x 64 x 41 job,
  // most with few counts: 29 + 31 us, in one kernel 40 us).  Above, the small
  // blocks walk the few counts faster (5376 LORs of the 256 x 256 x 81 job at
  // 1 % bins with counts: the pass 500 -> 444 us; 3984 LORs of a 128 x 128 x
  // 41 job: 141 -> 128 us).
  // With so few sinograms that a block has few warps anyway (37 and 19 of a
  // 128 x 128 image: 388 and 358 us with the queue, 304 and 181 without) there
  // is nothing to defer to small blocks either.
  //
  // A list costs a block about 2600 warp instructions and the walk along it
  // 250 and 17 a step, whether one lane has a ray or 32; a lane's own walk 300
  // and some 30 a step for 32 rays together.  So the bins of LORs with up to 32
  // counts, or 64 where a block of eight warps would take them, are walked one
  // a lane; of up to 40 sinograms all are (34 of a 256 x 256 image, 70 % bins
  // with counts: 326 us all listed, 331 us in part, 250 us).  Us of the listed
  // pass on the padded pair / with every LOR listed / with this, bins with
  // counts 1 %, 20 %, 70 %: 128 x 128 image, 27,556 LORs of 146 sinograms 177,
  // 521, 1054 / 433, 567, 744 / 134, 516, 749; of 34 sinograms 122, 186, 318 /
  // 135, 294, 303 / 73, 164, 259; of 310 sinograms 231, 1001, 2091 / 447, 720,
  // 1294 / 204, 726, 1294.  Between the two kernels lies the walk of the last
  // rays, 8 us: below 8000 LORs, or 1.5e6 LORs times voxels of a row and a
  // column, a pass is too short for it (6889 LORs of 310 sinograms, 64 x 64: 95,
  // 144, 225 us without, 61, 152, 233 with; on the padded pair 103, 188, 336;
  // 6240 of 34 sinograms, 320 x 320: 223, 294, 297 without, 199, 194, 229 with,
  // 250, 268, 317).
  const int64_t lors = lors_of(t, s), line = col_direct_lors(g);
  const bool queued = lors > line && t.n_sinos <= kColWindow && lors * t.n_sinos <= INT_MAX;
  const int direct = queued ? col_direct(t.n_sinos) : 0;
  const int few = lors > 2 * sms * kColBlocks && lors <= line && t.n_sinos > 4 * kColFew &&
                          t.n_sinos <= kColWindow ? kColFew : 0;
  k_em_cols_listed<CT><<<grid, block_of(t), smem, st>>>(g, d, t, s, counts, counts_packed, add, c.img, c.acc, back,
                                                       partials, skip_zero, few, direct, queue);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (direct) {
    k_em_cols_direct<CT><<<(unsigned)(sms * kColDirectBlocks), kColDirectBlock, 0, st>>>(
        g, d, t, s, counts, counts_packed, add, c.img, c.acc, back, partials, skip_zero, queue);
    return cudaGetLastError();
  }
  if (!few) return cudaSuccess;
  const unsigned resident = (unsigned)(sms * kColFewBlocks);
  k_em_cols_few<CT><<<grid < resident ? grid : resident, kColFewBlock, smem, st>>>(g, d, t, s, counts, counts_packed, add, c.img,
                                                                        c.acc, back, partials, skip_zero, queue);
  return cudaGetLastError();
}

cudaError_t launch_em_cols(const ImgGeom& g, const ColBuffers& c, const LorTable& t, SubsetSel s, const void* counts,
                           int counts_dtype, int counts_packed, const float* add, int back, double* partials,
                           int skip_zero, const ColQueue& queue, cudaStream_t st) {
  if (lors_of(t, s) == 0) return cudaSuccess;
  switch (counts_dtype) {
    case APIRL_F32:
      return em_cols(g, c, t, s, (const float*)counts, counts_packed, add, back, partials, skip_zero, queue, st);
    case APIRL_U32:
      return em_cols(g, c, t, s, (const uint32_t*)counts, counts_packed, add, back, partials, skip_zero, queue, st);
    case APIRL_U16:
      return em_cols(g, c, t, s, (const uint16_t*)counts, counts_packed, add, back, partials, skip_zero, queue, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace apirl
