// TOF projections by basic bin with the timing bins over the lanes (lines of at most 16 axial positions).
//
// With TOF only the z shift is left of the symmetries, so a basic bin has one line of a few axial positions (8 to 1 on an
// 8-ring scanner) and dozens of timing bins, and every row element a weight per timing bin (ProjParams::tof_w, tof_ws
// floats an element).  A warp takes a basic bin; lane (kg, a) holds axial position a and the kl timing bins from kg kl on,
// kg = lane / nax: 32 / nax groups share an axial position's voxel.  (With lanes on (line, axial position) only, as in the
// TOF-grouped kernels of project.cu, 1 to 8 lanes work; they remain for longer lines and for more timing bins than fit.)
//
// 16 row elements at a time: their weights come as one contiguous block by 16-byte asynchronous copies, two blocks in
// shared memory; their voxels are gathered by the lanes with kg over the elements, coalesced along z.
//   forward: every lane adds voxel x weight for its timing bins: kl multiply-adds on kl / 4 16-byte reads per element;
//   back:    every lane sums weight x datum over its timing bins, the groups' sums go through shared memory and one
//            reduction per (element, axial position) adds them to the image, in a fixed order.
// Forward sums add their products in row order (bit-identical to the grouped kernels); the back projection takes the timing
// bins in the grouped kernels' passes (tof_group_size), one reduction each, so that a voxel's float sum has the same terms.
// (All timing bins at once: 2.78 ms instead of 3.65 for the pair below at the time, and a smaller error against the
// fixed-point sum, 8e-7 against 1.3e-6; but the result moves by as much as the present error.)
//
// 33 timing bins, 8 rings x 288 detectors, all 19.5 M TOF bins: forward 3.59 -> 0.92 ms, back 3.19 -> 1.62 ms.  The weights
// are read once a projection: 2.9 GB, 0.45 ms at the copy bandwidth.  Both are bound by shared memory (77 and 95 % of the
// l1tex data path): the weights' 16-byte reads, the staged voxels and the groups' sums.
#include <cstdint>

#include "epilogue.cuh"
#include "internal.hpp"

namespace b200 {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kTlWarps = 4;
constexpr int kTlBatch = 16;   // row elements at a time
constexpr int kTlMaxKl = 24;   // timing bins of a lane
constexpr int kTlPad = 32;     // floats past a block that the last group of timing bins may read
constexpr int kTlMaxWs = 96;

// timing bins of a lane for lines of nax axial positions: all K over 32 / nax groups, in 16-byte pieces
__host__ __device__ inline int tl_kl(int K, int nax) {
  const int groups = 32 / nax;
  return ((K + groups - 1) / groups + 3) & ~3;
}
__host__ __device__ inline int tl_block(int ws) { return kTlBatch * ws + kTlPad; }  // floats
// two weight blocks, the elements (image index without z, z), voxels or partial sums
__host__ __device__ inline int tl_warp_smem(int ws) { return 8 * tl_block(ws) + 8 * kTlBatch + 4 * 32 * kTlBatch; }

// (offsets from one base, so that every access is known to be to shared memory)
struct TlStage {
  unsigned char* base;
  int block;  // floats
  __device__ __forceinline__ TlStage(unsigned char* smem, int ws) : base(smem), block(tl_block(ws)) {}
  __device__ __forceinline__ float* w(int b) const { return reinterpret_cast<float*>(base) + (b & 1) * block; }
  __device__ __forceinline__ int2* xs() const { return reinterpret_cast<int2*>(base + 8 * block); }
  __device__ __forceinline__ float* xv() const { return reinterpret_cast<float*>(base + 8 * block + 8 * kTlBatch); }
};

__device__ __forceinline__ void tl_fetch(float* dst, const float* src, int cnt, int ws, int lane) {
  const int pieces = cnt * ws / 4;
  for (int i = lane; i < pieces; i += 32) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + 4 * i));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + 4 * i) : "memory");
  }
}
// `words` 16-byte pieces from every element's weights (element stride ws) to a block of that stride
__device__ __forceinline__ void tl_fetch_part(float* dst, const float* src, int cnt, int ws, int words, int lane) {
  int r = lane / words, c = lane - r * words;
  const int dr = 32 / words, dc = 32 - dr * words;
  while (r < cnt) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + 4 * (r * words + c)));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + r * ws + 4 * c) : "memory");
    r += dr;
    c += dc;
    if (c >= words) {
      c -= words;
      ++r;
    }
  }
}
__device__ __forceinline__ void tl_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tl_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// a line of the basic bin, the same in every lane; false: outside the projection data
struct TlLine {
  int64_t out_base;
  int nax, npa, seg, view, flags, q;
};
__device__ __forceinline__ bool tl_line(const ProjParams& p, const ProjBinDev& pb, int l, TlLine& t) {
  const LineDev L = p.lines[pb.first_line + l];
  const int tang = static_cast<int>(L.tang_sign) * pb.tang;
  if (tang < p.min_tang || tang > p.max_tang) return false;
  const SegDev sd = p.segs[L.seg + p.S];
  t.nax = sd.nax;
  t.npa = sd.npa;
  t.seg = L.seg;
  t.view = L.view;
  t.flags = L.flags;
  t.q = L.q;
  t.out_base = sd.dev_offset + (static_cast<int64_t>(L.view) * p.num_tang + (tang - p.min_tang)) * sd.nax;
  return true;
}
// (image index without z, z - min_z at axial position 0) of an element under the line's symmetry operation
__device__ __forceinline__ int2 tl_transform(const ProjParams& p, const RowElem& e, const TlLine& t) {
  int z, y, x;
  unpack_zyx(e.zyx, z, y, x);
  const int xt = ((t.flags & 1) ? y : x) * ((t.flags & 2) ? -1 : 1);
  const int yt = ((t.flags & 1) ? x : y) * ((t.flags & 4) ? -1 : 1);
  const int zt = ((t.flags & 8) ? t.q - z : z) - p.min_z;
  return make_int2(((yt - p.min_y) * p.nx + (xt - p.min_x)) * p.nz, zt);
}

__device__ __forceinline__ void tl_store(const ProjParams& p, const TlLine& t, int k, int64_t idx, int a, float v,
                                         float* __restrict__ out, const FwdEpilogue& ep, double& ll, unsigned& nc) {
  switch (ep.mode) {
    case kEpiNone: forward_store<kEpiNone>(p, t.seg, t.view, k, t.nax, idx, a, v, out, ep, ll, nc); break;
    case kEpiRatio: forward_store<kEpiRatio>(p, t.seg, t.view, k, t.nax, idx, a, v, out, ep, ll, nc); break;
    case kEpiGradient: forward_store<kEpiGradient>(p, t.seg, t.view, k, t.nax, idx, a, v, out, ep, ll, nc); break;
    default: forward_store<kEpiLoglik>(p, t.seg, t.view, k, t.nax, idx, a, v, out, ep, ll, nc); break;
  }
}

template <int KL>
__device__ __forceinline__ void tl_forward(const ProjParams& p, const ProjBinDev& pb, const TlLine& t, const TlStage& S,
                                           const float* __restrict__ img, float* __restrict__ out, const FwdEpilogue& ep,
                                           double& ll, unsigned& nc, int lane) {
  const int K = p.num_tof, ws = p.tof_ws, nax = t.nax, groups = 32 / nax;
  const RowElem* row = p.tof_basic_rows + pb.row_offset;
  const float* wrow = p.tof_w + pb.row_offset * ws;
  const int kg = lane / nax, a = lane - kg * nax;
  const bool gather = kg < groups, on = gather && kg * KL < K;
  const int koff = on ? kg * KL : 0;
  const int n = pb.row_len;
  float acc[KL];
#pragma unroll
  for (int k = 0; k < KL; ++k) acc[k] = 0.f;
  __syncwarp();
  tl_fetch(S.w(0), wrow, min(kTlBatch, n), ws, lane);
  tl_commit();
  RowElem e{};
  if (lane < min(kTlBatch, n)) e = row[lane];
  for (int e0 = 0, b = 0; e0 < n; e0 += kTlBatch, ++b) {
    const int cnt = min(kTlBatch, n - e0), next = min(kTlBatch, n - e0 - kTlBatch);
    if (next > 0) tl_fetch(S.w(b + 1), wrow + static_cast<int64_t>(e0 + kTlBatch) * ws, next, ws, lane);
    tl_commit();
    if (lane < cnt) S.xs()[lane] = tl_transform(p, e, t);
    if (lane < next) e = row[e0 + kTlBatch + lane];
    __syncwarp();
    if (gather)
      for (int i = kg; i < cnt; i += groups) {
        const int2 X = S.xs()[i];
        const int zz = X.y + a * t.npa;
        S.xv()[i * nax + a] = (zz >= 0 && zz < p.nz) ? __ldg(img + X.x + zz) : 0.f;
      }
    tl_wait<1>();
    __syncwarp();
    const float* w = S.w(b) + koff;
    const float* xv = S.xv() + a;
#pragma unroll 2
    for (int i = 0; i < cnt; ++i) {
      const float x = xv[i * nax];
      const float4* wq = reinterpret_cast<const float4*>(w + i * ws);
#pragma unroll
      for (int q = 0; q < KL / 4; ++q) {
        const float4 v = wq[q];
        acc[4 * q] += x * v.x;
        acc[4 * q + 1] += x * v.y;
        acc[4 * q + 2] += x * v.z;
        acc[4 * q + 3] += x * v.w;
      }
    }
    __syncwarp();
  }
  tl_wait<0>();
  if (on)
#pragma unroll
    for (int k = 0; k < KL; ++k)
      if (koff + k < K)
        tl_store(p, t, koff + k, t.out_base + static_cast<int64_t>(koff + k) * p.tof_stride + a, a, acc[k], out, ep, ll, nc);
}

// the contributions to a voxel of one (line, axial position), summed in float in a fixed order, added to the image, or
// rounded once to the fixed-point grid (a power-of-two scale: exact) and added as a 64-bit integer
struct TlFloatSink {
  float* img;
  __device__ __forceinline__ void add(int64_t i, float v) const {
    if (v != 0.f) atomicAdd(img + i, v);
  }
};
struct TlFixedSink {
  unsigned long long* acc;
  float scale;
  __device__ __forceinline__ void add(int64_t i, float v) const {
    if (v != 0.f) atomicAdd(acc + i, static_cast<unsigned long long>(__float2ll_rn(v * scale)));
  }
};

template <int KL, typename Sink>
__device__ __forceinline__ void tl_back(const ProjParams& p, const ProjBinDev& pb, const TlLine& t, const TlStage& S,
                                        const float* __restrict__ pd, const Sink& sink, int zero_ends, int k0, int K,
                                        int lane) {
  const int ws = p.tof_ws, nax = t.nax, groups = 32 / nax, words = (K + 3) / 4;
  const RowElem* row = p.tof_basic_rows + pb.row_offset;
  const float* wrow = p.tof_w + pb.row_offset * ws + k0;
  const int kg = lane / nax, a = lane - kg * nax;
  const bool scatter = kg < groups, on = scatter && kg * KL < K;
  const int koff = on ? kg * KL : 0, used = (K + KL - 1) / KL;
  const bool zend = zero_ends && t.seg == 0 && (a == 0 || a == nax - 1);
  const int n = pb.row_len;
  float d[KL];
  bool any = false;
#pragma unroll
  for (int k = 0; k < KL; ++k) {
    d[k] = 0.f;
    if (on && !zend && koff + k < K)
      d[k] = pd ? __ldg(pd + t.out_base + static_cast<int64_t>(k0 + koff + k) * p.tof_stride + a) : 1.f;
    any |= d[k] != 0.f;
  }
  if (!__any_sync(kFull, any)) return;
  __syncwarp();
  tl_fetch_part(S.w(0), wrow, min(kTlBatch, n), ws, words, lane);
  tl_commit();
  RowElem e{};
  if (lane < min(kTlBatch, n)) e = row[lane];
  for (int e0 = 0, b = 0; e0 < n; e0 += kTlBatch, ++b) {
    const int cnt = min(kTlBatch, n - e0), next = min(kTlBatch, n - e0 - kTlBatch);
    if (next > 0)
      tl_fetch_part(S.w(b + 1), wrow + static_cast<int64_t>(e0 + kTlBatch) * ws, next, ws, words, lane);
    tl_commit();
    if (lane < cnt) S.xs()[lane] = tl_transform(p, e, t);
    if (lane < next) e = row[e0 + kTlBatch + lane];
    tl_wait<1>();
    __syncwarp();
    const float* w = S.w(b) + koff;
#pragma unroll 2
    for (int i = 0; i < cnt; ++i) {
      const float4* wq = reinterpret_cast<const float4*>(w + 4 * i * words);
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < KL / 4; ++q) {
        const float4 v = wq[q];
        sum += v.x * d[4 * q];
        sum += v.y * d[4 * q + 1];
        sum += v.z * d[4 * q + 2];
        sum += v.w * d[4 * q + 3];
      }
      S.xv()[i * 32 + lane] = sum;
    }
    __syncwarp();
    if (scatter)
      for (int i = kg; i < cnt; i += groups) {
        const int2 X = S.xs()[i];
        const int zz = X.y + a * t.npa;
        if (zz < 0 || zz >= p.nz) continue;
        float v = S.xv()[i * 32 + a];
        for (int g = 1; g < used; ++g) v += S.xv()[i * 32 + g * nax + a];
        sink.add(X.x + zz, v);
      }
    __syncwarp();
  }
  tl_wait<0>();
}

#define TL_SWITCH(kl, CALL)                           \
  switch (kl) {                                       \
    case 4: { constexpr int KL = 4; CALL; break; }    \
    case 8: { constexpr int KL = 8; CALL; break; }    \
    case 12: { constexpr int KL = 12; CALL; break; }  \
    case 16: { constexpr int KL = 16; CALL; break; }  \
    case 20: { constexpr int KL = 20; CALL; break; }  \
    default: { constexpr int KL = 24; CALL; break; }  \
  }

__device__ __forceinline__ void tl_forward_bin(const ProjParams& p, const ProjBinDev& pb, const TlStage& S,
                                               const float* __restrict__ img, float* __restrict__ out, const FwdEpilogue& ep,
                                               double& ll, unsigned& nc, int lane) {
  for (int l = 0; l < pb.num_lines; ++l) {
    TlLine t;
    if (!tl_line(p, pb, l, t)) continue;
    TL_SWITCH(tl_kl(p.num_tof, t.nax), tl_forward<KL>(p, pb, t, S, img, out, ep, ll, nc, lane));
  }
}
template <typename Sink>
__device__ __forceinline__ void tl_back_bin(const ProjParams& p, const ProjBinDev& pb, const TlStage& S,
                                            const float* __restrict__ pd, const Sink& sink, int zero_ends, int lane) {
  const int pass = tof_group_size(p.num_tof);
  for (int l = 0; l < pb.num_lines; ++l) {
    TlLine t;
    if (!tl_line(p, pb, l, t)) continue;
    // the timing bins in as many passes as the TOF-grouped kernels take, with a reduction each
    for (int k0 = 0; k0 < p.num_tof; k0 += pass) {
      const int K = min(pass, p.num_tof - k0);
      TL_SWITCH(tl_kl(K, t.nax), (tl_back<KL, Sink>(p, pb, t, S, pd, sink, zero_ends, k0, K, lane)));
    }
  }
}
// zeros where the last group of timing bins reads past an element's weights (its data there are 0)
__device__ __forceinline__ void tl_clear(const TlStage& S, int ws, int lane) {
  for (int i = lane; i < 2 * tl_block(ws); i += 32) S.w(0)[i] = 0.f;
  __syncwarp();
}

__global__ void __launch_bounds__(kTlWarps * 32, 7)
    forward_tof_lanes_kernel(ProjParams p, const int* __restrict__ items, int nitems, const float* __restrict__ img,
                             float* __restrict__ out, FwdEpilogue ep) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int i = blockIdx.x * kTlWarps + warp;
  if (i >= nitems) return;  // whole warps: no block-wide synchronisation below
  const TlStage S(smem + warp * tl_warp_smem(p.tof_ws), p.tof_ws);
  double ll = 0.0;
  unsigned nc = 0;
  tl_forward_bin(p, p.tof_basic[items[i]], S, img, out, ep, ll, nc, lane);
  if (ep.mode == kEpiRatio || ep.mode == kEpiGradient) {
    for (int o = 16; o > 0; o >>= 1) nc += __shfl_xor_sync(kFull, nc, o);
    if (lane == 0 && nc && ep.cancelled) atomicAdd(ep.cancelled, nc);
  }
  if (ep.mode == kEpiLoglik) {
    // one partial per basic bin (all its timing bins), reduced in a fixed order by the caller
    for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(kFull, ll, o);
    if (lane == 0) ep.partials[i] = ll;
  }
}

template <bool FIXED>
__global__ void __launch_bounds__(kTlWarps * 32, 7)
    back_tof_lanes_kernel(ProjParams p, const int* __restrict__ items, int nitems, const float* __restrict__ pd,
                          float* __restrict__ img, unsigned long long* __restrict__ acc, const double* __restrict__ scale,
                          int zero_ends) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int i = blockIdx.x * kTlWarps + warp;
  if (i >= nitems) return;
  const TlStage S(smem + warp * tl_warp_smem(p.tof_ws), p.tof_ws);
  tl_clear(S, p.tof_ws, lane);
  if constexpr (FIXED)
    tl_back_bin(p, p.tof_basic[items[i]], S, pd, TlFixedSink{acc, static_cast<float>(*scale)}, zero_ends, lane);
  else
    tl_back_bin(p, p.tof_basic[items[i]], S, pd, TlFloatSink{img}, zero_ends, lane);
}

// batched reconstructions: persistent warps over (frame, basic bin) items
template <bool FORWARD>
__global__ void __launch_bounds__(kTlWarps * 32, 7)
    batch_tof_lanes_kernel(const ProjParams* __restrict__ geoms, const BatchFrameDev* __restrict__ frames,
                           const BatchItem* __restrict__ items, int nitems, unsigned* counter, int ws) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const TlStage S(smem + warp * tl_warp_smem(ws), ws);
  tl_clear(S, ws, lane);
  for (;;) {
    __syncwarp();
    int k = 0;
    if (lane == 0) k = static_cast<int>(atomicAdd(counter, 1u));
    k = __shfl_sync(kFull, k, 0);
    if (k >= nitems) return;
    const BatchItem wi = items[k];
    const BatchFrameDev& f = frames[wi.frame];
    const ProjParams& p = geoms[f.geom];
    const ProjBinDev pb = p.tof_basic[wi.bin];
    if constexpr (FORWARD) {
      double ll = 0.0;
      unsigned nc = 0;
      tl_forward_bin(p, pb, S, f.x, f.ratio, f.ep, ll, nc, lane);
      for (int o = 16; o > 0; o >>= 1) nc += __shfl_xor_sync(kFull, nc, o);
      if (lane == 0 && nc && f.ep.cancelled) atomicAdd(f.ep.cancelled, nc);
    } else {
      tl_back_bin(p, pb, S, f.ratio, TlFloatSink{f.u}, 0, lane);
    }
  }
}

cudaError_t tl_prepare(const void* fn, int smem) {
  return smem > 48 * 1024 ? cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) : cudaSuccess;
}

}  // namespace

int tof_weight_stride(int num_tof) { return (num_tof + 3) & ~3; }

bool tof_lanes(const ProjParams& p) {
  return p.tof_w && p.max_nax <= 16 && p.tof_ws <= kTlMaxWs && tl_kl(p.num_tof, p.max_nax) <= kTlMaxKl;
}

cudaError_t launch_forward_tof_lanes(const ProjParams& p, const int* items, int nitems, const float* image, float* projdata,
                                     cudaStream_t st, const FwdEpilogue& ep) {
  const int sm = kTlWarps * tl_warp_smem(p.tof_ws);
  const cudaError_t e = tl_prepare(reinterpret_cast<const void*>(forward_tof_lanes_kernel), sm);
  if (e != cudaSuccess) return e;
  forward_tof_lanes_kernel<<<(nitems + kTlWarps - 1) / kTlWarps, kTlWarps * 32, sm, st>>>(p, items, nitems, image, projdata,
                                                                                         ep);
  return cudaGetLastError();
}

cudaError_t launch_back_tof_lanes(const ProjParams& p, const int* items, int nitems, const float* projdata, float* image,
                                  unsigned long long* acc, const double* scale, cudaStream_t st, int zero_ends) {
  const int sm = kTlWarps * tl_warp_smem(p.tof_ws), grid = (nitems + kTlWarps - 1) / kTlWarps;
  auto kernel = acc ? back_tof_lanes_kernel<true> : back_tof_lanes_kernel<false>;
  const cudaError_t e = tl_prepare(reinterpret_cast<const void*>(kernel), sm);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kTlWarps * 32, sm, st>>>(p, items, nitems, projdata, image, acc, scale, zero_ends);
  return cudaGetLastError();
}

cudaError_t launch_batch_tof_lanes(bool forward, const ProjParams* geoms, int num_tof, const BatchFrameDev* frames,
                                   const BatchItem* items, int nitems, unsigned* counter, int grid, cudaStream_t st) {
  const int ws = tof_weight_stride(num_tof), sm = kTlWarps * tl_warp_smem(ws);
  auto kernel = forward ? batch_tof_lanes_kernel<true> : batch_tof_lanes_kernel<false>;
  const cudaError_t e = tl_prepare(reinterpret_cast<const void*>(kernel), sm);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kTlWarps * 32, sm, st>>>(geoms, frames, items, nitems, counter, ws);
  return cudaGetLastError();
}

int batch_tof_lanes_max_ctas_per_sm(int num_tof, bool forward) {
  const int sm = kTlWarps * tl_warp_smem(tof_weight_stride(num_tof));
  auto kernel = forward ? batch_tof_lanes_kernel<true> : batch_tof_lanes_kernel<false>;
  if (tl_prepare(reinterpret_cast<const void*>(kernel), sm) != cudaSuccess) return 0;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kTlWarps * 32, sm) != cudaSuccess) return 0;
  return n;
}

}  // namespace b200
