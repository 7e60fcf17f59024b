// Tables and launchers of the z-frame projections (zframe.cu).
//
// A path item is a transaxial path (basic view, tangential position) under one transaxial symmetry operation, with the
// lines of all its basic segments in both z orientations.  Its rows are cut into chains: along the path a chain has at
// most one element per column and plane, and its plane never decreases, so that a register file which holds a line's
// sums (or data) in image planes has to be moved by one plane only where the chain crosses one (an event).
#pragma once

#include "internal.hpp"

namespace b200 {

constexpr int kZChains = 6;      // chains of an item (one warp); more go to further items of the path
constexpr int kZBatch = 8;       // records staged at a time
constexpr int kZWarps = 4;       // items (warps) per CTA

// One column of the path for every chain of the group: w1 before the column's events, w2 after them.
struct __align__(16) ZRec {
  float w1[2 * kZChains];  // each twice: the packed multiply-adds take pairs
  float w2[kZChains];
  int32_t leave[kZChains];  // forward: the axial positions of the up (low half) and down line whose sums leave the planes
                            // at the event, -1: none
  uint32_t xy;   // (x + 1024) | (y + 1024) << 11
  uint32_t op;   // bits 0..5: chain m moves up one plane (its event); 6..11: that event needs the edge code (a position
                 // leaves or enters the planes, or w2 is 0);
                 // bit 12: some w1 is 0 (that product is left out: 0 x inf would make a NaN)
  uint32_t pad[2];
};
static_assert(sizeof(ZRec) == 112, "a record is seven 16-byte pieces");
constexpr uint32_t kZGuard = 1u << 12;
constexpr int kZTurn = 8;

// slot 2 m: the line of chain m whose planes grow with the basic row's, slot 2 m + 1: the z-reflected one
struct ZItemDev {
  int rec0, nrec;       // the path group's records (nrec a multiple of 4)
  int flags;            // T: bit 0 swap x/y, bit 1 negate x, bit 2 negate y; from bit kZTurn on: the item's turn (ZParams::copies)
  int path;             // the path group's planes (ZParams::sixteenths)
  int2 slot[2 * kZChains];         // (index into lines[], basic bin) or (-1, -1)
  int16_t boff[2 * kZChains];      // back projection: the slot's datum 0 in the item's shared buffer (max_back floats)
  int8_t owner[4 * ((2 * kZChains + 3) / 4)];  // the slot whose sums this one shares (two chains of one line)
};

// stored plane (z + 512) of each chain of a path group before each sixteenth of its batches, where a warp may take over, and
// at the end
constexpr int kZSixteenths = 16;
struct ZPlanes {
  int16_t z[kZSixteenths + 1][8];
};

struct ZParams {
  const ZRec* recs;
  const ZPlanes* sixteenths;
  const ZItemDev* items;
  int nm;         // chains per item the kernels are compiled for: 4 or 6
  int planes;     // planes per lane: 1, 2 or 4 (32 x planes >= nz)
  int mean_rec;   // mean records of a path's groups
  // images that the back projection's sums are spread over (1, 2 or 4), added at the end.  A path's chain groups add to a voxel
  // one by one, where the column-staged kernels added their sum, so a voxel's float sum has as many times the terms and sqrt
  // of that times the rounding error.  Spread over c images it has 1 / c of it: 2 images for up to 3 groups, 4 beyond.
  int copies;
  int max_out;    // most projection values of one item
  int max_back;   // longest shared buffer of an item's data with the zeros around them
};

// How a call's items are walked: the forward projection sums an item's path in `segs` segments, taken by `parts` warps, and
// the back projection's warps take a part each.  The results depend on segs (and on parts = 1 or more), not on how many
// warps take the segments.
struct ZSplit {
  int segs, parts;
  int fold;  // batches whose products are summed by themselves
};
constexpr int kZManyWarps = kZSixteenths;  // most warps of an item
// value buffers of a forward warp: one, or one a segment where the segments' sums are added by several warps
__host__ __device__ inline int z_buffers(ZSplit sp) { return sp.parts > 1 ? sp.segs / sp.parts : 1; }
// the split as the batched kernels take it, whose CTAs have kZWarps warps: the same segments, so the same sums
inline ZSplit z_batch_split(ZSplit sp) {
  sp.parts = sp.parts < kZWarps ? sp.parts : kZWarps;
  return sp;
}
// shared memory of a forward warp, and the warps of a projection that the GPU runs at a time
int z_forward_smem(const ZParams& z, int buffers);
int z_resident_warps(const ZParams& z, bool forward);

// floats of an image of columns `stride` apart, in whole 16-byte pieces: how far the images that take the items in turn are apart
__host__ __device__ inline int64_t z_image_floats(int64_t ncols, int stride) { return (ncols * stride + 3) & ~int64_t(3); }

// column stride (floats) of the padded images the kernels use when planes > 1
inline int z_stride(const ZParams& z) { return 32 * z.planes; }

// image [col][nz] -> padded [col][stride] (planes past nz are zeros), `batch` images at the given strides
cudaError_t launch_pad_image(const float* in, int64_t in_stride, float* out, int64_t out_stride, int64_t ncols, int nz,
                             int stride, int batch, cudaStream_t st);
// image = the sum of `copies` images of columns `stride` apart (nz, or padded) that stand behind one another
cudaError_t launch_collect_images(const float* in, int64_t in_stride, int copies, float* out, int64_t out_stride,
                                  int64_t ncols, int nz, int stride, int batch, cudaStream_t st);

// padded != 0: image has column stride z_stride(z) (16-byte aligned), else nz; the forward projection takes padded images
// with sp.parts = 1 only
cudaError_t launch_forward_z(const ProjParams& p, const ZParams& z, const int* list, int n, ZSplit sp, const float* image,
                             int64_t img_stride, int padded, float* out, int64_t out_stride, int batch, cudaStream_t st,
                             const FwdEpilogue* ep);
// copies: images behind one another that take the items in turn (1: the image itself)
cudaError_t launch_back_z(const ProjParams& p, const ZParams& z, const int* list, int n, int parts, const float* pd,
                          int64_t pd_stride, float* image, int64_t img_stride, int copies, int padded, int batch,
                          cudaStream_t st, int zero_ends);
cudaError_t launch_back_z_fixed(const ProjParams& p, const ZParams& z, const int* list, int n, int parts, const float* pd,
                                unsigned long long* acc, const double* scale, cudaStream_t st, int zero_ends);

// batched reconstructions of frames whose geometries share a kernel variant (z: one of them): persistent CTAs over units
// of kZWarps (frame, item) work items; smem: the largest z_batch_smem of the frames' geometries
inline bool z_same_variant(const ZParams& a, const ZParams& b) {
  return a.nm == b.nm && a.planes == b.planes;
}
// BatchItem::frame with the split of the frame's items: the frame in the low 20 bits, log2 of segs, parts, fold above it
constexpr int kZFrameBits = 20;
__host__ __device__ inline int z_frame_of(int f) { return f & ((1 << kZFrameBits) - 1); }
__host__ __device__ inline ZSplit z_split_of(int f) {
  return ZSplit{1 << (f >> 20 & 7), 1 << (f >> 23 & 7), 1 << (f >> 26 & 7)};
}
inline int z_frame_split(int frame, ZSplit sp) {
  auto lg = [](int v) {
    int k = 0;
    while (1 << k < v) ++k;
    return k;
  };
  return frame | lg(sp.segs) << 20 | lg(sp.parts) << 23 | lg(sp.fold) << 26;
}
int z_batch_smem(const ZParams& z, bool forward, int buffers);
int z_batch_max_ctas_per_sm(const ZParams& z, bool forward, int smem);
// shared: the units hold items that warps share (forward: a kernel of its own)
cudaError_t launch_z_batch(const ZParams& z, bool forward, bool shared, const ProjParams* geoms, const ZParams* zgeoms,
                           const BatchFrameDev* frames, const BatchItem* items, int nunits, unsigned* counter, int smem,
                           int grid, cudaStream_t st);

}  // namespace b200
