// z-frame projections: a path item's lines held in image planes.
//
// A warp owns a path item (zframe.hpp).  Its lanes hold the planes of a voxel column (32, 64 or 128 planes, 1, 2 or 4 a
// lane) and, for every chain of the item, sums or data in the same planes: the axial position a of a line sees plane
// zt + npa a, zt the plane of axial position 0 in the current column.  Along the path zt stays for many columns (a ray of
// the clinical scanner crosses 0 to 120 planes in 200 to 500 columns), so a column costs one multiply-add per plane and
// chain straight from registers, shared by the chain's two lines (the z orientations, which have the same weights).
// Where a chain crosses a plane (an event) its lines move by one plane against the image, one up and one down.  The
// column-staged kernels (paths.cu) read every (element, line, plane) from shared memory instead: 4-byte reads for every
// multiply-add, which bounds them.
//
//   forward: G_m += w c for chain m; at an event both lines' sums U_m, D_m take G_m up while they move (one shuffle and
//            register renaming), and G_m starts again at w2 c;
//   back:    E_m = the two lines' data of chain m, from shared memory; u = sum_m w E_m is added to the image column.
//
// Clinical scanner (72.6 M lines, 344 x 344 x 127 image), all lines: forward 9.20 -> 4.53 ms, back 10.07 -> 3.64
// ms, deterministic back of one of 7 subsets 1.67 -> 1.02 ms.  Both are bound by latency and issue: 87 (forward) and 90
// instructions a column, of which the 12 packed multiply-adds (6 chains, 4 planes a lane) cannot be done without; 48 and 53 %
// of the issue slots, the l1tex data pipe below half and L2 below a fifth of their peaks, 16 and 20 warps per SM (the
// registers and the data in shared memory).  Tried: two warps per forward item
// with three chains each (80 registers, 24 warps: 66 % of the slots, but nearly twice the instructions, 6.3 ms); more
// registers per thread (12 warps: 6.0 ms); data in registers in the back projection too, moved at the events (4.8 ms).
#include <cstddef>
#include <cstdint>

#include "epilogue.cuh"
#include "zframe.hpp"

namespace b200 {

namespace {

constexpr unsigned kFull = 0xffffffffu;

using u64 = unsigned long long;
__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// two float multiply-adds in one instruction, each rounded as fmaf
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// a lane's P planes: pairs for the packed instructions
template <int P>
struct Planes {
  u64 h[P / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < P / 2; ++i) h[i] = 0;
  }
  __device__ __forceinline__ void get(float f[P]) const {
#pragma unroll
    for (int i = 0; i < P / 2; ++i) unpack2(h[i], f[2 * i], f[2 * i + 1]);
  }
  __device__ __forceinline__ void set(const float f[P]) {
#pragma unroll
    for (int i = 0; i < P / 2; ++i) h[i] = pack2(f[2 * i], f[2 * i + 1]);
  }
  __device__ __forceinline__ void fma(u64 ww, const Planes& c) {
#pragma unroll
    for (int i = 0; i < P / 2; ++i) h[i] = fma2(ww, c.h[i], h[i]);
  }
  __device__ __forceinline__ void mul(u64 ww, const Planes& c) {
#pragma unroll
    for (int i = 0; i < P / 2; ++i) h[i] = mul2(ww, c.h[i]);
  }
};
template <>
struct Planes<1> {
  float f0;
  __device__ __forceinline__ void zero() { f0 = 0.f; }
  __device__ __forceinline__ void get(float f[1]) const { f[0] = f0; }
  __device__ __forceinline__ void set(const float f[1]) { f0 = f[0]; }
  __device__ __forceinline__ void fma(u64 ww, const Planes& c) { f0 = fmaf(__uint_as_float(static_cast<unsigned>(ww)), c.f0, f0); }
  __device__ __forceinline__ void mul(u64 ww, const Planes& c) { f0 = __uint_as_float(static_cast<unsigned>(ww)) * c.f0; }
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// planes per axial position npa and ceil(2^15 / npa): d / npa = d * reciprocal >> 15 for d < 2^15 / npa
__device__ __forceinline__ int npa_code(int npa) { return npa | ((32768 + npa - 1) / npa) << 16; }
// axial position of plane offset d = z - zt, or -1
__device__ __forceinline__ int axial_at(int d, int code, int nax) {
  const int a = (d * static_cast<int>(static_cast<unsigned>(code) >> 16)) >> 15;
  return d >= 0 && a < nax && a * (code & 0xffff) == d ? a : -1;
}

// a slot's line (shared memory)
struct __align__(16) ZSlot {
  int zadd, npa, nax, off;  // npa: planes per axial position | reciprocal << 16; off: the values in the warp's buffer
  int64_t out_base;
  int zsign, seg, view, owner;
  uint32_t addr;            // shared address of the values (0: no line)
};

// the slots' lines, one lane each; `buf` offsets of the owners' values (a slot that shares takes its owner's)
__device__ __forceinline__ void setup_slots(const ProjParams& p, const ZItemDev& it, int nslots, ZSlot* sl,
                                            const float* buf, int lane) {
  ZSlot s;
  s.nax = 0;
  s.npa = npa_code(1);
  s.zadd = 0;
  s.zsign = (lane & 1) ? -1 : 1;  // (also of a slot without a line: the back projection's addresses move with it)
  s.seg = s.view = 0;
  s.out_base = 0;
  s.owner = lane;
  int full_nax = 0;
  if (lane < nslots) {
    const int2 lb = it.slot[lane];
    s.owner = it.owner[lane];
    if (lb.x >= 0) {
      const LineDev L = p.lines[lb.x];
      const int tang = static_cast<int>(L.tang_sign) * p.bins[lb.y].tang;
      // the line's view in the data's layout: a view shard holds some views only, the others' lines are inactive
      const int slot = p.view_slot ? __ldg(p.view_slot + L.view) : L.view;
      const SegDev sd = p.segs[L.seg + p.S];
      s.seg = L.seg;
      s.view = L.view;
      s.npa = npa_code(sd.npa);
      full_nax = sd.nax;
      if (tang >= p.min_tang && tang <= p.max_tang && slot >= 0) {
        s.nax = sd.nax;
        s.out_base = sd.dev_offset + (static_cast<int64_t>(slot) * p.num_tang + (tang - p.min_tang)) * sd.nax;
      }
      // plane of axial position 0: zsign z + zadd for a stored plane z (z + 512)
      s.zsign = (L.flags & 8) ? -1 : 1;
      s.zadd = (L.flags & 8) ? static_cast<int>(L.q) + 512 - p.min_z : -512 - p.min_z;
    }
  }
  // (an inactive line has room too: the records' leaving positions do not know which lines are)
  const int own = (lane < nslots && s.owner == lane && it.slot[lane].x >= 0) ? full_nax : 0;
  int pre = own;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, pre, o);
    if (lane >= o) pre += t;
  }
  s.off = __shfl_sync(kFull, pre - own, s.owner);
  s.addr = lane < nslots && it.slot[lane].x >= 0 ? smem_addr(buf) + 4 * s.off : 0;
  if (lane < nslots) sl[lane] = s;
  __syncwarp();
}

constexpr int kZRing = 4 * kZBatch;  // records in shared memory
// columns loaded ahead (forward), at most 4: more where few warps of an item are to hide the loads, and registers are left
constexpr int columns_ahead(int NM, int P, bool shared) { return shared && NM * P <= 8 ? 4 : 2; }

// shared memory of a warp: the records' ring, their column offsets, the slots, the lines' values (`buffers` of them) or data
__host__ __device__ inline int forward_smem(const ZParams& z, int buffers) {
  return kZRing * static_cast<int>(sizeof(ZRec) + sizeof(int)) + 2 * kZChains * static_cast<int>(sizeof(ZSlot)) +
         path_align16(z.max_out * buffers * 4);
}
__host__ __device__ inline int back_smem(const ZParams& z) {
  return 2 * kZBatch * static_cast<int>(sizeof(ZRec) + sizeof(int)) + 2 * kZChains * static_cast<int>(sizeof(ZSlot)) +
         path_align16(z.max_back * 4);
}

// The item's records through a ring of batches.  Forward, four: one in use, the next complete with its column offsets
// (columns are loaded ahead across the boundary), the one after on its way; back, two: one in use, the next on its way.
template <int NB>
struct ZRing {
  ZRec* ring;
  int* offs;  // the records' columns as float offsets
  const ZRec* src;
  int nrec, cx, cy, c0;

  __device__ __forceinline__ void init(const ProjParams& p, const ZParams& z, const ZItemDev& it, ZRec* r, int stride) {
    ring = r;
    offs = reinterpret_cast<int*>(r + NB * kZBatch);
    src = z.recs + it.rec0;
    nrec = it.nrec;
    const int swap = it.flags & 1;
    const int sx = (it.flags & 2) ? -1 : 1, sy = (it.flags & 4) ? -1 : 1;
    // column (x, y) under T: ((sy (swap ? x : y) - min_y) nx + sx (swap ? y : x) - min_x) stride
    cx = (swap ? sy * p.nx : sx) * stride;
    cy = (swap ? sx : sy * p.nx) * stride;
    c0 = (-p.min_y * p.nx - p.min_x) * stride - 1024 * (cx + cy);
  }
  __device__ __forceinline__ void fetch(int b, int lane) {
    if (b * kZBatch < nrec) {
      int4* d = reinterpret_cast<int4*>(batch(b));
      const int4* g = reinterpret_cast<const int4*>(src + b * kZBatch);
      constexpr int kPieces = kZBatch * sizeof(ZRec) / 16;
#pragma unroll
      for (int i = 0; i < kPieces; i += 32)
        if (i + 32 <= kPieces || lane < kPieces - i) cp_async16(d + i + lane, g + i + lane);
    }
    cp_commit();
  }
  // the columns of batch b (0 past the last record: loaded ahead, not used)
  __device__ __forceinline__ void offsets(int b, int lane) {
    if (lane < kZBatch) {
      const uint32_t pk = batch(b)[lane].xy;
      const int x = static_cast<int>(pk & 2047u), y = static_cast<int>((pk >> 11) & 2047u);
      offs[(b & (NB - 1)) * kZBatch + lane] = b * kZBatch + lane < nrec ? x * cx + y * cy + c0 : 0;
    }
  }
  __device__ __forceinline__ ZRec* batch(int b) const { return ring + (b & (NB - 1)) * kZBatch; }
};

template <int P, bool PAD>
__device__ __forceinline__ void load_column(const float* __restrict__ img, int off, int z, int nz, Planes<P>& c) {
  if constexpr (PAD && P == 4) {
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(img + off));
    c.h[0] = v.x, c.h[1] = v.y;
  } else if constexpr (PAD && P == 2) {
    c.h[0] = __ldg(reinterpret_cast<const unsigned long long*>(img + off));
  } else {
    float f[P];
#pragma unroll
    for (int j = 0; j < P; ++j) f[j] = z + j < nz ? __ldg(img + off + j) : 0.f;
    c.set(f);
  }
}

// what a lane needs at the events: lane 0 has to do with the up line's last plane (what rotates to it leaves there), lane
// 31 with the down line's first one
struct ZLane {
  int down, up;     // the lanes the planes below and above come from
  uint32_t slots;   // shared address of this lane's slot of chain 0 (lane 31: the down line's)
  int shift;        // of the leaving positions' packed pair (ZRec::leave): 16 for the up line's, 0 for the down line's
  int sign;         // -1: lane 0, 1: lane 31, 0: the others
};

// edge part of a forward event (text of the assembly): u0 / dl, the registers that took the leaving sums; rec, leave: the
// record and the offset of the leaving positions; slot, values: ZLane's slots and the offset of the chain's entry in them
#define Z_LEAVE(u0, dl, rec, leave, slot, values, shift, sign)                                                       \
  "{\n .reg .pred in, f, l;\n .reg .b32 a, q;\n .reg .f32 v, o;\n"                                                   \
  " ld.shared.b32 a, [" rec " + " leave "];\n ld.shared.b32 q, [" slot " + " values "];\n"                            \
  " shl.b32 a, a, " shift ";\n shr.s32 a, a, 16;\n"                                                                 \
  " setp.lt.s32 f, " sign ", 0;\n setp.gt.s32 l, " sign ", 0;\n setp.ne.s32 in, " sign ", 0;\n"               \
  " setp.ge.and.s32 in, a, 0, in;\n setp.ne.and.u32 in, q, 0, in;\n selp.f32 v, " u0 ", " dl ", f;\n shl.b32 a, a, 2;\n add.s32 a, a, q;\n"           \
  " @in ld.shared.f32 o, [a];\n @in add.f32 o, o, v;\n @in st.shared.f32 [a], o;\n"                                  \
  " selp.f32 " u0 ", 0f00000000, " u0 ", f;\n selp.f32 " dl ", 0f00000000, " dl ", l;\n}\n"

template <int NM, int P>
struct ZForward {
  float U[NM][P], D[NM][P];
  Planes<P> G[NM];

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
      for (int j = 0; j < P; ++j) U[m][j] = D[m][j] = 0.f;
#pragma unroll
    for (int m = 0; m < NM; ++m) G[m].zero();
  }
  // G += w1 c.  The branches of a column (a chain without an element, an event, an edge) are inside the assembly: as C++
  // control flow every register of the lines was copied where they join (19 moves a column of 80 instructions)
  __device__ __forceinline__ void multiply(uint32_t op, const u64* w, const Planes<P>& c) {
    if constexpr (P == 4 && NM == 6) {
      asm("{\n .reg .pred p, q0, q1, q2, q3, q4, q5;\n .reg .b32 t;\n"
          " and.b32 t, %20, 4096;\n setp.ne.u32 p, t, 0;\n @p bra.uni GUARD;\n"
          " fma.rn.f32x2 %0, %12, %18, %0;\n fma.rn.f32x2 %1, %12, %19, %1;\n"
          " fma.rn.f32x2 %2, %13, %18, %2;\n fma.rn.f32x2 %3, %13, %19, %3;\n"
          " fma.rn.f32x2 %4, %14, %18, %4;\n fma.rn.f32x2 %5, %14, %19, %5;\n"
          " fma.rn.f32x2 %6, %15, %18, %6;\n fma.rn.f32x2 %7, %15, %19, %7;\n"
          " fma.rn.f32x2 %8, %16, %18, %8;\n fma.rn.f32x2 %9, %16, %19, %9;\n"
          " fma.rn.f32x2 %10, %17, %18, %10;\n fma.rn.f32x2 %11, %17, %19, %11;\n"
          " bra.uni DONE;\nGUARD:\n"
          " setp.ne.u64 q0, %12, 0;\n setp.ne.u64 q1, %13, 0;\n setp.ne.u64 q2, %14, 0;\n"
          " setp.ne.u64 q3, %15, 0;\n setp.ne.u64 q4, %16, 0;\n setp.ne.u64 q5, %17, 0;\n"
          " @q0 fma.rn.f32x2 %0, %12, %18, %0;\n @q0 fma.rn.f32x2 %1, %12, %19, %1;\n"
          " @q1 fma.rn.f32x2 %2, %13, %18, %2;\n @q1 fma.rn.f32x2 %3, %13, %19, %3;\n"
          " @q2 fma.rn.f32x2 %4, %14, %18, %4;\n @q2 fma.rn.f32x2 %5, %14, %19, %5;\n"
          " @q3 fma.rn.f32x2 %6, %15, %18, %6;\n @q3 fma.rn.f32x2 %7, %15, %19, %7;\n"
          " @q4 fma.rn.f32x2 %8, %16, %18, %8;\n @q4 fma.rn.f32x2 %9, %16, %19, %9;\n"
          " @q5 fma.rn.f32x2 %10, %17, %18, %10;\n @q5 fma.rn.f32x2 %11, %17, %19, %11;\n"
          "DONE:\n}\n"
          : "+l"(G[0].h[0]), "+l"(G[0].h[1]), "+l"(G[1].h[0]), "+l"(G[1].h[1]), "+l"(G[2].h[0]), "+l"(G[2].h[1]),
            "+l"(G[3].h[0]), "+l"(G[3].h[1]), "+l"(G[4].h[0]), "+l"(G[4].h[1]), "+l"(G[5].h[0]), "+l"(G[5].h[1])
          : "l"(w[0]), "l"(w[1]), "l"(w[2]), "l"(w[3]), "l"(w[4]), "l"(w[5]), "l"(c.h[0]), "l"(c.h[1]), "r"(op));
    } else if constexpr (P == 4 && NM == 4) {
      asm("{\n .reg .pred p, q0, q1, q2, q3;\n .reg .b32 t;\n"
          " and.b32 t, %14, 4096;\n setp.ne.u32 p, t, 0;\n @p bra.uni GUARD;\n"
          " fma.rn.f32x2 %0, %8, %12, %0;\n fma.rn.f32x2 %1, %8, %13, %1;\n"
          " fma.rn.f32x2 %2, %9, %12, %2;\n fma.rn.f32x2 %3, %9, %13, %3;\n"
          " fma.rn.f32x2 %4, %10, %12, %4;\n fma.rn.f32x2 %5, %10, %13, %5;\n"
          " fma.rn.f32x2 %6, %11, %12, %6;\n fma.rn.f32x2 %7, %11, %13, %7;\n"
          " bra.uni DONE;\nGUARD:\n"
          " setp.ne.u64 q0, %8, 0;\n setp.ne.u64 q1, %9, 0;\n setp.ne.u64 q2, %10, 0;\n setp.ne.u64 q3, %11, 0;\n"
          " @q0 fma.rn.f32x2 %0, %8, %12, %0;\n @q0 fma.rn.f32x2 %1, %8, %13, %1;\n"
          " @q1 fma.rn.f32x2 %2, %9, %12, %2;\n @q1 fma.rn.f32x2 %3, %9, %13, %3;\n"
          " @q2 fma.rn.f32x2 %4, %10, %12, %4;\n @q2 fma.rn.f32x2 %5, %10, %13, %5;\n"
          " @q3 fma.rn.f32x2 %6, %11, %12, %6;\n @q3 fma.rn.f32x2 %7, %11, %13, %7;\n"
          "DONE:\n}\n"
          : "+l"(G[0].h[0]), "+l"(G[0].h[1]), "+l"(G[1].h[0]), "+l"(G[1].h[1]), "+l"(G[2].h[0]), "+l"(G[2].h[1]),
            "+l"(G[3].h[0]), "+l"(G[3].h[1])
          : "l"(w[0]), "l"(w[1]), "l"(w[2]), "l"(w[3]), "l"(c.h[0]), "l"(c.h[1]), "r"(op));
    } else if (!(op & kZGuard)) {
#pragma unroll
      for (int m = 0; m < NM; ++m) G[m].fma(w[m], c);
    } else {
#pragma unroll
      for (int m = 0; m < NM; ++m)
        if (static_cast<unsigned>(w[m])) G[m].fma(w[m], c);
    }
  }
  // Chain M's event where its bit is set: both lines take G up while they move by one plane, and G starts again at w2 c.
  // What rotates into the first plane (up line, lane 0) and the last (down line, lane 31) is the sum of the position
  // that leaves at the other end.  At an edge event (its bit set) that sum goes to the line's values, and the position
  // that enters starts at 0.
  template <int M>
  __device__ __forceinline__ void event(uint32_t op, uint32_t rec, const Planes<P>& c, const ZLane& k) {
    if constexpr (P == 4) {
      asm volatile(
          "{\n .reg .pred p, e;\n .reg .b32 t;\n .reg .f32 a, b, w, g0, g1, g2, g3;\n .reg .b64 ww;\n"
          " and.b32 t, %14, %15;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " ld.shared.f32 w, [%16 + %17];\n mov.b64 {g0, g1}, %8;\n mov.b64 {g2, g3}, %9;\n"
          " add.f32 a, %3, g3;\n add.f32 %3, %2, g2;\n add.f32 %2, %1, g1;\n add.f32 %1, %0, g0;\n"
          " shfl.sync.idx.b32 %0, a, %12, 31, -1;\n"
          " add.f32 b, %4, g0;\n add.f32 %4, %5, g1;\n add.f32 %5, %6, g2;\n add.f32 %6, %7, g3;\n"
          " shfl.sync.idx.b32 %7, b, %13, 31, -1;\n"
          " mov.b64 ww, {w, w};\n mul.rn.f32x2 %8, ww, %10;\n mul.rn.f32x2 %9, ww, %11;\n"
          " and.b32 t, %14, %18;\n setp.eq.u32 e, t, 0;\n @e bra.uni SKIP;\n"
          Z_LEAVE("%0", "%7", "%16", "%19", "%20", "%21", "%22", "%23")
          " setp.eq.f32 e, w, 0f00000000;\n @e mov.b64 %8, 0;\n @e mov.b64 %9, 0;\n"
          "SKIP:\n}\n"
          : "+f"(U[M][0]), "+f"(U[M][1]), "+f"(U[M][2]), "+f"(U[M][3]), "+f"(D[M][0]), "+f"(D[M][1]), "+f"(D[M][2]),
            "+f"(D[M][3]), "+l"(G[M].h[0]), "+l"(G[M].h[1])
          : "l"(c.h[0]), "l"(c.h[1]), "r"(k.down), "r"(k.up), "r"(op), "n"(1 << M), "r"(rec),
            "n"(offsetof(ZRec, w2) + 4 * M), "n"(64 << M), "n"(offsetof(ZRec, leave) + 4 * M), "r"(k.slots),
            "n"(2 * M * sizeof(ZSlot) + offsetof(ZSlot, addr)), "r"(k.shift), "r"(k.sign)
          : "memory");
    } else if constexpr (P == 2) {
      asm volatile(
          "{\n .reg .pred p, e;\n .reg .b32 t;\n .reg .f32 a, b, w, g0, g1;\n .reg .b64 ww;\n"
          " and.b32 t, %8, %9;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " ld.shared.f32 w, [%10 + %11];\n mov.b64 {g0, g1}, %4;\n"
          " add.f32 a, %1, g1;\n add.f32 %1, %0, g0;\n shfl.sync.idx.b32 %0, a, %6, 31, -1;\n"
          " add.f32 b, %2, g0;\n add.f32 %2, %3, g1;\n shfl.sync.idx.b32 %3, b, %7, 31, -1;\n"
          " mov.b64 ww, {w, w};\n mul.rn.f32x2 %4, ww, %5;\n"
          " and.b32 t, %8, %12;\n setp.eq.u32 e, t, 0;\n @e bra.uni SKIP;\n"
          Z_LEAVE("%0", "%3", "%10", "%13", "%14", "%15", "%16", "%17")
          " setp.eq.f32 e, w, 0f00000000;\n @e mov.b64 %4, 0;\n"
          "SKIP:\n}\n"
          : "+f"(U[M][0]), "+f"(U[M][1]), "+f"(D[M][0]), "+f"(D[M][1]), "+l"(G[M].h[0])
          : "l"(c.h[0]), "r"(k.down), "r"(k.up), "r"(op), "n"(1 << M), "r"(rec), "n"(offsetof(ZRec, w2) + 4 * M),
            "n"(64 << M), "n"(offsetof(ZRec, leave) + 4 * M), "r"(k.slots),
            "n"(2 * M * sizeof(ZSlot) + offsetof(ZSlot, addr)), "r"(k.shift), "r"(k.sign)
          : "memory");
    } else {
      asm volatile(
          "{\n .reg .pred p, e;\n .reg .b32 t;\n .reg .f32 a, b, w;\n"
          " and.b32 t, %6, %7;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " ld.shared.f32 w, [%8 + %9];\n"
          " add.f32 a, %0, %2;\n shfl.sync.idx.b32 %0, a, %4, 31, -1;\n"
          " add.f32 b, %1, %2;\n shfl.sync.idx.b32 %1, b, %5, 31, -1;\n"
          " mul.f32 %2, w, %3;\n"
          " and.b32 t, %6, %10;\n setp.eq.u32 e, t, 0;\n @e bra.uni SKIP;\n"
          Z_LEAVE("%0", "%1", "%8", "%11", "%12", "%13", "%14", "%15")
          " setp.eq.f32 e, w, 0f00000000;\n @e mov.f32 %2, 0f00000000;\n"
          "SKIP:\n}\n"
          : "+f"(U[M][0]), "+f"(D[M][0]), "+f"(G[M].f0)
          : "f"(c.f0), "r"(k.down), "r"(k.up), "r"(op), "n"(1 << M), "r"(rec), "n"(offsetof(ZRec, w2) + 4 * M),
            "n"(64 << M), "n"(offsetof(ZRec, leave) + 4 * M), "r"(k.slots),
            "n"(2 * M * sizeof(ZSlot) + offsetof(ZSlot, addr)), "r"(k.shift), "r"(k.sign)
          : "memory");
    }
  }
  template <int M>
  __device__ __forceinline__ void events(uint32_t op, uint32_t rec, const Planes<P>& c, const ZLane& k) {
    if constexpr (M < NM) {
      event<M>(op, rec, c, k);
      events<M + 1>(op, rec, c, k);
    }
  }
  __device__ __forceinline__ void column(const ZRec* r, const Planes<P>& c, const ZLane& k) {
    const uint32_t op = r->op;
    multiply(op, reinterpret_cast<const u64*>(r->w1), c);
    if (op & 63u) events<0>(op, smem_addr(r), c, k);
  }
  // G into the lines' sums without a move: a chain that crosses few planes would else add hundreds of products one by one
  __device__ __forceinline__ void fold() {
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      float g[P];
      G[m].get(g);
#pragma unroll
      for (int j = 0; j < P; ++j) {
        U[m][j] += g[j];
        D[m][j] += g[j];
      }
      G[m].zero();
    }
  }
  // the sums in registers (folded) to the lines' values, the chains at planes zr
  template <int M>
  __device__ __forceinline__ void flush(const ZSlot* sl, const int16_t* planes, float* buf, int lane) {
    if constexpr (M < NM) {
      const int zr = planes[M];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const ZSlot& s = sl[2 * M + d];
        const int z0 = P * lane - (s.zsign * zr + s.zadd), nax = s.nax;
        __syncwarp();
        if (s.npa == npa_code(1)) {
          float* v = buf + (s.off + z0);
#pragma unroll
          for (int j = 0; j < P; ++j)
            if (static_cast<unsigned>(z0 + j) < static_cast<unsigned>(nax)) v[j] += d ? D[M][j] : U[M][j];
        } else {
#pragma unroll
          for (int j = 0; j < P; ++j) {
            const int a = axial_at(z0 + j, s.npa, nax);
            if (a >= 0) buf[s.off + a] += d ? D[M][j] : U[M][j];
          }
        }
      }
      flush<M + 1>(sl, planes, buf, lane);
    }
  }
};

// the value of one axial position, through the epilogue
__device__ __forceinline__ void store_value(const ProjParams& p, const ZSlot& s, int a, float v, float* __restrict__ out,
                                            const FwdEpilogue& ep, double& ll, unsigned& ncancel) {
  const int seg = s.seg, view = s.view, nax = s.nax;
  const int64_t i = s.out_base + a;
  switch (ep.mode) {
    case kEpiNone: forward_store<kEpiNone>(p, seg, view, 0, nax, i, a, v, out, ep, ll, ncancel); break;
    case kEpiRatio: forward_store<kEpiRatio>(p, seg, view, 0, nax, i, a, v, out, ep, ll, ncancel); break;
    case kEpiLoglik: forward_store<kEpiLoglik>(p, seg, view, 0, nax, i, a, v, out, ep, ll, ncancel); break;
    case kEpiGradient: forward_store<kEpiGradient>(p, seg, view, 0, nax, i, a, v, out, ep, ll, ncancel); break;
    default: forward_store<kEpiLoglikRatio>(p, seg, view, 0, nax, i, a, v, out, ep, ll, ncancel); break;
  }
}

// the lines' values of a warp's item
__device__ __forceinline__ void store_values(const ProjParams& p, const ZSlot* sl, int nslots, const float* buf, int lane,
                                             float* __restrict__ out, const FwdEpilogue& ep, double& ll, unsigned& ncancel) {
  for (int k = 0; k < nslots; ++k) {
    if (sl[k].owner != k) continue;
    for (int a = lane; a < sl[k].nax; a += 32) store_value(p, sl[k], a, buf[sl[k].off + a], out, ep, ll, ncancel);
  }
}
// the same of a shared item: its warps take the lines in turn and add the segments' buffers in order (per of a part, max_out
// floats each, parts `stride` floats apart; the slots' offsets are those of the last one)
__device__ __forceinline__ void store_shared(const ProjParams& p, const ZSlot* sl, int nslots, const float* buf, ZSplit sp,
                                             int part, int per, int max_out, int stride, int lane, float* __restrict__ out,
                                             const FwdEpilogue& ep, double& ll, unsigned& ncancel) {
  buf -= part * stride + (per - 1) * max_out;
  for (int k = part; k < nslots; k += sp.parts) {
    if (sl[k].owner != k) continue;
    for (int a = lane; a < sl[k].nax; a += 32) {
      const float* q = buf + (sl[k].off + a);
      float v = 0.f;
      for (int w = 0; w < sp.parts; ++w, q += stride)
        for (int j = 0; j < per; ++j) v += q[j * max_out];
      store_value(p, sl[k], a, v, out, ep, ll, ncancel);
    }
  }
}

// the `parts` warps of a CTA that share an item meet
__device__ __forceinline__ void parts_sync(int warp, int parts) {
  // (two barriers by number: with one in a register the kernel would take all 16, and fewer CTAs fit on an SM)
  if (warp < parts)
    asm volatile("bar.sync 1, %0;" ::"r"(32 * parts) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"r"(32 * parts) : "memory");
}

// An item's path in sp.segs segments of its batches, sp.parts warps with as many segments each (1: this warp alone).  A
// segment's sums go to the lines' values at its end: short sums, so that their rounding stays small, and the same numbers
// whoever takes the segment where each has a buffer of its own.  smem: this warp's, warp_smem bytes a warp.
template <int NM, int P, bool PAD, bool SHARED>
__device__ __forceinline__ void forward_z_item(const ProjParams& p, const ZParams& z, const ZItemDev& it, ZSplit sp,
                                               unsigned char* smem, int warp_smem, const float* __restrict__ img,
                                               float* __restrict__ out, const FwdEpilogue& ep, double& ll,
                                               unsigned& ncancel, int warp, int lane) {
  ZRing<4> rg;
  rg.init(p, z, it, reinterpret_cast<ZRec*>(smem), PAD ? 32 * P : p.nz);
  ZSlot* sl = reinterpret_cast<ZSlot*>(rg.offs + kZRing);
  float* buf = reinterpret_cast<float*>(sl + 2 * kZChains);
  const int part = SHARED ? warp % sp.parts : 0, per = SHARED ? sp.segs / sp.parts : sp.segs;
  for (int i = lane; i < z.max_out * (SHARED ? per : 1); i += 32) buf[i] = 0.f;
  const int nb = (it.nrec + kZBatch - 1) / kZBatch;
  const int s0 = part * per, s1 = s0 + per;
  int b = nb * s0 / sp.segs;
  rg.fetch(b, lane);
  setup_slots(p, it, 2 * NM, sl, buf, lane);
  const int zlane = P * lane;
  const float* im = img + zlane;
  ZLane k_;
  k_.down = (lane + 31) & 31;
  k_.up = (lane + 1) & 31;
  k_.slots = smem_addr(sl + (lane == 31 ? 1 : 0));
  k_.shift = lane == 31 ? 0 : 16;
  k_.sign = lane == 0 ? -1 : lane == 31 ? 1 : 0;
  ZForward<NM, P> f;
  f.reset();
  cp_wait<0>();
  __syncwarp();
  rg.offsets(b, lane);
  rg.fetch(b + 1, lane);
  __syncwarp();
  constexpr int kAhead = columns_ahead(NM, P, SHARED);
  Planes<P> c[kAhead];
#pragma unroll
  for (int k = 0; k < kAhead; ++k) load_column<P, PAD>(im, rg.offs[(b & 3) * kZBatch + k], zlane, p.nz, c[k]);
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    const int b1 = nb * (s + 1) / sp.segs;
#pragma unroll 1
    while (b < b1) {
      const int be = min(b + sp.fold, b1);
#pragma unroll 1
      for (; b < be; ++b) {
        cp_wait<0>();  // batch b + 1, on its way since the batch before
        __syncwarp();
        rg.offsets(b + 1, lane);
        rg.fetch(b + 2, lane);
        __syncwarp();
        const ZRec* cur = rg.batch(b);
        const int n = min(kZBatch, it.nrec - b * kZBatch);
#pragma unroll 1
        for (int k = 0; k < n; k += kAhead) {
          // the columns kAhead on, across the end of the ring
          const int* ahead = rg.offs + ((b * kZBatch + k + kAhead) & (kZRing - 1));
#pragma unroll
          for (int i = 0; i < kAhead; ++i) {
            f.column(cur + k + i, c[i], k_);
            load_column<P, PAD>(im, ahead[i], zlane, p.nz, c[i]);
          }
        }
      }
      f.fold();
    }
    f.template flush<0>(sl, z.sixteenths[it.path].z[kZSixteenths / sp.segs * (s + 1)], buf, lane);
    f.reset();
    if (SHARED && s + 1 < s1) {  // on to the next segment's buffer
      __syncwarp();
      if (lane < 2 * NM) {
        sl[lane].off += z.max_out;
        if (sl[lane].addr) sl[lane].addr += 4 * z.max_out;
      }
      __syncwarp();
    }
  }
  cp_wait<0>();
  if constexpr (SHARED) {
    parts_sync(warp, sp.parts);
    store_shared(p, sl, 2 * NM, buf, sp, part, per, z.max_out, warp_smem / 4, lane, out, ep, ll, ncancel);
  } else {
    __syncwarp();
    store_values(p, sl, 2 * NM, buf, lane, out, ep, ll, ncancel);
  }
}

// CTAs per SM the forward kernels are compiled for
constexpr int forward_ctas(int NM, int P) { return P == 4 ? (NM > 4 ? 4 : 5) : P == 2 ? 6 : 7; }

// W: the CTA's warps, kZWarps or (a few items shared by more warps each) up to kZManyWarps
template <int NM, int P, bool PAD, bool SHARED, int W>
__global__ void __launch_bounds__(W * 32, W == kZWarps ? forward_ctas(NM, P) : 1)
    forward_z_kernel(ProjParams p, ZParams z, const int* __restrict__ list, int n, ZSplit sp, const float* __restrict__ img,
                     int64_t img_stride, float* __restrict__ out, int64_t out_stride, FwdEpilogue ep) {
  extern __shared__ __align__(16) unsigned char smem[];
  // one warp's values are the same in all its lanes, which the compiler takes from the broadcast
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int i = SHARED ? (blockIdx.x * (blockDim.x >> 5) + warp) / sp.parts : blockIdx.x * W + warp;
  if (i >= n) return;  // all the warps of an item
  if (blockIdx.y > 0) {  // image blockIdx.y of a batch
    const int64_t b = blockIdx.y;
    img += b * img_stride;
    if (out) out += b * out_stride;
    ep.y += b * ep.y_stride;
    if (ep.add) ep.add += b * ep.add_stride;
    if (ep.mult) ep.mult += b * ep.mult_stride;
    if (ep.small_value) ep.small_value += b * ep.sv_stride;
  }
  double ll = 0.0;
  unsigned ncancel = 0;
  const int warp_smem = forward_smem(z, z_buffers(sp));
  forward_z_item<NM, P, PAD, SHARED>(p, z, z.items[list[i]], sp, smem + warp * warp_smem, warp_smem, img, out, ep, ll, ncancel, warp,
                             lane);
  if (ep.mode == kEpiRatio || ep.mode == kEpiGradient || ep.mode == kEpiLoglikRatio) {
    // cancelled singularities (distributable.cxx:590-594)
    for (int o = 16; o > 0; o >>= 1) ncancel += __shfl_xor_sync(kFull, ncancel, o);
    if (lane == 0 && ncancel && ep.cancelled) atomicAdd(ep.cancelled, ncancel);
  }
  if (ep.mode == kEpiLoglik || ep.mode == kEpiLoglikRatio) {
    // one partial sum per item, reduced in a fixed order by the caller: deterministic
    for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(kFull, ll, o);
    if constexpr (SHARED) {
      __shared__ double red[W];
      if (lane == 0) red[warp] = ll;
      parts_sync(warp, sp.parts);
      if (warp % sp.parts) return;
      ll = 0.0;
      for (int w = 0; w < sp.parts; ++w) ll += red[warp + w];
    }
    if (lane == 0) ep.partials[static_cast<int64_t>(blockIdx.y) * n + i] = ll;
  }
}

// ---- back projection ----------------------------------------------------------------------------------------------

// What becomes of a column's sums u (planes lane + 32 j): floats added to the padded or the plain image, or rounded once
// per item to the fixed-point grid (a power-of-two scale: exact) and added as 64-bit integers, in any order the same sum.
// PAD: the columns hold every plane of the lanes, so none has to be left out.  TURNS: `copies` images (a power of two, `apart`
// floats apart) take the items in turn; an instance of its own, since a base address that depends on the item costs an
// addition a reduction (all clinical lines 3.60 -> 3.71 ms).
template <bool PAD, bool TURNS>
struct ZFloatSink {
  static constexpr bool kWhole = PAD;
  float* img;
  int copies;
  int64_t apart;
  __device__ __forceinline__ void load() {}
  __device__ __forceinline__ void batch(int64_t o) { img += o; }
  __device__ __forceinline__ void item(const ZItemDev& it) {
    if constexpr (TURNS) img += ((it.flags >> kZTurn) & (copies - 1)) * apart;
  }
  __device__ __forceinline__ void add(int i, float v) const { atomicAdd(img + i, v); }
};
struct ZFixedSink {
  static constexpr bool kWhole = false;
  unsigned long long* acc;
  const double* scale_ptr;
  float scale;
  __device__ __forceinline__ void load() { scale = static_cast<float>(*scale_ptr); }
  __device__ __forceinline__ void batch(int64_t) {}  // one image per launch
  __device__ __forceinline__ void item(const ZItemDev&) {}
  __device__ __forceinline__ void add(int i, float v) const {
    if (v != 0.f) atomicAdd(acc + i, static_cast<unsigned long long>(__float2ll_rn(v * scale)));
  }
};

// The lines' data stay in shared memory, every line's with zeros around it (ZItemDev::boff) so that plane z of the image
// reads datum z - zt without a test.  A lane holds planes lane + 32 j of E_m = the two lines' data of chain m, read again
// at the chain's events only: eight shared reads instead of moving eight registers, and no edge code.
template <int NM, int P>
struct ZBack {
  Planes<P> E[NM];
  uint32_t U[NM], D[NM];  // shared addresses of the lines' datum for plane `lane`

  template <int M>
  __device__ __forceinline__ void init(const ZSlot* sl, const ZItemDev& it, const int16_t* planes, uint32_t buf, int lane) {
    if constexpr (M < NM) {
      const int zr = planes[M];
      U[M] = buf + 4 * (it.boff[2 * M] + lane - (sl[2 * M].zsign * zr + sl[2 * M].zadd));
      D[M] = buf + 4 * (it.boff[2 * M + 1] + lane - (sl[2 * M + 1].zsign * zr + sl[2 * M + 1].zadd));
      float e[P];
#pragma unroll
      for (int j = 0; j < P; ++j) {
        float a, b;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(a) : "r"(U[M] + 128 * j) : "memory");
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(b) : "r"(D[M] + 128 * j) : "memory");
        e[j] = a + b;
      }
      E[M].set(e);
      init<M + 1>(sl, it, planes, buf, lane);
    }
  }
  // chain M's event where its bit is set (the branch in the assembly: see ZForward): E one plane on, and the column's
  // second element
  template <int M>
  __device__ __forceinline__ void event(uint32_t op, uint32_t rec, Planes<P>& u) {
    if constexpr (P == 4) {
      asm volatile(
          "{\n .reg .pred p, q;\n .reg .b32 t;\n .reg .f32 w, a0, a1, a2, a3, b0, b1, b2, b3;\n .reg .b64 ww, x, y;\n"
          " and.b32 t, %6, %7;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " add.s32 %4, %4, -4;\n add.s32 %5, %5, 4;\n ld.shared.f32 w, [%8 + %9];\n"
          " ld.shared.f32 a0, [%4];\n ld.shared.f32 a1, [%4 + 128];\n ld.shared.f32 a2, [%4 + 256];\n"
          " ld.shared.f32 a3, [%4 + 384];\n ld.shared.f32 b0, [%5];\n ld.shared.f32 b1, [%5 + 128];\n"
          " ld.shared.f32 b2, [%5 + 256];\n ld.shared.f32 b3, [%5 + 384];\n"
          " mov.b64 x, {a0, a1};\n mov.b64 y, {b0, b1};\n add.rn.f32x2 %0, x, y;\n"
          " mov.b64 x, {a2, a3};\n mov.b64 y, {b2, b3};\n add.rn.f32x2 %1, x, y;\n"
          " setp.neu.f32 q, w, 0f00000000;\n mov.b64 ww, {w, w};\n"
          " @q fma.rn.f32x2 %2, ww, %0, %2;\n @q fma.rn.f32x2 %3, ww, %1, %3;\n"
          "SKIP:\n}\n"
          : "+l"(E[M].h[0]), "+l"(E[M].h[1]), "+l"(u.h[0]), "+l"(u.h[1]), "+r"(U[M]), "+r"(D[M])
          : "r"(op), "n"(1 << M), "r"(rec), "n"(offsetof(ZRec, w2) + 4 * M)
          : "memory");
    } else if constexpr (P == 2) {
      asm volatile(
          "{\n .reg .pred p, q;\n .reg .b32 t;\n .reg .f32 w, a0, a1, b0, b1;\n .reg .b64 ww, x, y;\n"
          " and.b32 t, %4, %5;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " add.s32 %2, %2, -4;\n add.s32 %3, %3, 4;\n ld.shared.f32 w, [%6 + %7];\n"
          " ld.shared.f32 a0, [%2];\n ld.shared.f32 a1, [%2 + 128];\n"
          " ld.shared.f32 b0, [%3];\n ld.shared.f32 b1, [%3 + 128];\n"
          " mov.b64 x, {a0, a1};\n mov.b64 y, {b0, b1};\n add.rn.f32x2 %0, x, y;\n"
          " setp.neu.f32 q, w, 0f00000000;\n mov.b64 ww, {w, w};\n @q fma.rn.f32x2 %1, ww, %0, %1;\n"
          "SKIP:\n}\n"
          : "+l"(E[M].h[0]), "+l"(u.h[0]), "+r"(U[M]), "+r"(D[M])
          : "r"(op), "n"(1 << M), "r"(rec), "n"(offsetof(ZRec, w2) + 4 * M)
          : "memory");
    } else {
      asm volatile(
          "{\n .reg .pred p, q;\n .reg .b32 t;\n .reg .f32 w, a0, b0;\n"
          " and.b32 t, %4, %5;\n setp.eq.u32 p, t, 0;\n @p bra.uni SKIP;\n"
          " add.s32 %2, %2, -4;\n add.s32 %3, %3, 4;\n ld.shared.f32 w, [%6 + %7];\n"
          " ld.shared.f32 a0, [%2];\n ld.shared.f32 b0, [%3];\n add.f32 %0, a0, b0;\n"
          " setp.neu.f32 q, w, 0f00000000;\n @q fma.rn.f32 %1, w, %0, %1;\n"
          "SKIP:\n}\n"
          : "+f"(E[M].f0), "+f"(u.f0), "+r"(U[M]), "+r"(D[M])
          : "r"(op), "n"(1 << M), "r"(rec), "n"(offsetof(ZRec, w2) + 4 * M)
          : "memory");
    }
  }
  template <int M>
  __device__ __forceinline__ void events(uint32_t op, uint32_t rec, Planes<P>& u) {
    if constexpr (M < NM) {
      event<M>(op, rec, u);
      events<M + 1>(op, rec, u);
    }
  }
  __device__ __forceinline__ void column(const ZRec* r, uint32_t rec, Planes<P>& u) {
    const uint32_t op = r->op;
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(r->w1);
    if (!(op & kZGuard)) {
#pragma unroll
      for (int m = 0; m < NM; m += 2) {
        const ulonglong2 ww = w[m / 2];
        if (m == 0)
          u.mul(ww.x, E[0]);
        else
          u.fma(ww.x, E[m]);
        u.fma(ww.y, E[m + 1]);
      }
    } else {
      u.zero();
#pragma unroll
      for (int m = 0; m < NM; ++m)
        if (r->w1[2 * m] != 0.f) u.fma(reinterpret_cast<const u64*>(r->w1)[m], E[m]);
    }
    if (op & 63u) events<0>(op, rec, u);
  }
};

template <int NM, int P, typename Sink>
__device__ __forceinline__ void back_z_item(const ProjParams& p, const ZParams& z, const ZItemDev& it, ZRec* ring,
                                            int part, int parts, const float* __restrict__ pd, const Sink& sink,
                                            int stride, int zero_ends, int lane) {
  ZRing<2> rg;
  rg.init(p, z, it, ring, stride);
  ZSlot* sl = reinterpret_cast<ZSlot*>(rg.offs + 2 * kZBatch);
  float* buf = reinterpret_cast<float*>(sl + 2 * kZChains);
  // this warp's part of the path's records
  const int nb = (it.nrec + kZBatch - 1) / kZBatch;
  const int b0 = nb * part / parts, b1 = nb * (part + 1) / parts;
  rg.fetch(b0, lane);
  setup_slots(p, it, 2 * NM, sl, buf, lane);
  for (int i = lane; i < z.max_back; i += 32) buf[i] = 0.f;
  __syncwarp();
  for (int k = 0; k < 2 * NM; ++k) {
    const int nax = sl[k].nax, seg = sl[k].seg, npa = sl[k].npa & 0xffff, off = it.boff[k];
    if (sl[k].owner != k) continue;
    const int64_t base = sl[k].out_base;
    for (int a = lane; a < nax; a += 32) {
      float d = 0.f;
      if (!(zero_ends && seg == 0 && (a == 0 || a == nax - 1)))
        d = pd ? __ldg(pd + base + a) : 1.f;  // pd == nullptr back-projects ones
      buf[off + a * npa] = d;
    }
  }
  __syncwarp();
  ZBack<NM, P> f;
  f.template init<0>(sl, it, z.sixteenths[it.path].z[kZSixteenths / parts * part], smem_addr(buf), lane);
#pragma unroll 1
  for (int b = b0; b < b1; ++b) {
    cp_wait<0>();
    __syncwarp();
    rg.offsets(b, lane);
    rg.fetch(b + 1, lane);
    __syncwarp();
    const ZRec* cur = rg.batch(b);
    const int* offs = rg.offs + (b & 1) * kZBatch;
    const int n = min(kZBatch, it.nrec - b * kZBatch);
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      Planes<P> u;
      f.column(cur + k, smem_addr(cur + k), u);
      float v[P];
      u.get(v);
      const int i = offs[k] + lane;
#pragma unroll
      for (int j = 0; j < P; ++j)
        if (Sink::kWhole || lane + 32 * j < p.nz) sink.add(i + 32 * j, v[j]);
    }
  }
  cp_wait<0>();
}

// CTAs per SM the back kernels are compiled for
constexpr int back_ctas(int P) { return P == 4 ? 6 : 8; }

template <int NM, int P, typename Sink>
__global__ void __launch_bounds__(kZWarps * 32, back_ctas(P))
    back_z_kernel(ProjParams p, ZParams z, const int* __restrict__ list, int n, int parts, const float* __restrict__ pd,
                  int64_t pd_stride, Sink sink0, int64_t img_stride, int stride, int zero_ends) {
  extern __shared__ __align__(16) unsigned char smem[];
  // one warp's values are the same in all its lanes, which the compiler takes from the broadcast
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int w = blockIdx.x * kZWarps + warp, i = w / parts;
  if (i >= n) return;
  ZRec* ring = reinterpret_cast<ZRec*>(smem + warp * back_smem(z));
  Sink sink = sink0;
  sink.load();
  if (blockIdx.y > 0) {  // image blockIdx.y of a batch
    if (pd) pd += static_cast<int64_t>(blockIdx.y) * pd_stride;
    sink.batch(static_cast<int64_t>(blockIdx.y) * img_stride);
  }
  const ZItemDev& it = z.items[list[i]];
  sink.item(it);
  back_z_item<NM, P, Sink>(p, z, it, ring, w % parts, parts, pd, sink, stride, zero_ends, lane);
}

// ---- batched reconstructions: persistent CTAs over units of kZWarps (frame, item) work items of one frame ----------------
// A unit holds kZWarps entries: items (bin -1: none), or items repeated for each of the warps that share one.

// the CTA's next unit, or -1
__device__ __forceinline__ int next_z_unit(unsigned* counter, int nunits) {
  __shared__ int s_unit;
  __syncthreads();  // every warp has finished with the previous unit
  if (threadIdx.x == 0) s_unit = static_cast<int>(atomicAdd(counter, 1u));
  __syncthreads();
  return s_unit < nunits ? s_unit : -1;
}

// (SHARED: see forward_z_item; an instance of its own, as one kernel with both forms ran out of registers)
template <int NM, int P, bool SHARED>
__global__ void __launch_bounds__(kZWarps * 32, forward_ctas(NM, P))
    forward_z_batch_kernel(const ProjParams* __restrict__ geoms, const ZParams* __restrict__ zgeoms,
                           const BatchFrameDev* __restrict__ frames, const BatchItem* __restrict__ items, int nunits,
                           unsigned* counter, int warp_smem) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  for (int k; (k = next_z_unit(counter, nunits)) >= 0;) {
    const BatchItem wi = items[k * kZWarps + warp];
    if (wi.bin < 0) continue;
    const BatchFrameDev& f = frames[z_frame_of(wi.frame)];
    const ZParams& z = zgeoms[f.geom];
    double ll = 0.0;
    unsigned ncancel = 0;
    constexpr bool kPad = P > 1;
    const ZSplit sp = z_split_of(wi.frame);
    const float* x = kPad ? f.xpad : f.x;
    forward_z_item<NM, P, kPad, SHARED>(geoms[f.geom], z, z.items[wi.bin], sp, smem + warp * warp_smem, warp_smem, x, f.ratio,
                                        f.ep, ll, ncancel, warp, lane);
    for (int o = 16; o > 0; o >>= 1) ncancel += __shfl_xor_sync(kFull, ncancel, o);
    if (lane == 0 && ncancel && f.ep.cancelled) atomicAdd(f.ep.cancelled, ncancel);
  }
}

template <int NM, int P>
__global__ void __launch_bounds__(kZWarps * 32, back_ctas(P))
    back_z_batch_kernel(const ProjParams* __restrict__ geoms, const ZParams* __restrict__ zgeoms,
                        const BatchFrameDev* __restrict__ frames, const BatchItem* __restrict__ items, int nunits,
                        unsigned* counter, int warp_smem) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  ZRec* ring = reinterpret_cast<ZRec*>(smem + warp * warp_smem);
  for (int k; (k = next_z_unit(counter, nunits)) >= 0;) {
    const BatchItem wi = items[k * kZWarps + warp];
    if (wi.bin < 0) continue;
    const BatchFrameDev& f = frames[z_frame_of(wi.frame)];
    const ProjParams& p = geoms[f.geom];
    const ZParams& z = zgeoms[f.geom];
    const int parts = z_split_of(wi.frame).parts, part = warp % parts;
    if (f.acc64) {  // a deterministic frame: the same fixed-point integers as its own back projection
      ZFixedSink sink{f.acc64, f.fixed_scale, 0.f};
      sink.load();
      back_z_item<NM, P>(p, z, z.items[wi.bin], ring, part, parts, f.ratio, sink, p.nz, 0, lane);
    } else {
      constexpr bool kPad = P > 1;
      const int stride = kPad ? 32 * P : p.nz;
      ZFloatSink<kPad, true> sink{f.usums ? f.usums : f.u, f.usums ? z.copies : 1,
                                  z_image_floats(static_cast<int64_t>(p.ny) * p.nx, stride)};
      sink.item(z.items[wi.bin]);
      back_z_item<NM, P>(p, z, z.items[wi.bin], ring, part, parts, f.ratio, sink, stride, 0, lane);
    }
  }
}

template <typename K, typename... A>
cudaError_t launch_z(K kernel, int sm, int ctas, int warps, int batch, cudaStream_t st, A... args) {
  if (ctas <= 0 || batch <= 0) return cudaSuccess;
  if (batch > 65535) return cudaErrorInvalidValue;
  if (sm > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
  }
  kernel<<<dim3(ctas, batch), warps * 32, sm, st>>>(args...);
  return cudaGetLastError();
}

// CTAs of kZWarps warps for n items shared by `parts` warps each
int z_ctas(int n, int parts) { return static_cast<int>((static_cast<int64_t>(n) * parts + kZWarps - 1) / kZWarps); }

// planes of a column, four per thread: rows of `stride` floats from / to rows of nz
__global__ void pad_image_kernel(const float* __restrict__ in, int64_t in_stride, float* __restrict__ out,
                                 int64_t out_stride, int64_t ncols, int nz, int stride) {
  in += blockIdx.y * in_stride;
  out += blockIdx.y * out_stride;
  const int64_t n4 = ncols * (stride / 4);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t c = i / (stride / 4);
    const int z = static_cast<int>(i - c * (stride / 4)) * 4;
    const float* q = in + c * nz + z;
    float4 v;
    v.x = z < nz ? q[0] : 0.f;
    v.y = z + 1 < nz ? q[1] : 0.f;
    v.z = z + 2 < nz ? q[2] : 0.f;
    v.w = z + 3 < nz ? q[3] : 0.f;
    reinterpret_cast<float4*>(out)[i] = v;
  }
}
__global__ void unpad_image_kernel(const float* __restrict__ in, int64_t in_stride, int copies, float* __restrict__ out,
                                   int64_t out_stride, int64_t ncols, int nz, int stride) {
  in += blockIdx.y * in_stride;
  out += blockIdx.y * out_stride;
  const int64_t n4 = ncols * (stride / 4);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t c = i / (stride / 4);
    const int z = static_cast<int>(i - c * (stride / 4)) * 4;
    if (z >= nz) continue;
    float4 v = reinterpret_cast<const float4*>(in)[i];
    for (int k = 1; k < copies; ++k) {
      const float4 w = reinterpret_cast<const float4*>(in)[k * n4 + i];
      v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
    }
    float* q = out + c * nz + z;
    q[0] = v.x;
    if (z + 1 < nz) q[1] = v.y;
    if (z + 2 < nz) q[2] = v.z;
    if (z + 3 < nz) q[3] = v.w;
  }
}

// the sum of `copies` images of n floats, `apart` (a multiple of 4) floats apart, four at a time; the output wherever it is
__global__ void sum_images_kernel(const float* __restrict__ in, int64_t in_stride, int copies, int64_t apart,
                                  float* __restrict__ out, int64_t out_stride, int64_t n) {
  in += blockIdx.y * in_stride;
  out += blockIdx.y * out_stride;
  const bool aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < apart / 4;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float4 v = reinterpret_cast<const float4*>(in)[i];
    for (int k = 1; k < copies; ++k) {
      const float4 w = reinterpret_cast<const float4*>(in + k * apart)[i];
      v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
    }
    float* q = out + 4 * i;
    if (aligned && 4 * i + 3 < n) {
      *reinterpret_cast<float4*>(q) = v;
    } else {
      q[0] = v.x;
      if (4 * i + 1 < n) q[1] = v.y;
      if (4 * i + 2 < n) q[2] = v.z;
      if (4 * i + 3 < n) q[3] = v.w;
    }
  }
}

int pad_blocks(int64_t n4) {
  const int64_t b = (n4 + 255) / 256;
  return static_cast<int>(b < 148 * 16 ? b : 148 * 16);
}

// calls f.template operator()<NM, P>() for the geometry's chains per item and planes per lane
template <typename F>
cudaError_t z_variant(const ZParams& z, F&& f) {
  auto planes = [&]<int NM>() {
    switch (z.planes) {
      case 1: return f.template operator()<NM, 1>();
      case 2: return f.template operator()<NM, 2>();
      case 4: return f.template operator()<NM, 4>();
      default: return cudaErrorInvalidValue;
    }
  };
  if (z.nm == 4) return planes.template operator()<4>();
  if (z.nm == 6) return planes.template operator()<6>();
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_pad_image(const float* in, int64_t in_stride, float* out, int64_t out_stride, int64_t ncols, int nz,
                             int stride, int batch, cudaStream_t st) {
  pad_image_kernel<<<dim3(pad_blocks(ncols * (stride / 4)), batch), 256, 0, st>>>(in, in_stride, out, out_stride, ncols, nz,
                                                                                 stride);
  return cudaGetLastError();
}
cudaError_t launch_collect_images(const float* in, int64_t in_stride, int copies, float* out, int64_t out_stride,
                                  int64_t ncols, int nz, int stride, int batch, cudaStream_t st) {
  if (stride == nz) {
    const int64_t apart = z_image_floats(ncols, nz);
    sum_images_kernel<<<dim3(pad_blocks(apart / 4), batch), 256, 0, st>>>(in, in_stride, copies, apart, out, out_stride,
                                                                         ncols * nz);
  } else
    unpad_image_kernel<<<dim3(pad_blocks(ncols * (stride / 4)), batch), 256, 0, st>>>(in, in_stride, copies, out, out_stride,
                                                                                     ncols, nz, stride);
  return cudaGetLastError();
}

cudaError_t launch_forward_z(const ProjParams& p, const ZParams& z, const int* list, int n, ZSplit sp, const float* image,
                             int64_t img_stride, int padded, float* out, int64_t out_stride, int batch,
                             cudaStream_t st, const FwdEpilogue* ep) {
  FwdEpilogue e{};
  if (ep) e = *ep;
  const int sm = forward_smem(z, z_buffers(sp));
  if (padded && sp.parts > 1) return cudaErrorInvalidValue;
  return z_variant(z, [&]<int NM, int P>() {
    auto run = [&](auto kernel, int ctas, int warps) {
      return launch_z(kernel, warps * sm, ctas, warps, batch, st, p, z, list, n, sp, image, img_stride, out, out_stride, e);
    };
    if (sp.parts > kZWarps) return run(forward_z_kernel<NM, P, false, true, kZManyWarps>, n, sp.parts);
    if (sp.parts > 1) return run(forward_z_kernel<NM, P, false, true, kZWarps>, z_ctas(n, sp.parts), kZWarps);
    if constexpr (P > 1) {
      if (padded) return run(forward_z_kernel<NM, P, true, false, kZWarps>, z_ctas(n, 1), kZWarps);
    }
    return run(forward_z_kernel<NM, P, false, false, kZWarps>, z_ctas(n, 1), kZWarps);
  });
}

cudaError_t launch_back_z(const ProjParams& p, const ZParams& z, const int* list, int n, int parts, const float* pd,
                          int64_t pd_stride, float* image, int64_t img_stride, int copies, int padded, int batch,
                          cudaStream_t st, int zero_ends) {
  const int64_t ncols = static_cast<int64_t>(p.ny) * p.nx;
  return z_variant(z, [&]<int NM, int P>() {
    auto run = [&](auto kernel, auto sink, int stride) {
      return launch_z(kernel, kZWarps * back_smem(z), z_ctas(n, parts), kZWarps, batch, st, p, z, list, n, parts, pd,
                      pd_stride, sink, img_stride, stride, zero_ends);
    };
    if constexpr (P > 1) {
      if (padded && copies == 1)
        return run(back_z_kernel<NM, P, ZFloatSink<true, false>>, ZFloatSink<true, false>{image, 1, 0}, z_stride(z));
      if (padded)
        return run(back_z_kernel<NM, P, ZFloatSink<true, true>>,
                   ZFloatSink<true, true>{image, copies, z_image_floats(ncols, z_stride(z))}, z_stride(z));
    }
    if (copies == 1) return run(back_z_kernel<NM, P, ZFloatSink<false, false>>, ZFloatSink<false, false>{image, 1, 0}, p.nz);
    return run(back_z_kernel<NM, P, ZFloatSink<false, true>>,
               ZFloatSink<false, true>{image, copies, z_image_floats(ncols, p.nz)}, p.nz);
  });
}

cudaError_t launch_back_z_fixed(const ProjParams& p, const ZParams& z, const int* list, int n, int parts, const float* pd,
                                unsigned long long* acc, const double* scale, cudaStream_t st, int zero_ends) {
  return z_variant(z, [&]<int NM, int P>() {
    return launch_z(back_z_kernel<NM, P, ZFixedSink>, kZWarps * back_smem(z), z_ctas(n, parts), kZWarps, 1, st, p, z, list, n,
                    parts, pd, int64_t(0), ZFixedSink{acc, scale, 0.f}, int64_t(0), p.nz, zero_ends);
  });
}

int z_forward_smem(const ZParams& z, int buffers) { return forward_smem(z, buffers); }
int z_resident_warps(const ZParams& z, bool forward) {
  // (as compiled, or as many as an SM's 227 KB hold: the clinical back projection's data leave room for 5 CTAs of 6)
  const int smem = kZWarps * (forward ? forward_smem(z, 1) : back_smem(z)) + 1024;
  const int fit = 227 * 1024 / smem, compiled = forward ? forward_ctas(z.nm, z.planes) : back_ctas(z.planes);
  return 148 * kZWarps * (fit < 1 ? 1 : fit < compiled ? fit : compiled);
}

int z_batch_smem(const ZParams& z, bool forward, int buffers) {
  return kZWarps * (forward ? forward_smem(z, buffers) : back_smem(z));
}

cudaError_t launch_z_batch(const ZParams& z, bool forward, bool shared, const ProjParams* geoms, const ZParams* zgeoms,
                           const BatchFrameDev* frames, const BatchItem* items, int nunits, unsigned* counter, int smem,
                           int grid, cudaStream_t st) {
  if (nunits <= 0) return cudaSuccess;
  auto run = [&](auto kernel) {
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return e;
    }
    kernel<<<grid, kZWarps * 32, smem, st>>>(geoms, zgeoms, frames, items, nunits, counter, smem / kZWarps);
    return cudaGetLastError();
  };
  return z_variant(z, [&]<int NM, int P>() {
    if (!forward) return run(back_z_batch_kernel<NM, P>);
    return shared ? run(forward_z_batch_kernel<NM, P, true>) : run(forward_z_batch_kernel<NM, P, false>);
  });
}

int z_batch_max_ctas_per_sm(const ZParams& z, bool forward, int smem) {
  int n = 0;
  auto count = [&](auto kernel) {
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return e;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kZWarps * 32, smem);
  };
  const cudaError_t e = forward ? z_variant(z, [&]<int NM, int P>() { return count(forward_z_batch_kernel<NM, P, false>); })
                                : z_variant(z, [&]<int NM, int P>() { return count(back_z_batch_kernel<NM, P>); });
  return e == cudaSuccess ? n : 0;
}

}  // namespace b200
