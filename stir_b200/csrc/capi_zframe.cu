// Set-up of the z-frame tables and the dispatch between the two path-item projections (z-frame, column-staged).
#include "capi.hpp"
#include "zchains.hpp"

using namespace b200;

namespace {

constexpr size_t kPadLimit = size_t(1) << 26;  // floats of padded images or image sums at a time (256 MiB)

size_t most_groups(const std::vector<ZPath>& paths) {
  size_t most = 1;
  for (const ZPath& p : paths) most = std::max(most, p.recs.size());
  return most;
}

}  // namespace

namespace capi {

// The chains and records of every path (zframe.hpp).  Returns false, leaving no tables, where the z-frame kernels do not
// apply: more than 128 planes, a column outside the image, or a basic bin with more chains than a warp takes.
bool build_zframe(b200rt_projector& h, const std::vector<RowElem>& hr, const std::vector<LineDev>& lines, int nviews,
                  int nsegs, int ntangs, const std::vector<int>& bviews) {
  const Geometry& g = *h.geo;
  const ProjParams& p = h.params;
  if (g.num_tof() != 1 || p.nz < 1) return false;
  ZParams z{};
  if (p.nz > 128) return false;  // more planes than a warp holds
  z.planes = p.nz <= 32 ? 1 : p.nz <= 64 ? 2 : 4;
  const int64_t padded = static_cast<int64_t>(z_stride(z)) * p.ny * p.nx;
  if (padded >= (int64_t(1) << 31)) return false;
  const int ngroups = nviews * ntangs;
  const int planes = 32 * z.planes;
  ZPathLines fit;
  fit.S = g.S();
  fit.min_z = p.min_z;
  fit.planes = planes;
  for (int sg = -g.S(); sg <= g.S(); ++sg) {
    fit.nax.push_back(g.nax(sg));
    fit.npa.push_back(g.npa(sg));
  }
  // pass 0 counts the chains a path needs, pass 1 builds the records for groups of z.nm chains
  std::vector<ZPath> groups(ngroups);
  std::vector<int> chains_of(ngroups, 0), chains_max(ngroups, 0);
  auto work = [&](int gi, int cap) {
    ZPath& G = groups[gi];
    try {
      const int vi = gi / ntangs, ti = gi % ntangs;
      std::vector<ZMember> members(nsegs);
      for (int si = 0; si < nsegs; ++si) {
        const ProjBinDev& pb = h.h_bins[(static_cast<size_t>(vi) * nsegs + si) * ntangs + ti];
        members[si] = ZMember{hr.data() + pb.row_offset, pb.row_len, lines.data() + pb.first_line, pb.num_lines};
      }
      build_path(members, fit, cap, G);
      chains_of[gi] = G.total;
      chains_max[gi] = G.most;
    } catch (const std::exception&) {
      G.ok = false;
    }
  };
  const int nthreads = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
  auto run = [&](int stride, int cap) {
    std::vector<std::thread> pool;
    for (int t = 0; t < nthreads; ++t)
      pool.emplace_back([&, t] {
        // interleaved: neighbouring paths cost about the same
        for (int gi = t * stride; gi < ngroups; gi += nthreads * stride) work(gi, cap);
      });
    for (auto& th : pool) th.join();
  };
  // chains a warp takes (4 or 6), from a sample of the paths: as few groups of chains as possible, evenly filled
  run(7, 0);
  int total = 1, most = 1;
  auto count = [&]() {
    for (int gi = 0; gi < ngroups; ++gi) {
      total = std::max(total, chains_of[gi]);
      most = std::max(most, chains_max[gi]);
    }
  };
  count();
  if (most > kZChains) return false;
  const int ng = (total + kZChains - 1) / kZChains;
  z.nm = std::max((total + ng - 1) / ng, most) <= 4 ? 4 : kZChains;
  // Several groups of six chains with few elements each, four planes a lane: a record costs the same whether one chain or six
  // have an element, and the column-staged kernels only pay for the elements.  221 x 222 x 117 image, two rays, three groups,
  // 2.5 elements a record, one of 4 subsets: forward 844 / 650 us, back 554 / 657; 260 x 260 x 109, three groups, 4.6 elements: 94 /
  // 107 and 75 / 127.
  int64_t walked = 0, paths = 0, parts = 0, elements = 0;
  for (const ZPath& G : groups)
    if (G.total > 0) {
      const int n = (G.total + z.nm - 1) / z.nm;
      ++paths;
      parts += n;
      walked += static_cast<int64_t>(G.columns) * n;
      elements += G.elements;
    }
  if (z.planes == 4 && z.nm == kZChains && 2 * parts >= 3 * paths && 5 * elements < 13 * walked) return false;
  run(1, z.nm);
  count();
  if (most > kZChains) return false;
  if (most > z.nm) {  // a path outside the sample needs more
    z.nm = kZChains;
    for (ZPath& G : groups) G = ZPath{};
    run(1, z.nm);
  }
  int64_t nrecs = 0;
  for (int gi = 0; gi < ngroups; ++gi) {
    if (!groups[gi].ok) return false;
    for (const auto& r : groups[gi].recs) nrecs += static_cast<int64_t>(r.size());
  }
  if (nrecs >= (int64_t(1) << 31) - 64) return false;

  std::vector<ZItemDev> items;
  std::vector<int> item_view, item_out_view;
  std::vector<char> item_lead;  // the first item of a (path, T)
  std::vector<int> item_block;
  std::vector<PathItemDev> path_items;
  std::vector<char> led(static_cast<size_t>(ntangs));
  std::vector<int> base(ngroups), path0(ngroups);
  std::vector<ZPlanes> sixteenths;
  int64_t at = 0;
  for (int gi = 0; gi < ngroups; ++gi) {
    path0[gi] = static_cast<int>(sixteenths.size());
    sixteenths.insert(sixteenths.end(), groups[gi].planes.begin(), groups[gi].planes.end());
    base[gi] = static_cast<int>(at);
    for (const auto& r : groups[gi].recs) at += static_cast<int64_t>(r.size());
  }
  // items by (block of kZWarps tangential positions, view, T, chain group): the warps of a CTA take neighbouring paths,
  // whose columns overlap in L1, the CTAs that run together share their paths' records, and the longest paths (through
  // the middle of the field of view) come first
  for (int t0 = 0; t0 < ntangs; t0 += kZWarps)
    for (int vi = 0; vi < nviews; ++vi)
      for (int T = 0; T < 8; ++T) {
        const int t1 = std::min(t0 + kZWarps, ntangs);
        std::fill(led.begin(), led.end(), 0);
        size_t most_groups = 0;
        for (int ti = t0; ti < t1; ++ti) most_groups = std::max(most_groups, groups[vi * ntangs + ti].recs.size());
        for (size_t gr = 0; gr < most_groups; ++gr)
          for (int ti = t0; ti < t1; ++ti) {
            const ZPath& G = groups[vi * ntangs + ti];
            if (gr >= G.recs.size()) continue;
            int rec0 = base[vi * ntangs + ti];
            for (size_t k = 0; k < gr; ++k) rec0 += static_cast<int>(G.recs[k].size());
            const auto& cm = G.chain_member[gr];
            const int16_t* const ends[2] = {G.planes[gr].z[0], G.planes[gr].z[kZSixteenths]};  // planes at both ends
            // the k-th line of each orientation under T of every member
            for (int k = 0;; ++k) {
              ZItemDev it{};
              it.rec0 = rec0;
              it.nrec = static_cast<int>(G.recs[gr].size());
              it.flags = T | static_cast<int>((gr + ti + vi) & 3u) << kZTurn;
              it.path = path0[vi * ntangs + ti] + static_cast<int>(gr);
              int out = 0, nl = 0, ov = -2;
              for (int s = 0; s < 2 * kZChains; ++s) {
                it.slot[s] = make_int2(-1, -1);
                it.owner[s] = static_cast<int8_t>(s);
              }
              for (size_t m = 0; m < cm.size(); ++m) {
                const int b = (vi * nsegs + cm[m]) * ntangs + ti;
                const ProjBinDev& pb = h.h_bins[b];
                int seen[2] = {0, 0};
                for (int l = 0; l < pb.num_lines; ++l) {
                  const LineDev& L = lines[pb.first_line + l];
                  if ((L.flags & 7) != T) continue;
                  const int d = (L.flags & 8) ? 1 : 0;
                  if (seen[d]++ != k) continue;
                  const int s = 2 * static_cast<int>(m) + d;
                  it.slot[s] = make_int2(pb.first_line + l, b);
                  bool own = true;
                  for (size_t m2 = 0; m2 < m; ++m2)
                    if (cm[m2] == cm[m]) {
                      it.owner[s] = static_cast<int8_t>(2 * m2 + d);
                      own = false;
                      break;
                    }
                  if (own) {
                    out += g.nax(L.seg);
                    ++nl;
                  }
                  ov = ov == -2 ? L.view : ov == L.view ? ov : -1;
                }
              }
              if (nl == 0) break;
              // the back projection's buffer: every line's data with the zeros around them that its planes reach, the zeros
              // between two lines shared; first the zeros of the slots without a line
              const int nplanes = planes;
              int bend = 0, bzeros = 0;
              for (int s = 0; s < 2 * kZChains; ++s) {
                if (it.slot[s].x >= 0) continue;
                const size_t m = static_cast<size_t>(s / 2);
                const int z0 = ends[0][m], up = ends[1][m] - z0;
                // zt = z0 (slot 2 m) or -z0 at the first column (setup_slots), one up or down an event: read from `up`
                // down to 0, or from 0 up
                it.boff[s] = static_cast<int16_t>(s % 2 ? -z0 : z0 + up);
                bzeros = std::max(bzeros, nplanes + up);
              }
              for (size_t m = 0; m < cm.size(); ++m)
                for (int d = 0; d < 2; ++d) {
                  const int s = 2 * static_cast<int>(m) + d;
                  if (it.slot[s].x < 0 || it.owner[s] != s) continue;
                  const LineDev& L = lines[it.slot[s].x];
                  const int reach = (g.nax(L.seg) - 1) * g.npa(L.seg);
                  int lo = 0, hi = 0;  // planes read below datum 0 and above the last one, by any chain of the line
                  for (size_t m2 = m; m2 < cm.size(); ++m2) {
                    if (cm[m2] != cm[m]) continue;
                    for (int zr : {ends[0][m2], ends[1][m2]}) {
                      const int zt = (L.flags & 8) ? L.q + 512 - p.min_z - zr : zr - 512 - p.min_z;
                      lo = std::max(lo, zt);
                      hi = std::max(hi, nplanes - 1 - zt - reach);
                    }
                  }
                  const int at = bend + std::max(bzeros, lo);
                  if (at + reach + hi > 30000) return false;
                  it.boff[s] = static_cast<int16_t>(at);
                  bend = at + reach + 1;
                  bzeros = hi;
                }
              for (int s = 0; s < 2 * kZChains; ++s)
                if (it.owner[s] != s) it.boff[s] = it.boff[static_cast<int>(it.owner[s])];
              z.max_back = std::max(z.max_back, bend + bzeros);
              z.max_out = std::max(z.max_out, out);
              items.push_back(it);
              item_view.push_back(bviews[vi]);
              item_lead.push_back(!led[ti]);
              item_block.push_back(t0 / kZWarps);
              led[ti] = 1;
              item_out_view.push_back(ov);
              PathItemDev pi{};
              pi.ncols = it.nrec;
              pi.num_lines = nl;
              path_items.push_back(pi);
            }
            // every column inside the image under T
            const int swap = T & 1, sx = (T & 2) ? -1 : 1, sy = (T & 4) ? -1 : 1;
            for (const ZRec& r : G.recs[gr]) {
              const int x = static_cast<int>(r.xy & 2047u) - 1024, y = static_cast<int>(r.xy >> 11) - 1024;
              const int xi = (swap ? y : x) * sx - p.min_x, yi = (swap ? x : y) * sy - p.min_y;
              if (xi < 0 || xi >= p.nx || yi < 0 || yi >= p.ny) return false;
            }
          }
      }
  if (items.empty()) return false;
  if (kZWarps * (std::max(z.max_out, z.max_back) * 4 + 8192) > 200 * 1024) return false;

  h.z_recs.alloc(static_cast<size_t>(nrecs) + 2 * kZBatch);  // batches are fetched whole
  std::vector<ZRec> all(static_cast<size_t>(nrecs) + 2 * kZBatch);
  for (int gi = 0; gi < ngroups; ++gi) {
    size_t o = static_cast<size_t>(base[gi]);
    for (auto& r : groups[gi].recs) {
      std::copy(r.begin(), r.end(), all.begin() + o);
      o += r.size();
      std::vector<ZRec>().swap(r);
    }
  }
  h.z_recs.upload(all, h.stream);
  h.z_items.upload(items, h.stream);
  h.z_planes.upload(sixteenths, h.stream);
  h.dev_status.alloc(1);
  ck(cudaMemsetAsync(h.dev_status.p, 0, sizeof(unsigned), h.stream), "memset");
  ck(cudaStreamSynchronize(h.stream), "path tables");
  int64_t ngrp = 0;
  for (const ZPath& G : groups) ngrp += static_cast<int64_t>(G.recs.size());
  const size_t ng_most = most_groups(groups);
  z.copies = ng_most == 1 ? 1 : ng_most <= 3 ? 2 : 4;
  z.mean_rec = static_cast<int>(nrecs / std::max<int64_t>(1, ngrp));
  z.recs = h.z_recs.p;
  z.items = h.z_items.p;
  z.sixteenths = h.z_planes.p;
  h.zparams = z;
  h.z_work.alloc(items.size());
  h.z_partials.alloc(items.size());
  h.h_item_lead = std::move(item_lead);
  h.h_item_block = std::move(item_block);
  h.h_item_view = std::move(item_view);
  h.h_item_out_view = std::move(item_out_view);
  h.h_path_items = std::move(path_items);
  h.paths_view_split =
      std::find(h.h_item_out_view.begin(), h.h_item_out_view.end(), -1) == h.h_item_out_view.end();
  // padded images and image sums come from a pool of the handle's own, in stream order: calls on several streams or threads
  // have their own.  The pool keeps what one call needs (kPadLimit, or one image's where that is more); what calls side by
  // side had beyond that goes back to the device at the next synchronisation, and all of it with the handle.
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = h.device;
  ck(cudaMemPoolCreate(&h.z_pool, &props), "cudaMemPoolCreate");
  uint64_t keep = sizeof(float) * std::max<uint64_t>(kPadLimit, static_cast<uint64_t>(padded) * z.copies);
  ck(cudaMemPoolSetAttribute(h.z_pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute");
  h.use_paths = h.use_z = true;
  return true;
}

namespace {

// Warps that share each of n items with paths of `rec` records, `resident` warps on the GPU at a time.  A call with few items
// leaves most of the GPU idle while each warp walks its path, so the warps are doubled while what they add runs beside the
// others (m: warps wanted over resident ones) and a part still has enough records for its set-up (list, item, lines, the first
// records: about what 20 records cost).  Measured, us, one image: forward 1 / 2 / 4 / 8 / 16 warps an item, 62 items of 152
// records 42 / 22 / 13.5 / 10.4 / 10.3; 438 of 83 30 / 18 / 12.4 / 10.4 / 16.5; 630 of 146 37 / 21 / 13.5 / 16.5 / 23; 1972 of 173
// 45 / 27 / 27 / 37; 3423 of 391 97 / 72 / 66 / 80; 4158 of 68 27 / 29 / 33; 15892 of 355 282 / 268 / 288; 49350 of 49 196 / 243.
// Back: 243 of 241 70 / 41 / 27 / 19 / 16.5; 833 of 175 53 / 33 / 24 / 21 / 25; 2618 of 65 28 / 20 / 22 / 28; 4158 of 68 26 / 27 / 30.
// `far`: also worth it where each warp's own latency is what bounds it (long paths, few registers); `heavy`: not for short parts
// where a warp's set-up and sums are long (four planes a lane, 1764 items of 39 records: 34 / 41)
int sharing_warps(int n, int rec, int resident, bool far, bool heavy) {
  int parts = 1;
  while (parts < kZManyWarps) {
    const int next = 2 * parts;
    const double m = static_cast<double>(n) * next / resident;
    const int r = rec / next;
    const bool ok = m <= 1.0                ? r >= 5
                    : next >= 8             ? false
                    : m <= 1.5              ? r >= (heavy ? 30 : 16)
                    : m <= 2.3              ? r >= 30
                    : far && m <= 4.0       ? r >= 90
                    : far && m <= 12.0      ? next == 2 && r >= 125
                                            : false;
    if (!ok) break;
    parts = next;
  }
  return parts;
}

constexpr int kSharedLimit = 200 * 1024;

}  // namespace

// Segments and folds are there for the rounding: a line's sum takes the products of 16 (fold) columns at a time and starts again
// at every segment, so that no sum is long.  Error of the forward projection against 64 bits (2-norm, one subset), with one sum
// a path in products of 32 columns / as here: 172 x 172 x 127, 64 rings, span 11 2.5e-7 / 5.9e-8; 344 x 344 x 127 2.4e-7 /
// 1.1e-7; 171 x 171 x 63 9.7e-8 / 6.1e-8; 101 x 92 x 23 7.2e-8 / 4.9e-8; short paths (34 x 34 x 41) 7.2e-8 / 4.8e-8 with 8 columns
// (16: 5.2e-8).  The column-staged kernels, which add the sums of 58 columns by eight warps: 1.0e-7, 2.1e-7, 6.9e-8, 5.7e-8,
// 5.3e-8.  Steep paths of medium length need four segments (two: 1.2e-7 in the first case).  A segment costs 1 to 2 % of the time
// (all clinical lines: 4.41 ms with one segment in products of 32, 4.53 as here, 4.71 with four segments), 7 % on paths of 123
// records.
ZSplit z_split(const b200rt_projector& h, int n) {
  const ZParams& z = h.zparams;
  ZSplit sp;
  sp.parts = sharing_warps(n, z.mean_rec, z_resident_warps(z, true), z.planes == 1 || (z.planes == 2 && z.nm == 4),
                           z.planes == 4);
  // 16 warps a CTA: two CTAs an SM where the registers allow it, one elsewhere
  if (sp.parts == 16 && n > 148 && (z.nm > 4 || z.planes == 4)) sp.parts = 8;
  while (sp.parts > 1 && std::max(sp.parts, kZWarps) * z_forward_smem(z, 2) > kSharedLimit) sp.parts /= 2;
  sp.segs = std::max(sp.parts, z.planes == 4 && z.mean_rec >= 128 && z.mean_rec < 256 ? 4 : 2);
  sp.fold = z.planes > 1 && z.mean_rec < 64 ? 1 : 2;
  return sp;
}
int z_back_parts(const b200rt_projector& h, int n, int images) {
  const int items = static_cast<int>(std::min<int64_t>(static_cast<int64_t>(n) * images, 1 << 30));
  return sharing_warps(items, h.zparams.mean_rec, z_resident_warps(h.zparams, false), h.zparams.planes == 1, false);
}

// Whether a call is worth padded images, which save instructions and cache lines per column walked and cost a pass over the
// image each way, the launches and an allocation.  Forward, one warp an item, padded / plain, us: clinical, one of 21 subsets (4140
// items of 373 records, 118336 columns) 291 / 298, all lines 4694 / 5290; 4117 items of 218 records, 62500 columns 166 / 169;
// 742 of 245, 109392 columns 112 / 119 and shared 56 / 39; two planes a lane: 41356 of 181, 29241 columns 606 / 623; 9312 of
// 259, 111556 columns 188 / 177; 4032 of 145, 15776 columns 73 / 69.
bool pad_forward(const b200rt_projector& h, int n, int batch) {
  const ZParams& z = h.zparams;
  const int64_t ncols = static_cast<int64_t>(h.params.ny) * h.params.nx * batch;
  const int64_t walked = static_cast<int64_t>(n) * z.mean_rec * batch;
  return z.planes == 4 ? walked >= 200000 + 8 * ncols : z.planes == 2 && walked >= 1000000 + 20 * ncols;
}
// Back, where the planes fill the lanes (a plain column has a reduction for every 32 planes or part of them, a padded one for
// all of the lanes' planes: 79 of 128 planes 1020 / 775 us).  127 of 128 planes: all clinical lines 3635 / 4044, one of 21 subsets 273 /
// 275; 4950 items of 110 records, 15876 columns 76 / 64; 28050 of 31, 1296 columns 120 / 135; 63 of 64 planes: 41356 of 181 415 /
// 457; 9312 of 259, 111556 columns 153 / 142.
bool pad_back(const b200rt_projector& h, int n, int batch) {
  const ZParams& z = h.zparams;
  const int64_t ncols = static_cast<int64_t>(h.params.ny) * h.params.nx * batch;
  const int64_t walked = static_cast<int64_t>(n) * z.mean_rec * batch;
  return z.planes > 1 && 4 * h.params.nz > 3 * z_stride(z) && walked >= 500000 + 20 * ncols;
}

namespace {

// Device memory of one call (given back to the handle's pool in stream order), or null: the kernels then take the plain image.
// None while the stream is captured: allocation nodes would keep a graph from being instantiated twice, cloned or a child.
float* pool_alloc(b200rt_projector& h, size_t n, cudaStream_t st) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) cudaGetLastError();
  if (capturing != cudaStreamCaptureStatusNone) return nullptr;
  float* p = nullptr;
  if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p), n * sizeof(float), h.z_pool, st) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
  return p;
}
struct PoolBuf {
  float* p;
  cudaStream_t st;
  PoolBuf(b200rt_projector& h, size_t n, cudaStream_t s) : p(pool_alloc(h, n, s)), st(s) {}
  PoolBuf(const PoolBuf&) = delete;
  ~PoolBuf() {
    if (p) cudaFreeAsync(p, st);
  }
};

}  // namespace

void forward_paths(b200rt_projector& h, const int* list, int n, const float* images, int64_t img_stride, float* out,
                   int64_t out_stride, int batch, cudaStream_t st, const FwdEpilogue* ep, bool may_alloc, int n_call) {
  if (n <= 0 || batch <= 0) return;
  if (!h.use_z) {
    ck(launch_forward_paths_batch(h.params, h.pparams, list, n, images, img_stride, out, out_stride, batch, st, ep),
       "forward projection");
    return;
  }
  const ZParams& z = h.zparams;
  const ZSplit sp = z_split(h, n_call >= 0 ? n_call : n);
  if (!may_alloc || sp.parts > 1 || !pad_forward(h, n_call >= 0 ? n_call : n, batch)) {
    ck(launch_forward_z(h.params, z, list, n, sp, images, img_stride, 0, out, out_stride, batch, st, ep), "forward projection");
    return;
  }
  const int64_t ncols = static_cast<int64_t>(h.params.ny) * h.params.nx, per = ncols * z_stride(z);
  const int step = static_cast<int>(std::min<int64_t>(batch, std::max<int64_t>(1, static_cast<int64_t>(kPadLimit) / per)));
  PoolBuf pad(h, static_cast<size_t>(per) * step, st);
  for (int b = 0; b < batch; b += step) {
    const int nb = std::min(step, batch - b);
    FwdEpilogue e{};
    if (ep) {
      e = *ep;
      e.y += b * e.y_stride;
      if (e.add) e.add += b * e.add_stride;
      if (e.mult) e.mult += b * e.mult_stride;
      if (e.small_value) e.small_value += b * e.sv_stride;
      if (e.partials) e.partials += static_cast<int64_t>(b) * n;
    }
    const float* x = images + b * img_stride;
    float* o = out ? out + b * out_stride : nullptr;
    if (pad.p) {
      ck(launch_pad_image(x, img_stride, pad.p, per, ncols, h.params.nz, z_stride(z), nb, st), "image planes");
      ck(launch_forward_z(h.params, z, list, n, sp, pad.p, per, 1, o, out_stride, nb, st, &e), "forward projection");
    } else {
      ck(launch_forward_z(h.params, z, list, n, sp, x, img_stride, 0, o, out_stride, nb, st, &e), "forward projection");
    }
  }
}

// The order of a back projection's items.  As built, the paths through the middle come first: the longest, and the ones that add
// most to a voxel, whose float sum is then large, and rounds coarsely, while the many small values of the outer paths come
// (images of projected phantoms: 7 to 17 % more rounding error than in an order without a preference).  Where the items run in
// many waves, the blocks of tangential positions take turns (bit-reversed) up to the outer quarter, whose short paths stay last
// to even out the end (all clinical lines 3.64 ms in either order; 24102 items of 162 records 175 / 188 us).  Error against the
// fixed-point sums, longest first / in turns, over the column-staged kernels': 1.09 / 1.03 (344 x 344 x 127), 1.10 / 1.02 (171 x 171 x
// 63), 1.17 / 1.03 (332 x 336 x 11).  Calls of few waves, which have few terms a voxel, keep the longest first (4158 items of 68
// records: 26 us, in turns 30).
void back_order(const b200rt_projector& h, std::vector<int>& items) {
  if (!h.use_z || items.empty() || static_cast<int64_t>(items.size()) < 4 * z_resident_warps(h.zparams, false)) return;
  const int blocks = *std::max_element(h.h_item_block.begin(), h.h_item_block.end()) + 1, inner = blocks - blocks / 4;
  int bits = 0;
  while (1 << bits < inner) ++bits;
  std::vector<int> turn(blocks);
  for (int b = 0; b < blocks; ++b) {
    turn[b] = b < inner ? 0 : (1 << bits) + b;
    for (int k = 0; b < inner && k < bits; ++k) turn[b] |= (b >> k & 1) << (bits - 1 - k);
  }
  std::stable_sort(items.begin(), items.end(),
                   [&](int a, int b) { return turn[h.h_item_block[a]] < turn[h.h_item_block[b]]; });
}

// Memory of the call's own where its reductions go to padded columns or to several images, which collect() adds up.
// images: at a time.
BackSums::BackSums(b200rt_projector& h, int n, int images, cudaStream_t st) : h_(h), st_(st) {
  if (!h.use_z || n <= 0) return;
  const ZParams& z = h.zparams;
  const bool padded = pad_back(h, n, images);
  if (!padded && z.copies == 1) return;
  const int64_t ncols = static_cast<int64_t>(h.params.ny) * h.params.nx;
  stride_ = padded ? z_stride(z) : h.params.nz;
  per_ = z_image_floats(ncols, stride_) * z.copies;
  step_ = static_cast<int>(std::min<int64_t>(images, std::max<int64_t>(1, static_cast<int64_t>(kPadLimit) / per_)));
  sums_ = pool_alloc(h, static_cast<size_t>(per_) * step_, st);
}
BackSums::~BackSums() {
  if (sums_) cudaFreeAsync(sums_, st_);
}
void BackSums::clear(int images) {
  ck(cudaMemsetAsync(sums_, 0, sizeof(float) * per_ * images, st_), "memset");
}
void BackSums::add(const int* list, int n, const float* pd, int64_t pd_stride, int images, int zero_ends) {
  if (n > 0)
    ck(launch_back_z(h_.params, h_.zparams, list, n, z_back_parts(h_, n, images), pd, pd_stride, sums_, per_, h_.zparams.copies,
                     stride_ != h_.params.nz, images, st_, zero_ends),
       "back projection");
}
void BackSums::collect(float* images, int64_t img_stride, int n) {
  ck(launch_collect_images(sums_, per_, h_.zparams.copies, images, img_stride,
                           static_cast<int64_t>(h_.params.ny) * h_.params.nx, h_.params.nz, stride_, n, st_),
     "image sums");
}

// image b (overwritten) = the back projection of the list's items from projection data b
void back_paths(b200rt_projector& h, const int* list, int n, const float* pd, int64_t pd_stride, float* images,
                int64_t img_stride, int batch, cudaStream_t st, int zero_ends) {
  const int64_t ni = h.geo->image_size();
  BackSums sums(h, n, batch, st);
  if (sums.own()) {
    for (int b = 0; b < batch; b += sums.step()) {
      const int nb = std::min(sums.step(), batch - b);
      sums.clear(nb);
      sums.add(list, n, pd ? pd + b * pd_stride : nullptr, pd_stride, nb, zero_ends);
      sums.collect(images + b * img_stride, img_stride, nb);
    }
    return;
  }
  for (int b = 0; b < batch; ++b) ck(cudaMemsetAsync(images + b * img_stride, 0, sizeof(float) * ni, st), "memset");
  add_back_paths(h, list, n, pd, pd_stride, images, img_stride, batch, st, zero_ends);
}

// the same, added to the images
void add_back_paths(b200rt_projector& h, const int* list, int n, const float* pd, int64_t pd_stride, float* images,
                    int64_t img_stride, int batch, cudaStream_t st, int zero_ends) {
  if (n <= 0) return;
  if (h.use_z)
    ck(launch_back_z(h.params, h.zparams, list, n, z_back_parts(h, n, batch), pd, pd_stride, images, img_stride, 1, 0, batch, st,
                     zero_ends),
       "back projection");
  else
    ck(launch_back_paths_atomic_batch(h.params, h.pparams, list, n, pd, pd_stride, images, img_stride, batch, st, zero_ends),
       "back projection");
}

void back_paths_fixed(b200rt_projector& h, const int* list, int n, const float* pd, unsigned long long* acc,
                      const double* scale, cudaStream_t st, int zero_ends) {
  if (h.use_z)
    ck(launch_back_z_fixed(h.params, h.zparams, list, n, z_back_parts(h, n, 1), pd, acc, scale, st, zero_ends), "back projection");
  else
    ck(launch_back_paths_fixed(h.params, h.pparams, list, n, pd, acc, scale, st, zero_ends), "back projection");
}

}  // namespace capi
