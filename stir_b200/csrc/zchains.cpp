// Cuts the rows of a path's members into chains and lays out the records of its chain groups.
#include "zchains.hpp"

#include <algorithm>
#include <utility>

namespace b200 {

namespace {

struct Elem {
  int z;
  float v;
};

// a chain of one member
struct Chain {
  int member;
  int cur, z0;  // stored plane (z + 512) now and at the first column
};

// An event from stored plane zr to zr + 1 of a line (zt: plane of axial position 0 before it; dz: its move, 1 or -1):
// the axial position that leaves the planes [0, planes), or -1, and whether one enters
void edge_event(int zt, int dz, int nax, int npa, int planes, int& leave, bool& enters) {
  auto at = [&](int d) { return d >= 0 && d % npa == 0 && d / npa < nax ? d / npa : -1; };
  leave = dz > 0 ? at(planes - 1 - zt) : at(-zt);
  enters = (dz > 0 ? at(-(zt + 1)) : at(planes - 1 - (zt - 1))) >= 0;
}

}  // namespace

void build_path(const std::vector<ZMember>& members, const ZPathLines& fit, int cap, ZPath& path) {
  path = ZPath{};
  const int nsegs = static_cast<int>(members.size());
  std::vector<uint32_t> keys;
  std::vector<int> order;
  for (const ZMember& pb : members)
    for (int k = 0; k < pb.row_len; ++k) keys.push_back(pb.row[k].zyx & 0x3fffffu);  // x, y bits
  std::sort(keys.begin(), keys.end());
  keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
  const int ncols = static_cast<int>(keys.size());
  // every member's elements by column, planes ascending within a column
  std::vector<std::vector<std::vector<Elem>>> el(nsegs, std::vector<std::vector<Elem>>(ncols));
  for (int si = 0; si < nsegs; ++si) {
    const ZMember& pb = members[si];
    for (int k = 0; k < pb.row_len; ++k) {
      const RowElem e = pb.row[k];
      const size_t c = std::lower_bound(keys.begin(), keys.end(), e.zyx & 0x3fffffu) - keys.begin();
      el[si][c].push_back(Elem{static_cast<int>(e.zyx >> 22), e.v});
    }
    for (auto& v : el[si])
      std::stable_sort(v.begin(), v.end(), [](const Elem& a, const Elem& b) { return a.z < b.z; });
  }
  // the columns along the path: a ray steps in x or in y, so x + y (or x - y) orders them; away from the end where
  // the steepest member's planes are higher
  double mx = 0, my = 0, cov = 0;
  for (uint32_t k : keys) mx += k & 2047u, my += k >> 11;
  mx /= ncols, my /= ncols;
  for (uint32_t k : keys) cov += ((k & 2047u) - mx) * ((k >> 11) - my);
  const int sy = cov >= 0 ? 1 : -1;
  auto along = [&](int c) { return static_cast<int>(keys[c] & 2047u) + sy * static_cast<int>(keys[c] >> 11); };
  order.resize(ncols);
  for (int c = 0; c < ncols; ++c) order[c] = c;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return along(a) < along(b); });
  {
    double s0 = 0, s1 = 0, n0 = 0, n1 = 0;  // mean plane of the last member in the two halves
    for (int i = 0; i < ncols; ++i)
      for (const Elem& e : el[nsegs - 1][order[i]]) (i < ncols / 2 ? s0 : s1) += e.z, (i < ncols / 2 ? n0 : n1) += 1;
    if (n0 > 0 && n1 > 0 && s0 / n0 > s1 / n1) std::reverse(order.begin(), order.end());
  }
  // chains: each element goes to the member's chain with the highest plane not above it (one element per plane)
  struct Link {
    int chain;
    Elem e;
  };
  std::vector<std::vector<Chain>> chains(nsegs);
  std::vector<std::vector<std::vector<Link>>> links(nsegs, std::vector<std::vector<Link>>(ncols));
  int total = 0, most = 0;
  for (int si = 0; si < nsegs; ++si) {
    for (int i = 0; i < ncols; ++i)
      for (const Elem& e : el[si][order[i]]) {
        int best = -1;
        for (int c = 0; c < static_cast<int>(chains[si].size()); ++c) {
          const int cz = chains[si][c].cur;
          // a chain that is at this plane already in this column has taken the element of a merged ray
          if (cz <= e.z && (best < 0 || cz > chains[si][best].cur)) best = c;
        }
        if (best < 0) {
          best = static_cast<int>(chains[si].size());
          chains[si].push_back(Chain{si, e.z, e.z});
        }
        chains[si][best].cur = e.z;
        links[si][i].push_back(Link{best, e});
      }
    // lines of an empty row are projected too (to 0): a chain without elements
    if (chains[si].empty()) chains[si].push_back(Chain{si, 512, 512});
    total += static_cast<int>(chains[si].size());
    most = std::max(most, static_cast<int>(chains[si].size()));
  }
  path.total = total;
  path.most = most;
  path.columns = ncols;
  for (const ZMember& pb : members) path.elements += pb.row_len;
  if (cap == 0 || most > cap) return;  // a record has room for cap chains
  // members into groups of at most cap chains, in order
  std::vector<std::vector<int>> parts;
  int fill = cap + 1;
  for (int si = 0; si < nsegs; ++si) {
    const int n = static_cast<int>(chains[si].size());
    if (fill + n > cap) {
      parts.emplace_back();
      fill = 0;
    }
    parts.back().push_back(si);
    fill += n;
  }
  for (const auto& mem : parts) {
    std::vector<int> cm, cz0, first(nsegs, 0);
    for (int si : mem) {
      first[si] = static_cast<int>(cm.size());
      for (const Chain& c : chains[si]) {
        cm.push_back(si);
        cz0.push_back(c.z0);
      }
    }
    const int nc = static_cast<int>(cm.size());
    std::vector<int> cur = cz0;
    std::vector<ZRec> recs;
    for (int i = 0; i < ncols; ++i) {
      const size_t head = recs.size();
      auto fresh = [&]() {
        ZRec r{};
        r.xy = keys[order[i]];
        recs.push_back(r);
      };
      fresh();
      for (int si : mem)
        for (const Link& l : links[si][i]) {
          const int m = first[si] + l.chain;
          // up to the element's plane: one event a record, in further records of the column where one is not enough
          size_t k = head;
          while (cur[m] < l.e.z) {
            while (k < recs.size() && (recs[k].op & (1u << m))) ++k;
            if (k == recs.size()) fresh();
            recs[k].op |= 1u << m;
            // what leaves and enters: the same for every line of the member in one z orientation (checked)
            const ZMember& pb = members[si];
            int leave[2] = {-2, -2};
            for (int q = 0; q < pb.num_lines; ++q) {
              const LineDev& L = pb.lines[q];
              const int d = (L.flags & 8) ? 1 : 0;
              const int zt = d ? L.q + 512 - fit.min_z - cur[m] : cur[m] - 512 - fit.min_z;
              int out = -1;
              bool in = false;
              edge_event(zt, d ? -1 : 1, fit.nax[L.seg + fit.S], fit.npa[L.seg + fit.S], fit.planes, out, in);
              if (leave[d] != -2 && leave[d] != out) path.ok = false;
              leave[d] = out;
              if (out >= 0 || in) recs[k].op |= 1u << (6 + m);
            }
            recs[k].leave[m] = static_cast<int32_t>((static_cast<uint32_t>(std::max(leave[1], -1)) << 16) |
                                                    (static_cast<uint32_t>(std::max(leave[0], -1)) & 0xffffu));
            ++cur[m];
          }
          // the element: before the column's events at the chain's first plane here, after the event otherwise
          bool placed = false;
          for (size_t q = recs.size(); q-- > head;)
            if (recs[q].op & (1u << m)) {
              recs[q].w2[m] += l.e.v;
              placed = true;
              break;
            }
          if (!placed) recs[head].w1[2 * m] += l.e.v;
        }
    }
    while (recs.size() % 4) {  // the kernels take four records at a time
      ZRec r{};
      r.xy = recs.back().xy;
      recs.push_back(r);
    }
    for (ZRec& r : recs) {
      for (int m = 0; m < nc; ++m) {
        if (r.w1[2 * m] == 0.f) r.op |= kZGuard;
        r.w1[2 * m + 1] = r.w1[2 * m];
        if ((r.op >> m & 1u) && r.w2[m] == 0.f) r.op |= 1u << (6 + m);
      }
    }
    // the chains' planes where the kernels cut the batches
    ZPlanes planes;
    const int nrec = static_cast<int>(recs.size()), nb = (nrec + kZBatch - 1) / kZBatch;
    for (int m = 0; m < 8; ++m)
      for (int q = 0, r = 0, zr = m < nc ? cz0[m] : 512; q <= kZSixteenths; ++q) {
        for (; r < std::min(nb * q / kZSixteenths * kZBatch, nrec); ++r) zr += m < nc ? recs[r].op >> m & 1u : 0;
        planes.z[q][m] = static_cast<int16_t>(zr);
      }
    path.planes.push_back(planes);
    path.recs.push_back(std::move(recs));
    path.chain_member.push_back(std::move(cm));
  }
}

}  // namespace b200
