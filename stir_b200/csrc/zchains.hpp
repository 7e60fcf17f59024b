// Chains and records of one transaxial path (zframe.hpp), on the host.
#pragma once

#include <vector>

#include "zframe.hpp"

namespace b200 {

// A member of a path: the basic bin of one segment, with its row and its related lines.
struct ZMember {
  const RowElem* row;
  int row_len;
  const LineDev* lines;
  int num_lines;
};

// What the edge events depend on besides the rows (per segment: index segment + S).
struct ZPathLines {
  int S, min_z;
  int planes;  // planes of a warp: 32, 64 or 128
  std::vector<int> nax, npa;
};

struct ZPath {
  int total = 0, most = 0;                           // chains of the path, most of one member
  int columns = 0, elements = 0;                     // of all members
  std::vector<std::vector<ZRec>> recs;               // per chain group
  std::vector<std::vector<int>> chain_member;        // per chain group: the member of every chain
  std::vector<ZPlanes> planes;                       // per chain group
  bool ok = true;
};

// Counts the path's chains and, with cap > 0, builds the records of groups of at most cap chains (cap <= kZChains).  A path
// with a member of more than cap chains gets no records: `most` tells.
void build_path(const std::vector<ZMember>& members, const ZPathLines& fit, int cap, ZPath& path);

}  // namespace b200
