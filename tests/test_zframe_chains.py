"""The chains of a path (csrc/zchains.cpp) on the host: a member with more chains than a record has room for gets no records,
whatever the other paths of the geometry looked like when the chains a warp takes were chosen."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stir_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>

#include "zchains.hpp"

using namespace b200;

// two members: planes falling along the path by one a column (a chain each), and rising (one chain)
int main(int argc, char** argv) {
  const int falling = std::atoi(argv[1]), cap = std::atoi(argv[2]);
  std::vector<RowElem> a, b;
  for (int x = 0; x < falling; ++x) {
    a.push_back(RowElem{pack_zyx(falling - x, 0, x), 1.f});
    b.push_back(RowElem{pack_zyx(x, 0, x), 1.f});
  }
  LineDev line{};
  ZPathLines fit;
  fit.S = 0;
  fit.min_z = 0;
  fit.planes = 32;
  fit.nax = {8};
  fit.npa = {1};
  const std::vector<ZMember> members = {{a.data(), falling, &line, 1}, {b.data(), falling, &line, 1}};
  ZPath path;
  build_path(members, fit, cap, path);
  size_t records = 0;
  for (const auto& g : path.recs) records += g.size();
  std::printf("%d %d %zu %d\n", path.total, path.most, records, path.ok);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx, cuda = shutil.which("g++"), "/usr/local/cuda/include"
    if cxx is None or not os.path.isdir(cuda):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("chains")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "chains")
    # the sanitizers end the program at a write outside a record
    subprocess.run([cxx, "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all", "-I", CSRC,
                    "-isystem", cuda, str(d / "main.cpp"), os.path.join(CSRC, "zchains.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("falling,cap", [(4, 4), (5, 4), (6, 6), (7, 6), (10, 6), (20, 6), (20, 4)])
def test_members_of_many_chains(program, falling, cap):
    r = subprocess.run([program, str(falling), str(cap)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    total, most, records, ok = (int(v) for v in r.stdout.split())
    assert (total, most, ok) == (falling + 1, falling, 1)
    assert (records > 0) == (falling <= cap)
