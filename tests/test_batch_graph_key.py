"""CPU: captured bucket graphs are kept per device and shape."""
import os
import subprocess

from conftest import ROOT

HARNESS = r"""
#include <map>
#include "gl_batch_plan.h"
int main() {
  std::map<gl_bucket_key, int> graphs;
  for (int device : {1, 0, 7})
    for (uint64_t len : {8, 16})
      for (int dir : {0, 1}) graphs[{device, {{len, dir}, {4096, 0}}}] = 100 * device + (int)len + dir;
  bool ok = graphs.size() == 12 && !graphs.count({2, {{8, 0}, {4096, 0}}}) && !graphs.count({0, {{8, 0}}});
  for (auto &g : graphs)
    ok = ok && g.second == 100 * g.first.device + (int)g.first.sig[0].first + g.first.sig[0].second;
  return ok ? 0 : 1;
}
"""


def test_graphs_of_two_devices_are_apart(tmp_path):
    (tmp_path / "k.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"),
                    str(tmp_path / "k.cpp"), "-o", str(tmp_path / "k")], check=True)
    assert subprocess.run([str(tmp_path / "k")]).returncode == 0
    src = open(os.path.join(ROOT, "goldilocks_gb300", "csrc", "gl_batch.cu")).read()
    assert "std::map<gl_bucket_key, std::unique_ptr<bucket_graph>> g_graphs" in src
