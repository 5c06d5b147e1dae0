"""Task order of the all-slices kernel (msx_stream.cuh) on the CPU: every row and
column tile of every slice appears once, and the counter value that a task waits
for is exactly what the earlier tasks of the order will have added, so that the
first unfinished task can always run."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "msx_stream.cuh"
#include <cstdio>
#include <vector>
using namespace msx;
int main() {
  for (int wpt : {2, 4, 8})
    for (int G : {1, 2, 3, 7, 8, 9, 16, 21})
      for (int tiles_x : {1, 5, 22})
        for (int slices : {1, 2, 5})
          for (int last : {0, 1}) {
            const StreamShape sh{G, wpt, 16 / wpt, 64, tiles_x, slices, last};
            std::vector<int> row(sh.chunks(), 0), col(sh.chunks(), 0), seen(slices * sh.per_slice(), 0);
            for (long long u = 0; u < sh.tasks(); ++u) {
              const StreamTask t = stream_task(sh, u);
              if (t.slice < 0 || t.slice >= slices || t.chunk < 0 || t.chunk >= sh.chunks()) return printf("range\n"), 1;
              if (t.row ? (t.a < 0 || t.a + sh.ypt > sh.Ny || t.a % sh.ypt) : (t.a < 0 || t.a >= G || t.b < 0 ||
                          t.b >= tiles_x || t.a / wpt != t.chunk)) return printf("tile\n"), 1;
              if (!t.row && !last && t.slice == slices - 1) return printf("last column pass\n"), 1;
              int& c = t.row ? col[t.chunk] : row[t.chunk];
              if (t.need != c) return printf("need %d has %d\n", t.need, c), 1;  // all that it waits for comes before it
              const int at = t.slice * sh.per_slice() + (t.row ? t.chunk * sh.row_tiles() + t.a / sh.ypt
                                                               : sh.chunks() * sh.row_tiles() + t.a * tiles_x + t.b);
              if (seen[at]++) return printf("twice\n"), 1;
              const int4 d = task_desc(sh, u);
              if ((d.x & 1) != (t.row ? 1 : 0) || (d.x >> 1) != t.slice || d.y != t.chunk || d.z != t.a || d.w != t.b)
                return printf("descriptor\n"), 1;
              (t.row ? row : col)[t.chunk] += 1;
            }
            for (size_t i = 0; i < seen.size(); ++i) {
              const bool wanted = last || i < (size_t)(slices - 1) * sh.per_slice() + sh.chunks() * sh.row_tiles();
              if (seen[i] != (wanted ? 1 : 0)) return printf("missing\n"), 1;
            }
          }
  return 0;
}
'''


def test_task_order(tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not found')
    src, exe = tmp_path / 'tasks.cu', tmp_path / 'tasks'
    src.write_text(SRC)
    r = subprocess.run([nvcc, '-std=c++17', '-O1', '-w', '-I', os.path.join(ROOT, 'namsa_gb300', 'csrc'), str(src),
                        '-o', str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
