"""Functions of the D2Q9 cut-link kernel (csrc/d2q9.cu), compiled from that file for the CPU.

band_kernel stages segment_of(w, j) for every slot of every solid, used or not. The reads must stay
inside the world's vertex array [n_objects][max_segments][2]: here it ends at an unreadable page.

A cell's candidate segments are noted in any order. The cut found from them must be the one that
get_cutcell finds over all segments in their order.
"""
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.join(HERE, "..", "openhomelbm_b200", "csrc", "d2q9.cu")

PRELUDE = """
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/mman.h>
#define __device__
#define __forceinline__ inline
struct float4 { float x, y, z, w; };
static inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
struct World {
  int n_objects, max_segments, nx;
  const int *line_num;
  const float *tf, *position, *scale, *max_radius;
};
"""


def function(name):
    """The text of a device function of d2q9.cu ("" if there is none of that name)."""
    src = open(SOURCE).read()
    m = re.search(r"^__device__[^\n;]*\b%s\(.*?^}\n" % name, src, re.S | re.M)
    return m.group(0) if m else ""


def run(tmp_path, body, *args, flags=()):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PRELUDE + body)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", *flags, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True)


MAIN = """
int main(int argc, char** argv) {
  const int max_segments = atoi(argv[1]), n = argc - 2;
  int line_num[64];
  for (int s = 0; s < n; ++s) line_num[s] = atoi(argv[2 + s]);
  const size_t bytes = sizeof(float) * n * max_segments * 2, room = (bytes + 4095) / 4096 * 4096;
  char* m = static_cast<char*>(mmap(nullptr, room + 4096, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  if (m == MAP_FAILED || mprotect(m + room, 4096, PROT_NONE)) return 9;
  float* tf = reinterpret_cast<float*>(m + room - bytes);
  for (int k = 0; k < n * max_segments * 2; ++k) tf[k] = float(k);
  World w{};
  w.n_objects = n, w.max_segments = max_segments, w.line_num = line_num, w.tf = tf;
  for (int j = 0; j < n * max_segments; ++j) {
    volatile float4 g;
    const float4 v = segment_of(w, j);
    g.x = v.x, g.y = v.y, g.z = v.z, g.w = v.w;
    const int s = j / max_segments, i = j % max_segments;
    if (i >= line_num[s]) continue;
    const int a = 2 * j, b = 2 * (s * max_segments + (i + 1) % line_num[s]);
    if (g.x != a || g.y != a + 1 || g.z != b || g.w != b + 1) return 2;
  }
  return 0;
}
"""


@pytest.mark.parametrize("max_segments,counts", [(10, (4,)), (10, (10,)), (10, (10, 4)), (32, (32, 0)), (32, (32, 31)),
                                                 (7, (7, 1, 3)), (1, (1, 0))])
def test_staging_reads_only_the_outline_array(tmp_path, max_segments, counts):
    r = run(tmp_path, function("segment_of") + MAIN, max_segments, *counts)
    assert r.returncode == 0, (r.returncode, r.stderr)


SEARCH = """
#include <algorithm>
#include <random>
#include <vector>
constexpr int BAND_CAND = 16;
struct Cut {
  float t, ratio;
  int solid, seg;
};
"""

# Two or three solids of one segment each (an outline of two vertices, there and back): the first crosses a
# link at the cell's own point with t < 0, the others cross it further on. Every order of the
# candidates, and both orders of the solids.
SEARCH_MAIN = """
int main() {
  std::mt19937 g(1);
  auto uni = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(g); };
  int found = 0, wrong = 0;
  for (long trial = 0; trial < 3000000 && found < 300; ++trial) {
    const float x = float(g() % 500 + 2), y = float(g() % 500 + 2);
    const int d = g() % 8, dx = (d < 4 ? d : d + 1) / 3 - 1, dy = (d < 4 ? d : d + 1) % 3 - 1;
    const float a = uni(0.f, 6.2831853f), l0 = uni(.05f, 2.f), l1 = uni(.05f, 2.f);
    const float s0[4] = {x + l0 * cosf(a), y + l0 * sinf(a), x - l1 * cosf(a), y - l1 * sinf(a)};
    const int n = 2 + int(g() % 2);
    for (int turned = 0; turned < 2; ++turned) {
      float tf[3 * 4], position[6] = {x, y, x, y, x, y}, scale[3] = {1, 1, 1}, radius[3] = {100, 100, 100};
      const int line_num[3] = {2, 2, 2};
      for (int s = 0; s < n; ++s) {
        const float by = s == 0 ? 0.f : s == 1 ? .3f : .6f;
        float* t = tf + 4 * (turned ? n - 1 - s : s);
        for (int k = 0; k < 4; ++k) t[k] = s0[k] - by * float(k & 1 ? dy : dx);
      }
      World w{n, 2, 1, line_num, tf, position, scale, radius};
      World alone = w;
      alone.n_objects = 1;
      alone.tf = turned ? tf + 4 * (n - 1) : tf;
      const Cut near = get_cutcell(alone, x, y, float(dx), float(dy));
      if (!(near.solid >= 0 && near.t < 0.f)) continue;
      ++found;
      const Cut want = get_cutcell(w, x, y, float(dx), float(dy));
      std::vector<int> order(2 * n);
      for (int k = 0; k < 2 * n; ++k) order[k] = k;
      do {
        int cand[6];
        std::copy(order.begin(), order.end(), cand);
        const Cut got = get_cutcell_list(w, nullptr, cand, 2 * n, x, y, float(dx), float(dy));
        wrong += got.t != want.t || (want.t >= 0.f && (got.solid != want.solid || got.seg != want.seg || got.ratio != want.ratio));
      } while (std::next_permutation(order.begin(), order.end()));
    }
  }
  printf("%d near crossings, %d wrong cuts\\n", found, wrong);
  return found < 20 ? 3 : wrong ? 2 : 0;
}
"""


@pytest.mark.parametrize("flags", [(), ("-mfma", "-ffp-contract=fast")])
def test_cut_does_not_depend_on_the_candidates_order(tmp_path, flags):
    if flags and "fma" not in open("/proc/cpuinfo").read():
        pytest.skip("no fused multiply-add on this CPU")
    body = "#include <cmath>\n" + SEARCH + function("segment_of") + function("get_cutcell") + function("get_cutcell_list")
    r = run(tmp_path, body + SEARCH_MAIN, flags=flags)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(40, 5), (33, 0), (4, 3, 0)])
def test_outlines_of_different_lengths(counts):
    """The last outline shorter than the others, or never configured: one step against the binary32
    oracle. Tolerance: both sides round a stored moment at most 40 operations on terms summing to 2 over
    rho >= 0.8, 2 x 200 eps (eps = 2^-24)."""
    import numpy as np
    import torch

    from openhomelbm_b200.lbm import LBM_Solver
    from oracle import oracle as orc

    nx, ny, n = 90, 64, len(counts)
    rng = np.random.default_rng(3)
    m = np.zeros((6, nx, ny))
    m[0] = 1.0 + 0.02 * rng.uniform(-1, 1, (nx, ny))
    m[1:3] = 0.05 * rng.uniform(-1, 1, (2, nx, ny))
    for k, (a, b) in enumerate([(0, 0), (1, 1), (0, 1)]):
        m[3 + k] = m[1 + a] * m[1 + b] + 1e-3 * rng.uniform(-1, 1, (nx, ny))
    m = m.astype(np.float32)
    s = LBM_Solver(nx, ny, solid_num=n, use_graph=False)
    f = s.flows[0]
    f.vis_shear = 0.05
    for buf in f.moments:
        buf.copy_(torch.tensor(m))
    most = max(10, *counts)
    line, pos = np.zeros((n, most, 2), np.float32), np.zeros((n, 2), np.float32)
    scale = np.zeros(n, np.float32)
    for k, c in enumerate(counts):
        if c == 0:
            continue
        th = np.linspace(0, 2 * np.pi, c, endpoint=False) + 0.1
        line[k, :c] = np.stack([np.cos(th), 0.8 * np.sin(th)], 1)
        pos[k], scale[k] = (20.3 + 25.1 * k, 30.7 + 1.3 * k), 7.0 / nx
        f.configure_solid(k, line[k, :c], tuple(pos[k]), scale=7.0 / nx)
    assert f.max_segments_per_object == most
    sol = orc.Solids2D(line=line, line_num=np.array(counts), position=pos, angle=np.zeros(n), scale=scale,
                       mass_center=np.zeros((n, 2)), max_radius=f.solid_max_radius.cpu().numpy()).cast(np.float32)
    s.step()
    new, loads = orc.step_2d(m, m.copy(), vis_shear=np.float32(0.05), bc_type=f.bc_type, bc_value=f.bc_value,
                             flag=orc.border_flags_2d(nx, ny), solids=sol)
    assert np.abs(loads[:, :2]).max() > 0
    assert np.abs(f.cur.cpu().numpy() - new).max() <= 400 * 2.0 ** -24
