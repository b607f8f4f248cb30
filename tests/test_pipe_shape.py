"""Launch shapes of the pipelined LU-SGS sweeps (pipe_launch and pipe_sa_launch
of aero_topology.cpp, compiled here as plain C++): over blocks of every
proportion, long thin ones among them, cluster sizes and numbers of CTAs, each
accepted shape keeps what its kernel relies on."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cmath>
using std::fabs; using std::fma;
#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
#include "aero_topology.cpp"
#include <cstdio>
using namespace aero;

static int fails = 0, accepted = 0, refused = 0;
#define EXPECT(x) do { if (!(x)) { if (++fails <= 10) std::printf("failed: %s (%s %d x %d x %d, C %d, ctas %ld: P %d W %d NG %d NST %d D %d L %d)\n", #x, sa ? "sa" : "mean", nx, ny, nz, C, ctas, s.P, s.W, s.NG, s.NST, s.D, s.L); } } while (0)

static void check(int nx, int ny, int nz, int C, long ctas, int sms) {
  PipeNeed need;
  need.add(Box{1, nx, 1, ny, 1, nz}, C);
  for (int sa = 0; sa < 2; ++sa) {
    const PipeLaunch f = sa ? pipe_sa_launch(need) : pipe_launch(need, ctas, sms);
    const PipeShape& s = f.sh;
    if (!f.ok) { ++refused; continue; }
    ++accepted;
    EXPECT(s.P >= 1 && s.P <= 1022 && s.W >= 1 && s.NG >= 1);
    // a group's barriers: the planes of one round of the groups have one each
    EXPECT(s.NG <= 7 && s.NST >= s.NG && s.NST >= 2);
    EXPECT(f.threads == 32 * (s.W * s.NG + 1) && s.W * s.NG + 1 <= 16);
    EXPECT(sa || f.two == (ctas > sms) || !f.two);
    if (f.two) EXPECT(s.W * s.NG + 1 <= kPipeWarps[kPipeVariants - 1]);
    EXPECT(f.smem <= (size_t)(f.two ? 113 : 226) * 1024);
    EXPECT((s.D & (s.D - 1)) == 0 && s.D >= 8 && s.D <= 64);
    // The groups post their counts of messages read, one post per `lot`
    // messages, each after its plane, so that the last value in place may be
    // that of the group which is NG - 1 planes behind: (NG - 1) / lot posts.
    // A sender of message m has to see a count above m - D when all messages
    // before m have been read, of which the last m - lot + 1 .. may be unposted.
    const int lot = pipe_lot(s.D);
    EXPECT(lot + (s.NG - 1) / lot * lot < s.D);
  }
}

int main() {
  const int ext[] = {1, 2, 3, 5, 7, 9, 10, 15, 31, 40, 63, 127, 191, 500, 2000, 9000};
  for (int nx : ext)
    for (int ny : ext)
      for (int nz : ext) {
        if ((long)nx * ny * nz > 4000000) continue;
        for (int C : {1, 2, 4, 8, 16})
          for (long n : {1L, 8L, 64L, 300L}) check(nx, ny, nz, C, n * C, 148);
      }
  for (int n = 10000; n <= 30000; n += 250)  // a slab's planes fill most of the shared memory
    for (int w : {1, 2, 3, 5, 8, 9, 10})
      for (int C : {1, 2}) {
        check(n, w, w, C, C, 148);
        check(w, w, n, C, 200, 148);
      }
  // the number of SMs decides between one and two CTAs per SM
  PipeNeed need;
  need.add(Box{1, 31, 1, 15, 1, 3}, 4);
  if (pipe_launch(need, 148, 148).two || !pipe_launch(need, 149, 148).two || !pipe_launch(need, 148, 100).two) ++fails;
  std::printf("accepted %d refused %d fails %d\n", accepted, refused, fails);
  return fails != 0 || accepted < 1000 || refused < 100;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_launch_shapes(tmp_path):
    src = tmp_path / "shape.cpp"
    src.write_text(SRC)
    exe = tmp_path / "shape"
    csrc = os.path.join(ROOT, "aerocfd_b200", "csrc")
    subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O2", "-w", "-I" + csrc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_the_device_gives_the_number_of_sms():
    """No launch shape is made for a number of SMs written into the source."""
    import re
    csrc = os.path.join(ROOT, "aerocfd_b200", "csrc")
    for name in ("aero_runtime.cu", "aero_topology.cpp", "aero_topology.h", "aero_kernels.h"):
        code = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, name)).read())
        assert not re.search(r"\b148\b", code), name
