"""The faces of the queued brick CG kernels (csrc/afl_brick.cuh): every packet that a CTA sends
is one that its receiver waits for, and the other way round.  A packet that is not waited for
could arrive after its receiver has left the system and cleared its inbox for the next one of
its list.  The address functions of the kernels, run on the host over every CTA, thread and
plane."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
#include "afl_brick.cuh"
#include <cstdio>
#include <cstdlib>
#include <set>
using namespace afl;

template <int BX, int CZ>
int check(int nx, int ny, int nz, int cz) {
  using S = BrickShape<BX>;
  Dims g{};
  g.nx = nx, g.ny = ny, g.nz = nz, g.nxy = nx * ny, g.n = nx * ny * nz;
  const int nbx = (nx + S::BX - 1) / S::BX, nby = (ny + S::BY - 1) / S::BY,
            nbz = (nz + cz - 1) / cz;
  for (int czp : {(cz + 3) / 4 * 4, CZ}) {  // a system of its own, one of a queue
    std::set<int> sent, waited;
    for (int b = 0; b < nbx * nby * nbz; ++b)
      for (int t = 0; t < kBT; ++t) {
        const BrickCells<S> cl(g, nbx, nby, cz, t, b);
        const BrickFaces<S, true> fc(g, cl, nbx, nby, nbz, czp, t);
        auto send = [&](int at) {
          if (at >= 0 && !sent.insert(at).second) printf("sent twice\n"), exit(1);
        };
        for (int m = 0; m < CZ && m < (cz + 3) / 4 * 4; ++m)
          send(S::y_at(fc.ydst, m, cl.nzb));
        for (int n = 0; n < CZ / S::kXLanes || n == 0; ++n)
          send(S::template x_at<true>(fc.xdst, t, n, cz, cl.nzb));
        send(fc.zlo_dst);
        send(fc.zhi_dst);
        constexpr int NI = (CZ + S::kLanes - 1) / S::kLanes;
        for (int n = 0; n < NI; ++n)
          if (S::side_on(n, fc.side_lim)) waited.insert(fc.own + t + n * S::kLanes * S::kSide);
        if (fc.zlo_dst >= 0) waited.insert(fc.own + t + S::kSide * czp);
        if (fc.zhi_dst >= 0) waited.insert(fc.own + t + S::kSide * czp + kBT);
      }
    int lost = 0, stray = 0;
    for (int at : sent) stray += !waited.count(at);
    for (int at : waited) lost += !sent.count(at);
    if (stray || lost)
      return printf("%dx%dx%d BX %d cz %d: %d sent and not waited for, %d waited for and not sent\n",
                    nx, ny, nz, BX, cz, stray, lost), 1;
  }
  return 0;
}

template <int BX>
int shape(int nx, int ny, int nz) {
  int bad = 0;
  for (int cz = 1; cz <= (BX == 64 ? 16 : 32) && cz <= nz; ++cz)
    bad |= cz <= 4    ? check<BX, 4>(nx, ny, nz, cz)
           : cz <= 8  ? check<BX, 8>(nx, ny, nz, cz)
           : cz <= 16 ? check<BX, 16>(nx, ny, nz, cz)
                      : check<BX, 32>(nx, ny, nz, cz);
  return bad;
}

int main(int, char **v) {
  const int nx = atoi(v[1]), ny = atoi(v[2]), nz = atoi(v[3]);
  return shape<16>(nx, ny, nz) | shape<32>(nx, ny, nz) | shape<64>(nx, ny, nz);
}
"""


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    from aether_fluid import build
    d = tmp_path_factory.mktemp("faces")
    src, exe = d / "t.cu", d / "t"
    src.write_text(CODE)
    subprocess.check_call([build.nvcc(), *build.ARCH, "-std=c++17", "-O1",
                           "--expt-relaxed-constexpr", "-extended-lambda", "-I", build.CSRC,
                           str(src), "-o", str(exe)])
    return exe


# whole bricks; 48 rows in bricks of 32 and of 16; one row, column and plane past a brick;
# the smallest grid; several ragged bricks along every axis
@pytest.mark.parametrize("shape", [(32, 32, 32), (48, 48, 48), (33, 33, 33), (6, 6, 6),
                                   (65, 17, 35), (100, 37, 41)],
                         ids=lambda s: "x".join(map(str, s)))
def test_every_packet_sent_is_waited_for(checker, shape):
    out = subprocess.run([str(checker), *map(str, shape)], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr
