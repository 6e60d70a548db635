"""Host arithmetic of the few-row product kernel (gemm_ks_shape.h), compiled and swept: whatever tile and split the choice arrives at, every
block has a K-block, every column an owner inside the cluster, and ring, exchange and tensor memory their room."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SWEEP = r"""
#include <cstdio>
#include "gemm_ks_shape.h"
using namespace ac::gemm_ks;
static bool sound(const Shape& s, int64_t k, bool wide) {
  const int nkb = k_blocks(k, wide), quads = s.bn / s.split / 4;
  const size_t stage = (wide ? 1 : 2) * (size_t)kAHalf + (size_t)s.bn * KB * 4, ex = (size_t)s.split * quads * (BM + 1) * 16;
  if (s.split * s.kper < nkb || (s.split - 1) * s.kper >= nkb || quads * s.split * 4 != s.bn) return false;
  if (s.stages < 1 || s.stages > kMaxStages || s.stages > s.kper || (s.kper > 1 && s.stages < 2)) return false;
  // alignment, then the ring with the exchange behind it, or over it in a cluster of one
  if (s.smem > kSmemMax || s.smem < 1024 + (s.split > 1 ? s.stages * stage + ex : std::max(s.stages * stage, ex))) return false;
  for (int c = 0; c < s.bn / 4; ++c)
    if ((int)(((unsigned)c * (unsigned)s.inv) >> 20) != c / quads) return false;
  for (int rank = 0; rank < s.split; ++rank) {     // accumulators of the block: cross terms, main terms, and A's two buffers
    const int kbs = std::min(nkb, (rank + 1) * s.kper) - rank * s.kper, extra = wide ? 128 : 0;
    const int mains = std::min((512 - extra) / s.bn - 1, kbs);
    if (kbs < 1 || mains < 1 || s.bn * (mains + 1) + extra > 512) return false;
  }
  return true;
}
int main() {
  long long shapes = 0, picks = 0;
  for (bool wide : {false, true})
    for (int64_t k = 4; k <= 20000; k += k < 4200 ? 4 : 1004) {
      for (int bn : {0, 16, 32, 48, 64, 96, 128, 256})
        for (int split : {0, 1, 2, 3, 4, 8, 16}) {
          Shape s;
          if (!make_shape(bn, split, k, wide, &s)) continue;
          ++shapes;
          if (!sound(s, k, wide)) { std::printf("bn %d split %d k %lld wide %d\n", bn, split, (long long)k, wide); return 1; }
        }
      if (k % 32 == 0)
        for (int64_t m : {1, 64, 198, 1386, 9456, 1 << 20})
          for (int64_t n : {4, 96, 192, 768, 1000, 3072}) {
            const Shape s = pick_shape(m, n, k, wide, [](int split) { return split == 1 ? 148 : split == 2 ? 74 : split == 4 ? 33 : 15; });
            ++picks;
            if (!s.bn || s.clocks >= 1e30 || !sound(s, k, wide)) { std::printf("%lld x %lld x %lld wide %d\n", (long long)m, (long long)k, (long long)n, wide); return 2; }
          }
    }
  std::printf("ok %d\n", shapes > 10000 && picks > 5000);
}
"""


def test_every_shape_is_sound(tmp_path):
    src = tmp_path / "s.cpp"
    src.write_text(SWEEP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "altius_b200", "csrc"), str(src), "-o", str(tmp_path / "s")], check=True)
    r = subprocess.run([str(tmp_path / "s")], capture_output=True, text=True)
    assert r.stdout == "ok 1\n", r.stdout
