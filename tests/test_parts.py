"""The cut of a range into parts of about equal size (csrc/eb_parts.h) against 64-bit integers, for
leaves beyond the 262,144 points from which the product of part and size leaves 32 bits."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = r"""
#include "eb_parts.h"
#include <cstdio>
int main() {
  const int big[] = {262143, 262144, 262145, 262400, 1000003, 2097152, 40000001, 2000000000};
  for (int t = 1; t < 3000 + 8; ++t) {
    const int n = t < 3000 ? t : big[t - 3000], c = (int)((n + 31ll) / 32);
    EbParts p(n, c);
    for (long long i = 0; i < c; ++i) {
      const int at = p.at, m = p.next();
      if (at != i * n / c || at + m != (i + 1) * n / c || m < 1 || m > 32 || (p.at < n) != (i + 1 < c)) {
        std::printf("n %d part %lld: %d + %d\n", n, i, at, m);
        return 1;
      }
    }
  }
  return 0;
}
"""


def test_parts(tmp_path):
    src, exe = tmp_path / "parts.cpp", tmp_path / "parts"
    src.write_text(CODE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "electricbubbles_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
