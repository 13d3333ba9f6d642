"""Launch shapes of the partitioned path's pass 1 (cudf_b200/csrc/gb_record_shape.h),
compiled for the host: every record size gets one that fits shared memory, for
every partition count it may be given and every number of validity masks (no GPU
needed)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cstdio>
#include "gb_record_shape.h"
int main()
{
  const int optin = 227 * 1024;  // shared memory a CTA may opt into on sm_100
  int bad = 0, seen = 0;
  for (int words : gb::kRecSizes)
    for (int kw = 1; kw <= 2; ++kw)
      for (int masks = 0; masks <= 8; ++masks)
        for (int parts = 2; parts <= gb::kMaxParts; parts += parts < 2048 ? 1 : 2048) {
          if (words > 8 && parts > gb::kAllParts) continue;  // the widest records keep to fewer
          const gb::RecShape s = gb::rec_shape(kw, words, parts, masks, optin);
          const bool ok = s.threads * s.ctas == 1024 && s.rows >= 1 && s.rows <= 8 && s.rows != 7 && !(s.rows == 8 && kw == 2) &&
                          gb::rec_shape_fits(s, words, parts, masks, optin);
          if (!ok && ++bad < 10)
            std::printf("words %d key words %d masks %d partitions %d: %d x %d x %d\n", words, kw, masks, parts, s.threads, s.rows, s.ctas);
          ++seen;
        }
  std::printf("%d shapes, %d bad\n", seen, bad);
  return bad != 0;
}
'''


def test_every_record_size_and_partition_count_has_a_launch_shape(tmp_path):
    src, exe = tmp_path / "shapes.cpp", tmp_path / "shapes"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "cudf_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
