// gb_record_shape.h -- launch shapes of the partitioned path's pass 1
// (k_rec_scatter).  Plain C++: which shape a record size and a partition count
// get is checked on the host alone.
#pragma once
#include <stddef.h>

#include <initializer_list>

namespace gb {

constexpr int kRecSizes[] = {2, 4, 6, 8, 12};  // 8-byte words of a record
// Partitions of one call: every record size has a launch shape up to kAllParts
// of them, those of up to 64 bytes (96 without validity masks) up to kMaxParts.
constexpr int kAllParts = 8192;
constexpr int kMaxParts = 16384;

// A launch of pass 1: CTAs of `threads` threads, `rows` rows per thread, of
// which `ctas` share an SM.
struct RecShape {
  int threads, rows, ctas;  // threads = 0: no shape fits
};

// Dynamic shared memory of a CTA on tiles of `tile` rows: the sorted records,
// two histograms and the tile's validity words.
inline size_t rec_scatter_smem(int tile, int words, int nparts, int nmask)
{
  return (size_t)tile * words * 8 + (size_t)nparts * 8 + (size_t)nmask * (tile / 32 + 1) * 4;
}

inline bool rec_shape_fits(const RecShape& s, int words, int nparts, int nmask, int smem_optin)
{
  // 2 KB: the kernel's static shared memory and what an SM keeps per CTA
  return (rec_scatter_smem(s.threads * s.rows, words, nparts, nmask) + 2048) * s.ctas <= (size_t)smem_optin;
}

// The largest tile of a kind that fits: `ctas` = 2, 512-thread CTAs, or 1, 1024.
inline RecShape rec_shape_of(int ctas, int key_words, int words, int nparts, int nmask, int smem_optin)
{
  for (int rows : {8, 6, 5, 4, 3, 2, 1}) {
    if (rows == 8 && key_words == 2) continue;  // two words of 8 keys take too many registers
    const RecShape s{1024 / ctas, rows, ctas};
    if (rec_shape_fits(s, words, nparts, nmask, smem_optin)) return s;
  }
  return RecShape{0, 0, 0};
}

// Two CTAs per SM on the largest tile of which two fit, so that one loads while
// the other reserves or writes.  With many partitions the reservations and the
// clearing of the histograms are paid per tile, and one CTA on a tile as large
// as shared memory is faster.  Where the line lies, two CTAs / one CTA in ms:
//   16 bytes, 40M rows, 4096 partitions 0.85 / 0.68; 32 bytes, 100M rows, 740
//   partitions 1.58 / 1.63; then 20M rows each
//   48 bytes   592: 0.44 / 0.44   1036: 0.49 / 0.47   1480: 0.52 / 0.48   8192: 1.45 / 0.76
//   64 bytes   592: 0.61 / 0.65   1036: 0.68 / 0.69   1332: 0.71 / 0.69   8192: 1.57 / 1.06
//   96 bytes   740: 0.74 / 0.80   1332: 0.82 / 0.85   1776: 0.85 / 0.84   4096: 1.26 / 0.97
inline RecShape rec_shape(int key_words, int words, int nparts, int nmask, int smem_optin)
{
  const int first = nparts > (words <= 4 ? 6144 / words : 500 + 100 * words) ? 1 : 2;
  const RecShape s = rec_shape_of(first, key_words, words, nparts, nmask, smem_optin);
  return s.threads ? s : rec_shape_of(3 - first, key_words, words, nparts, nmask, smem_optin);
}

}  // namespace gb
