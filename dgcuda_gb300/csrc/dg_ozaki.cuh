// dg_ozaki.cuh -- the digit tables of the basis contractions as exact integer
// slices for f16 tensor-core MMAs (exact-slice emulation after Ozaki, Ogita
// and Oishi, "Error-free transformations of matrix multiplication by using
// fast routines of matrix multiplication and its applications", Numer.
// Algorithms 59, 2012; slices held as small integers, as in Ootomo, Ozaki and
// Yokota, IJHPCA 2024): what dg_oz_table_image returns.  The element stage
// itself contracts in fixed point on the integer pipe (dg_fixed.cuh), which
// measures faster.
//
//  * a table column shares the exponent of its largest entry; each entry
//    becomes a 53-bit integer X (truncated), and X is written in 7 balanced
//    base-256 digits d_j in [-128, 127] (X + 0x80808080808080 has the unsigned
//    digits d_j + 128);
//  * one warp contracts 16 rows (rows g and g + 8 of the MMA, g = lane / 4);
//    the 4 lanes of a quad hold K slots {2t, 2t+1, 2t+8, 2t+9} (t = lane % 4),
//    the positions 0..3 of the thread, and items (modes, area points, edge
//    points) fill position 0 of t = 0..3, position 1 of t = 0..3, and so on.
#pragma once
#include <cstdint>

#include "dg_device.cuh"

namespace dg {
namespace oz {

constexpr int kDigits = 7;
constexpr unsigned long long kBias = 0x80808080808080ull;

// tables: EVAL (K = modes, N = area points), PROJ (3 K blocks: GR and GS
// over the area points, E over the edge points; N = modes; one exponent per
// column across the three), TRACE (K = modes, N = edge points).  Words are
// the B fragments of each lane: word[digit][kblock][colgroup][lane] =
// {k 2t..2t+1, k 2t+8..2t+9} of column colgroup * 8 + g, as f16 pairs.
enum { kEval = 0, kProj = 1, kTrace = 2 };
// word offset of each table: 7 digits x 2 column groups x 32 lanes per K
// block, K blocks 1, 3, 1
__host__ __device__ constexpr int word_off(int tab) { return 7 * 2 * 32 * (tab == 0 ? 0 : tab == 1 ? 1 : 4); }
constexpr int kWords = 7 * 5 * 2 * 32;      // 2240 uint2
struct Tabs {
  uint2 w[kWords];
  int colexp[3][16];                         // biased exponent of each table column
  int pad[16];
};

// position p of lane quad index t -> slot (0..15)
__host__ __device__ constexpr int slot_of(int pos, int t) { return pos < 2 ? 2 * t + pos : 2 * t + 8 + (pos - 2); }

}  // namespace oz
}  // namespace dg
