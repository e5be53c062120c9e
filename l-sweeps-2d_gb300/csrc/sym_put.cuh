// How the factorisations write symmetric tiles (read by sweep_sym.cuh).
#pragma once
#include "common.cuh"
#include "internal.h"

#include <cuda_bf16.h>

namespace lsw {

// bf16 hi/lo terms of x: hi = rn(x), lo = rn(x - hi)
__device__ __forceinline__ void bf16_split(float x, unsigned& hi, unsigned& lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  hi = (unsigned)__bfloat16_as_ushort(h);
  lo = (unsigned)__bfloat16_as_ushort(l);
}

// Entry (i, j) of a line's factor into its symmetric tile (tab:
// SymTable::column of the cell); complex64: the tiles of (i, j), i's tile row not
// above j's; split: of (j, i), so that neighbouring threads (i) write
// neighbouring values of a row.
__device__ __forceinline__ void sym_put(float2* blk, const unsigned char* tab, int i, int j, float2 v, bool split) {
  const int bi = i >> 4, bj = j >> 4;
  if (split ? bi > bj : bi < bj) return;
  const int hi = max(bi, bj), lo = min(bi, bj);
  const int tile = tab[((bi + bj) & 3) * kSymTilesMax + lo] + ((hi - lo) >> 2);
  if (!split) {
    blk[tile * 256 + (j & 15) * 16 + ((i & 15) ^ SymTiles::swz(j & 15))] = v;
    return;
  }
  // planes re hi, im hi, re lo, im lo of four 8 x 8 blocks (by column, then row) of bf16, row j mod 16, column i mod 16
  unsigned short* p = reinterpret_cast<unsigned short*>(blk) + tile * 1024 +
                      (((j >> 3) & 1) + ((i >> 3) & 1) * 2) * 64 + (j & 7) * 8 + (i & 7);
  unsigned h, l;
  bf16_split(v.x, h, l);
  p[0] = (unsigned short)h;
  p[512] = (unsigned short)l;
  bf16_split(v.y, h, l);
  p[256] = (unsigned short)h;
  p[768] = (unsigned short)l;
}

}  // namespace lsw
