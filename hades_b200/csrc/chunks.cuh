// How the entries of a sort are cut: CTA r takes chunk r, in tiles.  Entries are numbered with 32 bits and there
// are fewer than 2^31; where a chunk would begin or a tile end may lie a round per CTA and a tile beyond, which
// unsigned numbers still hold.  The chunk of a CTA that gets nothing begins and ends at the last entry.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define HB_BOTH __host__ __device__ __forceinline__
#else
#define HB_BOTH inline
#endif

namespace hb {

struct SortChunks {
  uint32_t count;
  uint32_t chunk;
  HB_BOTH SortChunks(uint32_t n, uint32_t per_cta) : count(n), chunk(per_cta) {}
  // (of whole rounds of a CTA)
  HB_BOTH SortChunks(uint32_t n, uint32_t ctas, uint32_t round)
      : count(n), chunk(((n + ctas - 1) / ctas + round - 1) / round * round) {}
  HB_BOTH uint32_t begin(uint32_t rank) const { return least(rank * chunk); }
  HB_BOTH uint32_t end(uint32_t rank) const { return least(rank * chunk + chunk); }
  // entry `at` of tile `t` of a chunk: taken when it is below end(rank)
  HB_BOTH uint32_t entry(uint32_t rank, uint32_t t, uint32_t tile, uint32_t at) const { return rank * chunk + t * tile + at; }

 private:
  HB_BOTH uint32_t least(uint32_t e) const { return e < count ? e : count; }
};

}  // namespace hb
