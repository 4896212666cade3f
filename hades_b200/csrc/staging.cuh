// What other files use of the staging table (staging.cu).
#pragma once

#include "common.cuh"

namespace hb {

// hb_staging_insert_rows with a nullable device count that caps n.  early: the launch before is one of this call's,
// and none that writes emb_rows (HB_LAUNCH_NEXT, load_settled)
int staging_insert_rows(const hb_staging_t* s, const void* emb_rows, const int64_t* row_index, int64_t n,
                        const int64_t* n_dev, void* cache_rows, int64_t row_bytes, const int64_t* locs,
                        const uint8_t* last_writer, bool early, cudaStream_t st);

}  // namespace hb
