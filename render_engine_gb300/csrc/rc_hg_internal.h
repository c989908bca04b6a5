// Library-internal access to a hash-grid cache (for passes of the frame runtime that feed it).
#pragma once

#include <cuda_runtime.h>

#include "../../include/rc_hashgrid.h"

namespace rc {
cudaStream_t hg_stream(rc_hg* hg);   // the stream the cache's work is issued on
const rc_hg_config& hg_config(const rc_hg* hg);
bool hg_has_voxels(const rc_hg* hg);
// rc_hg_insert on the cache's stream, the entries also into v[i].entry
cudaError_t hg_insert_vertices(rc_hg* hg, const float* pos, const float* nrm, int n, uint32_t* entry, rc_hg_vertex* v);
// rc_hg_mark_paths_strided and rc_hg_voxels_mark of the same paths in one launch (the cache has voxel masks)
cudaError_t hg_path_marks(rc_hg* hg, const rc_hg_vertex* v, const int* len, int stride, int npaths);
}  // namespace rc
