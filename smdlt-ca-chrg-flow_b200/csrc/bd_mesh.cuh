// Spreading and interpolation of the particle-mesh mobility (bd_mesh.cu).
#pragma once

#include "bd_ctx.cuh"

namespace bd {
int mesh_alloc(bd_ctx* c);
int mesh_prepare(bd_ctx* c);
int mesh_spread(bd_ctx* c, int k, const VecIn& v, size_t vr, void* grid);
int mesh_gather(bd_ctx* c, int k, const void* grid);
void mesh_free(bd_ctx* c);
}  // namespace bd
