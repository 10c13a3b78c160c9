// Host-side mesh preparation (dem_mesh_host.cu).
#pragma once
#include <vector_types.h>

#include <cstdint>
#include <vector>

namespace gb300 {

struct MeshHost {
  int ntri = 0;
  std::vector<double> tri;     // [t*kTriStride] geometry, layout of MeshDev::tri
  std::vector<int> meta;       // obtuse index + edge/corner activity bits
  std::vector<uint8_t> edge_active, corner_active;  // [t*3]
  std::vector<int> cn_start, cn_list;               // coplanar node-neighbours
  std::vector<double> bbox;    // [t*6]: lower then upper corner of each triangle (initial mesh)
};

// Geometry, topology (unless edge/corner activity are given) and coplanar
// neighbour lists of a triangle mesh, nodes[ntri][3][3] in element order.
int mesh_prepare(int ntri, const double *nodes, const uint8_t *edge_active,
                 const uint8_t *corner_active, MeshHost &out);

// FP32 copies of one triangle (geometry record g, out[kTrif]): node 0; unit
// normal; then per edge q its outward in-plane unit normal en_q and, in w, its
// offset en_q.(n_q - n_0), so that en_q.(x - n_0) - w is the distance beyond
// the edge.  Triangles whose edges 0 and 1 are within 1e-5 of parallel get
// zero edge normals: their normals carry too much rounding to bound anything
// (the test then never rejects by an edge).
void tri_floats(const double *g, float4 *out);

}  // namespace gb300
