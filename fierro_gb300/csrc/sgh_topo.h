// Mesh topology built on the GPU (sgh_topo.cu).
#ifndef FIERRO_SGH_TOPO_H
#define FIERRO_SGH_TOPO_H

#include <vector>

#include "fierro_sgh.h"
#include "sgh_internal.h"

struct fierro_sgh;

namespace fierro {
namespace topo {

// Fills the handle's device topology (d_nie, d_cin_start, d_cin, d_eie_start,
// d_eie, d_bc and the four renumbering maps; d_eie is allocated here) and the
// host renumbering maps (topo.node_int2ext, topo.elem_int2ext) from the caller's
// mesh, read by the GPU in place.  The boundary deck must be validated already.
int build_device(fierro_sgh* h, const fierro_mesh* mesh, const fierro_boundary* bcs, int64_t num_bcs);

// The same topologies as build_topology's (renumbered), built on the GPU one after the
// other and brought to the host; built[k] is 0 for a mesh that was refused (what
// build_topology refuses, and elements of very many neighbours) or did not fit.  The
// mesh arrays lie on 8-byte boundaries.
struct ToHost {
  const fierro_mesh* mesh;
  const fierro_boundary* bcs;
  int64_t num_bcs;
  HostTopo* out;
};
void build_to_host(const std::vector<ToHost>& list, std::vector<char>* built);

}  // namespace topo
}  // namespace fierro

#endif
