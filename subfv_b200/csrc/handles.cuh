// Opaque handle types of the C-ABI, shared by the translation units that implement it.
#pragma once
#include <memory>
#include <mutex>

#include "../../include/subfv.h"
#include "common.cuh"
#include "mesh_dev.cuh"

// What a state keeps of its mesh, so that either may be destroyed first, also from another
// thread. While the mesh lives, `stream` is its stream. Destroying it clears `stream` and
// leaves in `last` the end of the work queued by then, which may still write the state's
// buffers: freed memory of the pool can belong to another state at once, and neither
// cudaFree nor the stream's destruction waits for that work.
struct MeshLife {
  std::mutex mu;
  cudaStream_t stream = nullptr;
  cudaEvent_t last = nullptr;
  ~MeshLife() {
    if (last) cudaEventDestroy(last);
  }
};

// A device mesh plus the scratch buffers the stateless reference-shaped calls need.
struct subfv_mesh {
  subfv::DevMesh d;
  double* stage = nullptr;  // host-layout staging, max(5*ne, 3*nv) doubles
  double* sol6 = nullptr;   // [ne][kRec] cell records
  double* rhs6 = nullptr;   // [ne][kRhs]
  double* mass = nullptr;   // [ne]
  subfv::LagScalars* sc = nullptr;
  // the backward-Euler Jacobian's host pattern, built on first use and kept with the mesh
  void* imp_pattern = nullptr;
  void (*imp_pattern_free)(void*) = nullptr;
  std::shared_ptr<MeshLife> life = std::make_shared<MeshLife>();
};

namespace subfv {
int handle_check_status(DevMesh& d);
int handle_clear_status(DevMesh& d);
int handle_ensure_scratch(subfv_mesh* m);
// full geometry when Lagrangian steps left only the step's subset current
int handle_ensure_full_geometry(DevMesh& d);
// the Lagrangian step's per-mesh arrays (allocated on the mesh's stream)
int handle_ensure_lag_arrays(DevMesh& d);
}  // namespace subfv
