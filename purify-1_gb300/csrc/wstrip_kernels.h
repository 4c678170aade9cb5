// Host-callable launchers of the tensor-core row kernels: G, G^H and the sum
// of the task windows on the strip plan (wplan.h WStripPlan), complex<float>.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdint>

#include "pg_types.h"

namespace pg {

struct WStripArgs {
  const void *grid = nullptr;   // G input, Nv x Nu complex
  const void *vis_in = nullptr; // G^H input in caller order
  void *vis_out = nullptr;      // G output in caller order
  void *windows = nullptr;      // G^H output, the task windows
  const void *factors = nullptr;
  const WStripTask *tasks = nullptr;
  const int32_t *order = nullptr;
  const int32_t *group_oct = nullptr;
  const WTerm *terms = nullptr;
  int ntasks = 0, Nu = 0, Nv = 0;
  int tiles = 0, rows = 0;      // plan's tiles and rows
  bool wide = false;            // set by the launcher: the grid is read 16 bytes at a time
  bool early = true;            // may start before the kernel ahead of it is done
};

struct WStripFoldArgs {
  const void *windows = nullptr;
  const WStripTask *tasks = nullptr;
  const int2 *owner = nullptr;  // strips x cols
  void *grid = nullptr;
  int strips = 0, cols = 0, tiles = 0, rows = 0, Nu = 0, Nv = 0;
};

// Values of slack before and after the factors (WStripArgs::factors).
constexpr int kStripSlack = 64;
cudaError_t launch_wstrip_degrid(const WStripArgs &a, cudaStream_t s);
cudaError_t launch_wstrip_grid(const WStripArgs &a, cudaStream_t s);
cudaError_t launch_wstrip_fold(const WStripFoldArgs &f, cudaStream_t s);

}  // namespace pg
