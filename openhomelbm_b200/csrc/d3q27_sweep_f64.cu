// The binary64 kernels of d3q27_sweep.cuh, in a module of their own: a program's first step loads the
// module of its kernel, and these are large.

#include <cstring>

#include "d3q27_sweep.cuh"

namespace hl {
namespace d3 {

int launch_sweep_f64(const hl_world3d* w, double vis, const hl_diag* diag, const sw::Maps* maps, cudaStream_t st) {
  if (maps != nullptr) return sw::dispatch<StoreF64, true>(w, vis, diag, *maps, st);
  sw::Maps unused;
  std::memset(&unused, 0, sizeof(unused));
  return sw::dispatch<StoreF64, false>(w, vis, diag, unused, st);
}

}  // namespace d3
}  // namespace hl
