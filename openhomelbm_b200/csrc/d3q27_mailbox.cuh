// Launchers of the 16-bit stream-collide (d3q27_mailbox.cu).
#pragma once

#include "d3q27_sweep.cuh"

namespace hl {
namespace d3 {

int launch_mailbox(const hl_world3d* w, double vis, const hl_diag* diag, const sw::Maps& maps, cudaStream_t st);
int launch_mailbox_batch(const sw::BatchDomain* doms, int n_doms, int n_items, double vis, const hl_storage& storage,
                         int parity, int* status, cudaStream_t st);

}  // namespace d3
}  // namespace hl
