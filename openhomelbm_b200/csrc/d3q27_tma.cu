// Launchers of the D3Q27 sweep kernel (d3q27_sweep.cuh) for domains whose rows are multiples of 16 bytes
// (walled tiles may reach past the domain; periodic domains are whole tiles), staged by the tensor memory
// accelerator: binary32, alone or many domains in one launch, and binary64 (d3q27_sweep_f64.cu). The
// 16-bit storages go on to d3q27_mailbox.cu with tensor maps from here.
//
// Staging: per plane one thread issues a box copy of the tile's rows with the one beyond either end and
// a 16-byte wide box for the column before and after the tile. Periodic wrap-around along x and z is a
// coordinate; a row beyond y's ends comes as boxes of its own. Boxes outside a walled domain are
// zero-filled by the copy. Completion is tracked by one mbarrier per stage with bounded waits. No
// multicast: every block loads its own boxes.

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "d3q27_mailbox.cuh"
#include "d3q27_sweep.cuh"

namespace hl {
namespace d3 {
namespace tma {

using sw::BatchDomain;
using sw::Maps;
constexpr int TY = sw::tile_y<float>(), TZ = sw::TZ;

// ---------------------------------------------------------------- host side
CUtensorMapDataType tmap_dtype(hl_dtype d) {
  switch (d) {
    case HL_F32: return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    case HL_F64: return CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    case HL_F16: return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    default: return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  }
}

size_t esize(hl_dtype d) { return d == HL_F64 ? 8 : d == HL_F32 ? 4 : 2; }

// Tensor maps over the (nz, ny, nx, 10) moment array (innermost first); cached per buffer.
int encode_maps(const hl_world3d* w, bool mailbox, Maps* out) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int, int, int, bool>, Maps> cache;
  const auto key = std::make_tuple(w->cur, w->nx, w->ny, w->nz, int(w->storage.dtype), mailbox);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return HL_OK;
    }
  }
  const size_t es = esize(w->storage.dtype);
  const int wz = int(16 / es);
  const cuuint64_t dims[4] = {cuuint64_t(w->nz), cuuint64_t(w->ny), cuuint64_t(w->nx), 10};
  const cuuint64_t strides[3] = {cuuint64_t(w->nz) * es, cuuint64_t(w->ny) * w->nz * es,
                                 cuuint64_t(w->nx) * w->ny * w->nz * es};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  // rows per box: the tile's and one beyond either end (the mailbox kernel takes those apart)
  const cuuint32_t rows = mailbox ? TY : (w->storage.dtype == HL_F64 ? sw::tile_y<double>() : TY) + 2;
  const cuuint32_t boxes[4][4] = {{TZ, rows, 1, 10}, {cuuint32_t(wz), rows, 1, 10}, {TZ, 1, 1, 10}, {cuuint32_t(wz), 1, 1, 10}};
  // the driver entry point is resolved at run time, so the library loads without a driver
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (encode == nullptr) {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || fn == nullptr) {
      set_error("d3q27: cuTensorMapEncodeTiled is unavailable (%s)", cudaGetErrorString(e));
      return HL_ERR_CUDA;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  CUtensorMap* dst[4] = {&out->rows, &out->column, &out->row, &out->corner};
  for (int k = 0; k < 4; ++k) {
    void* base = const_cast<void*>(w->cur);
    const CUresult r = encode(dst[k], tmap_dtype(w->storage.dtype), 4, base, dims,
                                              strides, boxes[k], estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error("d3q27: cuTensorMapEncodeTiled failed (%d)", int(r));
      return HL_ERR_CUDA;
    }
  }
  std::lock_guard<std::mutex> lk(mu);
  if (cache.size() > 64) cache.clear();
  cache[key] = *out;
  return HL_OK;
}

// ---------------------------------------------------------------- batched domains
// Prepared descriptor arrays (device address -> domains, items), so that a launch can only
// use counts that match what was written there.
std::mutex g_batch_mu;
std::map<const void*, std::pair<int, int>> g_batches;

template <class S>
int launch_batch(const BatchDomain* doms, int n_doms, int n_items, double vis, int parity, int* status, cudaStream_t st) {
  using G = sw::Geo<S, true, false>;
  constexpr int NST = sw::stages<S, true>(), SMEM = sw::smem_bytes<G, NST>();
  StepArgs a{};
  a.n_items = n_items;
  a.vis_shear = vis;
  a.status = status;
  Maps maps;
  std::memset(&maps, 0, sizeof(maps));
  auto kern = sw::sweep_kernel<S, true, NST, sw::BLOCKS_PER_SM, false, false, false, false, true>;
  const int rc = set_smem_attr(reinterpret_cast<const void*>(kern), SMEM, "cudaFuncSetAttribute(d3q27 tma batch)");
  if (rc != HL_OK) return rc;
  const int slots = sw::BLOCKS_PER_SM * num_sms();
  kern<<<n_items < slots ? n_items : slots, sw::THREADS, SMEM, st>>>(a, maps, doms, n_doms, parity);
  HL_LAUNCH_CHECK("d3q27 stream_collide (tma batch) launch");
  return HL_OK;
}

}  // namespace tma

bool tma_eligible(const hl_world3d* w) {
  if (w->storage.dtype == HL_F64) return false;
  if (w->ny % tma::TY != 0 || w->nz % tma::TZ != 0) return false;
  const size_t es = tma::esize(w->storage.dtype);
  if ((reinterpret_cast<uintptr_t>(w->cur) & 15) != 0 || (reinterpret_cast<uintptr_t>(w->post) & 15) != 0) return false;
  return (size_t(w->nz) * es) % 16 == 0;
}

// Domains whose planes the tensor copies can deliver: 16-byte rows and buffers; periodic ones of
// whole tiles (a box cannot wrap inside a tile; walled tiles that reach past the domain are
// zero-filled there).
bool box_eligible(const hl_world3d* w) {
  const size_t es = tma::esize(w->storage.dtype);
  const int ty = w->storage.dtype == HL_F64 ? sw::tile_y<double>() : tma::TY;
  if ((reinterpret_cast<uintptr_t>(w->cur) & 15) != 0 || (reinterpret_cast<uintptr_t>(w->post) & 15) != 0) return false;
  if ((size_t(w->nz) * es) % 16 != 0) return false;
  return !w->periodic || (w->ny % ty == 0 && w->nz % tma::TZ == 0);
}

int launch_step_tma(const hl_world3d* w, double vis, const hl_diag* diag, cudaStream_t st) {
  // the 16-bit storages, whatever the call's options: see d3q27_mailbox.cu
  const hl_dtype dt = w->storage.dtype;
  const bool mailbox = dt == HL_F16 || dt == HL_BF16;
  sw::Maps maps;
  const int rc = tma::encode_maps(w, mailbox, &maps);
  if (rc != HL_OK) return rc;
  if (mailbox) return launch_mailbox(w, vis, diag, maps, st);
  switch (dt) {
    case HL_F32: return sw::dispatch<StoreF32, true>(w, vis, diag, maps, st);
    case HL_F64: return launch_sweep_f64(w, vis, diag, &maps, st);
    default: break;
  }
  set_error("d3q27 (tma): dtype not supported");
  return HL_ERR_UNSUPPORTED;
}

}  // namespace d3
}  // namespace hl

using namespace hl;

extern "C" size_t hl_d3q27_batch_bytes(int n_domains) {
  return n_domains > 0 ? size_t(n_domains) * sizeof(d3::tma::BatchDomain) : 0;
}

extern "C" int hl_d3q27_batch_prepare(const hl_world3d* worlds, int n_domains, void* desc, size_t desc_bytes,
                                      int* n_items, hl_stream stream) {
  using d3::tma::BatchDomain;
  HL_CHECK_ARG(worlds != nullptr && n_items != nullptr, "d3q27 batch: worlds or n_items is NULL");
  HL_CHECK_ARG(n_domains >= 1 && n_domains <= 4096, "d3q27 batch: %d domains (1 .. 4096)", n_domains);
  HL_CHECK_ARG(desc != nullptr && (reinterpret_cast<uintptr_t>(desc) & 63) == 0,
               "d3q27 batch: descriptor buffer NULL or not 64-byte aligned");
  HL_CHECK_ARG(desc_bytes >= hl_d3q27_batch_bytes(n_domains), "d3q27 batch: descriptor buffer too small (%zu < %zu)",
               desc_bytes, hl_d3q27_batch_bytes(n_domains));
  const hl_world3d& w0 = worlds[0];
  HL_CHECK_ARG(w0.storage.dtype == HL_F32 || w0.storage.dtype == HL_F16 || w0.storage.dtype == HL_BF16,
               "d3q27 batch: storage dtype %d (float32, float16 or bfloat16)", int(w0.storage.dtype));
  std::vector<BatchDomain> h;
  h.resize(size_t(n_domains));
  long long total = 0;
  for (int k = 0; k < n_domains; ++k) {
    const hl_world3d& w = worlds[k];
    HL_CHECK_ARG(w.nx >= 3 && w.ny >= 3 && w.nz >= 3, "d3q27 batch: domain %d has dims %d x %d x %d", k, w.nx, w.ny,
                 w.nz);
    HL_CHECK_ARG(w.cur != nullptr && w.post != nullptr && w.cur != w.post, "d3q27 batch: domain %d buffers", k);
    HL_CHECK_ARG(d3::tma_eligible(&w), "d3q27 batch: domain %d is not TMA-eligible (ny %% 16, nz %% 32, alignment)",
                 k);
    HL_CHECK_ARG(!w.periodic && w.force == nullptr && w.flag == nullptr,
                 "d3q27 batch: domain %d must be walled, without force or flag fields", k);
    HL_CHECK_ARG(w.storage.dtype == w0.storage.dtype && w.storage.u_scale == w0.storage.u_scale &&
                     w.storage.s_scale == w0.storage.s_scale,
                 "d3q27 batch: domain %d has another storage type or scale than domain 0", k);
    BatchDomain& d = h[size_t(k)];
    hl_world3d flip = w;
    flip.cur = w.post;
    flip.post = const_cast<void*>(w.cur);
    int rc = d3::tma::encode_maps(&w, w.storage.dtype != HL_F32, &d.maps[0]);
    if (rc != HL_OK) return rc;
    rc = d3::tma::encode_maps(&flip, w.storage.dtype != HL_F32, &d.maps[1]);
    if (rc != HL_OK) return rc;
    d.buf[0] = const_cast<void*>(w.cur);
    d.buf[1] = w.post;
    d.N = (long long)w.nx * w.ny * w.nz;
    d.nx = w.nx;
    d.ny = w.ny;
    d.nz = w.nz;
    d.tiles_z = w.nz / d3::tma::TZ;
    d.n_tiles = (w.ny / d3::tma::TY) * d.tiles_z;
    // x chunks of about 32 planes (or the "d3q27_chunks" override): with the items of every
    // domain to spread over the SMs, the chunks only need to be long against the two halo
    // planes each one reads
    const int chunks = g_tune_d3_chunks > 0 ? std::min(g_tune_d3_chunks, w.nx) : std::max(1, (w.nx + 16) / 32);
    d.chunk_len = (w.nx + chunks - 1) / chunks;
    d.n_items = d.n_tiles * ((w.nx + d.chunk_len - 1) / d.chunk_len);
    d.item_base = int(total);
    total += d.n_items;
    HL_CHECK_ARG(total < (1ll << 30), "d3q27 batch: too many items");
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(desc, h.data(), h.size() * sizeof(BatchDomain), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_status(e, "d3q27 batch: descriptor upload");
  {
    std::lock_guard<std::mutex> lk(d3::tma::g_batch_mu);
    d3::tma::g_batches[desc] = {n_domains, int(total)};
  }
  *n_items = int(total);
  return HL_OK;
}

extern "C" int hl_d3q27_stream_collide_batch(const void* desc, int n_domains, int n_items, double vis_shear,
                                             const hl_storage* storage, int parity, int* status, hl_stream stream) {
  HL_CHECK_ARG(desc != nullptr && storage != nullptr, "d3q27 batch: descriptors or storage is NULL");
  HL_CHECK_ARG(vis_shear > 0.0, "d3q27 batch: viscosity must be positive");
  HL_CHECK_ARG(parity == 0 || parity == 1, "d3q27 batch: parity %d", parity);
  {
    std::lock_guard<std::mutex> lk(d3::tma::g_batch_mu);
    auto it = d3::tma::g_batches.find(desc);
    HL_CHECK_ARG(it != d3::tma::g_batches.end() && it->second.first == n_domains && it->second.second == n_items,
                 "d3q27 batch: descriptors not prepared for %d domains and %d items", n_domains, n_items);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* doms = static_cast<const d3::tma::BatchDomain*>(desc);
  switch (storage->dtype) {
    case HL_F32: return d3::tma::launch_batch<StoreF32>(doms, n_domains, n_items, vis_shear, parity, status, st);
    case HL_F16:
    case HL_BF16: return d3::launch_mailbox_batch(doms, n_domains, n_items, vis_shear, *storage, parity, status, st);
    default: break;
  }
  set_error("d3q27 batch: storage dtype %d not supported", int(storage->dtype));
  return HL_ERR_UNSUPPORTED;
}
