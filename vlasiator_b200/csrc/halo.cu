// Packing and unpacking the blocks of some cells of a batch, on the device,
// for the ghost-layer exchange of a spatial grid split over several batches
// (one per GPU and rank).  No reference counterpart as an entry point: it is
// the data movement of update_remote_mapping_contribution_amr and the dccrg
// remote-neighbour updates (vlasovsolver/cpu_trans_map_amr.cpp:493-810),
// rebuilt as a pack into a caller's device buffer, a transfer the caller
// makes (NCCL send/recv, or any other), and an unpack into the receiving
// batch.
#include "batch_internal.cuh"

namespace vlgpu {

// Copies chunks of blocks (IDs and 64 values) to their places, a chunk (first
// list entry, first output block, blocks) per CTA and half a warp per block.
// The host cuts the selected cells into chunks of one size, so a large cell
// spreads over many CTAs.  An indirect state is read through src_index (a
// block without data gives zeros), so packing moves nothing in the batch.
//
// Bound by HBM reads and writes.  A CTA per cell took 561 us for 13 cells of 12000 blocks
// and 404 us for 1024 cells of 30 to 9000 blocks (1.8 TB/s, the largest cells
// last); in chunks the packing, adjustment and moments of the latter together
// went from 1280 to 1036 us.
constexpr int PACK_THREADS = 256;
constexpr uint32_t PACK_BLOCKS = 4 * PACK_THREADS / 16;  // blocks a CTA moves per pass, four per half-warp
constexpr uint32_t PACK_CHUNK = 4 * PACK_BLOCKS;         // largest chunk
__global__ void __launch_bounds__(PACK_THREADS) pack_cells_kernel(const uint32_t* __restrict__ gids,
                                                                  const uint32_t* __restrict__ src_index,
                                                                  const float4* __restrict__ data,
                                                                  const uint32_t* __restrict__ desc,
                                                                  uint32_t* __restrict__ out_gids,
                                                                  float4* __restrict__ out_data) {
   const uint32_t src = desc[3 * blockIdx.x], dst = desc[3 * blockIdx.x + 1], n = desc[3 * blockIdx.x + 2];
   const uint32_t sub = threadIdx.x & 15, hw = threadIdx.x >> 4;
   for (uint32_t b0 = 0; b0 < n; b0 += PACK_BLOCKS) {
      float4 v[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
         const uint32_t b = b0 + hw + u * (PACK_THREADS / 16);
         v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
         if (b < n) {
            const uint32_t row = src_index ? src_index[src + b] : src + b;
            if (row != 0xffffffffu) v[u] = __ldg(data + 16 * (size_t)row + sub);
         }
      }
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
         const uint32_t b = b0 + hw + u * (PACK_THREADS / 16);
         if (b < n) out_data[16 * ((size_t)dst + b) + sub] = v[u];
      }
   }
   for (uint32_t b = threadIdx.x; b < n; b += PACK_THREADS) out_gids[dst + b] = gids[src + b];
}

// Every block ID below max_gid; a bad one sets *bad.
__global__ void check_gids_range_kernel(const uint32_t* __restrict__ gids, uint64_t n, uint32_t max_gid,
                                        uint32_t* __restrict__ bad) {
   for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
      if (gids[i] >= max_gid) *bad = 1u;
}

// Words of the chunk list of any selection that names a cell once: at most a
// partial chunk per cell, and 16 full ones per SM or one per PACK_CHUNK blocks.
size_t pack_scratch_words(uint64_t capacity, uint32_t n_cells, int sm_count) {
   return 3 * ((size_t)n_cells + 16 * (size_t)sm_count + capacity / PACK_CHUNK);
}

}  // namespace vlgpu

using namespace vlgpu;
using namespace vlgpu_batch_ops;

namespace {

// The batch's current state made direct (list entry p holds data row p of
// the current pool), and its cell slots and rows in use on the host.
int direct_state_slots(vlgpu_batch* b, std::vector<CellSlot>& slots, uint32_t rows[4]) {
   const int st = materialize_async(b);
   if (st != VLGPU_OK) return st;
   slots.resize(b->n_cells);
   VL_CHECK(cudaMemcpyAsync(slots.data(), b->st_slots, sizeof(CellSlot) * b->n_cells, cudaMemcpyDeviceToHost,
                            b->stream));
   VL_CHECK(cudaMemcpyAsync(rows, b->rows_used, sizeof(uint32_t) * 4, cudaMemcpyDeviceToHost, b->stream));
   VL_CHECK(cudaStreamSynchronize(b->stream));
   return VLGPU_OK;
}

// Room for n uint32 words of the per-batch exchange scratch (more than the
// batch was made with only where cells are named several times).
int halo_scratch(vlgpu_batch* b, size_t n) {
   if (n <= b->halo_words) return VLGPU_OK;
   uint32_t* more = nullptr;
   VL_CHECK(cudaMalloc(&more, sizeof(uint32_t) * n));
   cudaFree(b->halo_scratch);
   b->halo_scratch = more;
   b->halo_words = n;
   return VLGPU_OK;
}

// Whether the selection names every cell of the batch.
bool replaces_all(const vlgpu_batch* b, uint32_t n_sel, const uint32_t* cells) {
   if (n_sel < b->n_cells) return false;
   std::vector<char> seen(b->n_cells, 0);
   uint32_t n = 0;
   for (uint32_t i = 0; i < n_sel; ++i) {
      n += !seen[cells[i]];
      seen[cells[i]] = 1;
   }
   return n == b->n_cells;
}

// Unpacking that replaces every cell: nothing of the current state is kept,
// so it is not made direct (a copy of the whole VDF after an adjustment), and
// the blocks go to the start of the idle pool.  The current state stays as it
// is until the block IDs are known to be good, so one wait serves the whole
// call.
int unpack_all(vlgpu_batch* b, uint32_t n_sel, const uint32_t* cells, const uint32_t* counts, const uint32_t* gids,
               const float* data, uint64_t total) {
   if (total > b->capacity) return VLGPU_ENOMEM;
   const int pool = 1 - b->cur;
   uint32_t bad = 0, used = 0;
   std::vector<CellSlot> slots(b->n_cells);
   uint32_t o = 0;
   for (uint32_t i = 0; i < n_sel; ++i) {
      slots[cells[i]] = CellSlot{o, counts[i]};
      o += counts[i];
   }
   VL_CHECK(cudaMemcpyAsync(b->slots[pool], slots.data(), sizeof(CellSlot) * b->n_cells, cudaMemcpyHostToDevice,
                            b->stream));
   if (total > 0) {
      VL_CHECK(cudaMemsetAsync(b->halo_scratch, 0, sizeof(uint32_t), b->stream));
      const uint32_t max_gid = b->mesh.len[0] * b->mesh.len[1] * b->mesh.len[2];
      check_gids_range_kernel<<<b->sm_count * 2, 256, 0, b->stream>>>(gids, total, max_gid, b->halo_scratch);
      b->launches += 1;
      VL_CHECK(cudaGetLastError());
      VL_CHECK(cudaMemcpyAsync(b->gids[pool], gids, sizeof(uint32_t) * total, cudaMemcpyDeviceToDevice, b->stream));
      VL_CHECK(cudaMemcpyAsync(b->data[pool], data, sizeof(float) * WID3 * total, cudaMemcpyDeviceToDevice, b->stream));
      VL_CHECK(cudaMemcpyAsync(&bad, b->halo_scratch, sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream));
   }
   VL_CHECK(cudaMemcpyAsync(&used, b->rows_used + b->st_list, sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream));
   VL_CHECK(cudaStreamSynchronize(b->stream));
   // the same room is asked for as when some cells are replaced: behind the
   // rows in use
   if (used + total > b->capacity) return VLGPU_ENOMEM;
   if (bad) return VLGPU_EINVAL;
   const uint32_t now = (uint32_t)total;
   VL_CHECK(cudaMemcpyAsync(b->rows_used + pool, &now, sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream));
   set_direct_state(b, pool);
   b->content_valid = false;
   return VLGPU_OK;
}

}  // namespace

extern "C" {

int vlgpu_batch_pack_cells(vlgpu_batch* b, uint32_t n_sel, const uint32_t* cells, uint32_t* counts, uint32_t* gids,
                           float* data, uint64_t capacity, uint64_t* used) {
   if (!b || !used || (n_sel > 0 && (!cells || !counts))) return VLGPU_EINVAL;
   VL_CHECK(cudaSetDevice(b->device));
   std::vector<CellSlot> slots(b->n_cells);
   VL_CHECK(cudaMemcpyAsync(slots.data(), b->st_slots, sizeof(CellSlot) * b->n_cells, cudaMemcpyDeviceToHost,
                            b->stream));
   VL_CHECK(cudaStreamSynchronize(b->stream));
   uint64_t total = 0;
   for (uint32_t i = 0; i < n_sel; ++i) {
      if (cells[i] >= b->n_cells) return VLGPU_EINVAL;
      counts[i] = slots[cells[i]].count;
      total += counts[i];
   }
   *used = total;
   if (total > capacity) return VLGPU_ENOMEM;
   if (total > 0 && (!gids || !data)) return VLGPU_EINVAL;
   if (total == 0) return VLGPU_OK;
   // chunks small enough that a small selection still reaches every SM
   const uint64_t even = total / (8 * (uint64_t)b->sm_count);
   const uint32_t chunk = even <= PACK_BLOCKS ? PACK_BLOCKS : std::min<uint32_t>(PACK_CHUNK, (uint32_t)even);
   std::vector<uint32_t> desc;
   desc.reserve(3 * ((size_t)n_sel + total / chunk));
   uint32_t dst = 0;
   for (uint32_t i = 0; i < n_sel; ++i) {
      const CellSlot s = slots[cells[i]];
      for (uint32_t q = 0; q < s.count; q += chunk) {
         const uint32_t n = std::min(chunk, s.count - q);
         desc.insert(desc.end(), {s.off + q, dst, n});
         dst += n;
      }
   }
   const int st = halo_scratch(b, desc.size());
   if (st != VLGPU_OK) return st;
   VL_CHECK(cudaMemcpyAsync(b->halo_scratch, desc.data(), sizeof(uint32_t) * desc.size(), cudaMemcpyHostToDevice,
                            b->stream));
   pack_cells_kernel<<<(unsigned)(desc.size() / 3), PACK_THREADS, 0, b->stream>>>(
      b->st_gids, b->st_src, reinterpret_cast<const float4*>(b->data[b->cur]), b->halo_scratch, gids,
      reinterpret_cast<float4*>(data));
   b->launches += 1;
   VL_CHECK(cudaGetLastError());
   VL_CHECK(cudaStreamSynchronize(b->stream));
   return VLGPU_OK;
}

int vlgpu_batch_unpack_cells(vlgpu_batch* b, uint32_t n_sel, const uint32_t* cells, const uint32_t* counts,
                             const uint32_t* gids, const float* data) {
   if (!b || (n_sel > 0 && (!cells || !counts))) return VLGPU_EINVAL;
   VL_CHECK(cudaSetDevice(b->device));
   uint64_t total = 0;
   for (uint32_t i = 0; i < n_sel; ++i) {
      if (cells[i] >= b->n_cells) return VLGPU_EINVAL;
      total += counts[i];
   }
   if (total > 0 && (!gids || !data)) return VLGPU_EINVAL;
   if (replaces_all(b, n_sel, cells)) return unpack_all(b, n_sel, cells, counts, gids, data, total);
   std::vector<CellSlot> slots;
   uint32_t rows[4];
   int st = direct_state_slots(b, slots, rows);
   if (st != VLGPU_OK) return st;
   const uint64_t L = rows[b->st_list];
   if (L + total > b->capacity) return VLGPU_ENOMEM;
   if (total > 0) {
      // the blocks' IDs must lie on the batch's mesh
      VL_CHECK(cudaMemsetAsync(b->halo_scratch, 0, sizeof(uint32_t), b->stream));
      const uint32_t max_gid = b->mesh.len[0] * b->mesh.len[1] * b->mesh.len[2];
      check_gids_range_kernel<<<b->sm_count * 2, 256, 0, b->stream>>>(gids, total, max_gid, b->halo_scratch);
      b->launches += 1;
      VL_CHECK(cudaGetLastError());
      uint32_t bad = 0;
      VL_CHECK(cudaMemcpyAsync(&bad, b->halo_scratch, sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream));
      VL_CHECK(cudaStreamSynchronize(b->stream));
      if (bad) return VLGPU_EINVAL;
      // appended behind the rows in use of the current list and pool; the
      // cells' earlier rows become unreferenced (the next sweep compacts)
      VL_CHECK(cudaMemcpyAsync(const_cast<uint32_t*>(b->st_gids) + L, gids, sizeof(uint32_t) * total,
                               cudaMemcpyDeviceToDevice, b->stream));
      VL_CHECK(cudaMemcpyAsync(b->data[b->cur] + L * WID3, data, sizeof(float) * WID3 * total,
                               cudaMemcpyDeviceToDevice, b->stream));
   }
   uint64_t o = L;
   for (uint32_t i = 0; i < n_sel; ++i) {
      slots[cells[i]] = CellSlot{(uint32_t)o, counts[i]};
      o += counts[i];
   }
   rows[b->st_list] = (uint32_t)(L + total);
   rows[b->cur] = (uint32_t)(L + total);
   VL_CHECK(cudaMemcpyAsync(const_cast<CellSlot*>(b->st_slots), slots.data(), sizeof(CellSlot) * b->n_cells,
                            cudaMemcpyHostToDevice, b->stream));
   VL_CHECK(cudaMemcpyAsync(b->rows_used, rows, sizeof(uint32_t) * 4, cudaMemcpyHostToDevice, b->stream));
   VL_CHECK(cudaStreamSynchronize(b->stream));
   b->content_valid = false;
   b->pivot_valid = false;
   return VLGPU_OK;
}

}  // extern "C"
