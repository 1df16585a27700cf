// SLICE-3D one-dimensional acceleration remap on sparse 4x4x4 velocity blocks
// for sm_100a.  One sweep is two kernels:
//
//   columnize_kernel  one CTA per cell.  Builds the cell's column structure
//                     for the sweep dimension from 96-bit occupancy masks in
//                     shared memory (one mask per transverse block pair),
//                     computes each column's target block range with the
//                     reference's rule (cpu_acc_map.cpp:258-324), allocates
//                     the cell's output blocks and writes one ColumnSet record
//                     per transverse pair plus the source permutation.
//
//   remap_pair_kernel (fused arithmetic, PPM and PLM), remap_walk_kernel
//                     (fused, PQM) or remap_kernel (the exact mode):
//                     persistent; eight lanes (pair) or a half-warp take one
//                     ColumnSet and walk it along the sweep dimension, two
//                     columns or one of the 4x4 block face per lane.  The
//                     reconstruction is built in registers from a sliding
//                     window of the column; each source cell's mass goes to
//                     the Lagrangian target cells it overlaps in a per-lane
//                     ring of 8 target blocks in shared memory, and completed
//                     target blocks are streamed out.  Every output block is
//                     written exactly once, so no zero fill and no atomics are
//                     needed.
//
// remap_kernel follows the reference's scalar build operation by operation
// (round-to-nearest intrinsics, no contraction, the double-precision products
// of cpu_face_estimates.hpp:163 and cpu_acc_map.cpp:585), so its results are
// bit-identical to the reference's map_1d on the same inputs.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "fused_ppm.cuh"
#include "vlgpu_common.cuh"

namespace vlgpu {

// ---------------------------------------------------------------------------
// exact IEEE single-precision helpers (never contracted into FMA)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }
// double constant times float, rounded once to float (VecSimple<float> * double)
__device__ __forceinline__ float dmf(double c, float x) { return __double2float_rn(__dmul_rn(c, (double)x)); }

// h4 left face value, cpu_face_estimates.hpp:160-167
__device__ __forceinline__ float h4_face(float vm2, float vm1, float v0, float vp1) {
   float s = fa(-vm2, fm(7.0f, vm1));
   s = fa(s, fm(7.0f, v0));
   s = fs(s, vp1);
   return dmf(1.0 / 12.0, s);
}

__device__ __forceinline__ float minmod(float s1, float s2) {
   const float slope = (fabsf(s1) < fabsf(s2)) ? s1 : s2;
   return (fm(s1, s2) <= 0.0f) ? 0.0f : slope;
}
__device__ __forceinline__ float maxmod(float s1, float s2) {
   const float slope = (fabsf(s1) > fabsf(s2)) ? s1 : s2;
   return (fm(s1, s2) <= 0.0f) ? 0.0f : slope;
}

// PPM coefficients of cpu_1d_ppm.hpp:35-54 (filtered h4 faces, superbee,
// Colella-Woodward monotonicity) for the cell with neighbours vm1, vp1 and
// raw faces fl (left) / fr (right).
__device__ __forceinline__ void ppm_coeff(float vm1, float v0, float vp1, float fl, float fr, float threshold,
                                          float scale, float& a0, float& a1, float& a2) {
   const float l = fm(vm1, scale), m = fm(v0, scale), r = fm(vp1, scale);
   const float a = fs(r, m), b = fs(m, l);
   const float s1 = minmod(a, fm(2.0f, b));
   const float s2 = minmod(fm(2.0f, a), b);
   const float slope = maxmod(s1, s2);
   const float slope_abs = fm(fabsf(slope), threshold);
   const float slope_sign = (slope > 0.0f) ? 1.0f : -1.0f;
   if (slope_abs == 0.0f) {
      fr = v0;
      fl = v0;
   }
   const float half_slope = fm(fm(slope_sign, 0.5f), slope_abs);
   if (fm(fs(vm1, fl), fs(fl, v0)) < 0.0f) fl = fs(v0, half_slope);
   if (fm(fs(vp1, fr), fs(fr, v0)) < 0.0f) fr = fa(v0, half_slope);
   const float one_sixth = (float)(1.0 / 6.0);
   {
      const float d = fs(fr, fl);
      const float e = fs(v0, fm(0.5f, fa(fl, fr)));
      if (fm(d, e) > fm(fm(d, d), one_sixth)) fl = fs(fm(3.0f, v0), fm(2.0f, fr));
   }
   {
      const float d = fs(fr, fl);
      const float e = fs(v0, fm(0.5f, fa(fl, fr)));
      if (fm(fm(-d, d), one_sixth) > fm(d, e)) fr = fs(fm(3.0f, v0), fm(2.0f, fl));
   }
   a0 = fl;
   a1 = fs(fs(fm(3.0f, v0), fm(2.0f, fl)), fr);
   a2 = fs(fa(fl, fr), fm(2.0f, v0));
}

// ---------------------------------------------------------------------------
// 96-bit mask helpers
// ---------------------------------------------------------------------------
// Word q (0..2) of a mask, chosen with selects so that a mask held in
// registers is never indexed dynamically (which would move it to local memory).
__device__ __forceinline__ uint32_t mask_word(const uint32_t m[3], int q) {
   return q == 0 ? m[0] : (q == 1 ? m[1] : m[2]);
}
__device__ __forceinline__ int mask_next_set(const uint32_t m[3], int k) {
   for (; k < 96; k = (k | 31) + 1) {
      const uint32_t w = mask_word(m, k >> 5) >> (k & 31);
      if (w) return k + __ffs(w) - 1;
   }
   return 96;
}
__device__ __forceinline__ int mask_next_clear(const uint32_t m[3], int k) {
   for (; k < 96; k = (k | 31) + 1) {
      const uint32_t w = (~mask_word(m, k >> 5)) >> (k & 31);
      if (w) return k + __ffs(w) - 1;
   }
   return 96;
}

// Target block range of one column (cpu_acc_map.cpp:307-338).  Returns true
// when the range violates the wall margin.
__device__ __forceinline__ bool column_extent(float mx, float mn, float dk, float dv, float v_min, int max_len,
                                              int first_k, int last_k, int wall_margin, int& fb, int& lb) {
   const float first_min_v = fa(fm((float)(WID * first_k), dv), v_min);
   const float last_max_v = fa(fm((float)(WID * (last_k + 1)), dv), v_min);
   const int first_gk = __float2int_rz(fd(fs(first_min_v, mx), dk));
   const int last_gk = __float2int_rz(fd(fs(last_max_v, mn), dk));
   fb = first_gk / WID;
   lb = last_gk / WID;
   fb = (fb >= 0) ? fb : 0;
   fb = (fb < max_len) ? fb : max_len - 1;
   lb = (lb >= 0) ? lb : 0;
   lb = (lb < max_len) ? lb : max_len - 1;
   return fb < wall_margin || fb >= max_len - wall_margin || lb < wall_margin || lb >= max_len - wall_margin;
}

// The set's corner extremes of the Lagrangian starting point
// (cpu_acc_map.cpp:258-288), evaluated exactly as the reference does.
__device__ __forceinline__ void set_corners(const SweepCell& P, uint32_t si, uint32_t sj, float& mx, float& mn) {
   const float A0 = (float)(si * WID), A1 = (float)(si * WID + WID - 1);
   const float B0 = (float)(sj * WID), B1 = (float)(sj * WID + WID - 1);
   const float c00 = fa(fa(P.intersection, fm(A0, P.di)), fm(B0, P.dj));
   const float c01 = fa(fa(P.intersection, fm(A0, P.di)), fm(B1, P.dj));
   const float c10 = fa(fa(P.intersection, fm(A1, P.di)), fm(B0, P.dj));
   const float c11 = fa(fa(P.intersection, fm(A1, P.di)), fm(B1, P.dj));
   mx = c00;
   mx = (mx < c01) ? c01 : mx;
   mx = (mx < c10) ? c10 : mx;
   mx = (mx < c11) ? c11 : mx;
   mn = c00;
   mn = (c01 < mn) ? c01 : mn;
   mn = (c10 < mn) ? c10 : mn;
   mn = (c11 < mn) ? c11 : mn;
}

// ---------------------------------------------------------------------------
// columnize: one CTA per cell
// ---------------------------------------------------------------------------
// Threads per CTA (launch_columnize_batch).  Where every cell has an SM to
// itself the largest cell is the launch's time, so its CTA is as large as can
// be; up to eight cells per SM the largest ones still decide; with more cells
// six small CTAs share an SM and hide one another's barriers.  A step of 13
// cells of 12000 blocks, with 1024 threads: 1215 -> 872 us; of 1024 drifting
// cells (512 against 256 threads, the adjustment's lists likewise): 1451 ->
// 1375 us; of 4096: 512 threads take 2% longer than 256.
constexpr int COL_THREADS = 256;
constexpr int COL_MID_THREADS = 512;
constexpr int COL_FEW_THREADS = 1024;
constexpr int COL_UNROLL = 4;  // list entries a thread has in flight
constexpr uint32_t NO_BLOCK = 0xffffffffu;  // a list entry without data: all zero

// Swapped indices of a block ID, by the mesh's reciprocals.
template <int DIM>
__device__ __forceinline__ void swapped_of(const MeshDev& mesh, uint32_t gid, uint32_t s[3]) {
   uint32_t x, y, z;
   block_xyz(mesh, gid, x, y, z);
   s[0] = (DIM == 0) ? z : x;
   s[1] = (DIM == 1) ? z : y;
   s[2] = (DIM == 0) ? x : (DIM == 1 ? y : z);
}

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   uint32_t x = v;
#pragma unroll
   for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
   }
   if (lane == 31) warp_sums[warp] = x;
   __syncthreads();
   if (warp == 0) {
      const int nw = blockDim.x >> 5;
      uint32_t s = (lane < nw) ? warp_sums[lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
         const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
         if (lane >= o) s += y;
      }
      if (lane < nw) warp_sums[lane] = s;
   }
   __syncthreads();
   total = warp_sums[(blockDim.x >> 5) - 1];
   const uint32_t before = (warp > 0) ? warp_sums[warp - 1] : 0u;
   __syncthreads();
   return before + x - v;
}

// The column structure of one cell, by the whole CTA (see the file header).
template <int DIM, bool FULL_PLANE>
__device__ __forceinline__ void columnize_cell(
   uint32_t cell, const uint32_t* __restrict__ gids, const uint32_t* __restrict__ src_index,
   const CellSlot* __restrict__ src_slots, CellSlot* __restrict__ dst_slots, uint32_t* __restrict__ perm,
   ColumnSet* __restrict__ sets, uint32_t set_capacity, uint32_t dst_capacity,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, SweepCounters* __restrict__ counters,
   BatchStats* __restrict__ stats, const MeshDev& mesh, int wall_margin, int first_of_step, uint32_t zero_row,
   uint32_t plane_cap, uint32_t* __restrict__ wide_cells) {
   extern __shared__ uint32_t smem[];
   __shared__ uint32_t warp_sums[32];
   __shared__ uint32_t s_bbox[4];
   __shared__ uint32_t s_set_base, s_dst_base, s_nsets, s_ntgt, s_flags;
   __shared__ uint32_t s_bin[MAX_LEN + 1];  // sets by length, longest first: count, then first record

   const CellSlot src = src_slots[cell];
   const SweepCell P = sweep_cells[cell];
   uint32_t li, lj;
   plane_lengths(mesh.len, DIM, li, lj);
   const int max_len = (int)mesh.len[DIM];

   if (threadIdx.x == 0) {
      s_bbox[0] = 0xffffffffu; s_bbox[1] = 0; s_bbox[2] = 0xffffffffu; s_bbox[3] = 0;
      s_flags = 0;
   }
   __syncthreads();
   if (src.count == 0) {
      if (threadIdx.x == 0) dst_slots[cell] = CellSlot{0u, 0u};
      return;
   }
   constexpr uint32_t FULL = 0xffffffffu;
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   // pass 1: bounding box of the transverse indices (warp reductions, one
   // shared min/max per warp).  With shared memory for the whole plane, a list
   // longer than the plane is not passed over for its box: six steps of 13 cells of
   // 12000 blocks 2724 -> 2610 us.  A short list's box is the cheaper one: one cell
   // of 412 blocks 680 us with it, 705 without.
   const bool whole = FULL_PLANE && src.count > li * lj;
   if (!whole) {
      uint32_t a0 = 0xffffffffu, a1 = 0, b0 = 0xffffffffu, b1 = 0;
      for (uint32_t t = threadIdx.x; t < src.count; t += blockDim.x * COL_UNROLL) {
         // (an entry past the end repeats the thread's first one)
         uint32_t g[COL_UNROLL];
#pragma unroll
         for (int u = 0; u < COL_UNROLL; ++u) {
            const uint32_t b = t + blockDim.x * u;
            g[u] = gids[src.off + (b < src.count ? b : t)];
         }
#pragma unroll
         for (int u = 0; u < COL_UNROLL; ++u) {
            uint32_t s[3];
            swapped_of<DIM>(mesh, g[u], s);
            a0 = min(a0, s[0]); a1 = max(a1, s[0]);
            b0 = min(b0, s[1]); b1 = max(b1, s[1]);
         }
      }
      a0 = __reduce_min_sync(FULL, a0); a1 = __reduce_max_sync(FULL, a1);
      b0 = __reduce_min_sync(FULL, b0); b1 = __reduce_max_sync(FULL, b1);
      if (lane == 0) {
         atomicMin(&s_bbox[0], a0); atomicMax(&s_bbox[1], a1);
         atomicMin(&s_bbox[2], b0); atomicMax(&s_bbox[3], b1);
      }
   }
   __syncthreads();
   const uint32_t a_lo = whole ? 0u : s_bbox[0], b_lo = whole ? 0u : s_bbox[2];
   const uint32_t na = whole ? li : s_bbox[1] - a_lo + 1, nb = whole ? lj : s_bbox[3] - b_lo + 1;
   const uint32_t plane = na * nb;
   if (plane > plane_cap) {
      // too wide for this launch's shared memory: left to columnize_wide_kernel
      if (threadIdx.x == 0) wide_cells[atomicAdd(&counters->n_wide, 1u)] = cell;
      return;
   }
   uint32_t* mask = smem;                   // 3 * plane
   uint32_t* prefix = smem + 3 * plane;     // plane
   uint16_t* set_t = (uint16_t*)(prefix + plane);  // plane (set index -> t)
   uint16_t* rank = (uint16_t*)(prefix + plane + (plane + 1) / 2);  // plane (set index -> record)
   uint32_t* tcount = prefix + plane + 2 * ((plane + 1) / 2);       // plane
   for (uint32_t q = threadIdx.x; q < 3 * plane; q += blockDim.x) mask[q] = 0;
   for (uint32_t q = threadIdx.x; q <= MAX_LEN; q += blockDim.x) s_bin[q] = 0;
   __syncthreads();
   // pass 2: occupancy masks along the sweep dimension; where the list runs
   // along the sweep (the x sweep of a list in ID order) the lanes that set
   // bits of one word combine them first
   for (uint32_t t = warp * 32; t < src.count; t += blockDim.x * COL_UNROLL) {
      uint32_t g[COL_UNROLL];
#pragma unroll
      for (int u = 0; u < COL_UNROLL; ++u) {
         const uint32_t b = t + blockDim.x * u + lane;
         g[u] = (b < src.count) ? gids[src.off + b] : 0u;
      }
#pragma unroll
      for (int u = 0; u < COL_UNROLL; ++u) {
         const uint32_t b = t + blockDim.x * u + lane;
         uint32_t key = 0xffffffffu, bit = 0u;
         if (b < src.count) {
            uint32_t s[3];
            swapped_of<DIM>(mesh, g[u], s);
            key = 3 * ((s[0] - a_lo) * nb + (s[1] - b_lo)) + (s[2] >> 5);
            bit = 1u << (s[2] & 31);
         }
         const uint32_t left = __shfl_up_sync(FULL, key, 1);
         const bool run = __popc(__ballot_sync(FULL, lane > 0 && key == left && key != 0xffffffffu)) >= 12;
         if (!run) {
            if (key != 0xffffffffu) atomicOr(&mask[key], bit);
            continue;
         }
         const uint32_t match = __match_any_sync(FULL, key);
         const bool big = key != 0xffffffffu && __popc(match) >= 4;
         if (key != 0xffffffffu && !big) atomicOr(&mask[key], bit);
         for (uint32_t leaders = __ballot_sync(FULL, big && (int)lane == __ffs(match) - 1); leaders;
              leaders &= leaders - 1) {
            const int leader = __ffs(leaders) - 1;
            const bool mine = (__shfl_sync(FULL, match, leader) >> lane) & 1u;
            const uint32_t bits = __reduce_or_sync(FULL, mine ? bit : 0u);
            if ((int)lane == leader) atomicOr(&mask[key], bits);
         }
      }
   }
   __syncthreads();
   // scan over the plane: source offsets and set indices
   const uint32_t chunk = (plane + blockDim.x - 1) / blockDim.x;
   const uint32_t t0 = min(plane, threadIdx.x * chunk), t1 = min(plane, t0 + chunk);
   uint32_t my_blocks = 0, my_sets = 0;
   for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t n = __popc(mask[3 * t]) + __popc(mask[3 * t + 1]) + __popc(mask[3 * t + 2]);
      my_blocks += n;
      my_sets += (n > 0);
   }
   uint32_t tot_blocks, tot_sets;
   uint32_t blk_base = block_exclusive_scan(my_blocks, warp_sums, tot_blocks);
   uint32_t set_base = block_exclusive_scan(my_sets, warp_sums, tot_sets);
   for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t n = __popc(mask[3 * t]) + __popc(mask[3 * t + 1]) + __popc(mask[3 * t + 2]);
      prefix[t] = blk_base;
      blk_base += n;
      if (n > 0) {
         set_t[set_base++] = (uint16_t)t;
         atomicAdd(&s_bin[MAX_LEN - n], 1u);
      }
   }
   if (threadIdx.x == 0) {
      const uint32_t base = atomicAdd(&counters->n_sets, tot_sets);
      s_set_base = base;
      s_nsets = tot_sets;
      if (base + tot_sets > set_capacity) s_flags |= VLGPU_CELL_NOMEM;
   }
   __syncthreads();
   // the records go by length, so that the sets a warp of the remap walks in
   // step are equally long (28 -> 30.5 of 32 lanes busy, 10% fewer instructions; six
   // steps of 4096 cells 31.5 -> 29.3 ms); the output keeps the sets' order
   if (warp == 0) {
      constexpr int PER = (MAX_LEN + 1 + 31) / 32;
      uint32_t n[PER], sum = 0;
#pragma unroll
      for (int q = 0; q < PER; ++q) {
         const int k = (int)lane * PER + q;
         n[q] = (k <= MAX_LEN) ? s_bin[k] : 0u;
         sum += n[q];
      }
      uint32_t x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
         const uint32_t y = __shfl_up_sync(FULL, x, o);
         if ((int)lane >= o) x += y;
      }
      x -= sum;
#pragma unroll
      for (int q = 0; q < PER; ++q) {
         const int k = (int)lane * PER + q;
         if (k <= MAX_LEN) s_bin[k] = x;
         x += n[q];
      }
   }
   __syncthreads();
   const bool sets_ok = !(s_flags & VLGPU_CELL_NOMEM);
   // per set: target mask from the column extents
   uint32_t wall = 0, baddk = 0;
   for (uint32_t s = threadIdx.x; s < tot_sets; s += blockDim.x) {
      const uint32_t t = set_t[s];
      const uint32_t si = a_lo + t / nb, sj = b_lo + t % nb;
      uint32_t m[3] = {mask[3 * t], mask[3 * t + 1], mask[3 * t + 2]};
      uint32_t tm[3] = {0u, 0u, 0u};
      if (P.flags & SWEEP_PASS) {
         // the cell's blocks pass through the sweep unchanged
         tm[0] = m[0]; tm[1] = m[1]; tm[2] = m[2];
      } else {
         float mx, mn;
         set_corners(P, si, sj, mx, mn);
         if (!(P.dk > 0.0f)) baddk = 1;
         int k = mask_next_set(m, 0);
         while (k < 96) {
            const int e = mask_next_clear(m, k) - 1;
            int fb, lb;
            if (column_extent(mx, mn, P.dk, mesh.dv[DIM], mesh.vmin[DIM], max_len, k, e, wall_margin, fb, lb))
               wall = 1;
#pragma unroll
            for (int w = 0; w < 3; ++w) {
               const int q0 = max(fb - 32 * w, 0), q1 = min(lb - 32 * w, 31);
               if (q0 <= q1) tm[w] |= (0xffffffffu << q0) & (0xffffffffu >> (31 - q1));
            }
            k = mask_next_set(m, e + 1);
         }
      }
      tcount[s] = __popc(tm[0]) + __popc(tm[1]) + __popc(tm[2]);
      if (sets_ok) {
         ColumnSet cs;
         cs.cell = cell;
         cs.sij = si | (sj << 16);
         cs.src_pos = src.off + prefix[t];
         cs.dst_pos = 0;
         cs.src_mask[0] = m[0]; cs.src_mask[1] = m[1]; cs.src_mask[2] = m[2];
         cs.tgt_mask[0] = tm[0]; cs.tgt_mask[1] = tm[1]; cs.tgt_mask[2] = tm[2];
         const uint32_t r = atomicAdd(&s_bin[MAX_LEN - (__popc(m[0]) + __popc(m[1]) + __popc(m[2]))], 1u);
         rank[s] = (uint16_t)r;
         sets[s_set_base + r] = cs;
      }
   }
   if (wall) atomicOr(&s_flags, VLGPU_CELL_WALL);
   if (baddk) atomicOr(&s_flags, VLGPU_CELL_BADDK);
   __syncthreads();
   // scan of target counts over sets -> output positions
   const uint32_t sch = (tot_sets + blockDim.x - 1) / blockDim.x;
   const uint32_t q0 = min(tot_sets, threadIdx.x * sch), q1 = min(tot_sets, q0 + sch);
   uint32_t my_t = 0;
   for (uint32_t s = q0; s < q1; ++s) my_t += tcount[s];
   uint32_t tot_t;
   uint32_t tbase = block_exclusive_scan(my_t, warp_sums, tot_t);
   if (threadIdx.x == 0) {
      const uint32_t base = atomicAdd(&counters->dst_top, tot_t);
      s_dst_base = base;
      s_ntgt = tot_t;
      if ((uint64_t)base + tot_t > dst_capacity) s_flags |= VLGPU_CELL_NOMEM;
   }
   __syncthreads();
   const bool ok = !(s_flags & VLGPU_CELL_NOMEM);
   if (ok) {
      for (uint32_t s = q0; s < q1; ++s) {
         sets[s_set_base + rank[s]].dst_pos = s_dst_base + tbase;
         tbase += tcount[s];
      }
      // source permutation in (set, k) order
      for (uint32_t e = threadIdx.x; e < src.count; e += blockDim.x * COL_UNROLL) {
         uint32_t g[COL_UNROLL], row[COL_UNROLL];
#pragma unroll
         for (int u = 0; u < COL_UNROLL; ++u) {
            const uint32_t b = e + blockDim.x * u, at = src.off + (b < src.count ? b : e);
            g[u] = gids[at];
            row[u] = src_index ? src_index[at] : at;
            row[u] = (row[u] == NO_BLOCK) ? zero_row : row[u];
         }
#pragma unroll
         for (int u = 0; u < COL_UNROLL; ++u) {
            if (e + blockDim.x * u >= src.count) break;
            uint32_t s[3];
            swapped_of<DIM>(mesh, g[u], s);
            const uint32_t t = (s[0] - a_lo) * nb + (s[1] - b_lo);
            perm[src.off + prefix[t] + (uint32_t)mask_popc_below(&mask[3 * t], s[2])] = row[u];
         }
      }
   } else if (sets_ok) {
      // no room for the output: neutralise this cell's sets
      for (uint32_t s = threadIdx.x; s < tot_sets; s += blockDim.x) {
         sets[s_set_base + s].tgt_mask[0] = 0;
         sets[s_set_base + s].tgt_mask[1] = 0;
         sets[s_set_base + s].tgt_mask[2] = 0;
         sets[s_set_base + s].src_mask[0] = 0;
         sets[s_set_base + s].src_mask[1] = 0;
         sets[s_set_base + s].src_mask[2] = 0;
      }
   }
   if (threadIdx.x == 0) {
      atomicAdd(&stats->src_blocks, (unsigned long long)src.count);
      atomicAdd(&stats->dst_blocks, (unsigned long long)(ok ? s_ntgt : 0u));
      atomicAdd(&stats->sweeps, 1ull);
      atomicAdd(&stats->sets, (unsigned long long)tot_sets);
      if (first_of_step) atomicAdd(&stats->step_blocks, (unsigned long long)src.count);
      dst_slots[cell] = ok ? CellSlot{s_dst_base, s_ntgt} : CellSlot{0u, 0u};
      if (s_flags) atomicOr(&status[cell], s_flags);
      if (!ok) atomicOr(&counters->overflow, 1u);
   }
}

// One CTA per cell of [cell_begin, cell_end).
template <int DIM, int THREADS>
__global__ void __launch_bounds__(THREADS) columnize_kernel(
   const uint32_t* __restrict__ gids, const uint32_t* __restrict__ src_index, const CellSlot* __restrict__ src_slots,
   CellSlot* __restrict__ dst_slots, uint32_t* __restrict__ perm, ColumnSet* __restrict__ sets,
   uint32_t set_capacity, uint32_t dst_capacity,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, SweepCounters* __restrict__ counters,
   BatchStats* __restrict__ stats, MeshDev mesh, int wall_margin, uint32_t cell_begin, uint32_t cell_end,
   int first_of_step, uint32_t zero_row, const uint32_t* __restrict__ order, uint32_t plane_cap,
   uint32_t* __restrict__ wide_cells, const uint32_t* __restrict__ stop) {
   if (cell_begin + blockIdx.x >= cell_end || (stop && *stop)) return;
   const uint32_t cell = order ? order[blockIdx.x] : cell_begin + blockIdx.x;
   columnize_cell<DIM, THREADS == COL_FEW_THREADS>(cell, gids, src_index, src_slots, dst_slots, perm, sets,
                                                   set_capacity, dst_capacity, sweep_cells, status, counters, stats,
                                                   mesh, wall_margin, first_of_step, zero_row, plane_cap, wide_cells);
}

// Persistent CTAs over the cells whose plane did not fit the capped launch
// (wide_cells, counters->n_wide of them), with a full plane of shared memory.
template <int DIM>
__global__ void __launch_bounds__(COL_FEW_THREADS) columnize_wide_kernel(
   const uint32_t* __restrict__ gids, const uint32_t* __restrict__ src_index, const CellSlot* __restrict__ src_slots,
   CellSlot* __restrict__ dst_slots, uint32_t* __restrict__ perm, ColumnSet* __restrict__ sets,
   uint32_t set_capacity, uint32_t dst_capacity,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, SweepCounters* __restrict__ counters,
   BatchStats* __restrict__ stats, MeshDev mesh, int wall_margin, int first_of_step, uint32_t zero_row,
   const uint32_t* __restrict__ wide_cells) {
   const uint32_t n = counters->n_wide;
   for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
      columnize_cell<DIM, true>(wide_cells[it], gids, src_index, src_slots, dst_slots, perm, sets, set_capacity,
                          dst_capacity, sweep_cells, status, counters, stats, mesh, wall_margin, first_of_step,
                          zero_row, 0xffffffffu, nullptr);
      __syncthreads();  // the next cell reuses the shared state
   }
}

// Dynamic shared memory of columnize for a full transverse plane.
size_t columnize_smem_bytes(uint32_t plane) {
   return sizeof(uint32_t) * (3 * plane + plane + 2 * ((plane + 1) / 2) + plane) + 16;
}

// ---------------------------------------------------------------------------
// remap: persistent, one half-warp per column set
// ---------------------------------------------------------------------------
constexpr int REMAP_THREADS = 256;
constexpr int RING_BLOCKS = 8;               // target blocks held per set
constexpr int RING_CELLS = RING_BLOCKS * WID;  // per lane
constexpr int RING_STRIDE = RING_CELLS * 16 + 16;  // floats per half-warp (+16 pad: bank shift)
// remap_walk_kernel keeps each lane's ring contiguous: 32 cells padded to 36
// floats, so a block's four cells are one aligned 16-byte access (lanes that
// store to the same slot share 8 bank groups, a conflict the measured kernel
// pays for less than it saves in flush instructions)
constexpr int WALK_LANE_STRIDE = RING_CELLS + 4;

template <int DIM>
__device__ __forceinline__ int cell_offset(int i, int j, int g) {
   if (DIM == 0) return i * WID2 + j * WID + g;
   if (DIM == 1) return i + j * WID2 + g * WID;
   return i + j * WID + g * WID2;
}

// How the workers of a remap launch (warps, half-warps) take the column sets.
// A worker's first sets follow from its number, neighbours on different SMs;
// only further ones come from the counter.  A launch with fewer sets than
// workers touches no counter: taking every set from it made the 592 CTAs of
// a one-cell sweep queue 9472 atomics on one address (15.3 us for 100 sets).
struct SetClaims {
   SweepCounters* counters;
   uint32_t begin, n_sets, dynamic;  // the launch's first set, the end, the first set given out by the counter
   __device__ __forceinline__ SetClaims(SweepCounters* c, uint32_t n) : counters(c), begin(c->first_set), n_sets(n), dynamic(n) {}
   // worker w of the CTA's `workers`, `each` sets at a time
   __device__ __forceinline__ uint32_t first(uint32_t w, uint32_t workers, uint32_t each) {
      dynamic = begin + workers * gridDim.x * each;
      return begin + (w * gridDim.x + blockIdx.x) * each;
   }
   // `leader` asks for the lanes of `mask` (aligned segments of `width` lanes)
   __device__ __forceinline__ uint32_t next(bool leader, unsigned mask, int width, uint32_t each) {
      if (dynamic >= n_sets) return n_sets;
      uint32_t s = 0;
      if (leader) s = dynamic + atomicAdd(&counters->work, each);
      return __shfl_sync(mask, s, 0, width);
   }
};


__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

template <int DIM>
__device__ __forceinline__ void load_lane(const float* __restrict__ data, uint32_t idx, int i, int j, float v[4]) {
   const float* __restrict__ blk = data + (size_t)idx * WID3;
   if (DIM == 0) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(blk + cell_offset<0>(i, j, 0)));
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
   } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) v[g] = __ldg(blk + cell_offset<DIM>(i, j, g));
   }
}

template <int DIM>
__device__ __forceinline__ void store_lane(float* __restrict__ blk, int i, int j, const float v[4]) {
   if (DIM == 0) {
      *reinterpret_cast<float4*>(blk + cell_offset<0>(i, j, 0)) = make_float4(v[0], v[1], v[2], v[3]);
   } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) blk[cell_offset<DIM>(i, j, g)] = v[g];
   }
}

// The set of a cell that is not accelerated in this step (SWEEP_PASS): its
// blocks are copied to the output in ascending k, which is the target mask's
// order (columnize gave the set its source mask as the target mask), with
// their block IDs and content flags.
template <int DIM>
__device__ __forceinline__ void pass_through_set(const ColumnSet& cs, const uint32_t* __restrict__ perm,
                                                 const float* __restrict__ src_data, float* __restrict__ dst_data,
                                                 uint32_t* __restrict__ dst_gids, uint8_t* __restrict__ content_out,
                                                 const MeshDev& mesh, float content_thr, int lane, unsigned hmask) {
   const int i = lane & 3, j = lane >> 2;
   uint32_t r = 0;
   for (int k = mask_next_set(cs.src_mask, 0); k < 96; k = mask_next_set(cs.src_mask, k + 1), ++r) {
      float v[4];
      load_lane<DIM>(src_data, perm[cs.src_pos + r], i, j, v);
      const uint32_t o = cs.dst_pos + r;
      store_lane<DIM>(dst_data + (size_t)o * WID3, i, j, v);
      const bool c = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])) >= content_thr;
      const unsigned any_c = __ballot_sync(hmask, c) & hmask;
      if (lane == 0) {
         dst_gids[o] = gid_from_swapped(cs.si(), cs.sj(), (uint32_t)k, mesh.len, DIM);
         content_out[o] = any_c ? 1 : 0;
      }
   }
}

// Reference argmax / argmin lane selection (cpu_acc_map.cpp:515-529): the
// first lane holding the largest value above DBL_MIN (default lane 0) and the
// first lane holding the smallest value below DBL_MAX (default lane 0).
__device__ __forceinline__ void select_lanes(float lag, int lane, unsigned hmask, int& max_lane, int& min_lane) {
   bool vmax = (double)lag > DBL_MIN;
   float xmax = lag;
   int imax = lane;
   bool vmin = (double)lag < DBL_MAX;
   float xmin = lag;
   int imin = lane;
#pragma unroll
   for (int o = 8; o >= 1; o >>= 1) {
      const bool ov = __shfl_xor_sync(hmask, vmax, o, 16);
      const float ox = __shfl_xor_sync(hmask, xmax, o, 16);
      const int oi = __shfl_xor_sync(hmask, imax, o, 16);
      if (ov && (!vmax || ox > xmax || (ox == xmax && oi < imax))) { vmax = true; xmax = ox; imax = oi; }
      const bool nv = __shfl_xor_sync(hmask, vmin, o, 16);
      const float nx = __shfl_xor_sync(hmask, xmin, o, 16);
      const int ni = __shfl_xor_sync(hmask, imin, o, 16);
      if (nv && (!vmin || nx < xmin || (nx == xmin && ni < imin))) { vmin = true; xmin = nx; imin = ni; }
   }
   max_lane = vmax ? imax : 0;
   min_lane = vmin ? imin : 0;
}

template <int DIM>
__global__ void __launch_bounds__(REMAP_THREADS, 3) remap_kernel(
   const ColumnSet* __restrict__ sets, SweepCounters* __restrict__ counters, const uint32_t* __restrict__ perm,
   const float* __restrict__ src_data, float* __restrict__ dst_data, uint32_t* __restrict__ dst_gids,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, MeshDev mesh, int wall_margin,
   uint32_t set_capacity, uint8_t* __restrict__ content_out, double content_threshold, const HandOver after) {
   hand_over(after, counters);
   __shared__ float ring_all[(REMAP_THREADS / 16) * RING_STRIDE];
   const int hw = threadIdx.x >> 4;
   const int lane = threadIdx.x & 15;
   const unsigned hmask = 0xffffu << (threadIdx.x & 16);
   float* ring = ring_all + hw * RING_STRIDE;
   const int i = lane & 3, j = lane >> 2;
   uint32_t n_sets = counters->n_sets;
   n_sets = (n_sets < set_capacity) ? n_sets : set_capacity;
   SetClaims claims(counters, n_sets);
   const int max_len = (int)mesh.len[DIM];
   const float dv = mesh.dv[DIM], v_min = mesh.vmin[DIM];
   const double i_dv = 1.0 / (double)dv;
   // (double)v >= content_threshold  <=>  v >= the smallest float >= the threshold
   const float content_thr = __double2float_ru(content_threshold);

   // the ring starts empty; every set flushes all its targets, and a flush
   // zeroes the slots it reads, so the ring is empty again at each set start
#pragma unroll
   for (int q = 0; q < RING_CELLS; ++q) ring[q * 16 + lane] = 0.0f;
   for (uint32_t sidx = claims.first(hw, REMAP_THREADS / 16, 1u); sidx < n_sets;
        sidx = claims.next(lane == 0, hmask, 16, 1u)) {
      const ColumnSet cs = sets[sidx];
      const SweepCell P = sweep_cells[cs.cell];
      if (P.flags & SWEEP_PASS) {
         pass_through_set<DIM>(cs, perm, src_data, dst_data, dst_gids, content_out, mesh, content_thr, lane, hmask);
         continue;
      }
      const float threshold = P.threshold;
      const float scale = __double2float_rn(1.0 / (double)threshold);
      const float dk = P.dk;
      // lane's Lagrangian starting point (cpu_acc_map.cpp:493-496)
      const float A = fa((float)(cs.si() * WID), (float)i);
      const float B = fa((float)(cs.sj() * WID), (float)j);
      const float im = fa(fa(P.intersection, fm(A, P.di)), fm(B, P.dj));
      float mx, mn;
      set_corners(P, cs.si(), cs.sj(), mx, mn);
      int next_flush = mask_next_set(cs.tgt_mask, 0);
      uint32_t out_idx = 0;
      bool range_err = false;

      // writes out every target block below `limit_block` that is still held
      auto flush_until = [&](int limit_block) {
         while (next_flush < 96 && next_flush < limit_block) {
            float v[4];
            const int slot = (next_flush & (RING_BLOCKS - 1)) * WID;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
               v[g] = ring[(slot + g) * 16 + lane];
               ring[(slot + g) * 16 + lane] = 0.0f;
            }
            const uint32_t o = cs.dst_pos + out_idx;
            store_lane<DIM>(dst_data + (size_t)o * WID3, i, j, v);
            // content flag of the finished block (compute_block_has_content)
            const bool c = (v[0] >= content_thr) | (v[1] >= content_thr) | (v[2] >= content_thr) |
                           (v[3] >= content_thr);
            const unsigned any_c = __ballot_sync(hmask, c) & hmask;
            if (lane == 0) {
               dst_gids[o] = gid_from_swapped(cs.si(), cs.sj(), (uint32_t)next_flush, mesh.len, DIM);
               content_out[o] = any_c ? 1 : 0;
            }
            ++out_idx;
            next_flush = mask_next_set(cs.tgt_mask, next_flush + 1);
         }
      };

      int src_rank = 0;
      int col_s = mask_next_set(cs.src_mask, 0);
      int col_e = (col_s < 96) ? mask_next_clear(cs.src_mask, col_s) - 1 : 95;
      int cf = 0, cl = 0;
      if (col_s < 96) column_extent(mx, mn, dk, dv, v_min, max_len, col_s, col_e, wall_margin, cf, cl);
      while (col_s < 96) {
         const int nxt_s = mask_next_set(cs.src_mask, col_e + 1);
         int nxt_e = 95, ncf = 1 << 20, ncl = 0;
         if (nxt_s < 96) {
            nxt_e = mask_next_clear(cs.src_mask, nxt_s) - 1;
            column_extent(mx, mn, dk, dv, v_min, max_len, nxt_s, nxt_e, wall_margin, ncf, ncl);
         }
         // ---- map one column (cpu_acc_map.cpp:395-631) ----
         float v_r = fa(fm((float)(WID * col_s), dv), v_min);
         int gk_r;
         int max_lane = 0, min_lane = 0;
         {
            const float lag = fd(fs(v_r, im), dk);
            gk_r = __float2int_rz(lag);
            select_lanes(lag, lane, hmask, max_lane, min_lane);
         }
         const int gk_lo_col = cf * WID, gk_hi_col = (cl + 1) * WID - 1;
         float pw[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // the previous block (zero padding at a column start)
         float cur[4], nxt[4];
         load_lane<DIM>(src_data, perm[cs.src_pos + src_rank], i, j, cur);
         if (col_e > col_s) {
            load_lane<DIM>(src_data, perm[cs.src_pos + src_rank + 1], i, j, nxt);
         } else {
            nxt[0] = nxt[1] = nxt[2] = nxt[3] = 0.0f;
         }
         // raw left face of the column's first cell
         float face = h4_face(pw[2], pw[3], cur[0], cur[1]);
         for (int kb = col_s; kb <= col_e; ++kb) {
            float nn[4];
            if (kb + 2 <= col_e) {
               load_lane<DIM>(src_data, perm[cs.src_pos + src_rank + 2], i, j, nn);
            } else {
               nn[0] = nn[1] = nn[2] = nn[3] = 0.0f;
            }
            // cell g of the block is w[g + 4]; the stencil reaches 2 cells each way
            const float w[12] = {pw[0], pw[1], pw[2], pw[3], cur[0], cur[1], cur[2], cur[3],
                                 nxt[0], nxt[1], nxt[2], nxt[3]};
#pragma unroll
            for (int g = 0; g < 4; ++g) {
               float a[3];
               const float fr = h4_face(w[g + 3], w[g + 4], w[g + 5], w[g + 6]);
               ppm_coeff(w[g + 3], w[g + 4], w[g + 5], face, fr, threshold, scale, a[0], a[1], a[2]);
               face = fr;
               const float v_l = v_r;
               v_r = fa(v_r, dv);
               const int gk_l = gk_r;
               gk_r = __float2int_rz(fd(fs(v_r, im), dk));
               int min_gk = __shfl_sync(hmask, gk_l, min_lane, 16);
               int max_gk = __shfl_sync(hmask, gk_r, max_lane, 16);
               min_gk = (min_gk > gk_lo_col) ? min_gk : gk_lo_col;
               max_gk = (max_gk < gk_hi_col) ? max_gk : gk_hi_col;
               if (max_gk >= min_gk) {
                  if ((min_gk >> 2) < next_flush || (max_gk >> 2) >= next_flush + RING_BLOCKS) {
                     range_err = true;
                  } else {
                     float dens_r = 0.0f;
                     for (int gk = min_gk; gk <= max_gk; ++gk) {
                        float x = fa(fm((float)(gk + 1), dk), im);
                        x = (x > v_l) ? x : v_l;
                        x = (x < v_r) ? x : v_r;
                        const float u = __double2float_rn(__dmul_rn((double)fs(x, v_l), i_dv));
                        const float dl = dens_r;
                        dens_r = fm(u, fa(a[0], fm(u, fa(a[1], fm(u, a[2])))));
                        float* t = &ring[(gk & (RING_CELLS - 1)) * 16 + lane];
                        *t = fa(*t, fs(dens_r, dl));
                     }
                  }
               }
            }
            // targets below the next source cell's lower bound are complete
            int lb = ncf * WID;
            if (kb < col_e) {
               int nl = __shfl_sync(hmask, gk_r, min_lane, 16);
               nl = (nl > gk_lo_col) ? nl : gk_lo_col;
               lb = (nl < lb) ? nl : lb;
            }
            flush_until(lb >> 2);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
               pw[g] = cur[g];
               cur[g] = nxt[g];
               nxt[g] = nn[g];
            }
            ++src_rank;
         }
         col_s = nxt_s;
         col_e = nxt_e;
         cf = ncf;
         cl = ncl;
      }
      flush_until(1 << 20);
      if (__any_sync(hmask, range_err)) {
         if (lane == 0) atomicOr(&status[cs.cell], VLGPU_CELL_RANGE);
         // deposits past the ring window may have landed in slots no flush
         // reads: clear the ring so that the next set starts empty
#pragma unroll
         for (int q = 0; q < RING_CELLS; ++q) ring[q * 16 + lane] = 0.0f;
      }
   }
}

// ---------------------------------------------------------------------------
// remap_walk: the fused arithmetic as a single-accumulator walk (PQM)
// ---------------------------------------------------------------------------
// The same column sets, lanes, ring and flushes as remap_kernel, with the
// distribution of mass over the target cells reduced to what the fused mode
// needs:
//
//  - Distribution: each lane keeps one pending target g (the lowest target
//    cell not yet complete), its accumulated mass and the position u of the
//    target's right edge (g+1) dk + im relative to the current source cell,
//    in units of dv.  A source cell with the edge inside (u < 1) completes
//    target g with the integral up to the edge and starts target g+1 with the
//    rest of the cell (v0 - D(u), so the cell's mass is kept exactly as a
//    sum); otherwise the whole cell goes to target g.  A second edge inside
//    one source cell (dk < dv) takes a rare loop.
//  - Ring traffic: a completed target is stored once into the lane's ring
//    slot.  Within a column a lane completes each target cell once, and the
//    targets of different columns of a set never share a cell while dk < 4 dv
//    (a target would have to span the empty block between them); the first
//    target of a column starts from what its slot already holds (the last
//    target of the column before it, when dk >= 4 dv), so targets shared by
//    two columns are summed in every case.  A flush zeroes the slots it reads.
//  - Target limits of the column (cpu_acc_map.cpp:559-569): a lane whose first
//    target lies below the column's lowest target cell starts at that cell,
//    which then receives all mass below its right edge, as in the reference;
//    mass of targets above the column's highest cell is moved into it when
//    the column ends.
template <int DIM>
__global__ void __launch_bounds__(REMAP_THREADS, 3) remap_walk_kernel(
   const ColumnSet* __restrict__ sets, SweepCounters* __restrict__ counters, const uint32_t* __restrict__ perm,
   const float* __restrict__ src_data, float* __restrict__ dst_data, uint32_t* __restrict__ dst_gids,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, MeshDev mesh, int wall_margin,
   uint32_t set_capacity, uint8_t* __restrict__ content_out, double content_threshold, const HandOver after) {
   hand_over(after, counters);
   __shared__ __align__(16) float ring_all[REMAP_THREADS * WALK_LANE_STRIDE];
   const int hw = threadIdx.x >> 4;
   const int lane = threadIdx.x & 15;
   const unsigned hmask = 0xffffu << (threadIdx.x & 16);
   // this lane's slots ring[t], t = target cell mod RING_CELLS, contiguous so
   // that a target block's four cells are one 16-byte access
   float* ring = ring_all + (size_t)threadIdx.x * WALK_LANE_STRIDE;
   const int i = lane & 3, j = lane >> 2;
   uint32_t n_sets = counters->n_sets;
   n_sets = (n_sets < set_capacity) ? n_sets : set_capacity;
   SetClaims claims(counters, n_sets);
   const int max_len = (int)mesh.len[DIM];
   const float dv = mesh.dv[DIM], v_min = mesh.vmin[DIM];
   const float inv_dv = (float)(1.0 / (double)dv);
   const float content_thr = __double2float_ru(content_threshold);
   constexpr int RMASK = RING_CELLS - 1;
   constexpr uint32_t SMASK = RING_CELLS - 1;  // slot offsets wrap around the ring

#pragma unroll
   for (int q = 0; q < RING_CELLS; ++q) ring[q] = 0.0f;
   for (uint32_t sidx = claims.first(hw, REMAP_THREADS / 16, 1u); sidx < n_sets;
        sidx = claims.next(lane == 0, hmask, 16, 1u)) {
      const ColumnSet cs = sets[sidx];
      const SweepCell P = sweep_cells[cs.cell];
      if (P.flags & SWEEP_PASS) {
         pass_through_set<DIM>(cs, perm, src_data, dst_data, dst_gids, content_out, mesh, content_thr, lane, hmask);
         continue;
      }
      const float dk = P.dk;
      const float A = fa((float)(cs.si() * WID), (float)i);
      const float B = fa((float)(cs.sj() * WID), (float)j);
      const float im = fa(fa(P.intersection, fm(A, P.di)), fm(B, P.dj));
      float mx, mn;
      set_corners(P, cs.si(), cs.sj(), mx, mn);
      const uint32_t gid0 = gid_from_swapped(cs.si(), cs.sj(), 0u, mesh.len, DIM);
      const uint32_t gid_step = gid_from_swapped(cs.si(), cs.sj(), 1u, mesh.len, DIM) - gid0;
      // the next target block to write and the end of the run of consecutive
      // target blocks it belongs to
      int next_flush = mask_next_set(cs.tgt_mask, 0);
      int run_end = mask_next_clear(cs.tgt_mask, next_flush);
      uint32_t out_idx = 0;
      bool range_err = false;

      auto flush_until = [&](int limit_block) {
         while (next_flush < 96 && next_flush < limit_block) {
            const int slot = (next_flush & (RING_BLOCKS - 1)) * WID;
            const float4 v4 = *reinterpret_cast<const float4*>(ring + slot);
            *reinterpret_cast<float4*>(ring + slot) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float v[4] = {v4.x, v4.y, v4.z, v4.w};
            const uint32_t o = cs.dst_pos + out_idx;
            store_lane<DIM>(dst_data + (size_t)o * WID3, i, j, v);
            const bool c = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])) >= content_thr;
            const unsigned any_c = __ballot_sync(hmask, c) & hmask;
            if (lane == 0) {
               dst_gids[o] = gid0 + (uint32_t)next_flush * gid_step;
               content_out[o] = any_c ? 1 : 0;
            }
            ++out_idx;
            if (++next_flush >= run_end) {
               next_flush = mask_next_set(cs.tgt_mask, next_flush);
               run_end = mask_next_clear(cs.tgt_mask, next_flush);
            }
         }
      };

      // a cell whose Lagrangian cells do not advance (flagged by columnize)
      // gets its target blocks with zero values
      const bool walkable = dk > 0.0f;
      int src_rank = 0;
      int col_s = walkable ? mask_next_set(cs.src_mask, 0) : 96;
      int col_e = (col_s < 96) ? mask_next_clear(cs.src_mask, col_s) - 1 : 95;
      int cf = 0, cl = 0;
      if (col_s < 96) column_extent(mx, mn, dk, dv, v_min, max_len, col_s, col_e, wall_margin, cf, cl);
      while (col_s < 96) {
         const int nxt_s = mask_next_set(cs.src_mask, col_e + 1);
         int nxt_e = 95, ncf = 1 << 20, ncl = 0;
         if (nxt_s < 96) {
            nxt_e = mask_next_clear(cs.src_mask, nxt_s) - 1;
            column_extent(mx, mn, dk, dv, v_min, max_len, nxt_s, nxt_e, wall_margin, ncf, ncl);
         }
         const int lo = cf * WID, hi = (cl + 1) * WID - 1;
         // ---- the lane's first target: the lowest g with (g+1) dk + im > v_l ----
         float v_l = fa(fm((float)(WID * col_s), dv), v_min);
         int g = __float2int_rz(fd(fs(v_l, im), dk));
         float e = fa(fm((float)(g + 1), dk), im);
         for (int q = 0; q < 3 && e <= v_l; ++q) {
            ++g;
            e = fa(fm((float)(g + 1), dk), im);
         }
         for (int q = 0; q < 3; ++q) {
            const float ep = fa(fm((float)g, dk), im);
            if (!(ep > v_l)) break;
            --g;
            e = ep;
         }
         if (g < lo) {
            g = lo;
            e = fa(fm((float)(g + 1), dk), im);
         }
         float g1f = (float)(g + 1);   // the pending target's edge index (g + 1)
         uint32_t soff = (uint32_t)(g & RMASK);  // the pending target's slot
         float u = fs(e, v_l) * inv_dv;
         // minus the pending target's accumulated mass (kept negated so that
         // both branches of the per-cell update are one select and one add)
         float nacc = -ring[soff];  // what another column left in the slot
         float pw0 = 0.0f, pw1 = 0.0f, pw2 = 0.0f, pw3 = 0.0f;  // cells below the block (zero padding)
         float cur[4], nxt[4];
         load_lane<DIM>(src_data, perm[cs.src_pos + src_rank], i, j, cur);
         if (col_e > col_s) {
            load_lane<DIM>(src_data, perm[cs.src_pos + src_rank + 1], i, j, nxt);
         } else {
            nxt[0] = nxt[1] = nxt[2] = nxt[3] = 0.0f;
         }
         // face state of the column's first cell
         float face = h8_value(0.0f, 0.0f, 0.0f, 0.0f, cur[0], cur[1], cur[2], cur[3]);
         float face_d = h7_derivative(0.0f, 0.0f, 0.0f, 0.0f, cur[0], cur[1], cur[2], cur[3]);
         for (int kb = col_s; kb <= col_e; ++kb) {
            float nn[4];
            if (kb + 2 <= col_e) {
               load_lane<DIM>(src_data, perm[cs.src_pos + src_rank + 2], i, j, nn);
            } else {
               nn[0] = nn[1] = nn[2] = nn[3] = 0.0f;
            }
            const float w[12] = {pw0, pw1, pw2, pw3, cur[0], cur[1], cur[2], cur[3], nxt[0], nxt[1], nxt[2], nxt[3]};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
               const float vm1 = w[q + 3], v0 = w[q + 4], vp1 = w[q + 5];
               float a[5];
               const float fr = h8_value(w[q + 1], w[q + 2], w[q + 3], w[q + 4], w[q + 5], w[q + 6], w[q + 7],
                                         w[q + 8]);
               const float fdr = h7_derivative(w[q + 1], w[q + 2], w[q + 3], w[q + 4], w[q + 5], w[q + 6], w[q + 7],
                                               w[q + 8]);
               pqm_coeff_fused(vm1, v0, vp1, face, fr, face_d, fdr, a);
               face = fr;
               face_d = fdr;
               // ---- distribute the cell over the lane's targets ----
               const bool has = u < 1.0f;  // the pending target's right edge lies inside this cell
               float D = pqm_integral(u, a);  // used only when has
               if (has) ring[soff] = D - nacc;
               nacc = (has ? D : nacc) - v0;
               {
                  const float g1n = g1f + 1.0f;
                  const float un = fs(fa(fm(g1n, dk), im), v_l) * inv_dv;  // the next edge (reference's rounding)
                  g1f = has ? g1n : g1f;
                  u = has ? un : u;
                  soff = has ? ((soff + 1u) & SMASK) : soff;
               }
               if (u < 1.0f) {
                  // further edges inside the same source cell (dk < dv)
                  for (int guard = 0; u < 1.0f && guard < 8; ++guard) {
                     const float D2 = pqm_integral(u, a);
                     ring[soff] = D2 - D;
                     D = D2;
                     g1f += 1.0f;
                     soff = (soff + 1u) & SMASK;
                     u = fs(fa(fm(g1f, dk), im), v_l) * inv_dv;
                  }
                  // more than eight target edges in one source cell (dk < dv / 8):
                  // outside what the walk represents, reported with the cell
                  range_err |= u < 1.0f;
                  nacc = D - v0;
               }
               u -= 1.0f;
               v_l = fa(v_l, dv);
            }
            g = __float2int_rn(g1f) - 1;  // the pending target
            int top = g - 1;  // the highest target this block completed
            if (kb == col_e) {
               // column done: the pending target keeps the rest; targets
               // above the column's highest cell are folded into it
               if (g > hi) {
                  float extra = -nacc;
                  for (int t = hi + 1; t < g && t <= hi + RING_CELLS / 2; ++t) {
                     extra += ring[t & RMASK];
                     ring[t & RMASK] = 0.0f;
                  }
                  range_err |= g > hi + RING_CELLS / 2;
                  ring[hi & RMASK] += extra;
                  top = hi;
               } else {
                  // the slot holds nothing of this column's yet (its first
                  // target's earlier content is already in nacc)
                  ring[soff] = -nacc;
                  top = g;
               }
            }
            // everything this block wrote must lie inside the ring's window
            range_err |= top >= (next_flush + RING_BLOCKS) * WID;
            // targets below the next source cell's lower bound are complete
            int lb = ncf * WID;
            if (kb < col_e) {
               int nl = __reduce_min_sync(hmask, g < hi ? g : hi);
               lb = (nl < lb) ? nl : lb;
            }
            flush_until(lb >> 2);
            pw0 = cur[0]; pw1 = cur[1]; pw2 = cur[2]; pw3 = cur[3];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
               cur[q] = nxt[q];
               nxt[q] = nn[q];
            }
            ++src_rank;
         }
         col_s = nxt_s;
         col_e = nxt_e;
         cf = ncf;
         cl = ncl;
      }
      flush_until(1 << 20);
      if (__any_sync(hmask, range_err)) {
         if (lane == 0) atomicOr(&status[cs.cell], VLGPU_CELL_RANGE);
#pragma unroll
         for (int q = 0; q < RING_CELLS; ++q) ring[q] = 0.0f;
      }
   }
}

// ---------------------------------------------------------------------------
// remap_pair: the fused arithmetic, two columns per lane
// ---------------------------------------------------------------------------
// The walk of remap_walk_kernel (pending target, edges, column limits, flushes)
// with eight lanes per column set, four sets per warp, each lane walking two
// neighbouring columns whose values sit side by side in float2 registers:
//
//  - The arithmetic of both columns is one packed f32x2 instruction; loads,
//    stores and ring accesses move both columns' values at once, and the
//    bookkeeping of a block and of a set (about 80 and 300 instructions) is
//    shared by twice the cells.
//  - The limiter works on magnitudes: with L = |v0 - left face|, R = |right
//    face - v0| (a face outside the values of its two cells gives half the
//    superbee slope h = min(|a|, |b|, max(|a|, |b|) / 2) instead) the
//    Colella-Woodward corrections are L = min(L, 2R), R = min(R, 2L), and the
//    reconstruction is v0 - s (L + u ((R - 2L) + u (L - R))) with s the sign of
//    the slope, zero at an extremum.  v0 - face is the neighbour's value
//    minus the same face for the cell on the other side, so it is carried.
//    That takes 8 operations of the ALU pipe per cell where the selections of
//    faces took 14.
//  - The four sets of a warp walk in step (the loop count is the warp's), so
//    every vote covers the whole warp.
//  - The ring of target cells lies slot by slot in shared memory (a slot of
//    all the CTA's lanes is contiguous): a lane's slot is always in its own
//    banks, whatever slots the other lanes are at.
//  - The pending target's slot is written for every cell, complete or not,
//    which saves the test.  That needs the slot to be the target's own: the
//    pending target may not be a whole ring ahead of the oldest one that is
//    still to be flushed.  Where the columns of a block face start far apart
//    it can be, and those sets (PAIR_LEAN) write a target when it is complete.
//
// Bound by issue and the ALU pipe (72% and 60% busy with 24 warps per SM, the
// most the ring's 64 KB per CTA leave room for).  Measured on 4096 drifting
// Maxwellian cells (5.8 M blocks): 2870 GB/s of 8 B per cell against 2321 GB/s
// with half a warp per set (1145 against 1415 us), and with the sets by length
// (columnize_cell) 3197 GB/s; before that, 64 cells: 38 against 53 us; PLM on
// 1024 cells: 247 against 291 us.  Two CTAs per SM with
// 100 registers take 17% longer, a loop over two blocks that loads a block
// ahead 25% (instruction cache); prefetches to L2 change nothing.
constexpr int PAIR_THREADS = 256;
constexpr int PAIR_WARPS = PAIR_THREADS / 32;
constexpr uint32_t PAIR_SLOT_BYTES = PAIR_THREADS * sizeof(float2);  // one ring slot of the CTA
constexpr uint32_t PAIR_SLOT_MASK = (RING_CELLS - 1) * PAIR_SLOT_BYTES;
constexpr int PAIR_CTAS = 3;  // per SM: 72 to 80 registers, 192 KB of rings
constexpr size_t PAIR_SMEM = (size_t)RING_CELLS * PAIR_SLOT_BYTES;
// The columns of a set start within S = 3 (|di| + |dj|) / dk target cells of
// one another.  At the end of a block every target cell below the lowest
// pending one's block is flushed, so during the next the highest pending
// target is less than 3 + (S + 1) + (4 dv / dk + 1) cells above the oldest one
// in the ring; where flushing waits for the set's next column, whose lowest
// target block may lie below the highest one of this, less than 3 + 3 + 3 + S.
// With S + 4 dv / dk <= 20 both are less than the ring's 32, with room for the
// rounding of the edges.  (A step that turns by 22 degrees has 6.)
constexpr float PAIR_LEAN = 20.0f;
// A column's start is cut at this many target cells (the mesh has 384): one
// above is reported when the column ends, one below counts as the column's
// lowest target, and the slot's offset stays far from its 32 bits.  A start
// that a 32-bit cell index does not hold is reported on either side.
constexpr float PAIR_FAR = 1e6f;
constexpr float PAIR_INDEX = 2147483648.0f;

// The lane's two columns of the block at `row` (data: the lane's first cell of
// row 0): cells g = 0..3 along the sweep, .x and .y the two columns.
template <int DIM>
__device__ __forceinline__ void load_pair(const float* __restrict__ data, uint32_t row, float2 v[4]) {
   const float* __restrict__ blk = data + (size_t)row * WID3;
   if (DIM == 0) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(blk));
      const float4 b = __ldg(reinterpret_cast<const float4*>(blk) + 1);
      v[0] = make_float2(a.x, b.x);
      v[1] = make_float2(a.y, b.y);
      v[2] = make_float2(a.z, b.z);
      v[3] = make_float2(a.w, b.w);
   } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) v[g] = __ldg(reinterpret_cast<const float2*>(blk + g * (DIM == 1 ? WID : WID2)));
   }
}

template <int DIM>
__device__ __forceinline__ void store_pair(float* __restrict__ blk, const float2 v[4]) {
   if (DIM == 0) {
      reinterpret_cast<float4*>(blk)[0] = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
      reinterpret_cast<float4*>(blk)[1] = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
   } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) *reinterpret_cast<float2*>(blk + g * (DIM == 1 ? WID : WID2)) = v[g];
   }
}

// The set of a cell that is not accelerated in this step (pass_through_set)
// by its eight lanes.
template <int DIM>
__device__ __forceinline__ void pass_through_pair(const ColumnSet& cs, const uint32_t* __restrict__ perm,
                                                  const float* __restrict__ src_data, float* __restrict__ dst_data,
                                                  uint32_t* __restrict__ dst_gids, uint8_t* __restrict__ content_out,
                                                  const uint32_t len[3], float content_thr, int off, bool leader,
                                                  unsigned omask) {
   uint32_t r = 0;
   for (int k = mask_next_set(cs.src_mask, 0); k < 96; k = mask_next_set(cs.src_mask, k + 1), ++r) {
      float2 v[4];
      load_pair<DIM>(src_data + off, perm[cs.src_pos + r], v);
      const uint32_t o = cs.dst_pos + r;
      store_pair<DIM>(dst_data + (size_t)o * WID3 + off, v);
      bool c = false;
#pragma unroll
      for (int g = 0; g < 4; ++g) c |= fmaxf(v[g].x, v[g].y) >= content_thr;
      const unsigned any_c = __ballot_sync(omask, c) & omask;
      if (leader) {
         dst_gids[o] = gid_from_swapped(cs.si(), cs.sj(), (uint32_t)k, len, DIM);
         content_out[o] = any_c ? 1 : 0;
      }
   }
}

// First set bit of a mask (96: none) and first clear bit at or after k.
__device__ __forceinline__ int mask_first(const uint32_t m[3]) {
   return m[0] ? __ffs(m[0]) - 1 : (m[1] ? 31 + __ffs(m[1]) : (m[2] ? 63 + __ffs(m[2]) : 96));
}
__device__ __forceinline__ int mask_run_end(const uint32_t m[3], int k) {
   uint32_t c[3];
#pragma unroll
   for (int w = 0; w < 3; ++w) {
      const int s = k - 32 * w;  // bits of the word below k count as set
      c[w] = ~m[w] & (s <= 0 ? 0xffffffffu : (s >= 32 ? 0u : 0xffffffffu << s));
   }
   return mask_first(c);
}

// What the sweep's kernels read of the mesh, in the walk's precision.
struct PairMesh {
   uint32_t len[3];
   int wall_margin;
   float dv, v_min, inv_dv;
   float content_thr;  // the smallest float >= the threshold: v >= it exactly when (double)v >= the threshold
};

template <int DIM, int RECON>
__global__ void __launch_bounds__(PAIR_THREADS, PAIR_CTAS) remap_pair_kernel(
   const ColumnSet* __restrict__ sets, SweepCounters* __restrict__ counters, const uint32_t* __restrict__ perm,
   const float* __restrict__ src_data, float* __restrict__ dst_data, uint32_t* __restrict__ dst_gids,
   const SweepCell* __restrict__ sweep_cells, uint32_t* __restrict__ status, const PairMesh mesh,
   uint32_t set_capacity, uint8_t* __restrict__ content_out, const HandOver after) {
   hand_over(after, counters);
   static_assert(RECON == RECON_PPM || RECON == RECON_PLM, "the quartic reconstruction runs in remap_walk_kernel");
   extern __shared__ __align__(16) unsigned char pair_ring[];
   constexpr unsigned FULL = 0xffffffffu;
   const int lane = threadIdx.x & 31, l8 = threadIdx.x & 7;
   const unsigned oshift = lane & 24;  // the octet's first lane
   // the lane's columns (i0, j0) and its neighbour: i0 + 1, or j0 + 1 in the x
   // sweep, whose columns are rows of the block along y
   const int i0 = (DIM == 0) ? (l8 >> 1) : 2 * (l8 & 1);
   const int j0 = (DIM == 0) ? 2 * (l8 & 1) : (l8 >> 1);
   const int off = cell_offset<DIM>(i0, j0, 0);
   // this lane's ring slot at byte s (target cell times PAIR_SLOT_BYTES, mod the ring)
   const uint32_t lane_at = threadIdx.x * (uint32_t)sizeof(float2);
   auto slot_x = [&](uint32_t s) -> float& {
      return *reinterpret_cast<float*>(pair_ring + ((s & PAIR_SLOT_MASK) | lane_at));
   };
   auto slot_y = [&](uint32_t s) -> float& {
      return *reinterpret_cast<float*>(pair_ring + ((s & PAIR_SLOT_MASK) | lane_at) + 4);
   };
   auto slot2 = [&](uint32_t s) -> float2& {
      return *reinterpret_cast<float2*>(pair_ring + ((s & PAIR_SLOT_MASK) | lane_at));
   };

   uint32_t n_sets = counters->n_sets;
   n_sets = (n_sets < set_capacity) ? n_sets : set_capacity;
   SetClaims claims(counters, n_sets);
   const float2 zero2 = make_float2(0.0f, 0.0f);

   uint32_t base = claims.first(threadIdx.x >> 5, PAIR_WARPS, 4u);
   if (base >= n_sets) return;
#pragma unroll
   for (int q = 0; q < RING_CELLS; ++q) slot2(q * PAIR_SLOT_BYTES) = zero2;
   for (; base < n_sets; base = claims.next(lane == 0, FULL, 32, 4u)) {
      const uint32_t sidx = base + (oshift >> 3);
      float2 im = zero2;
      float dk = 1.0f;
      uint32_t out = 0, gid0 = 0, pos = 0;  // next output block; block ID of the set's k = 0; the set's first row
      int n_src = 0;                        // source blocks to walk
      int next_flush = 96, run_end = 96;    // next target block to write, end of its run of consecutive ones
      // the current column: source blocks from this one on, highest target
      // cell, and the next column's first target block (none: NO_COLUMN)
      constexpr int NO_COLUMN = 1 << 20;
      int left = 0, hi = 0, ncf = NO_COLUMN;
      int kb = 0, lo = 0;  // first block and lowest target cell of the column about to start
      bool lean = false;   // see PAIR_LEAN
      if (sidx < n_sets) {
         const ColumnSet cs = sets[sidx];
         const SweepCell P = sweep_cells[cs.cell];
         if (P.flags & SWEEP_PASS) {
            pass_through_pair<DIM>(cs, perm, src_data, dst_data, dst_gids, content_out, mesh.len, mesh.content_thr, off,
                                   l8 == 0, 0xffu << oshift);
         } else {
            dk = P.dk;
            const float A0 = fa((float)(cs.si() * WID), (float)i0), B0 = fa((float)(cs.sj() * WID), (float)j0);
            const float A1 = (DIM == 0) ? A0 : fa((float)(cs.si() * WID), (float)(i0 + 1));
            const float B1 = (DIM == 0) ? fa((float)(cs.sj() * WID), (float)(j0 + 1)) : B0;
            im.x = fa(fa(P.intersection, fm(A0, P.di)), fm(B0, P.dj));
            im.y = fa(fa(P.intersection, fm(A1, P.di)), fm(B1, P.dj));
            gid0 = gid_from_swapped(cs.si(), cs.sj(), 0u, mesh.len, DIM);
            out = cs.dst_pos;
            pos = cs.src_pos;
            next_flush = mask_first(cs.tgt_mask);
            run_end = mask_run_end(cs.tgt_mask, next_flush);
            // a cell whose Lagrangian cells do not advance (flagged by
            // columnize) gets its target blocks with zero values
            if (dk > 0.0f) n_src = __popc(cs.src_mask[0]) + __popc(cs.src_mask[1]) + __popc(cs.src_mask[2]);
            lean = !(fmaf(3.0f, fabsf(P.di) + fabsf(P.dj), 4.0f * mesh.dv) <= PAIR_LEAN * dk);
            if (n_src > 0) {
               kb = mask_first(cs.src_mask);
               const int e = mask_run_end(cs.src_mask, kb);
               left = e - kb;
               if (left == n_src) {
                  // one column: columnize marked exactly its targets
                  lo = next_flush * WID;
                  hi = run_end * WID - 1;
               } else {
                  float mx, mn;
                  int cf, cl, ncl;
                  set_corners(P, cs.si(), cs.sj(), mx, mn);
                  column_extent(mx, mn, dk, mesh.dv, mesh.v_min, (int)mesh.len[DIM], kb, e - 1, mesh.wall_margin, cf, cl);
                  lo = cf * WID;
                  hi = (cl + 1) * WID - 1;
                  const int s = mask_next_set(cs.src_mask, e);
                  column_extent(mx, mn, dk, mesh.dv, mesh.v_min, (int)mesh.len[DIM], s,
                                mask_run_end(cs.src_mask, s) - 1, mesh.wall_margin, ncf, ncl);
               }
            }
         }
      }
      __syncwarp();
      const int iters = __reduce_max_sync(FULL, n_src);
      const bool any_lean = __any_sync(FULL, lean);  // the warp's sets walk in step
      bool range_err = false;

      // writes out the target blocks below `limit` that all the lanes of the
      // octet have completed
      auto flush = [&](int limit) {
         limit = limit < 96 ? limit : 96;
         for (;;) {
            unsigned can = __ballot_sync(FULL, next_flush < limit);
            can &= can >> 4;
            can &= can >> 2;
            can &= (can >> 1) & 0x01010101u;  // bit 8 q: all of octet q's lanes
            if (can == 0u) break;
            float2 v[4];
            const uint32_t slot = (uint32_t)next_flush * (WID * PAIR_SLOT_BYTES);
#pragma unroll
            for (int g = 0; g < 4; ++g) v[g] = slot2(slot + g * PAIR_SLOT_BYTES);
            const float m = fmaxf(fmaxf(fmaxf(v[0].x, v[0].y), fmaxf(v[1].x, v[1].y)),
                                  fmaxf(fmaxf(v[2].x, v[2].y), fmaxf(v[3].x, v[3].y)));
            const unsigned any_c = __ballot_sync(FULL, m >= mesh.content_thr) >> oshift;
            if ((can >> oshift) & 1u) {
#pragma unroll
               for (int g = 0; g < 4; ++g) slot2(slot + g * PAIR_SLOT_BYTES) = zero2;
               store_pair<DIM>(dst_data + (size_t)out * WID3 + off, v);
               if (l8 == 0) {
                  dst_gids[out] = gid0 + (uint32_t)next_flush *
                                            (DIM == 0 ? 1u : (DIM == 1 ? mesh.len[0] : mesh.len[0] * mesh.len[1]));
                  content_out[out] = (any_c & 0xffu) ? 1 : 0;
               }
               ++out;
               if (++next_flush >= run_end) {
                  const ColumnSet& cs = sets[sidx];
                  const uint32_t tm[3] = {cs.tgt_mask[0], cs.tgt_mask[1], cs.tgt_mask[2]};
                  next_flush = mask_next_set(tm, next_flush);
                  run_end = mask_run_end(tm, next_flush);
               }
            }
         }
      };

      // the walk's state (see remap_walk_kernel): u the pending target's right
      // edge in the cell, g2f the index of the edge after it, nacc minus its
      // mass so far, so its slot (target cell times PAIR_SLOT_BYTES)
      float v_l = 0.0f;
      float2 g2f = zero2, u = zero2, nacc = zero2;
      uint32_t sox = 0, soy = 0;
      float2 vm1 = zero2;
      PpmWalk ppm{zero2, zero2, false, false};

      // the state at the start of the column whose first block is c
      auto start = [&](const float2 c[4]) {
         v_l = fa(fm((float)(WID * kb), mesh.dv), mesh.v_min);
         // each lane's first target: the lowest g with (g+1) dk + im > v_l
         auto first_target = [&](float imc, float& gf, float& uc, uint32_t& so) {
            const float q0 = fd(fs(v_l, imc), dk);
            range_err |= fabsf(q0) >= PAIR_INDEX;
            int g = __float2int_rz(fminf(fmaxf(q0, -PAIR_FAR), PAIR_FAR));
            float e = fa(fm((float)(g + 1), dk), imc);
#pragma unroll 1
            for (int q = 0; q < 3 && e <= v_l; ++q) {
               ++g;
               e = fa(fm((float)(g + 1), dk), imc);
            }
#pragma unroll 1
            for (int q = 0; q < 3; ++q) {
               const float ep = fa(fm((float)g, dk), imc);
               if (!(ep > v_l)) break;
               --g;
               e = ep;
            }
            if (g < lo) {
               g = lo;
               e = fa(fm((float)(g + 1), dk), imc);
            }
            gf = (float)(g + 2);
            uc = fs(e, v_l) * mesh.inv_dv;
            so = (uint32_t)g * PAIR_SLOT_BYTES;
         };
         first_target(im.x, g2f.x, u.x, sox);
         first_target(im.y, g2f.y, u.y, soy);
         // what another column left in the slots; a target above the ring's
         // window has none yet, its slot is an older target's
         const uint32_t end = (uint32_t)(next_flush + RING_BLOCKS) * (WID * PAIR_SLOT_BYTES);
         nacc.x = sox < end ? -slot_x(sox) : 0.0f;
         nacc.y = soy < end ? -slot_y(soy) : 0.0f;
         // zero padding below the column
         vm1 = zero2;
         if constexpr (RECON == RECON_PPM) ppm.start(zero2, zero2, c[0], c[1]);
         else ppm.b = c[0];
      };

      // one cell: v0 with its upper neighbours; `complete_only`: see PAIR_LEAN
      auto cell_step = [&](auto complete_only, const float2 v0, const float2 vp1, const float2 vp2) {
         // ---- reconstruction ----
         float2 s, l, r;
         if constexpr (RECON == RECON_PPM) {
            ppm_magnitudes_x2(ppm, vm1, v0, vp1, vp2, s, l, r);
            vm1 = v0;
         } else {
            const float2 a = p_minus(vp1, v0);
            half_slope_x2(a, ppm.b, l, s);
            r = l;
            ppm.b = a;
         }
         // ---- distribute the cell over the lane's targets ----
         const float2 um = __fadd2_rn(u, f2(-1.0f));
         const bool hx = um.x < 0.0f, hy = um.y < 0.0f;  // the pending target's right edge lies inside
         const float2 rl = p_minus(r, l);
         // used only where the edge lies inside
         const float2 T = (RECON == RECON_PPM) ? __ffma2_rn(u, rl, l) : l;
         const float2 D = __fmul2_rn(u, __ffma2_rn(__fmul2_rn(s, um), T, v0));
         // without an edge the slot is written again when its target is complete
         const float2 val = p_minus(D, nacc);
         if (!decltype(complete_only)::value || hx) slot_x(sox) = val.x;
         if (!decltype(complete_only)::value || hy) slot_y(soy) = val.y;
         nacc = p_minus(make_float2(hx ? D.x : nacc.x, hy ? D.y : nacc.y), v0);
         // the next edge, with the reference's roundings (the packed multiply
         // and add get contracted, so these are scalar)
         const float2 e = make_float2(fa(fm(g2f.x, dk), im.x), fa(fm(g2f.y, dk), im.y));
         const float2 un = __ffma2_rn(make_float2(fs(e.x, v_l), fs(e.y, v_l)), f2(mesh.inv_dv), f2(-1.0f));
         u = um;
         if (hx) {
            g2f.x += 1.0f;
            u.x = un.x;
            sox += PAIR_SLOT_BYTES;
         }
         if (hy) {
            g2f.y += 1.0f;
            u.y = un.y;
            soy += PAIR_SLOT_BYTES;
         }
         if (__builtin_expect(fminf(u.x, u.y) < 0.0f, 0)) {
            // further edges inside the same source cell (dk < dv); more than
            // eight (dk < dv / 8) lie outside what the walk represents and
            // are reported with the cell
            auto more = [&](float& uc, float& gf, uint32_t& so, float imc, float vc, float sc, float lc, float rlc,
                            float Dc, auto slot) {
#pragma unroll 1
               for (int guard = 0; uc < 0.0f && guard < 8; ++guard) {
                  const float ue = uc + 1.0f;
                  const float T2 = (RECON == RECON_PPM) ? fmaf(ue, rlc, lc) : lc;
                  const float D2 = ue * fmaf(sc * uc, T2, vc);
                  slot(so) = D2 - Dc;
                  Dc = D2;
                  so += PAIR_SLOT_BYTES;
                  uc = fmaf(fs(fa(fm(gf, dk), imc), v_l), mesh.inv_dv, -1.0f);
                  gf += 1.0f;
               }
               range_err |= uc < 0.0f;
               return Dc - vc;
            };
            if (u.x < 0.0f) nacc.x = more(u.x, g2f.x, sox, im.x, v0.x, s.x, l.x, rl.x, D.x, slot_x);
            if (u.y < 0.0f) nacc.y = more(u.y, g2f.y, soy, im.y, v0.y, s.y, l.y, rl.y, D.y, slot_y);
         }
         v_l = fa(v_l, mesh.dv);
      };

      // the values of block `it` and of the one after it
      float2 w[4] = {zero2, zero2, zero2, zero2}, n[4] = {zero2, zero2, zero2, zero2};
      uint32_t row = 0;  // data row of block it + 1
      if (n_src > 0) load_pair<DIM>(src_data + off, __ldg(perm + pos), w);
      if (n_src > 1) row = __ldg(perm + pos + 1);
      if (n_src > 0) start(w);
      // (one pass at least: a set without source blocks writes its targets)
      for (int it = 0; it == 0 || it < iters; ++it) {
         const bool active = it < n_src, last = left == 1;
         if (it + 1 < n_src) load_pair<DIM>(src_data + off, row, n);
         if (it + 2 < n_src) row = __ldg(perm + pos + it + 2);
         if (active) {
            // zero padding above the column
            const float2 n0 = last ? zero2 : n[0], n1 = last ? zero2 : n[1];
            if (__builtin_expect(any_lean, 0)) {
               // (a loop: a second unrolled copy would only lengthen the kernel)
               float2 v[6] = {w[0], w[1], w[2], w[3], n0, n1};
#pragma unroll 1
               for (int q = 0; q < 4; ++q) {
                  cell_step(std::true_type{}, v[0], v[1], v[2]);
#pragma unroll
                  for (int k = 0; k < 5; ++k) v[k] = v[k + 1];
               }
            } else {
               cell_step(std::false_type{}, w[0], w[1], w[2]);
               cell_step(std::false_type{}, w[1], w[2], w[3]);
               cell_step(std::false_type{}, w[2], w[3], n0);
               cell_step(std::false_type{}, w[3], n0, n1);
            }
         }
         int limit = NO_COLUMN;  // target blocks below it are complete in this lane's columns
         if (active) {
            const int gx = (int)(sox / PAIR_SLOT_BYTES), gy = (int)(soy / PAIR_SLOT_BYTES);  // the pending targets
            int top = max(gx, gy) - 1;  // the highest target this block completed
            limit = min(min(gx, gy), min(hi, ncf * WID)) >> 2;
            if (last) {
               // column done: the pending targets keep the rest; targets
               // above the column's highest cell are folded into it
               auto close = [&](int g, uint32_t so, float rest, auto slot) {
                  if (g > hi) {
#pragma unroll 1
                     for (int t = hi + 1; t < g && t <= hi + RING_CELLS / 2; ++t) {
                        rest += slot((uint32_t)t * PAIR_SLOT_BYTES);
                        slot((uint32_t)t * PAIR_SLOT_BYTES) = 0.0f;
                     }
                     range_err |= g > hi + RING_CELLS / 2;
                     if (!any_lean) slot(so) = 0.0f;  // what was written there while it was pending
                     slot((uint32_t)hi * PAIR_SLOT_BYTES) += rest;
                     return hi;
                  }
                  slot(so) = rest;
                  return g;
               };
               const int tx = close(gx, sox, -nacc.x, slot_x), ty = close(gy, soy, -nacc.y, slot_y);
               top = max(top, max(tx, ty));
               limit = ncf;
            }
            // everything this block wrote must lie inside the ring's window
            range_err |= top >= (next_flush + RING_BLOCKS) * WID;
            --left;
         }
         flush(limit);
         if (active && last && ncf != NO_COLUMN) {
            // the next column of the set
            const ColumnSet& cs = sets[sidx];
            const SweepCell P = sweep_cells[cs.cell];
            const uint32_t sm[3] = {cs.src_mask[0], cs.src_mask[1], cs.src_mask[2]};
            int e = 0;
            for (int done = it + 1;; done -= left) {
               kb = mask_next_set(sm, e);
               e = mask_run_end(sm, kb);
               left = e - kb;
               if (done == 0) break;
            }
            float mx, mn;
            int cf, cl;
            set_corners(P, cs.si(), cs.sj(), mx, mn);
            column_extent(mx, mn, dk, mesh.dv, mesh.v_min, (int)mesh.len[DIM], kb, e - 1, mesh.wall_margin, cf, cl);
            lo = cf * WID;
            hi = (cl + 1) * WID - 1;
            ncf = NO_COLUMN;
            const int s = mask_next_set(sm, e);
            if (s < 96)
               column_extent(mx, mn, dk, mesh.dv, mesh.v_min, (int)mesh.len[DIM], s, mask_run_end(sm, s) - 1,
                             mesh.wall_margin, ncf, cl);
            start(n);
         }
#pragma unroll
         for (int q = 0; q < 4; ++q) w[q] = n[q];
      }
      if ((__ballot_sync(FULL, range_err) >> oshift) & 0xffu) {
         // deposits past the ring's window may lie in slots no flush reads
         if (l8 == 0) atomicOr(&status[sets[sidx].cell], VLGPU_CELL_RANGE);
#pragma unroll
         for (int q = 0; q < RING_CELLS; ++q) slot2(q * PAIR_SLOT_BYTES) = zero2;
      }
   }
}

// ---------------------------------------------------------------------------
// host-side launch helpers (used by capi.cu)
// ---------------------------------------------------------------------------
// Columnize of the cells [cell_begin, cell_end) in launch order, each with room
// for the whole plane (at 67 x 67 two CTAs' worth of an SM's shared memory) and
// one CTA of 1024 threads per SM: for few cells, and for the per-cell calls,
// which bring one cell or a few.  (A call of map_1d_noalloc with many cells takes this form too:
// 592 cells of 30 blocks 96 us in all, 1024 of 14 blocks 110 us; 105 and 121 us
// with 256 threads, before its copies and waits were merged.)
cudaError_t launch_columnize(int dim, const uint32_t* gids, const uint32_t* src_index, const CellSlot* src_slots,
                             CellSlot* dst_slots,
                             uint32_t* perm, ColumnSet* sets, uint32_t set_capacity, uint32_t dst_capacity,
                             const SweepCell* sweep_cells, uint32_t* status, SweepCounters* counters,
                             BatchStats* stats, const MeshDev& mesh, int wall_margin, uint32_t cell_begin,
                             uint32_t cell_end, int first_of_step, uint32_t zero_row, const uint32_t* stop,
                             cudaStream_t stream) {
   uint32_t li, lj;
   plane_lengths(mesh.len, dim, li, lj);
   const size_t smem = columnize_smem_bytes(li * lj);
   const uint32_t n = cell_end - cell_begin;
   if (n == 0) return cudaSuccess;
   cudaError_t e = cudaSuccess;
#define VLGPU_COL(D)                                                                                             \
   e = cudaFuncSetAttribute(columnize_kernel<D, COL_FEW_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                            (int)smem);                                                                         \
   if (e != cudaSuccess) return e;                                                                              \
   columnize_kernel<D, COL_FEW_THREADS><<<n, COL_FEW_THREADS, smem, stream>>>(                                  \
      gids, src_index, src_slots, dst_slots, perm, sets, set_capacity, dst_capacity, sweep_cells, status, counters, \
      stats, mesh, wall_margin, cell_begin, cell_end, first_of_step, zero_row, nullptr, 0xffffffffu, nullptr, stop);
   if (dim == 0) { VLGPU_COL(0) } else if (dim == 1) { VLGPU_COL(1) } else { VLGPU_COL(2) }
#undef VLGPU_COL
   return cudaGetLastError();
}

// Columnize of every cell of a batch: one CTA per cell, the largest cells
// first (order), with shared memory for planes of up to COL_CAP_PLANE entries,
// which lets six CTAs share an SM; the cells with wider planes follow in
// columnize_wide_kernel.  The counters are zero before every sweep.
constexpr uint32_t COL_CAP_PLANE = 1024;
cudaError_t launch_columnize_batch(int dim, const uint32_t* gids, const uint32_t* src_index,
                                   const CellSlot* src_slots, CellSlot* dst_slots, uint32_t* perm, ColumnSet* sets,
                                   uint32_t set_capacity, uint32_t dst_capacity, const SweepCell* sweep_cells,
                                   uint32_t* status, SweepCounters* counters, BatchStats* stats, const MeshDev& mesh,
                                   int wall_margin, uint32_t n_cells, int first_of_step, uint32_t zero_row,
                                   uint32_t* wide_cells, const uint32_t* order, int wide_grid, uint32_t few_cells,
                                   cudaStream_t stream) {
   if (n_cells == 0) return cudaSuccess;
   uint32_t li, lj;
   plane_lengths(mesh.len, dim, li, lj);
   if (n_cells <= few_cells)
      return launch_columnize(dim, gids, src_index, src_slots, dst_slots, perm, sets, set_capacity, dst_capacity,
                              sweep_cells, status, counters, stats, mesh, wall_margin, 0, n_cells, first_of_step,
                              zero_row, nullptr, stream);
   const uint32_t cap = li * lj < COL_CAP_PLANE ? li * lj : COL_CAP_PLANE;
   const size_t smem_cap = columnize_smem_bytes(cap);
   const size_t smem = columnize_smem_bytes(li * lj);
   const uint32_t g2 = (uint32_t)wide_grid < n_cells ? (uint32_t)wide_grid : n_cells;
   cudaError_t e = cudaSuccess;
#define VLGPU_COLB(D, THREADS)                                                                                           \
   e = cudaFuncSetAttribute(columnize_kernel<D, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                            (int)smem);                                                                          \
   if (e != cudaSuccess) return e;                                                                               \
   e = cudaFuncSetAttribute(columnize_wide_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
   if (e != cudaSuccess) return e;                                                                               \
   columnize_kernel<D, THREADS><<<n_cells, THREADS, smem_cap, stream>>>(                                              \
      gids, src_index, src_slots, dst_slots, perm, sets, set_capacity, dst_capacity, sweep_cells, status, counters, \
      stats, mesh, wall_margin, 0, n_cells, first_of_step, zero_row, order, cap, wide_cells, nullptr);                              \
   columnize_wide_kernel<D><<<g2, COL_FEW_THREADS, smem, stream>>>(gids, src_index, src_slots, dst_slots, perm, sets, \
                                                               set_capacity, dst_capacity, sweep_cells, status,   \
                                                               counters, stats, mesh, wall_margin, first_of_step, \
                                                               zero_row, wide_cells);
   if (n_cells <= 8 * few_cells) {
      if (dim == 0) { VLGPU_COLB(0, COL_MID_THREADS) } else if (dim == 1) { VLGPU_COLB(1, COL_MID_THREADS) }
      else { VLGPU_COLB(2, COL_MID_THREADS) }
   } else {
      if (dim == 0) { VLGPU_COLB(0, COL_THREADS) } else if (dim == 1) { VLGPU_COLB(1, COL_THREADS) }
      else { VLGPU_COLB(2, COL_THREADS) }
   }
#undef VLGPU_COLB
   return cudaGetLastError();
}

// CTAs per SM of columnize_wide_kernel (the largest plane of the three
// dimensions).
int columnize_wide_blocks_per_sm(const MeshDev& mesh) {
   uint32_t li, lj, best = 0;
   for (int d = 0; d < 3; ++d) {
      plane_lengths(mesh.len, d, li, lj);
      best = li * lj > best ? li * lj : best;
   }
   const size_t smem = columnize_smem_bytes(best);
   int n = 0;
   cudaFuncSetAttribute(columnize_wide_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
   cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, columnize_wide_kernel<0>, COL_FEW_THREADS, smem);
   return n > 0 ? n : 1;
}

cudaError_t launch_remap(int dim, const ColumnSet* sets, SweepCounters* counters, const uint32_t* perm,
                         const float* src_data, float* dst_data, uint32_t* dst_gids, const SweepCell* sweep_cells,
                         uint32_t* status, const MeshDev& mesh, int wall_margin, uint32_t set_capacity,
                         uint8_t* content_out, double content_threshold, bool exact, int recon, int grid,
                         const HandOver& after, cudaStream_t stream) {
   PairMesh pm;
   for (int d = 0; d < 3; ++d) pm.len[d] = mesh.len[d];
   pm.wall_margin = wall_margin;
   pm.dv = mesh.dv[dim];
   pm.v_min = mesh.vmin[dim];
   pm.inv_dv = (float)(1.0 / (double)mesh.dv[dim]);
   pm.content_thr = (float)content_threshold;
   if ((double)pm.content_thr < content_threshold) pm.content_thr = std::nextafterf(pm.content_thr, FLT_MAX);
#define VLGPU_REMAP(D)                                                                                        \
   remap_kernel<D><<<grid, REMAP_THREADS, 0, stream>>>(sets, counters, perm, src_data, dst_data, dst_gids,          \
                                                       sweep_cells, status, mesh, wall_margin, set_capacity,        \
                                                       content_out, content_threshold, after)
#define VLGPU_WALK(D)                                                                                          \
   remap_walk_kernel<D><<<grid, REMAP_THREADS, 0, stream>>>(sets, counters, perm, src_data, dst_data, dst_gids, \
                                                               sweep_cells, status, mesh, wall_margin, set_capacity, \
                                                               content_out, content_threshold, after)
#define VLGPU_PAIR(D, R)                                                                                       \
   {                                                                                                           \
      const cudaError_t e = cudaFuncSetAttribute(remap_pair_kernel<D, R>,                                      \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM); \
      if (e != cudaSuccess) return e;                                                                          \
      remap_pair_kernel<D, R><<<grid, PAIR_THREADS, PAIR_SMEM, stream>>>(                                      \
         sets, counters, perm, src_data, dst_data, dst_gids, sweep_cells, status, pm, set_capacity, content_out, after); \
   }
#define VLGPU_PAIR_DIMS(R)                 \
   if (dim == 0) VLGPU_PAIR(0, R)          \
   else if (dim == 1) VLGPU_PAIR(1, R)     \
   else VLGPU_PAIR(2, R)
   if (exact) {
      if (recon != RECON_PPM) return cudaErrorInvalidValue;  // the exact mode is PPM only
      if (dim == 0) VLGPU_REMAP(0);
      else if (dim == 1) VLGPU_REMAP(1);
      else VLGPU_REMAP(2);
   } else if (recon == RECON_PLM) {
      VLGPU_PAIR_DIMS(RECON_PLM)
   } else if (recon == RECON_PQM) {
      if (dim == 0) VLGPU_WALK(0);
      else if (dim == 1) VLGPU_WALK(1);
      else VLGPU_WALK(2);
   } else {
      VLGPU_PAIR_DIMS(RECON_PPM)
   }
#undef VLGPU_PAIR_DIMS
#undef VLGPU_PAIR
#undef VLGPU_WALK
#undef VLGPU_REMAP
   return cudaGetLastError();
}

// Points the remap at the first set the next columnize launch will create
// (per-cell launch sequences share one set array).
__global__ void rebase_work_kernel(SweepCounters* counters) {
   counters->first_set = counters->n_sets;
   counters->work = 0u;
}

cudaError_t launch_rebase_work(SweepCounters* counters, cudaStream_t stream) {
   rebase_work_kernel<<<1, 1, 0, stream>>>(counters);
   return cudaGetLastError();
}

int remap_blocks_per_sm() {
   int n = 0;
   cudaFuncSetAttribute(remap_pair_kernel<2, RECON_PPM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM);
   cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, remap_pair_kernel<2, RECON_PPM>, PAIR_THREADS, PAIR_SMEM);
   return n > 0 ? n : 1;
}

}  // namespace vlgpu
