// Moves a lattice operator's vector between the tensor order and the
// reference order (device code, shared by the copies and the Q64 conversions).
//
// A reference index follows the occupied slots from the first orbital up, a
// tensor index (r_up * D_down + r_down, colex ranks) from the last orbital
// down, so neighbours in one order are far apart in the other: element by
// element, one side of the move is 8- or 16-byte accesses scattered over
// 32-byte sectors.  Both orders have runs, though.  Split the orbitals into a
// low part and the last kTileHigh ones: all states of one low occupation (both
// spins) are two runs of the reference order (the next slot is Up, or Down),
// in an order of their high occupations that depends on the high particle
// counts alone; and for fixed high occupations and a fixed low Up one, the low
// Down occupations of equal count are one run of the tensor order.  A tile is
// one low Up occupation, K consecutive low Down occupations and every high
// occupation: it passes through shared memory between runs of K elements on
// the tensor side and of about half its high occupations (18 at 2 + 2 particles
// on 4 orbitals) on the reference side.  (dim < 2^31: indices are 32 bits.)
//
// One move of 4x4 6+6, complex128 (1.03 GB): 1.2 ms element by element, 0.52 by
// tiles (2.31 GB moved, 4.4 TB/s, 0.66 of the measured copy); complex64 0.85 and
// 0.27 ms.  A block-wide tile with synchronous loads took 0.5 and 0.44: the warps
// waited at its barriers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mb_internal.h"

namespace mb {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t to, const void* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(BYTES)
               : "memory");
}
// the warp's copies are in shared memory, for every lane
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// e / d for e < 1024, d <= 1024 by ceil(2^20 / d): exact while e * d < 2^20
__device__ __forceinline__ uint32_t div_mul(int d) { return ((1u << 20) + d - 1) / d; }
__device__ __forceinline__ int div_by(int e, uint32_t mul) { return (int)(((uint32_t)e * mul) >> 20); }

// SCATTER: dst[perm[i]] = f(src[i]), else dst[i] = f(src[perm[i]]); a block a
// tile, each warp its own K columns, at its own pace: the elements and their
// reference indices go to the warp's shared memory as asynchronous copies, all
// in flight together, by their slot, the place in the reference side's order.
template <bool SCATTER, typename In, typename Out, typename F>
__global__ void __launch_bounds__(32 * kTileWarps)
k_tiles(RowOrder o, const In* __restrict__ src, Out* __restrict__ dst, F f) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int32_t s_base[kTilePairs];  // a (row, high Down occupation) pair's first element
  __shared__ int32_t s_place[kTilePairs];
  f.start();
  const OrderTile t = o.tiles[blockIdx.x];
  const int nt = t.n_rows * t.n_cols, stride = nt | 1;
  for (int q = threadIdx.x; q < nt; q += blockDim.x) {
    const int ur = q / t.n_cols, dc = q - ur * t.n_cols;
    s_base[q] = (int32_t)(o.rows[t.row + ur] * o.Dd) + o.cols[t.col + dc] + t.k0;
    s_place[q] = o.place[t.place + q];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = warp * t.kw, kn = min(t.kw, t.k - first);
  if (kn <= 0) return;
  In* vals = reinterpret_cast<In*>(smem + (size_t)warp * o.warp_bytes);
  int32_t* at = reinterpret_cast<int32_t*>(vals + o.warp_slots);  // reference indices
  const uint32_t vals_s = smem_addr(vals), at_s = smem_addr(at);
  const int total = nt * kn;
  const uint32_t mul_k = div_mul(kn), mul_n = div_mul(nt);
  auto tensor_side = [&](int e, int& slot) -> int32_t {
    const int pair = div_by(e, mul_k), k = e - pair * kn;
    slot = k * stride + s_place[pair];
    return s_base[pair] + first + k;
  };
  auto reference_side = [&](int s) { return stride == nt ? s : s + div_by(s, mul_n); };
#pragma unroll 4
  for (int e = lane; e < total; e += 32) {
    int slot;
    const int32_t i = tensor_side(e, slot);
    copy_async<4>(at_s + 4 * slot, o.perm + i);
    if (SCATTER) copy_async<(int)sizeof(In)>(vals_s + (int)sizeof(In) * slot, src + i);
  }
  copies_done();
  if constexpr (SCATTER) {
#pragma unroll 4
    for (int s = lane; s < total; s += 32) {
      const int slot = reference_side(s);
      dst[at[slot]] = f(vals[slot]);
    }
  } else {
#pragma unroll 4
    for (int s = lane; s < total; s += 32) {
      const int slot = reference_side(s);
      copy_async<(int)sizeof(In)>(vals_s + (int)sizeof(In) * slot, src + at[slot]);
    }
    copies_done();
#pragma unroll 4
    for (int e = lane; e < total; e += 32) {
      int slot;
      const int32_t i = tensor_side(e, slot);
      dst[i] = f(vals[slot]);
    }
  }
}

template <bool SCATTER, typename In, typename Out, typename F>
void launch_tiles(const RowOrder& o, const In* src, Out* dst, F f, cudaStream_t st) {
  if (o.n_tiles <= 0) return;
  auto kern = k_tiles<SCATTER, In, Out, F>;
  const size_t smem = (size_t)kTileWarps * o.warp_bytes;
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)o.n_tiles, 32 * kTileWarps, smem, st>>>(o, src, dst, f);
  MB_CUDA(cudaGetLastError());
}

}  // namespace mb
