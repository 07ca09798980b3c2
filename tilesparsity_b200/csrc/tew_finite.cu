// TEW layers run as one masked GEMM whose tiles are wider than the mask: a tile gathers every row any of its
// single weights lies in, and the packed weights are zero outside the mask.  0 * x adds nothing while x is finite;
// an infinity or a NaN in a gathered row would reach all columns of the tile instead of those that keep the row.
// This pass takes such results back (the reference multiplies by a dense 0/1 mask, Pruning/VGG/prune_algo.py:171-175,
// and gives no rule for them; here a weight outside the mask is no part of the product).
#include <mma.h>

#include <type_traits>

#include "ts_common.cuh"
#include "ts_kernels.h"

namespace ts {

namespace {

constexpr int kCheckRows = 256;       // batch rows a block looks at
constexpr int kGroup = 32;            // batch rows it computes again at a time
constexpr int kChunk = 32;            // kept rows staged at a time
constexpr int kXPitch = kGroup + 8, kOutPitch = kGroup + 4, kSpecPitch = kGroup + 1;

// A non-finite activation makes every column of its tile non-finite at that batch row (inf * 0 and NaN * w are
// NaN, inf * w is infinite), so one column per tile tells: 1/128 of Ct is read, and where it is finite (always, in
// a healthy program) the block is done.  What bounds it is a launch; it is made programmatically, so that its
// start and its read of the tile lie under the GEMM's tail.  2048 x 4096 at 6400 rows, 1.5 % single weights: 83.0 us
// a pass without it, 86.4 us with it.
//
// Where something is not finite the block computes 32 batch rows of the tile at a time again: the product over the finite
// activations on the tensor cores (wmma: the tile is small and the case rare), and beside it, entry by entry, what
// the others add in the columns whose mask bit is set.  The NaNs of Ct become the sum of the two.  (A plain loop over
// the rows per column took 1.3 ms a pass for a single NaN and 400 ms for one feature that is NaN in every batch row; so
// it is 0.2 and 2.0 ms, and 5 ms where no activation is finite.)
// grid (ceil(M / 256), tiles), block 128: a warp per 32 columns of the tile.
template <int DT>
__global__ void __launch_bounds__(128)
tew_finite_kernel(const TileDesc* __restrict__ tiles, const uint16_t* __restrict__ Wp, long long ldw, const uint8_t* __restrict__ bits,
                  long long bits_ld, const uint16_t* At, long long lda, uint16_t* Ct, long long ldc, int M, float alpha) {
  using namespace nvcuda;
  using T = typename std::conditional<DT == kBF16, __nv_bfloat16, __half>::type;
  constexpr uint32_t kExp = DT == kBF16 ? 0x7f80u : 0x7c00u;
  __shared__ __align__(4) uint8_t flags[kCheckRows / 8];
  __shared__ __align__(128) uint16_t xs[kChunk * kXPitch];      // the chunk's activations, zero where not finite
  __shared__ __align__(16) uint16_t raw[kChunk * kGroup];       // the chunk's activations
  __shared__ uint32_t bad_in[kChunk];                           // batch rows that are not finite, per staged row
  __shared__ __align__(32) float sums[128 * kOutPitch];
  __shared__ float special[128 * kSpecPitch];                   // what non-finite activations add
  grid_launch_dependents();
  const TileDesc t = tiles[blockIdx.y];     // (installed by a synchronous call: read ahead of the wait)
  const bool empty = t.n_count == 0 || t.k_count == 0;
  const int n_first = empty ? 0 : t.n_list[0];
  grid_dependency_wait();   // Ct comes from the kernel before this one
  if (empty) return;
  const int m0 = blockIdx.x * kCheckRows, tid = threadIdx.x, warp = tid >> 5;
  // bit e: element e of the piece is infinite or NaN
  auto not_finite = [](const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t bad = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (((w[e >> 1] >> (16 * (e & 1))) & kExp) == kExp) bad |= 1u << e;
    }
    return bad;
  };
  uint32_t bad = 0;
  if (tid < kCheckRows / 8 && m0 + tid * 8 < M) bad = not_finite(*reinterpret_cast<const uint4*>(Ct + n_first * ldc + m0 + tid * 8));
  if (!__syncthreads_or(bad != 0)) return;
  if (tid < kCheckRows / 8) flags[tid] = static_cast<uint8_t>(bad);
  __syncthreads();

  const bool active = tid < t.n_count;
  const int n = active ? t.n_list[tid] : 0;
  const uint16_t* const wrow = Wp + static_cast<long long>(t.w_row0 + tid) * ldw;
  const uint8_t* const mask = bits + n * bits_ld;
  for (int g = 0; g < kCheckRows / kGroup; ++g) {
    if (*reinterpret_cast<const uint32_t*>(flags + g * (kGroup / 8)) == 0) continue;     // (the same for the whole block)
    const int mg = m0 + g * kGroup;
    uint32_t todo = 0;                              // NaNs of this thread's column
    if (active) {
#pragma unroll
      for (int p = 0; p < kGroup / 8; ++p) {
        if (mg + p * 8 >= M) continue;
        const uint4 v = *reinterpret_cast<const uint4*>(Ct + n * ldc + mg + p * 8);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float c = unpack1<DT>(static_cast<uint16_t>(w[e >> 1] >> (16 * (e & 1))));
          if (c != c) todo |= 1u << (p * 8 + e);
        }
      }
    }
    if (!__syncthreads_or(todo != 0)) continue;     // results that are out of the type's range, no more
    wmma::fragment<wmma::accumulator, 16, 16, 16, float> acc[2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) wmma::fill_fragment(acc[i >> 1][i & 1], 0.0f);
    uint32_t touched = 0, nan = 0;                  // batch rows with an entry in `special`, and those that are NaN there
    for (int r0 = 0; r0 < t.k_count; r0 += kChunk) {
      {
        const int row = tid >> 2, p = tid & 3, m = mg + p * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r0 + row < t.k_count && m < M) v = *reinterpret_cast<const uint4*>(At + t.k_list[r0 + row] * lda + m);
        const uint32_t b = not_finite(v);
        *reinterpret_cast<uint4*>(raw + row * kGroup + p * 8) = v;
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if ((b >> e) & 1) w[e >> 1] &= (e & 1) ? 0x0000ffffu : 0xffff0000u;
        }
        *reinterpret_cast<uint4*>(xs + row * kXPitch + p * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        uint32_t all = b << (8 * p);
        all |= __shfl_xor_sync(0xffffffffu, all, 1);
        all |= __shfl_xor_sync(0xffffffffu, all, 2);
        if (p == 0) bad_in[row] = all;
        bad = all;
      }
      const bool any_bad = __syncthreads_or(bad != 0);
#pragma unroll
      for (int k = 0; k < kChunk; k += 16) {
        wmma::fragment<wmma::matrix_a, 16, 16, 16, T, wmma::row_major> a[2];
        wmma::fragment<wmma::matrix_b, 16, 16, 16, T, wmma::row_major> b[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          // (all 128 rows of the tile exist, zero past its last column and past its last kept row)
          wmma::load_matrix_sync(a[i], reinterpret_cast<const T*>(Wp + static_cast<long long>(t.w_row0 + warp * 32 + i * 16) * ldw + r0 + k),
                                 static_cast<unsigned>(ldw));
          wmma::load_matrix_sync(b[i], reinterpret_cast<const T*>(xs + k * kXPitch + i * 16), kXPitch);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) wmma::mma_sync(acc[i >> 1][i & 1], a[i >> 1], b[i & 1], acc[i >> 1][i & 1]);
      }
      if (any_bad && todo) {
        for (int row = 0; row < kChunk; ++row) {
          uint32_t here = bad_in[row] & todo & ~nan;              // (a NaN stays one)
          if (here == 0) continue;
          const int k = t.k_list[r0 + row];
          if (!((mask[k >> 3] >> (k & 7)) & 1)) continue;
          const float w = unpack1<DT>(wrow[r0 + row]);
          for (; here; here &= here - 1) {
            const int e = __ffs(here) - 1;
            float* const s = special + tid * kSpecPitch + e;
            const float v = w * unpack1<DT>(raw[row * kGroup + e]) + (((touched >> e) & 1) ? *s : 0.0f);
            *s = v;
            touched |= 1u << e;
            if (v != v) nan |= 1u << e;
          }
        }
      }
      __syncthreads();                              // xs, raw and bad_in are free again
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      wmma::store_matrix_sync(sums + (warp * 32 + (i >> 1) * 16) * kOutPitch + (i & 1) * 16, acc[i >> 1][i & 1], kOutPitch, wmma::mem_row_major);
    }
    __syncwarp();
    for (; todo; todo &= todo - 1) {
      const int e = __ffs(todo) - 1;
      const float v = sums[tid * kOutPitch + e] + (((touched >> e) & 1) ? special[tid * kSpecPitch + e] : 0.0f);
      Ct[n * ldc + mg + e] = static_cast<uint16_t>(pack2<DT>(alpha * v, 0.0f) & 0xffffu);
    }
    __syncthreads();
  }
}

}  // namespace

cudaError_t tew_finite_launch(int dtype, const TileDesc* tiles, int n_tiles, const void* Wp, long long ldw, const uint8_t* bits,
                              long long bits_ld, const void* At, long long lda, void* Ct, long long ldc, int M, float alpha,
                              cudaStream_t stream) {
  if (M <= 0 || n_tiles <= 0) return cudaSuccess;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(128);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto kern = dtype == kBF16 ? tew_finite_kernel<kBF16> : tew_finite_kernel<kF16>;
  for (int t0 = 0; t0 < n_tiles; t0 += 65535) {     // tiles are the grid's y dimension
    cfg.gridDim = dim3(static_cast<unsigned>((M + kCheckRows - 1) / kCheckRows), static_cast<unsigned>(n_tiles - t0 < 65535 ? n_tiles - t0 : 65535));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tiles + t0, static_cast<const uint16_t*>(Wp), ldw, bits, bits_ld,
                                             static_cast<const uint16_t*>(At), lda, static_cast<uint16_t*>(Ct), ldc, M, alpha);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ts
