// TEW layers run as one masked GEMM whose tiles are wider than the mask: a tile gathers every row any of its
// single weights lies in, and the packed weights are zero outside the mask.  0 * x adds nothing while x is finite;
// an infinity or a NaN in a gathered row would reach all columns of the tile instead of those that keep the row.
// This pass takes such results back (the reference multiplies by a dense 0/1 mask, Pruning/VGG/prune_algo.py:171-175,
// and gives no rule for them; here a weight outside the mask is no part of the product).
#include "ts_common.cuh"
#include "ts_kernels.h"

namespace ts {

namespace {

// A non-finite activation makes every column of its tile non-finite at that batch row (inf * 0 and NaN * w are
// NaN, inf * w is infinite), so one column per tile tells: 1/128 of Ct is read, and where it is finite (always, in
// a healthy program) the block is done.  What bounds it is a launch; it is made programmatically, so that its
// start and its read of the tile lie under the GEMM's tail.  2048 x 4096 at 6400 rows, 1.5 % single weights: 83.0 us
// a pass without it, 86.4 us with it.  Where a batch row is not finite, thread j computes column j's NaNs again over the mask's
// entries alone.
// grid (ceil(M / 1024), tiles), block 128.
template <int DT>
__global__ void __launch_bounds__(128)
tew_finite_kernel(const TileDesc* __restrict__ tiles, const uint16_t* __restrict__ Wp, long long ldw, const uint8_t* __restrict__ bits,
                  long long bits_ld, const uint16_t* At, long long lda, uint16_t* Ct, long long ldc, int M, float alpha) {
  constexpr uint32_t kExp = DT == kBF16 ? 0x7f80u : 0x7c00u;
  __shared__ uint8_t flags[128];
  grid_launch_dependents();
  const TileDesc t = tiles[blockIdx.y];     // (installed by a synchronous call: read ahead of the wait)
  const bool empty = t.n_count == 0 || t.k_count == 0;
  const int n_first = empty ? 0 : t.n_list[0];
  grid_dependency_wait();   // Ct comes from the kernel before this one
  if (empty) return;
  const int m0 = blockIdx.x * 1024, m = m0 + threadIdx.x * 8;
  uint32_t bad = 0;
  if (m < M) {
    const uint4 v = *reinterpret_cast<const uint4*>(Ct + n_first * ldc + m);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (((w[e >> 1] >> (16 * (e & 1))) & kExp) == kExp) bad |= 1u << e;
    }
  }
  if (!__syncthreads_or(bad != 0)) return;
  flags[threadIdx.x] = static_cast<uint8_t>(bad);
  __syncthreads();
  const int j = threadIdx.x;
  if (j >= t.n_count) return;
  const int n = t.n_list[j];
  const uint16_t* const wrow = Wp + static_cast<long long>(t.w_row0 + j) * ldw;
  const uint8_t* const mask = bits + n * bits_ld;
  for (int i = 0; i < 1024; ++i) {
    if (!((flags[i >> 3] >> (i & 7)) & 1)) continue;
    uint16_t* const c = Ct + n * ldc + m0 + i;
    const float had = unpack1<DT>(*c);
    if (had == had) continue;
    float acc = 0.0f;
    for (int r = 0; r < t.k_count; ++r) {
      const int k = t.k_list[r];
      if ((mask[k >> 3] >> (k & 7)) & 1) acc = fmaf(unpack1<DT>(wrow[r]), unpack1<DT>(At[k * lda + m0 + i]), acc);
    }
    *c = static_cast<uint16_t>(pack2<DT>(alpha * acc, 0.0f) & 0xffffu);
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
    cfg.gridDim = dim3(static_cast<unsigned>((M + 1023) / 1024), static_cast<unsigned>(n_tiles - t0 < 65535 ? n_tiles - t0 : 65535));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tiles + t0, static_cast<const uint16_t*>(Wp), ldw, bits, bits_ld,
                                             static_cast<const uint16_t*>(At), lda, static_cast<uint16_t*>(Ct), ldc, M, alpha);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ts
