// Weight packing and 16-bit transpose.
//
// pack: builds the per-tile compacted weight matrix the masked GEMM consumes, the device-side
// counterpart of the reference's host loop gen_masked_stream_weight
// (StreamMaskedGEMM/perf/basic_nn.cu:757-769) and of the kernel compaction in exportPrunedModel
// (Pruning/BERT/utils/MyHook.py:76-85):  Wp[w_row0 + j][i] = W[kept_k[i]][kept_col(j)], K contiguous.
// Rows and K positions beyond the kept counts stay zero (the caller clears Wp before the launch).
// HBM-bound: reads the kept entries of W once, writes 2 bytes per kept entry.
//
// transpose16: out[c][r] = in[r][c] for 16-bit elements; turns a row-major activation matrix
// [M][K] into the K-major [K][M] layout the GEMM gathers from (the reference keeps its activations
// in that layout throughout, basic_nn.cu:823,1014).
#include "ts_common.cuh"
#include "ts_kernels.h"

namespace ts {

namespace {

template <typename T>
__device__ __forceinline__ float load_as_float(const T* p);
template <>
__device__ __forceinline__ float load_as_float<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float load_as_float<__half>(const __half* p) { return __half2float(*p); }
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}

// grid: (ceil(max_k / 64), n_tiles); block 256.  Each block moves a 64 (kept rows) x 128 (kept
// columns) patch through shared memory so that both the read (along columns) and the write (along
// K) are coalesced.
template <typename TIn, int DT>
__global__ void __launch_bounds__(256)
pack_weights_kernel(const TIn* __restrict__ W, long long ld_w, const TileDesc* __restrict__ tiles,
                    uint16_t* __restrict__ Wp, long long ldw) {
  const TileDesc td = tiles[blockIdx.y];
  const int i0 = blockIdx.x * 64;
  if (i0 >= td.k_count) return;
  __shared__ uint16_t patch[64][130];
  const int tx = threadIdx.x & 127;   // column inside the tile
  const int ty = threadIdx.x >> 7;    // 0..1
  long long col = -1;
  if (tx < td.n_count) {
    col = td.c_row0 + (td.n_list ? td.n_list[tx] + (td.relative ? tx : 0) : tx);
  }
  for (int ii = ty; ii < 64; ii += 2) {
    const int i = i0 + ii;
    uint16_t v = 0;
    if (i < td.k_count && col >= 0) {
      const int kk = td.k_list[i] + (td.relative ? i : 0);
      const float f = load_as_float<TIn>(W + static_cast<long long>(kk) * ld_w + col);
      v = static_cast<uint16_t>(pack2<DT>(f, 0.0f) & 0xffffu);
    }
    patch[ii][tx] = v;
  }
  __syncthreads();
  const int wi = threadIdx.x & 63;    // K position inside the patch
  const int wj = threadIdx.x >> 6;    // 0..3
  if (i0 + wi < td.k_count) {
    for (int j = wj; j < td.n_count; j += 4) {
      Wp[static_cast<long long>(td.w_row0 + j) * ldw + i0 + wi] = patch[wi][j];
    }
  }
}

__global__ void __launch_bounds__(256)
transpose16_kernel(const uint16_t* __restrict__ in, long long ld_in, uint16_t* __restrict__ out,
                   long long ld_out, int rows, int cols) {
  __shared__ uint16_t t[64][66];
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  for (int rr = ty; rr < 64; rr += 4) {
    const int r = r0 + rr, c = c0 + tx;
    t[rr][tx] = (r < rows && c < cols) ? in[static_cast<long long>(r) * ld_in + c] : 0;
  }
  __syncthreads();
  for (int cc = ty; cc < 64; cc += 4) {
    const int c = c0 + cc, r = r0 + tx;
    if (c < cols && r < rows) out[static_cast<long long>(c) * ld_out + r] = t[tx][cc];
  }
}

// The same for matrices whose pointers, row pitches and sizes allow 16-byte accesses on both sides.  A block
// moves 128 x 128 elements: a thread loads an 8 x 8 block (eight 16-byte pieces, 256 contiguous bytes of a
// row per 16 lanes), transposes it in registers by byte permutes, and the block's 16-byte pieces change
// lanes through shared memory, so that the stores are runs of 256 bytes too; the pieces of a row are
// swizzled by its number, which keeps both sides free of bank conflicts.  Bound by the memory system:
// 3080 x 3072 (38 MB moved, most of it in L2) 5.4 us, against 15 us for the two-byte form above.
__global__ void __launch_bounds__(256)
transpose16_vec_kernel(const uint16_t* __restrict__ in, long long ld_in, uint16_t* __restrict__ out,
                       long long ld_out, int rows, int cols) {
  __shared__ uint4 t[128 * 16];            // [column][row / 8], 16-byte pieces
  const int r0 = blockIdx.y * 128, c0 = blockIdx.x * 128;
  const int c8 = threadIdx.x & 15, r8 = threadIdx.x >> 4;
  const int c = c0 + c8 * 8, r = r0 + r8 * 8;
  uint4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = (c < cols && r + i < rows) ? __ldg(reinterpret_cast<const uint4*>(in + static_cast<long long>(r + i) * ld_in + c))
                                      : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {             // columns 2q, 2q + 1: word q of every row
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 a = v[2 * i], b = v[2 * i + 1];
      const uint32_t wa = q == 0 ? a.x : (q == 1 ? a.y : (q == 2 ? a.z : a.w));
      const uint32_t wb = q == 0 ? b.x : (q == 1 ? b.y : (q == 2 ? b.z : b.w));
      lo[i] = __byte_perm(wa, wb, 0x5410);
      hi[i] = __byte_perm(wa, wb, 0x7632);
    }
    t[(c8 * 8 + 2 * q) * 16 + (r8 ^ c8)] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    t[(c8 * 8 + 2 * q + 1) * 16 + (r8 ^ c8)] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  }
  __syncthreads();
  const int p = threadIdx.x & 15;           // rows 8p .. of a column
  const bool r_ok = r0 + p * 8 < rows;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int cc = i * 16 + (threadIdx.x >> 4);
    if (r_ok && c0 + cc < cols) {
      *reinterpret_cast<uint4*>(out + static_cast<long long>(c0 + cc) * ld_out + r0 + p * 8) = t[cc * 16 + (p ^ (cc >> 3))];
    }
  }
}

// Ct[rows[blockIdx.y]][0 .. M) = 0, eight elements per thread.
__global__ void __launch_bounds__(256)
zero_rows_kernel(const int* __restrict__ rows, uint16_t* __restrict__ Ct, long long ldc, int M) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (m < M) *reinterpret_cast<uint4*>(Ct + static_cast<long long>(__ldg(rows + blockIdx.y)) * ldc + m) = make_uint4(0, 0, 0, 0);
}

}  // namespace

cudaError_t zero_rows_launch(const int* rows, int n_rows, void* Ct, long long ldc, int M, cudaStream_t stream) {
  const unsigned bx = static_cast<unsigned>((M / 8 + 255) / 256);
  for (int r = 0; r < n_rows; r += 65535) {     // rows are the grid's y dimension
    zero_rows_kernel<<<dim3(bx, static_cast<unsigned>(n_rows - r < 65535 ? n_rows - r : 65535)), 256, 0, stream>>>(
        rows + r, static_cast<uint16_t*>(Ct), ldc, M);
  }
  return cudaGetLastError();
}

cudaError_t pack_weights_launch(int w_dtype, int out_dtype, const void* W, long long ld_w,
                                const TileDesc* tiles, int n_tiles, int max_k, void* Wp,
                                long long ldw, cudaStream_t stream) {
  if (n_tiles <= 0 || max_k <= 0) return cudaSuccess;
  dim3 grid((max_k + 63) / 64, n_tiles);
  uint16_t* out = static_cast<uint16_t*>(Wp);
#define TS_PACK(TIN, DT) \
  pack_weights_kernel<TIN, DT><<<grid, 256, 0, stream>>>(static_cast<const TIN*>(W), ld_w, tiles, out, ldw)
  if (out_dtype == kBF16) {
    if (w_dtype == kF32) TS_PACK(float, kBF16);
    else if (w_dtype == kF16) TS_PACK(__half, kBF16);
    else TS_PACK(__nv_bfloat16, kBF16);
  } else {
    if (w_dtype == kF32) TS_PACK(float, kF16);
    else if (w_dtype == kF16) TS_PACK(__half, kF16);
    else TS_PACK(__nv_bfloat16, kF16);
  }
#undef TS_PACK
  return cudaGetLastError();
}

cudaError_t transpose16_launch(const void* in, long long ld_in, void* out, long long ld_out,
                               int rows, int cols, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const bool vec = ((rows | cols | ld_in | ld_out) & 7) == 0 &&
                   ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
  if (vec && (rows + 127) / 128 <= 65535) {
    transpose16_vec_kernel<<<dim3((cols + 127) / 128, (rows + 127) / 128), 256, 0, stream>>>(
        static_cast<const uint16_t*>(in), ld_in, static_cast<uint16_t*>(out), ld_out, rows, cols);
    return cudaGetLastError();
  }
  dim3 grid((cols + 63) / 64, (rows + 63) / 64);
  transpose16_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in), ld_in,
                                               static_cast<uint16_t*>(out), ld_out, rows, cols);
  return cudaGetLastError();
}

}  // namespace ts
