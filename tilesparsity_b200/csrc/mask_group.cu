// Mask construction for a whole group of layers in a handful of launches.
//
// The arithmetic is that of mask_build.cu (NumPy's float32 operations in NumPy's order, see there); what is
// different is the shape of the work.  A pruning step hands over anything from one 768 x 3072 matrix to the
// kernels of a whole network under one threshold, and none of its stages is long: per-layer launches, uploads
// of tile tables and a round trip to the host between the column and the row stage cost 1100 us for the 13
// kernels of a VGG16-shaped network (59 MB of scores: 9 us of HBM time).  Here every stage is one launch over
// all layers; the layer table travels in the kernel arguments; the percentile is one launch (a cluster of
// eight blocks, histograms in shared memory); the regrouping of surviving columns into tiles happens on
// the device; and the results land in page-locked host memory straight from the kernels.
#include <cooperative_groups.h>

#include "ts_common.cuh"
#include "ts_mask_kernels.h"

namespace cg = cooperative_groups;

namespace ts {

namespace {

__device__ __forceinline__ const MaskLayer& layer_at(const MaskGroup& g, int l) { return g.ext ? g.ext[l] : g.inl[l]; }

// Layer whose range of blocks holds `block` (ranges start at first(l), ascending).
template <typename F>
__device__ __forceinline__ int find_layer(const MaskGroup& g, int block, F first) {
  int lo = 0, hi = g.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first(layer_at(g, mid)) <= block) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Tiles of layer l, and where the norms of its first tile-row lie.
__device__ __forceinline__ int tiles_of(const MaskGroup& g, int l) { return g.n_tiles ? g.n_tiles[l] : layer_at(g, l).max_tiles; }
__device__ __forceinline__ long long norm_base(const MaskGroup& g, int l) {
  if (!g.n_tiles) return layer_at(g, l).norm0;
  long long b = 0;
  for (int i = 0; i < l; ++i) b += static_cast<long long>(g.n_tiles[i]) * layer_at(g, i).K;
  return b;
}
__device__ __forceinline__ int bound_of(const MaskGroup& g, const MaskLayer& L, int t) {
  return g.bounds ? g.bounds[L.tile0 + t] : min(L.N, t * g.G);
}

// ---------------------------------------------------------------------------------------------
// Column norms: sqrt(sum_k score[k][n]^2 in row order) / K
// ---------------------------------------------------------------------------------------------
// The sum of one column is a chain of K dependent additions (four cycles each: 10 us for 4608 rows), so all
// that counts is that nothing else slows the chain down: a block owns 32 columns, all four warps keep five
// slabs of 64 rows in flight (16-byte cp.async where the rows allow it; with 4-byte ones the warp that adds spent most
// of its time issuing its share of them), and one warp walks the slab that has landed with the next 16 values in
// registers ahead of the additions.  13 kernels of a VGG16-shaped network: 82 -> 36 us.
constexpr int kColsPerBlock = 32, kColRows = 64, kColSlabs = 6;

__global__ void __launch_bounds__(128)
group_col_norms_kernel(const __grid_constant__ MaskGroup g, float* __restrict__ out) {
  __shared__ __align__(16) float slab[kColSlabs][kColRows][kColsPerBlock];
  const int l = find_layer(g, blockIdx.x, [](const MaskLayer& m) { return m.col_blk0; });
  const MaskLayer& L = layer_at(g, l);
  const int n0 = (blockIdx.x - L.col_blk0) * kColsPerBlock;
  const int c = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool col_ok = n0 + c < L.N;
  const int K = L.K, n_slabs = (K + kColRows - 1) / kColRows;
  const float* src = L.score + n0 + c;
  const bool vec = (L.ld % 4) == 0 && (reinterpret_cast<uintptr_t>(L.score) & 15u) == 0 && n0 + kColsPerBlock <= L.N;
  auto fetch = [&](int s) {
    if (s < n_slabs && vec) {
#pragma unroll
      for (int i = 0; i < kColRows / 16; ++i) {        // four rows of 8 x 16 bytes per warp
        const int r = (w + i * 4) * 4 + (c >> 3), k = s * kColRows + r;
        if (k < K) cp_async_16_full(smem_u32(&slab[s % kColSlabs][r][(c & 7) * 4]), L.score + static_cast<long long>(k) * L.ld + n0 + (c & 7) * 4);
      }
    } else if (s < n_slabs && col_ok) {
#pragma unroll
      for (int i = 0; i < kColRows / 4; ++i) {
        const int r = w + i * 4, k = s * kColRows + r;
        if (k < K) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&slab[s % kColSlabs][r][c])),
                       "l"(src + static_cast<long long>(k) * L.ld));
        }
      }
    }
    cp_async_commit();
  };
  for (int s = 0; s < kColSlabs - 1; ++s) fetch(s);
  float acc = 0.0f;                        // (a square added to +0 is that square)
  for (int s = 0; s < n_slabs; ++s) {
    cp_async_wait_group<kColSlabs - 2>();
    __syncthreads();                       // slab s has landed; slab s - 1 has been consumed
    fetch(s + kColSlabs - 1);
    if (w == 0) {
      const int rows = min(kColRows, K - s * kColRows);
      const float(*row)[kColsPerBlock] = slab[s % kColSlabs];
      int r = 0;
      if (rows == kColRows) {              // the next 16 values are read while these are added
        float x[2][16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[0][i] = row[i][c];
#pragma unroll
        for (int b = 0; b < kColRows / 16; ++b) {
          if (b + 1 < kColRows / 16) {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[(b + 1) & 1][i] = row[(b + 1) * 16 + i][c];
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) acc = __fadd_rn(acc, __fmul_rn(x[b & 1][i], x[b & 1][i]));
        }
        r = kColRows;
      }
      for (; r < rows; ++r) acc = __fadd_rn(acc, __fmul_rn(row[r][c], row[r][c]));
    }
  }
  cp_async_wait_all();
  if (w == 0 && col_ok) out[L.col0 + n0 + c] = __fdiv_rn(__fsqrt_rn(acc), static_cast<float>(K));
}

// ---------------------------------------------------------------------------------------------
// np.percentile of a float32 array in one launch
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t key_of(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// One block of 1024 threads, or a cluster of eight of them for more values.  The two order statistics by
// digits of 11 bits over the range [min, max] of the order-preserving keys (counting from the bottom of the
// range spreads values that share their leading bits over the bins, so the shared-memory atomics rarely
// meet); every block adds up all blocks' histograms through distributed shared memory and makes the same
// choice, so nothing is sent back.  Then NumPy's rank arithmetic and _lerp, every step one IEEE operation in
// the type NumPy would use (wide: q is a NumPy float64).  18432 values: 23 us; 115 Ki: 25 us
// (what the passes wait for is each other: with the keys in registers and all remote reads in flight it was 26).
constexpr int kPctBins = 2048;

__global__ void __launch_bounds__(1024)
group_percentile_kernel(const float* __restrict__ vals, long long n_static, const __grid_constant__ MaskGroup g, double q, int wide,
                        double* __restrict__ thr_out, double* __restrict__ thr_host) {
  __shared__ unsigned int hist[kPctBins];
  __shared__ unsigned int lo_s, hi_s, above_s;
  __shared__ unsigned int warp_sum[32];
  __shared__ uint32_t sel_bin, sel_excl, sel_count, next_bin;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned int ranks = cluster.num_blocks(), rank = cluster.block_rank();
  const int t = threadIdx.x;
  long long n = n_static;
  if (g.n_tiles) {
    n = 0;
    for (int l = 0; l < g.n; ++l) n += static_cast<long long>(g.n_tiles[l]) * layer_at(g, l).K;
  }
  // ranks and interpolation weight (np.percentile, method "linear")
  long long pi, ni;
  float gamma_f = 0.0f;
  double gamma_d = 0.0;
  if (wide) {
    const double virt = __dmul_rn(static_cast<double>(n - 1), __ddiv_rn(q, 100.0));
    const double prev = floor(virt);
    pi = static_cast<long long>(prev);
    ni = pi + 1;
    if (virt >= static_cast<double>(n - 1)) pi = ni = n - 1;
    gamma_d = __dsub_rn(virt, prev);
  } else {
    const float virt = __fmul_rn(static_cast<float>(n - 1), __fdiv_rn(static_cast<float>(q), 100.0f));
    const float prev = floorf(virt);
    pi = static_cast<long long>(prev);
    ni = pi + 1;
    if (virt >= static_cast<float>(n - 1)) pi = ni = n - 1;
    gamma_f = __fsub_rn(virt, prev);
  }
  if (pi < 0) pi = ni = 0;
  if (ni > n - 1) ni = n - 1;
  if (pi > n - 1) pi = n - 1;

  const long long stride = 1024LL * ranks, first = rank * 1024LL + t;
  if (t == 0) {
    lo_s = 0xffffffffu;
    hi_s = 0u;
    above_s = 0xffffffffu;
  }
  __syncthreads();
  {
    unsigned int lo = 0xffffffffu, hi = 0u;
    for (long long i = first; i < n; i += stride) {
      const uint32_t k = key_of(__ldg(vals + i));
      lo = min(lo, k);
      hi = max(hi, k);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((t & 31) == 0) {
      atomicMin(&lo_s, lo);
      atomicMax(&hi_s, hi);
    }
  }
  cluster.sync();
  uint32_t lo = 0xffffffffu, hi = 0u;
  for (unsigned int r = 0; r < ranks; ++r) {
    lo = min(lo, *cluster.map_shared_rank(&lo_s, r));
    hi = max(hi, *cluster.map_shared_rank(&hi_s, r));
  }
  long long want = pi;              // rank inside [lo, hi]
  long long less = 0;               // keys below lo
  uint32_t key = lo, above = 0xffffffffu;
  long long count_le = n;
  bool have_above = false;
  for (int pass = 0; pass < 4; ++pass) {
    const uint32_t range = hi - lo;
    const int bits = 32 - __clz(range | 1u);
    const int shift = bits > 11 ? bits - 11 : 0;
    for (int b = t; b < kPctBins; b += 1024) hist[b] = 0;
    if (t == 0) next_bin = 0xffffffffu;
    __syncthreads();
    for (long long i = first; i < n; i += stride) {
      const uint32_t k = key_of(__ldg(vals + i));
      if (k >= lo && k <= hi) atomicAdd(&hist[(k - lo) >> shift], 1u);
    }
    cluster.sync();
    // bins 2t and 2t + 1 over all blocks, inclusive scan over the block
    unsigned int a = 0, b = 0;
    for (unsigned int r = 0; r < ranks; ++r) {
      const uint2 v = *reinterpret_cast<const uint2*>(cluster.map_shared_rank(hist, r) + 2 * t);
      a += v.x;
      b += v.y;
    }
    unsigned int incl = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int up = __shfl_up_sync(0xffffffffu, incl, o);
      if ((t & 31) >= o) incl += up;
    }
    if ((t & 31) == 31) warp_sum[t >> 5] = incl;
    __syncthreads();
    if (t < 32) {
      unsigned int s = warp_sum[t];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int up = __shfl_up_sync(0xffffffffu, s, o);
        if (t >= o) s += up;
      }
      warp_sum[t] = s;
    }
    __syncthreads();
    if (t >= 32) incl += warp_sum[(t >> 5) - 1];
    const unsigned int ex_a = incl - a - b, ex_b = incl - b;
    if (want >= ex_a && want < ex_b) {
      sel_bin = 2 * t;
      sel_excl = ex_a;
      sel_count = a;
    } else if (want >= ex_b && want < incl) {
      sel_bin = 2 * t + 1;
      sel_excl = ex_b;
      sel_count = b;
    }
    __syncthreads();
    const uint32_t bin = sel_bin;
    // the next key above the selected one, when single keys are bins
    if (shift == 0) {
      if (a && 2u * t > bin) atomicMin(&next_bin, 2u * t);
      if (b && 2u * t + 1u > bin) atomicMin(&next_bin, 2u * t + 1u);
    }
    cluster.sync();                 // every block has read every histogram; next_bin is complete
    less += sel_excl;
    want -= sel_excl;
    if (shift == 0) {
      key = lo + bin;
      count_le = less + sel_count;
      if (next_bin != 0xffffffffu) {
        above = lo + next_bin;
        have_above = true;
      }
      break;
    }
    lo += bin << shift;
    hi = lo + min(hi - lo, (1u << shift) - 1u);     // (no sum that wraps: keys reach 0xffffffff)
  }
  if (ni != pi && count_le < ni + 1 && !have_above) {   // (the same decision in every block)
    unsigned int m = 0xffffffffu;
    for (long long i = first; i < n; i += stride) {
      const uint32_t k = key_of(__ldg(vals + i));
      if (k > key) m = min(m, k);
    }
    m = __reduce_min_sync(0xffffffffu, m);
    if ((t & 31) == 0) atomicMin(&above_s, m);
    cluster.sync();
    for (unsigned int r = 0; r < ranks; ++r) above = min(above, *cluster.map_shared_rank(&above_s, r));
  }
  cluster.sync();                   // no block leaves while others read its shared memory
  if (rank == 0 && t == 0) {
    const float x = value_of(key);
    const float y = (ni != pi && count_le < ni + 1) ? value_of(above) : x;
    const float diff = __fsub_rn(y, x);
    double res;
    if (wide) {
      res = __dadd_rn(static_cast<double>(x), __dmul_rn(static_cast<double>(diff), gamma_d));
      if (gamma_d >= 0.5) res = __dsub_rn(static_cast<double>(y), __dmul_rn(static_cast<double>(diff), __dsub_rn(1.0, gamma_d)));
    } else {
      float r = __fadd_rn(x, __fmul_rn(diff, gamma_f));
      if (gamma_f >= 0.5f) r = __fsub_rn(y, __fmul_rn(diff, __fsub_rn(1.0f, gamma_f)));
      res = static_cast<double>(r);
    }
    *thr_out = res;
    if (thr_host) *thr_host = res;
  }
}

// ---------------------------------------------------------------------------------------------
// Column stage -> tiles: one block per layer
// ---------------------------------------------------------------------------------------------
// keep[c] = norm > threshold (strict, prune_algo.py:67).  A tile ends right after its G-th kept column unless
// that is the last column (prune_algo.py:72-89), so column c lies in tile floor(kept columns before c / G).
__global__ void __launch_bounds__(256)
group_columns_kernel(const __grid_constant__ MaskGroup g, const float* __restrict__ col_norms, const double* __restrict__ thr,
                     uint8_t* __restrict__ keep, int* __restrict__ tile_of_col, int* __restrict__ bounds, int* __restrict__ n_tiles,
                     uint8_t* __restrict__ keep_host, int* __restrict__ bounds_host, int* __restrict__ n_tiles_host) {
  __shared__ int warp_cnt[8];
  const int l = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const MaskLayer& L = layer_at(g, l);
  const double limit = *thr;
  int before = 0;                     // kept columns before this step
  if (t == 0) bounds[L.tile0] = bounds_host[L.tile0] = 0;
  for (int c0 = 0; c0 < L.N; c0 += 256) {
    const int c = c0 + t;
    const bool k = c < L.N && static_cast<double>(col_norms[L.col0 + c]) > limit;
    const unsigned int bal = __ballot_sync(0xffffffffu, k);
    if (lane == 0) warp_cnt[w] = __popc(bal);
    __syncthreads();
    int mine = before, total = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < w) mine += warp_cnt[i];
      total += warp_cnt[i];
    }
    mine += __popc(bal & ((1u << lane) - 1u));
    if (c < L.N) {
      keep[L.col0 + c] = keep_host[L.col0 + c] = k ? 1 : 0;
      tile_of_col[L.col0 + c] = mine / g.G;
      if (k && (mine + 1) % g.G == 0 && c + 1 < L.N) {
        bounds[L.tile0 + (mine + 1) / g.G] = bounds_host[L.tile0 + (mine + 1) / g.G] = c + 1;
      }
      if (c + 1 == L.N) {
        const int nt = mine / g.G + 1;
        n_tiles[l] = n_tiles_host[l] = nt;
        bounds[L.tile0 + nt] = bounds_host[L.tile0 + nt] = L.N;
      }
    }
    before += total;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Tile-row norms
// ---------------------------------------------------------------------------------------------
struct Run {
  const float* row;        // first element of the run
  const uint8_t* colmask;  // nullptr, or one byte per element (0: the element counts as +0)
};

__device__ __forceinline__ float square_at(const Run& s, int i) {
  if (s.colmask && !s.colmask[i]) return 0.0f;
  const float x = __ldg(s.row + i);
  return __fmul_rn(x, x);
}

// NumPy's pairwise sum of [o, o + n), 8 <= n <= 128, by the 8 lanes of a group (lane j: elements j, j + 8, ...).
// A plain loop: with its 16 loads written out ahead of the additions the kernel takes more registers and fewer blocks
// run (8192 x 8192 with pruned columns: 227 us, 182 us so; the 13 kernels of a VGG16-shaped network 274 -> 262 us a call).
__device__ __forceinline__ float leaf8(const Run& s, int o, int n, int j) {
  const int body = n - (n % 8);
  float r = square_at(s, o + j);
  for (int i = 8; i < body; i += 8) r = __fadd_rn(r, square_at(s, o + i + j));
  r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));   // r0+r1, r2+r3, r4+r5, r6+r7
  r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));
  r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 4));
  for (int i = body; i < n; ++i) r = __fadd_rn(r, square_at(s, o + i));
  return r;
}

// A run of any length; the control flow depends on n only, which is uniform across a warp.
__device__ float pairwise8(const Run& s, int o, int n, int j) {
  if (n < 8) {
    float r = 0.0f;
    for (int i = 0; i < n; ++i) r = __fadd_rn(r, square_at(s, o + i));
    return r;
  }
  if (n <= 128) return leaf8(s, o, n, j);
  int n2 = n / 2;
  n2 -= n2 % 8;
  const float a = pairwise8(s, o, n2, j);
  const float b = pairwise8(s, o + n2, n - n2, j);
  return __fadd_rn(a, b);
}

// norms[base + t*K + k] = ||score[k, tile t] (.* kept columns)|| / width.  A block takes 32 rows of one tile, one
// row per group of 8 lanes.  Tiles of exactly 128 columns without a column mask (all of tw1's when 128
// divides N) go through shared memory with 16-byte loads; bound by HBM there.
__global__ void __launch_bounds__(256)
group_row_norms_kernel(const __grid_constant__ MaskGroup g, const uint8_t* __restrict__ col_keep, float* __restrict__ norms) {
  constexpr int kPitch = 136;   // floats per staged row: rows 8 banks apart, 16-byte aligned
  __shared__ __align__(16) float stage[32 * kPitch];
  const int l = find_layer(g, blockIdx.x, [](const MaskLayer& m) { return m.norm_blk0; });
  const MaskLayer& L = layer_at(g, l);
  const int kb = (L.K + 31) / 32;
  const int rel = blockIdx.x - L.norm_blk0, t = rel / kb, k0 = (rel - t * kb) * 32;
  if (t >= tiles_of(g, l)) return;
  const int c0 = bound_of(g, L, t), width = bound_of(g, L, t + 1) - c0;
  const int group = threadIdx.x >> 3, j = threadIdx.x & 7, k = k0 + group;
  float v;
  if (width == 128 && !col_keep && (L.ld % 4) == 0 && (c0 % 4) == 0 && (reinterpret_cast<uintptr_t>(L.score) & 15u) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {                            // 32 rows x 32 float4
      const int r = (threadIdx.x >> 5) + i * 8, c4 = threadIdx.x & 31;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k0 + r < L.K) x = __ldg(reinterpret_cast<const float4*>(L.score + static_cast<long long>(k0 + r) * L.ld + c0 + c4 * 4));
      *reinterpret_cast<float4*>(&stage[r * kPitch + c4 * 4]) = x;
    }
    __syncthreads();
    const float* row = &stage[group * kPitch];
    float x = row[j];
    v = __fmul_rn(x, x);
#pragma unroll
    for (int i = 8; i < 128; i += 8) {
      x = row[i + j];
      v = __fadd_rn(v, __fmul_rn(x, x));
    }
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
  } else {
    const int kk = k < L.K ? k : L.K - 1;   // clamped rows keep the warp converged; their result is dropped
    Run s;
    s.row = L.score + static_cast<long long>(kk) * L.ld + c0;
    s.colmask = col_keep ? col_keep + L.col0 + c0 : nullptr;
    v = pairwise8(s, 0, width, j);
  }
  v = __fdiv_rn(__fsqrt_rn(v), static_cast<float>(width));
  if (k < L.K && j == 0) norms[norm_base(g, l) + static_cast<long long>(t) * L.K + k] = v;
}

// ---------------------------------------------------------------------------------------------
// Thresholded: kept-row lists and dense masks
// ---------------------------------------------------------------------------------------------
// Blocks below g.list_blocks: one tile each; its kept rows (norm > threshold, strict) in ascending order, at
// an offset drawn from a cursor, a multiple of kListAlign (the host puts the tiles back in order by their records).
// The list usually lies in page-locked host memory, where the number of writes counts and not their size: the rows
// are gathered in shared memory and leave as whole lines, up to 1 KiB at a time.  The blocks after
// them write the dense masks, 16 mask bytes per thread and step.  One 768 x 3072 matrix: 50 us with a write per row
// and eight steps, 11.5 us so.
constexpr int kDenseSteps = 2;

__global__ void __launch_bounds__(256)
group_apply_kernel(const __grid_constant__ MaskGroup g, const float* __restrict__ norms, const double* __restrict__ thr,
                   const uint8_t* __restrict__ col_keep, const int* __restrict__ tile_of_col, int* __restrict__ cursor,
                   int* __restrict__ list, int2* __restrict__ records) {
  const double limit = *thr;
  if (blockIdx.x < static_cast<unsigned>(g.list_blocks)) {
    __shared__ int warp_cnt[8];
    __shared__ int base_s;
    __shared__ __align__(16) int buf[512];
    const int l = find_layer(g, blockIdx.x, [](const MaskLayer& m) { return m.rec0; });
    const MaskLayer& L = layer_at(g, l);
    const int t = blockIdx.x - L.rec0;
    if (t >= tiles_of(g, l)) return;
    const float* v = norms + norm_base(g, l) + static_cast<long long>(t) * L.K;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int c = 0;
    for (int k = threadIdx.x; k < L.K; k += 256) c += static_cast<double>(v[k]) > limit ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) warp_cnt[w] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      int total = 0;
      for (int i = 0; i < 8; ++i) total += warp_cnt[i];
      base_s = atomicAdd(cursor, (total + kListAlign - 1) / kListAlign * kListAlign);
      records[blockIdx.x] = make_int2(base_s, total);
    }
    __syncthreads();
    int* out = list + base_s;
    int fill = 0;                         // rows waiting in buf, below 256 between the steps
    for (int k0 = 0; k0 < L.K; k0 += 256) {
      const int k = k0 + threadIdx.x;
      const bool f = k < L.K && static_cast<double>(v[k]) > limit;
      const unsigned int bal = __ballot_sync(0xffffffffu, f);
      if (lane == 0) warp_cnt[w] = __popc(bal);
      __syncthreads();
      int before = fill, total = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < w) before += warp_cnt[i];
        total += warp_cnt[i];
      }
      if (f) buf[before + __popc(bal & ((1u << lane) - 1u))] = k;
      fill += total;
      __syncthreads();
      if (fill >= 256) {
        if (threadIdx.x < 64) reinterpret_cast<int4*>(out)[threadIdx.x] = reinterpret_cast<const int4*>(buf)[threadIdx.x];
        const int rest = buf[256 + threadIdx.x];
        __syncthreads();
        buf[threadIdx.x] = rest;
        __syncthreads();
        out += 256;
        fill -= 256;
      }
    }
    // (whole pieces of four: what stands behind the last row lies inside the tile's rounded share)
    if (static_cast<int>(threadIdx.x) * 4 < fill) reinterpret_cast<int4*>(out)[threadIdx.x] = reinterpret_cast<const int4*>(buf)[threadIdx.x];
    return;
  }
  const int block = static_cast<int>(blockIdx.x) - g.list_blocks;
  const int l = find_layer(g, block, [](const MaskLayer& m) { return m.dense_blk0; });
  const MaskLayer& L = layer_at(g, l);
  const unsigned int per_row = static_cast<unsigned int>((L.N + 15) / 16);
  const unsigned int groups = per_row * static_cast<unsigned int>(L.K);   // (2^32 would be 275 GB of scores)
  const bool one_tile = !tile_of_col && g.G % 16 == 0;                    // 16 columns never straddle a tile
  const float* v = norms + norm_base(g, l);
  const bool vec = (L.N % 16) == 0 && (L.ld_mask % 16) == 0 && (reinterpret_cast<uintptr_t>(L.mask) & 15u) == 0;
  unsigned int i = static_cast<unsigned int>(block - L.dense_blk0) * (256u * kDenseSteps) + threadIdx.x;
  for (int step = 0; step < kDenseSteps && i < groups; ++step, i += 256) {
    const int k = static_cast<int>(i / per_row), n0 = static_cast<int>(i - k * per_row) * 16;
    const int n1 = min(L.N, n0 + 16);
    uint32_t out[4] = {0, 0, 0, 0};
    int tile = -1;
    uint32_t on = 0;
    if (one_tile) {
      on = static_cast<double>(v[static_cast<long long>(n0 / g.G) * L.K + k]) > limit ? 0x01010101u : 0u;
      out[0] = out[1] = out[2] = out[3] = on;
    } else if (tile_of_col && vec && ((L.col0 + n0) & 15) == 0 && tile_of_col[L.col0 + n0] == tile_of_col[L.col0 + n0 + 15]) {
      // (tile numbers ascend with the column: all 16 in one tile, their flags in one load)
      if (static_cast<double>(v[static_cast<long long>(tile_of_col[L.col0 + n0]) * L.K + k]) > limit) {
        const uint4 kept = __ldg(reinterpret_cast<const uint4*>(col_keep + L.col0 + n0));
        out[0] = kept.x;
        out[1] = kept.y;
        out[2] = kept.z;
        out[3] = kept.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        if (n0 + e < n1) {
          const int t = tile_of_col ? tile_of_col[L.col0 + n0 + e] : (n0 + e) / g.G;
          if (t != tile) {
            tile = t;
            on = static_cast<double>(v[static_cast<long long>(t) * L.K + k]) > limit ? 1u : 0u;
          }
          const uint32_t bit = col_keep ? (on & col_keep[L.col0 + n0 + e]) : on;
          out[e >> 2] |= bit << (8 * (e & 3));
        }
      }
    }
    uint8_t* dst = L.mask + static_cast<long long>(k) * L.ld_mask + n0;
    if (vec) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
    } else {
      for (int e = 0; e < n1 - n0; ++e) dst[e] = static_cast<uint8_t>(out[e >> 2] >> (8 * (e & 3)));
    }
  }
}

template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), unsigned grid, unsigned block, unsigned cluster, cudaStream_t s, A... args) {
  if (grid == 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace

int group_col_blocks(int N) { return (N + kColsPerBlock - 1) / kColsPerBlock; }
int group_norm_blocks(int K, int tiles) { return tiles * ((K + 31) / 32); }
long long group_dense_blocks(int K, int N) {
  return (static_cast<long long>((N + 15) / 16) * K + 256 * kDenseSteps - 1) / (256 * kDenseSteps);
}

cudaError_t group_col_norms_launch(const MaskGroup& g, int blocks, float* out, cudaStream_t s) {
  return launch(group_col_norms_kernel, blocks, 128, 1, s, g, out);
}

cudaError_t group_percentile_launch(const float* vals, long long n, long long n_max, const MaskGroup& g, double q, int wide,
                                    double* thr, double* thr_host, cudaStream_t s) {
  // up to 16 Ki values one block reads them all as fast as eight would start together
  const unsigned ranks = n_max > (1 << 14) ? 8 : 1;
  return launch(group_percentile_kernel, ranks, 1024, ranks, s, vals, n, g, q, wide, thr, thr_host);
}

cudaError_t group_columns_launch(const MaskGroup& g, const float* col_norms, const double* thr, uint8_t* keep, int* tile_of_col,
                                 int* bounds, int* n_tiles, uint8_t* keep_host, int* bounds_host, int* n_tiles_host, cudaStream_t s) {
  return launch(group_columns_kernel, g.n, 256, 1, s, g, col_norms, thr, keep, tile_of_col, bounds, n_tiles, keep_host, bounds_host,
                n_tiles_host);
}

cudaError_t group_row_norms_launch(const MaskGroup& g, int blocks, const uint8_t* col_keep, float* norms, cudaStream_t s) {
  return launch(group_row_norms_kernel, blocks, 256, 1, s, g, col_keep, norms);
}

cudaError_t group_apply_launch(const MaskGroup& g, int blocks, const float* norms, const double* thr, const uint8_t* col_keep,
                               const int* tile_of_col, int* cursor, int* list, int2* records, cudaStream_t s) {
  return launch(group_apply_kernel, blocks, 256, 1, s, g, norms, thr, col_keep, tile_of_col, cursor, list, records);
}

}  // namespace ts
