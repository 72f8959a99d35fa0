// Per-row, per-block transposition between the mul_ir and ir_mul layouts.
//
// Takes the place of the reference's closed `segmented_transpose`
// (cuequivariance_torch/primitives/transpose.py:155-183): block b of every row is a [u, v]
// tile at `offset` and is written back as [v, u].  The row is staged in shared memory so that both
// the global read and the global write are contiguous.
#include "common.cuh"

namespace {

// One warp per row, four elements per access.  Bound by HBM (a read and a write of every row); what the kernel below,
// one element per access and two block-wide barriers per row, takes three times as long for is the division per
// element and the wait for the slowest thread: 32,768 rows of 64x(0e+1o+2e) in bf16, 75 MB: 71 -> 21 us.
template <typename T> struct Quad;
template <> struct Quad<float> { using type = float4; };
template <> struct Quad<double> { using type = double4; };
template <> struct Quad<uint16_t> { using type = ushort4; };

template <typename T>
__global__ void __launch_bounds__(256) segmented_transpose_warp_kernel(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int dim,
                                                                       const int4* __restrict__ info, int num_blocks) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Q = typename Quad<T>::type;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  T* tile = reinterpret_cast<T*>(smem_raw) + (size_t)warp * dim;
  for (int64_t r = (int64_t)blockIdx.x * warps + warp; r < rows; r += (int64_t)gridDim.x * warps) {
    const Q* xr = reinterpret_cast<const Q*>(x + r * dim);
#pragma unroll 4
    for (int i = lane; i < dim / 4; i += 32) reinterpret_cast<Q*>(tile)[i] = xr[i];
    __syncwarp();
    for (int b = 0; b < num_blocks; ++b) {
      const int4 d = __ldg(info + b);
      const int off = d.x, u = d.y, v = d.z;
      if ((off | (u * v)) & 3) {                                             // an odd block: element by element
        for (int e = lane; e < u * v; e += 32) {
          const int j = e / u, i = e - j * u;
          y[r * dim + off + e] = tile[off + i * v + j];
        }
        continue;
      }
      Q* yr = reinterpret_cast<Q*>(y + r * dim + off);
      for (int e = lane; e < u * v / 4; e += 32) {
        int j = (int)((unsigned)(4 * e) / (unsigned)u), i = 4 * e - j * u;   // destination [j, i] of a [v, u] tile
        T a[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[q] = tile[off + i * v + j];
          if (++i == u) { i = 0; ++j; }
        }
        Q o;
        o.x = a[0]; o.y = a[1]; o.z = a[2]; o.w = a[3];
        yr[e] = o;
      }
    }
    __syncwarp();
  }
}

template <typename T>
__global__ void __launch_bounds__(256) segmented_transpose_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                                  int64_t rows, int dim,
                                                                  const int4* __restrict__ info, int num_blocks) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const T* xr = x + r * dim;
    T* yr = y + r * dim;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) tile[i] = xr[i];
    __syncthreads();
    for (int b = 0; b < num_blocks; ++b) {
      const int4 d = __ldg(info + b);
      const int off = d.x, u = d.y, v = d.z;
      for (int e = threadIdx.x; e < u * v; e += blockDim.x) {
        const int j = e / u, i = e - j * u;  // destination [j, i] of a [v, u] tile
        yr[off + e] = tile[off + i * v + j];
      }
    }
    __syncthreads();
  }
}

template <typename T>
int launch(const void* x, void* y, int64_t rows, int64_t dim, const int32_t* info, int nb, cudaStream_t st) {
  const size_t smem = (size_t)dim * sizeof(T);
  if (smem > 200 * 1024) return cueq::fail("segmented_transpose: row of %lld elements does not fit shared memory", (long long)dim);
  // Rows in whole groups of four elements, at the alignment of a group.  float64 only up to 6 KB: beyond, the gather of four
  // doubles per thread conflicts in shared memory and few warps hold their rows; 16 M elements in rows of 576 / 1,152 / 2,304:
  // 77 / 64 / 61 us by the kernel with a block per row, 63 / 73 / 75 us by this one (float32 72 / 58 / 52 and 28 / 32 / 37 us).
  if (dim % 4 == 0 && (((uintptr_t)x | (uintptr_t)y) % (4 * sizeof(T))) == 0 && smem <= (sizeof(T) == 8 ? 6 : 24) * 1024) {
    int warps = 8;
    while (warps > 1 && warps * smem > 48 * 1024) warps /= 2;
    const unsigned grid = (unsigned)std::min<int64_t>((rows + warps - 1) / warps, 148 * 32);
    segmented_transpose_warp_kernel<T><<<grid, warps * 32, warps * smem, st>>>(reinterpret_cast<const T*>(x), reinterpret_cast<T*>(y), rows, (int)dim,
                                                                              reinterpret_cast<const int4*>(info), nb);
    CUEQ_CUDA_OK(cudaGetLastError());
    return 0;
  }
  if (smem > 48 * 1024) CUEQ_CUDA_OK(cudaFuncSetAttribute(segmented_transpose_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const unsigned grid = (unsigned)std::min<int64_t>(rows, 148 * 8);
  segmented_transpose_kernel<T><<<grid, 256, smem, st>>>(reinterpret_cast<const T*>(x), reinterpret_cast<T*>(y), rows, (int)dim,
                                                        reinterpret_cast<const int4*>(info), nb);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace

extern "C" int cueq_b200_segmented_transpose(const void* x, void* y, int64_t rows, int64_t dim,
                                             const int32_t* info_dev, int32_t num_blocks, int32_t dtype,
                                             void* stream) {
  if (rows == 0 || dim == 0) return 0;
  if (!x || !y || !info_dev) return cueq::fail("segmented_transpose: null argument");
  if (x == y) return cueq::fail("segmented_transpose: x and y must not alias");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (dtype) {
    case CUEQ_F32: return launch<float>(x, y, rows, dim, info_dev, num_blocks, st);
    case CUEQ_F64: return launch<double>(x, y, rows, dim, info_dev, num_blocks, st);
    case CUEQ_BF16:
    case CUEQ_F16: return launch<uint16_t>(x, y, rows, dim, info_dev, num_blocks, st);
    default: return cueq::fail("segmented_transpose: invalid dtype %d", dtype);
  }
}
