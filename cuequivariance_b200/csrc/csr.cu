// Edges by receiver: rowptr[r] = first position, in the order of the receivers, whose receiver is >= r.
//
// csr_rowptr takes an ascending index (its rows are searched, one thread per row) and reports one that is not: the caller
// sorts it and asks again.  csr_small sorts as well, in one thread block, up to kSmall edges: nothing to read back, no
// further launches.  Both are bound by launch latency.  On new edge lists they replace six elementwise and search kernels
// (comparison, reduction, arange, search, two conversions), a read of the result and, for unsorted lists, a library sort in
// front of the first product.
#include "common.cuh"

namespace {

constexpr int kSmall = 4096, kSmallRows = 65536;

template <typename I>
__global__ void __launch_bounds__(256) csr_rowptr_kernel(const I* __restrict__ index, int n, int rows, int* __restrict__ rowptr, int* __restrict__ descends) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 < n && __ldg(index + i + 1) < __ldg(index + i)) *descends = 1;
  if (i > rows) return;
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((int64_t)__ldg(index + mid) < i) lo = mid + 1; else hi = mid;
  }
  rowptr[i] = lo;
}

// (receiver, position) pairs, sorted by a bitonic network in shared memory: the positions make the keys distinct, so the
// order is that of a stable sort.  `size`: n rounded up to a power of two.
template <typename I>
__global__ void __launch_bounds__(1024) csr_small_kernel(const I* __restrict__ index, int n, int size, int rows, int* __restrict__ order, int* __restrict__ rowptr) {
  __shared__ unsigned long long key[kSmall];
  for (int e = threadIdx.x; e < size; e += 1024) key[e] = e < n ? ((unsigned long long)(unsigned)__ldg(index + e) << 32) | (unsigned)e : ~0ull;
  for (int k = 2; k <= size; k <<= 1)
    for (int j = k >> 1; j; j >>= 1) {
      __syncthreads();
      for (int e = threadIdx.x; e < size; e += 1024) {
        const int f = e ^ j;
        if (f > e) {
          const unsigned long long a = key[e], b = key[f];
          if ((a > b) == !(e & k)) { key[e] = b; key[f] = a; }
        }
      }
    }
  __syncthreads();
  for (int e = threadIdx.x; e < n; e += 1024) order[e] = (int)(key[e] & 0xffffffffu);
  for (int r = threadIdx.x; r <= rows; r += 1024) {
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((unsigned)(key[mid] >> 32) < (unsigned)r) lo = mid + 1; else hi = mid;
    }
    rowptr[r] = lo;
  }
}

}  // namespace

extern "C" int cueq_b200_csr_rowptr(const void* index, int index_is_64, int64_t n, int64_t rows, int32_t* rowptr, int32_t* descends, void* stream) {
  if ((!index && n) || !rowptr || !descends) return cueq::fail("csr_rowptr: null argument");
  if (n < 0 || n > 2147483646LL || rows < 0 || rows > 2147483646LL) return cueq::fail("csr_rowptr: invalid size");
  const int64_t threads = n > rows + 1 ? n : rows + 1;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (index_is_64) csr_rowptr_kernel<long long><<<grid, 256, 0, st>>>(reinterpret_cast<const long long*>(index), (int)n, (int)rows, rowptr, descends);
  else csr_rowptr_kernel<int><<<grid, 256, 0, st>>>(reinterpret_cast<const int*>(index), (int)n, (int)rows, rowptr, descends);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int cueq_b200_csr_small(const void* index, int index_is_64, int64_t n, int64_t rows, int32_t* order, int32_t* rowptr, void* stream) {
  if ((n && (!index || !order)) || !rowptr) return cueq::fail("csr_small: null argument");
  if (n < 0 || n > kSmall || rows < 0 || rows > kSmallRows) return cueq::fail("csr_small: at most %d edges and %d rows", kSmall, kSmallRows);
  int size = 1;
  while (size < n) size <<= 1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (index_is_64) csr_small_kernel<long long><<<1, 1024, 0, st>>>(reinterpret_cast<const long long*>(index), (int)n, size, (int)rows, order, rowptr);
  else csr_small_kernel<int><<<1, 1024, 0, st>>>(reinterpret_cast<const int*>(index), (int)n, size, (int)rows, order, rowptr);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}
