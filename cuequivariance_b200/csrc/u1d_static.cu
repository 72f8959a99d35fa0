// Straight-line ("static") kernels for polynomials known at build time.
//
// Same contract as the generic uniform-1d executor (u1d_generic.cu; reference call site
// cuequivariance_torch/primitives/segmented_polynomial_uniform_1d.py:294-316), float32 only:
// one thread evaluates one (row, channel) pair, but instead of walking a path table it runs
// the code generated for that polynomial (generated/u1d_static.cuh): every operand segment is
// loaded once into a register, every path is a few multiplies.  Used for the symmetric
// contraction, whose ~2,000 paths make the table-driven kernel instruction- and L1-bound.
#include <cstring>

#include "common.cuh"
#include "generated/u1d_static.cuh"

namespace {

constexpr int kMaxBuf = 8;

struct StaticBuf {
  void* ptr;
  const void* index;
  int32_t mode;
  int32_t index_is_64;
  int32_t row_size;  // elements per row
  int32_t vec;       // 1: segments have a channel axis, 0: scalar segments
  int32_t mul_ir;    // 1: blocks of 1, 3, 5, ... segments, [channel][component] each
};

struct StaticParams {
  StaticBuf buf[kMaxBuf];
  int64_t batch;
  int32_t extent;
};

// Segment s of a row of irreps 0, 1, 2, ... (one block each) lies in block l = floor(sqrt(s)), whose first segment
// is l * l.  The generated code passes s as a literal, so this folds away.
constexpr int kMaxL = 3;
__host__ __device__ constexpr int block_of(int s) { return s < 1 ? 0 : s < 4 ? 1 : s < 9 ? 2 : 3; }

// Channel-major buffers are read and written in place.  A thread's components of a block are contiguous, so a warp's
// reads cover whole lines (the lines stay in L1 between the block's components); a block of an output goes through
// shared memory, so that every store of a warp is 128 contiguous bytes: stored component by component, each 32-byte
// sector would be written 2l+1 times.  A separate transposition of the rows in and out cost as much as the smaller
// kernels themselves: a read and a write of every feature, output and both their gradients.  No pipe
// bounds the kernels: 8 to 20 warps per SM (registers) wait for loads that a body makes once and nothing else overlaps, and
// use 47-64 % of the issue slots, 2.1-2.5 times the time of their instructions.  16,384 atoms x 128 channels of
// 0e+1o+2e+3o -> 0e+1o, degree 3: forward 93 us, weight gradient 109 us, feature gradient 267 us; the step 470 us, with
// transposed copies and without the factored sums (gen_u1d_static.py) 820 us.
template <class K>
__global__ void __launch_bounds__(128) u1d_static_kernel(const __grid_constant__ StaticParams P) {
  __shared__ float staging[4][32 * (2 * kMaxL + 1)];
  float* const stage = staging[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= P.batch * P.extent) return;
  const int64_t z = gid / P.extent;
  const int u = (int)(gid - z * P.extent);
  const int X = P.extent;
  const float* in_base[K::NUM_INPUTS];
  int in_stride[K::NUM_INPUTS];
#pragma unroll
  for (int b = 0; b < K::NUM_INPUTS; ++b) {
    const StaticBuf& s = P.buf[b];
    const int64_t row = s.mode == CUEQ_SHARED ? 0 : s.mode == CUEQ_BATCHED ? z : cueq::load_index(s.index, s.index_is_64, z);
    in_base[b] = reinterpret_cast<const float*>(s.ptr) + row * s.row_size + (s.vec ? u : 0);
    in_stride[b] = s.vec ? X : 1;
  }
  float* out_base[K::NUM_OUTPUTS];
  int out_stride[K::NUM_OUTPUTS];
  bool out_atomic[K::NUM_OUTPUTS];
#pragma unroll
  for (int j = 0; j < K::NUM_OUTPUTS; ++j) {
    const StaticBuf& s = P.buf[K::NUM_INPUTS + j];
    const int64_t row = s.mode == CUEQ_SHARED ? 0 : s.mode == CUEQ_BATCHED ? z : cueq::load_index(s.index, s.index_is_64, z);
    out_base[j] = reinterpret_cast<float*>(s.ptr) + row * s.row_size + (s.vec ? u : 0);
    out_stride[j] = s.vec ? X : 1;
    out_atomic[j] = s.mode != CUEQ_BATCHED || (!s.vec && X > 1);
  }
  auto in = [&](int b, int s) -> float {
    const int l = block_of(s), first = l * l;
    // in_base already points at channel u of segment 0
    if (s < (kMaxL + 1) * (kMaxL + 1) && P.buf[b].mul_ir) return __ldg(in_base[b] + first * X + u * (2 * l) + (s - first));
    return __ldg(in_base[b] + s * in_stride[b]);
  };
  float block[2 * kMaxL + 1];   // components of the output block being collected (constant indices only)
  auto out = [&](int j, int s, float v) {
    const int l = block_of(s), first = l * l, d = 2 * l + 1;
    if (s < (kMaxL + 1) * (kMaxL + 1) && P.buf[K::NUM_INPUTS + j].mul_ir) {
      // X is a multiple of 32: the lanes of a warp hold 32 consecutive channels of one row, all or none of them here
      block[s - first] = v;
      if (s - first == d - 1) {
#pragma unroll
        for (int i = 0; i < d; ++i) stage[lane * d + i] = block[i];
        __syncwarp();
        float* p = out_base[j] + first * X + (u - lane) * (2 * l);   // the warp's run of the block, at this lane (out_base is at u)
#pragma unroll
        for (int t = 0; t < d; ++t) p[t * 32] = stage[t * 32 + lane];
        __syncwarp();
      }
      return;
    }
    float* p = out_base[j] + s * out_stride[j];
    if (out_atomic[j]) atomicAdd(p, v); else *p = v;
  };
  K::run(in, out);
}

struct StaticEntry {
  const char* digest;
  const char* name;
  int num_inputs, num_outputs;
  void (*launch)(const StaticParams&, unsigned, cudaStream_t);
};

template <class K>
void launch_t(const StaticParams& P, unsigned grid, cudaStream_t st) { u1d_static_kernel<K><<<grid, 128, 0, st>>>(P); }

#define U1D_ENTRY(K) {K::digest(), K::name(), K::NUM_INPUTS, K::NUM_OUTPUTS, &launch_t<K>},
const StaticEntry kStatic[] = {U1D_STATIC_FOR_EACH(U1D_ENTRY)};
constexpr int kNumStatic = sizeof(kStatic) / sizeof(kStatic[0]);

}  // namespace

extern "C" int cueq_b200_u1d_static_find(const char* digest) {
  if (!digest) return -1;
  for (int i = 0; i < kNumStatic; ++i)
    if (std::strcmp(kStatic[i].digest, digest) == 0) return i;
  return -1;
}

extern "C" const char* cueq_b200_u1d_static_name(int id) { return (id >= 0 && id < kNumStatic) ? kStatic[id].name : nullptr; }

extern "C" int cueq_b200_u1d_static_launch(int id, int64_t batch, int32_t extent, const cueq_buffer* buffers,
                                           const int32_t* buffer_dim, const int32_t* buffer_num_segments, int32_t num_buffers,
                                           void* stream) {
  const int32_t layouts[kMaxBuf] = {};
  return cueq_b200_u1d_static_launch_layouts(id, batch, extent, buffers, buffer_dim, buffer_num_segments, num_buffers, layouts, stream);
}

extern "C" int cueq_b200_u1d_static_launch_layouts(int id, int64_t batch, int32_t extent, const cueq_buffer* buffers,
                                                   const int32_t* buffer_dim, const int32_t* buffer_num_segments, int32_t num_buffers,
                                                   const int32_t* layouts, void* stream) {
  if (id < 0 || id >= kNumStatic) return cueq::fail("u1d_static: kernel id %d out of range", id);
  const StaticEntry& e = kStatic[id];
  if (num_buffers != e.num_inputs + e.num_outputs) return cueq::fail("u1d_static: %s takes %d buffers, got %d", e.name, e.num_inputs + e.num_outputs, num_buffers);
  if (num_buffers > kMaxBuf) return cueq::fail("u1d_static: too many buffers");
  if (!buffers || !buffer_dim || !buffer_num_segments || !layouts) return cueq::fail("u1d_static: null argument");
  if (batch < 0 || extent < 1) return cueq::fail("u1d_static: invalid batch or extent");
  StaticParams P;
  std::memset(&P, 0, sizeof(P));
  for (int b = 0; b < num_buffers; ++b) {
    const cueq_buffer& s = buffers[b];
    if (s.dtype != CUEQ_F32) return cueq::fail("u1d_static: buffer %d is not float32", b);
    if (s.mode != CUEQ_SHARED && s.mode != CUEQ_BATCHED && s.mode != CUEQ_INDEXED) return cueq::fail("u1d_static: buffer %d has invalid mode", b);
    if (s.mode == CUEQ_BATCHED && s.rows != batch) return cueq::fail("u1d_static: batched buffer %d has %lld rows, batch is %lld", b, (long long)s.rows, (long long)batch);
    if (s.mode == CUEQ_SHARED && s.rows != 1) return cueq::fail("u1d_static: shared buffer %d must have one row", b);
    if (s.mode == CUEQ_INDEXED && !s.index && batch > 0) return cueq::fail("u1d_static: indexed buffer %d has no index", b);
    P.buf[b].ptr = s.ptr; P.buf[b].index = s.index; P.buf[b].mode = s.mode; P.buf[b].index_is_64 = s.index_is_64;
    P.buf[b].vec = buffer_dim[b];
    if (layouts[b] != 0 && layouts[b] != 1) return cueq::fail("u1d_static: buffer %d has invalid layout", b);
    P.buf[b].mul_ir = layouts[b];
    if (layouts[b]) {
      const int n = buffer_num_segments[b];
      if (!buffer_dim[b] || (n != 1 && n != 4 && n != 9 && n != 16))
        return cueq::fail("u1d_static: buffer %d cannot be channel-major (%d segments, channel axis %d)", b, n, buffer_dim[b]);
      if (b >= e.num_inputs && (s.mode != CUEQ_BATCHED || extent % 32))
        return cueq::fail("u1d_static: a channel-major output has to be batched with an extent that is a multiple of 32");
    }
    P.buf[b].row_size = buffer_num_segments[b] * (buffer_dim[b] ? extent : 1);
  }
  if (batch == 0) return 0;
  P.batch = batch;
  P.extent = extent;
  const int64_t grid = (batch * extent + 127) / 128;
  if (grid > 2147483647LL) return cueq::fail("u1d_static: batch too large for one launch");
  e.launch(P, (unsigned)grid, reinterpret_cast<cudaStream_t>(stream));
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}
