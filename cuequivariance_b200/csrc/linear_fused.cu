// Equivariant linear layer in float32 accuracy on the tensor cores, all irreps, components and weight classes in one
// launch (counterpart of the reference's cuequivariance_torch/operations/linear.py:30-191 and, with classes, of
// primitives/segmented_polynomial_indexed_linear.py:116-156,247-339):
//
//   linear_map  out[z, v, i] = c * sum_u W[class(z)][u, v] x[z, u, i]       forward, and with W transposed the input gradient
//   linear_gw   gW[class][u, v] += c * sum_{z in class, i} x[z, u, i] g[z, v, i]      partial sums, added in a fixed order
//
// What bounds them: the rows are read once and written once, 2 * 268 MB each for 32,768 nodes of 128x(0e+1o+2e+3o);
// 82 us at 6.5 TB/s against 46 us of three-pass TF32.  The layer used to be one GEMM launch per irrep and component
// (48 of them, the row reductions on 32 thread blocks), with layout transpositions around them and the weights split by
// elementwise kernels: 3.25 ms for forward and both gradients.  Now 0.62 ms: linear_map 195 us (2.75 TB/s), linear_gw 212 us.
// What is left is the latency between load, split and MMA: tensor pipe 23 % and HBM 45 % busy.
//
// The components of an irrep share its weight block, so rows (z, i) are folded into the M axis of the MMA (linear_map)
// or its K axis (linear_gw).  Eight warps fetch rows straight from the caller's layout: a thread owns 4 channels x d
// components, contiguous in a mul_ir row, so the transposition happens in registers on the way into the K-major,
// 128-byte-swizzled operand tiles; they split x = hi + lo into TF32 halves at the same time (see gemm_f32x3.cu).
// Thread blocks are persistent over a run of tiles: the split weight block stays in shared memory (128 KB at 128 x 128)
// until the run enters the next irrep or class.
//
// Accumulators: the tensor core's float32 sums are not rounded to nearest, so the chains are kept short.  linear_map:
// K blocks go in pairs to an accumulator of their own, small terms (hi*lo, lo*hi) of both blocks before the large ones,
// i.e. 8 additions at full magnitude per chain (the GEMMs before: 12 per accumulator).  linear_gw: hi*hi dealt to three
// accumulators, small terms to a fourth; at most kMaxRunGw blocks per run (about 160 additions, before: 192).
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

using namespace cueq_tc;

constexpr int kMaxPaths = CUEQ_LINEAR_MAX_PATHS, kMaxClasses = CUEQ_LINEAR_MAX_CLASSES;
constexpr int kBlk = 128 * 128;              // one operand block: 128 rows x 32 float32, 16 KiB
constexpr int kMaxRunGw = 128;               // K blocks per run of linear_gw

struct LPath { int x_off, o_off, w_off, K, N, d, w_sn, w_sk; float c; };

struct LParams {
  const float* x;       // linear_map: input rows; linear_gw: x rows (M side)
  const float* w;       // linear_map: weights
  float* out;           // linear_map: output rows; linear_gw: weight gradient
  float* parts;         // linear_gw: partial sums, one slot of `slot` floats per run
  int64_t slot;
  const float* g;       // linear_gw: cotangent rows (N side)
  int64_t ldx, ldo, w_class_stride;
  int x_mul_ir, o_mul_ir, num_paths, num_classes;
  int total;            // tiles (linear_map) or K blocks (linear_gw) over all paths and classes
  int* status;
  LPath path[kMaxPaths];
  int bounds[kMaxClasses + 1];
};

__host__ __device__ constexpr int rows_per_tile(int d) { return 128 / d; }     // nodes per tile of linear_map
__host__ __device__ constexpr int rows_per_block(int d) { return 32 / d; }     // nodes per K block of linear_gw

// The runs of consecutive items (tiles / K blocks) of one path and class that fall into [first, last): calls
// f(path, class, z of the run's first item, z end of the class, items).  Every role of a thread block walks the same runs.
template <class PerItem, class F>
__device__ __forceinline__ void for_each_run(const LParams& p, int first, int last, PerItem per_item, F f) {
  int start = 0;
  for (int q = 0; q < p.num_paths && start < last; ++q) {
    const int n = per_item(p.path[q].d);
    for (int c = 0; c < p.num_classes && start < last; ++c) {
      const int items = (p.bounds[c + 1] - p.bounds[c] + n - 1) / n;
      const int a = max(first, start), b = min(last, start + items);
      if (a < b) f(p.path[q], c, p.bounds[c] + (a - start) * n, p.bounds[c + 1], b - a);
      start += items;
    }
  }
}

__device__ __forceinline__ void umma_tf32(unsigned tmem_c, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
               ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// the four instructions of a 32-wide K block
__device__ __forceinline__ void umma_block(unsigned tmem_c, const void* a, const void* b, unsigned idesc, unsigned accumulate) {
  const unsigned long long da = smem_desc(a), db = smem_desc(b);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_c, da + 2ull * kk, db + 2ull * kk, idesc, kk ? 1u : accumulate);
}
__device__ __forceinline__ float tf32_hi(float v) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}
// 16 bytes (4 consecutive k) of one operand row, split, into the hi tile and its lo twin
__device__ __forceinline__ void store_split(unsigned char* hi_tile, unsigned char* lo_tile, int row, int chunk, const float (&v)[4]) {
  float h[4], l[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    h[c] = tf32_hi(v[c]);
    l[c] = tf32_hi(v[c] - h[c]);
  }
  const int off = row * 128 + ((chunk ^ (row & 7)) << 4);
  *reinterpret_cast<float4*>(hi_tile + off) = make_float4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4*>(lo_tile + off) = make_float4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&f)[32]) {
  unsigned v[32];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                 "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                 "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < 32; ++c) f[c] = __uint_as_float(v[c]);
}
__device__ __forceinline__ void tmem_ld16(unsigned t, float (&y)[16]) {
  unsigned v[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(t));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < 16; ++c) y[c] = __uint_as_float(v[c]);
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(s32(b)) : "memory");
}
// what a warp wrote to shared memory becomes visible to the tensor core, then one lane arrives
__device__ __forceinline__ void publish(unsigned long long* b, int lane) {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncwarp();
  if (lane == 0) bar_arrive(b);
}
__device__ __forceinline__ unsigned idesc_tf32(int n) {   // D = f32, A = B = tf32, both K-major, M = 128
  return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}
__device__ __forceinline__ unsigned tmem_alloc_all(unsigned* slot, int warp, int owner) {
  if (warp == owner) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s32(slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return *slot;
}
__device__ __forceinline__ void tmem_free_all(unsigned base, int warp, int owner) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == owner) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(512u) : "memory");
  }
}

// ---- linear_map -----------------------------------------------------------------------------------------------
// Warps 0-3 epilogue (TMEM lane quadrant = warp), 4 MMA issue and TMEM owner, 5-12 load and split.
constexpr int kMapLoaders = 256;
constexpr int kMapThreads = 160 + kMapLoaders;
constexpr int kMapB = 0;                                  // split weights: hi [4][16 KiB], lo [4][16 KiB]
constexpr int kMapA = 8 * kBlk;                           // 2 stages x (hi + lo)
constexpr int kMapStage = kMapA + 4 * kBlk;               // output staging: 128 rows x 32 columns, padded to 36 at most
constexpr int kMapBars = kMapStage + 128 * 36 * 4;
constexpr size_t kMapSmem = kMapBars + 128 + 1024;

struct MapShared {
  unsigned char* base;
  unsigned long long *full, *empty, *accfull, *accempty, *bready, *bdone;
};

template <int D, bool MUL_IR>
__device__ __forceinline__ void map_load(const LParams& p, const LPath& q, int z0, int zend, int tiles, const MapShared& sh, int tid,
                                         unsigned& it, bool& dead) {
  constexpr int NZ = rows_per_tile(D);
  constexpr int J = (NZ * 8 + kMapLoaders - 1) / kMapLoaders;   // (node, 4-channel chunk) units per thread
  const int lane = tid & 31, nkb = q.K / 32;
  const int total = tiles * nkb;
  float4 next[J][D];
  auto fetch = [&](int b) {
    const int t = b / nkb, kb = b - t * nkb;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int unit = tid + j * kMapLoaders, z = unit >> 3, ch = kb * 32 + (unit & 7) * 4;
      const int row = z0 + t * NZ + z;
      const bool in = z < NZ && row < zend;
      const float* src = p.x + (int64_t)row * p.ldx + q.x_off + (MUL_IR ? ch * D : ch);
#pragma unroll
      for (int i = 0; i < D; ++i)
        next[j][i] = in ? __ldg(reinterpret_cast<const float4*>(src + (MUL_IR ? 4 * i : i * q.K))) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  // rows of the tiles after the next on their way into L2: at the latency of HBM, the one block a thread has in registers
  // is not enough (239 us without, 195 us with; two loader groups of seven warps instead: 353 us, their registers spill)
  auto prefetch = [&](int t) {
    const int row = z0 + t * NZ + tid;
    if (tid < NZ && row < zend)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p.x + (int64_t)row * p.ldx + q.x_off), "r"(q.K * D * 4) : "memory");
  };
  prefetch(1);
  prefetch(2);
  fetch(0);
  for (int b = 0; b < total; ++b, ++it) {
    if (b % nkb == 0) prefetch(b / nkb + 3);
    float f[J][4 * D];
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
      for (int i = 0; i < D; ++i) { f[j][4 * i] = next[j][i].x; f[j][4 * i + 1] = next[j][i].y; f[j][4 * i + 2] = next[j][i].z; f[j][4 * i + 3] = next[j][i].w; }
    if (b + 1 < total) fetch(b + 1);
    const unsigned s = it & 1;
    if (!dead) dead = !bar_wait(sh.empty + s, ((it >> 1) & 1) ^ 1, p.status);
    unsigned char* hi = sh.base + kMapA + s * 2 * kBlk;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int unit = tid + j * kMapLoaders, z = unit >> 3, chunk = unit & 7;
      if (z < NZ && !dead) {
#pragma unroll
        for (int i = 0; i < D; ++i) {
          float v[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c] = MUL_IR ? f[j][c * D + i] : f[j][4 * i + c];
          store_split(hi, hi + kBlk, z * D + i, chunk, v);
        }
      }
    }
    publish(sh.full + s, lane);
  }
}

// Accumulator rows (z, i) -> global rows.  A pass moves 32 output channels through shared memory, written lane-per-row and
// read back as 16-byte pieces of the global rows.  mul_ir: a node's components and channels interleave at a pitch of
// 32 d + 4 floats (2-way bank conflicts for d > 1); ir_mul: 128-byte rows, 16-byte pieces swizzled (none).  Moved
// element by element, one dependent load and store after the other, the epilogue was four times the MMAs' time.
template <int D, bool MUL_IR>
__device__ __forceinline__ void map_store(const LParams& p, const LPath& q, int z0, int zend, int tiles, const MapShared& sh, int warp,
                                          int lane, unsigned tmem_base, unsigned& tile, bool& dead) {
  constexpr int NZ = rows_per_tile(D), PZ = 32 * D + 4;
  constexpr int NV = 8;                                              // 16-byte pieces per thread and pass: 128 rows x 8 / 128
  float* stage = reinterpret_cast<float*>(sh.base + kMapStage);
  const int r = warp * 32 + lane, z = r / D, i = r - z * D;
  for (int t = 0; t < tiles; ++t, ++tile) {
    const unsigned set = tile & 1;
    if (!dead) dead = !bar_wait(sh.accfull + set, (tile >> 1) & 1, p.status);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const bool good = !dead && status_clean(p.status);
    const int zt = z0 + t * NZ, nz = good ? min(NZ, zend - zt) : 0;
    float* base = p.out + (int64_t)zt * p.ldo + q.o_off;
#pragma unroll 1
    for (int part = 0; part < q.N / 32; ++part) {
      float v[32];
      const unsigned ta = tmem_base + ((unsigned)(warp * 32) << 16) + set * 256 + part * 32;
      tmem_ld32(ta, v);
      if (q.K > 64) {
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float v2[16];
          tmem_ld16(ta + 128 + h, v2);
#pragma unroll
          for (int c = 0; c < 16; ++c) v[h + c] += v2[c];
        }
      }
      if (part == q.N / 32 - 1) {                                    // everything of this accumulator set is in registers
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(sh.accempty + set);
      }
      asm volatile("bar.sync 1, 128;\n" ::: "memory");               // the previous pass has left the staging tile
      if (MUL_IR) {
        if (r < NZ * D) {
#pragma unroll
          for (int c = 0; c < 32; ++c) stage[z * PZ + c * D + i] = v[c];
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; c += 4)
          *reinterpret_cast<float4*>(stage + r * 32 + (((c >> 2) ^ (r & 7)) << 2)) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
      }
      asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
      for (int k0 = 0; k0 < NV; k0 += 4) {
        float4 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int e = r + (k0 + k) * 128;
          if (MUL_IR) o[k] = *reinterpret_cast<const float4*>(stage + min(e / (8 * D), NZ - 1) * PZ + e % (8 * D) * 4);
          else o[k] = *reinterpret_cast<const float4*>(stage + (e >> 3) * 32 + (((e & 7) ^ ((e >> 3) & 7)) << 2));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int e = r + (k0 + k) * 128;
          if (MUL_IR) {
            const int zz = e / (8 * D), rem = e % (8 * D) * 4;
            if (zz < nz) *reinterpret_cast<float4*>(base + (int64_t)zz * p.ldo + part * 32 * D + rem) = o[k];
          } else {
            const int row = e >> 3, zz = row / D, ii = row - zz * D;
            if (zz < nz) *reinterpret_cast<float4*>(base + (int64_t)zz * p.ldo + ii * q.N + part * 32 + (e & 7) * 4) = o[k];
          }
        }
      }
    }
  }
}

#define LINEAR_DISPATCH(FN, D, MUL, ...)                                                             \
  switch (D) {                                                                                       \
    case 1: FN<1, true>(__VA_ARGS__); break;                                                         \
    case 3: if (MUL) FN<3, true>(__VA_ARGS__); else FN<3, false>(__VA_ARGS__); break;                \
    case 5: if (MUL) FN<5, true>(__VA_ARGS__); else FN<5, false>(__VA_ARGS__); break;                \
    default: if (MUL) FN<7, true>(__VA_ARGS__); else FN<7, false>(__VA_ARGS__); break;               \
  }

__global__ void __launch_bounds__(kMapThreads, 1) linear_map_kernel(const __grid_constant__ LParams p) {
  extern __shared__ unsigned char smem_raw[];
  MapShared sh;
  sh.base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  sh.full = reinterpret_cast<unsigned long long*>(sh.base + kMapBars);
  sh.empty = sh.full + 2; sh.accfull = sh.empty + 2; sh.accempty = sh.accfull + 2; sh.bready = sh.accempty + 2; sh.bdone = sh.bready + 1;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(sh.bdone + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) { bar_init(sh.full + s, kMapLoaders / 32); bar_init(sh.empty + s, 1); bar_init(sh.accfull + s, 1); bar_init(sh.accempty + s, 4); }
    bar_init(sh.bready, kMapLoaders / 32);
    bar_init(sh.bdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const unsigned tmem_base = tmem_alloc_all(tmem_slot, warp, 4);
  const int first = (int)((int64_t)p.total * blockIdx.x / gridDim.x), last = (int)((int64_t)p.total * (blockIdx.x + 1) / gridDim.x);

  if (warp < 4) {
    unsigned tile = 0;
    bool dead = false;
    for_each_run(p, first, last, rows_per_tile, [&](const LPath& q, int, int z0, int zend, int tiles) {
      LINEAR_DISPATCH(map_store, q.d, p.o_mul_ir, p, q, z0, zend, tiles, sh, warp, lane, tmem_base, tile, dead)
    });
  } else if (warp == 4) {
    if (lane == 0) {
      unsigned it = 0, tile = 0, run = 0;
      bool ok = true;
      for_each_run(p, first, last, rows_per_tile, [&](const LPath& q, int, int, int, int tiles) {
        const int nkb = q.K / 32;
        const unsigned idesc = idesc_tf32(q.N);
        ok = ok && bar_wait(sh.bready, run & 1, p.status);
        ++run;
        for (int t = 0; t < tiles && ok; ++t, ++tile) {
          const unsigned set = tile & 1;
          ok = bar_wait(sh.accempty + set, ((tile >> 1) & 1) ^ 1, p.status);
          for (int kb = 0; kb < nkb && ok; kb += 2) {
            const unsigned acc = tmem_base + set * 256 + (kb >> 1) * 128;
            const int n = min(2, nkb - kb);
            for (int h = 0; h < n && ok; ++h) {                       // small terms of both blocks
              const unsigned s = (it + h) & 1;
              ok = bar_wait(sh.full + s, ((it + h) >> 1) & 1, p.status);
              if (!ok) break;
              asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
              const unsigned char* a = sh.base + kMapA + s * 2 * kBlk;
              const unsigned char* b = sh.base + kMapB + (kb + h) * kBlk;
              umma_block(acc, a + kBlk, b, idesc, h ? 1u : 0u);
              umma_block(acc, a, b + 4 * kBlk, idesc, 1u);
            }
            for (int h = 0; h < n && ok; ++h) {
              const unsigned s = (it + h) & 1;
              umma_block(acc, sh.base + kMapA + s * 2 * kBlk, sh.base + kMapB + (kb + h) * kBlk, idesc, 1u);
              umma_commit(sh.empty + s);
            }
            it += n;
          }
          if (ok) umma_commit(sh.accfull + set);
        }
        if (ok) umma_commit(sh.bdone);
      });
    }
  } else {
    const int tid = threadIdx.x - 160;
    unsigned it = 0, run = 0;
    bool dead = false;
    for_each_run(p, first, last, rows_per_tile, [&](const LPath& q, int cls, int z0, int zend, int tiles) {
      if (run && !dead) dead = !bar_wait(sh.bdone, (run - 1) & 1, p.status);
      ++run;
      // weight block, scaled by the path coefficient and split: row n, 4 consecutive k per 16-byte chunk
      const float* w = p.w + cls * p.w_class_stride + q.w_off;
#pragma unroll 1
      for (int e = tid; e < q.N * (q.K / 4); e += kMapLoaders) {
        const int n = e % q.N, k = (e / q.N) * 4;
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = __ldg(w + (int64_t)n * q.w_sn + (int64_t)(k + c) * q.w_sk) * q.c;
        unsigned char* hi = sh.base + kMapB + (k >> 5) * kBlk;
        if (!dead) store_split(hi, hi + 4 * kBlk, n, (k >> 2) & 7, v);
      }
      publish(sh.bready, lane);
      LINEAR_DISPATCH(map_load, q.d, p.x_mul_ir, p, q, z0, zend, tiles, sh, tid, it, dead)
    });
  }
  tmem_free_all(tmem_base, warp, 4);
}

// ---- linear_gw ------------------------------------------------------------------------------------------------
// Warps 0-3 epilogue, 4 MMA issue and TMEM owner, 5-20 transpose and split, 21 and 22 bulk copies of raw rows (x, g; one per
// node).  A K block is the (node, component) pairs of 32 / d whole nodes, padded with zeros to 32.  Eight transposing warps
// and one copying warp took 2.5 times the MMAs' time per block (5 times for scalars, 64 copies of 512 bytes); rows copied by
// cp.async instead: 460 us against 315 us.
constexpr int kGwWorkers = 512;
constexpr int kGwThreads = 224 + kGwWorkers;
constexpr int kGwOps = 0;                                  // 2 stages x (x hi, x lo, g hi, g lo)
constexpr int kGwRawStages = 3;
constexpr int kGwRaw = 2 * 4 * kBlk;                       // raw rows: x part [16 KiB], g part [16 KiB] per stage
constexpr int kGwBars = kGwRaw + kGwRawStages * 2 * kBlk;
constexpr size_t kGwSmem = kGwBars + 128 + 1024;

// raw rows of the block's nodes -> K-major split tile; thread = (channel, quarter of the k range).  Reads are free of bank
// conflicts: neighbouring channels are d (odd) or 1 floats apart.
template <int D, bool MUL_IR, int QUARTER>
__device__ __forceinline__ void gw_transpose_quarter(const float* raw, unsigned char* hi, int ch, int C, int nodes) {
#pragma unroll
  for (int gg = 0; gg < 2; ++gg) {
    const int chunk = QUARTER * 2 + gg;
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int k = chunk * 4 + c, z = k / D, i = k - z * D;
      v[c] = (z < rows_per_block(D) && z < nodes) ? raw[z * (C * D) + (MUL_IR ? ch * D + i : i * C + ch)] : 0.f;
    }
    store_split(hi, hi + kBlk, ch, chunk, v);
  }
}
template <int D, bool MUL_IR>
__device__ __forceinline__ void gw_transpose(const float* raw, unsigned char* hi, int C, int nodes, int tid) {
  const int ch = tid & 127;
  if (ch >= C) return;
  switch (tid >> 7) {
    case 0: gw_transpose_quarter<D, MUL_IR, 0>(raw, hi, ch, C, nodes); break;
    case 1: gw_transpose_quarter<D, MUL_IR, 1>(raw, hi, ch, C, nodes); break;
    case 2: gw_transpose_quarter<D, MUL_IR, 2>(raw, hi, ch, C, nodes); break;
    default: gw_transpose_quarter<D, MUL_IR, 3>(raw, hi, ch, C, nodes); break;
  }
}

__global__ void __launch_bounds__(kGwThreads, 1) linear_gw_kernel(const __grid_constant__ LParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned long long* rawfull = reinterpret_cast<unsigned long long*>(base + kGwBars);
  unsigned long long* rawempty = rawfull + kGwRawStages;
  unsigned long long* opfull = rawempty + kGwRawStages;
  unsigned long long* opempty = opfull + 2;
  unsigned long long* accfull = opempty + 2;
  unsigned long long* accempty = accfull + 1;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(accempty + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kGwRawStages; ++s) { bar_init(rawfull + s, 2); bar_init(rawempty + s, kGwWorkers / 32); }
    for (int s = 0; s < 2; ++s) { bar_init(opfull + s, kGwWorkers / 32); bar_init(opempty + s, 1); }
    bar_init(accfull, 1);
    bar_init(accempty, 4);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const unsigned tmem_base = tmem_alloc_all(tmem_slot, warp, 4);
  const int first = (int)((int64_t)p.total * blockIdx.x / gridDim.x), last = (int)((int64_t)p.total * (blockIdx.x + 1) / gridDim.x);

  if (warp < 4) {
    unsigned run = 0;
    bool dead = false;
    for_each_run(p, first, last, rows_per_block, [&](const LPath& q, int cls, int, int, int blocks) {
      if (!dead) dead = !bar_wait(accfull, run & 1, p.status);
      ++run;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int m = warp * 32 + lane;
      const bool good = !dead && status_clean(p.status) && m < q.K;
      // runs in order: from one to the next the thread block, the (path, class) or both move on, so their sum numbers them
      float* dst = p.parts + (int64_t)((int)blockIdx.x + (int)(&q - p.path) * p.num_classes + cls) * p.slot + (int64_t)m * q.N;
      for (int part = 0; part < q.N / 32; ++part) {
        float v[32];
        const unsigned ta = tmem_base + ((unsigned)(warp * 32) << 16) + part * 32;
        tmem_ld32(ta + 3 * 128, v);                                  // small terms
        for (int a = 0; a < 3 && a < blocks; ++a) {
          float v2[32];
          tmem_ld32(ta + a * 128, v2);
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] += v2[c];
        }
        if (good) {
#pragma unroll
          for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(dst + part * 32 + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(accempty);
    });
  } else if (warp == 4) {
    if (lane == 0) {
      unsigned it = 0, run = 0;
      bool ok = true;
      for_each_run(p, first, last, rows_per_block, [&](const LPath& q, int, int, int, int blocks) {
        const unsigned idesc = idesc_tf32(q.N);
        ok = ok && bar_wait(accempty, (run & 1) ^ 1, p.status);
        ++run;
        for (int b = 0; b < blocks && ok; ++b, ++it) {
          const unsigned s = it & 1;
          ok = bar_wait(opfull + s, (it >> 1) & 1, p.status);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const unsigned char* st = base + kGwOps + s * 4 * kBlk;
          umma_block(tmem_base + 3 * 128, st + kBlk, st + 2 * kBlk, idesc, b ? 1u : 0u);
          umma_block(tmem_base + 3 * 128, st, st + 3 * kBlk, idesc, 1u);
          umma_block(tmem_base + (b % 3) * 128, st, st + 2 * kBlk, idesc, b >= 3 ? 1u : 0u);
          umma_commit(opempty + s);
        }
        if (ok) umma_commit(accfull);
      });
    }
  } else if (warp >= 21) {
    const bool is_g = warp == 22;
    unsigned it = 0;
    bool ok = true;
    for_each_run(p, first, last, rows_per_block, [&](const LPath& q, int, int z0, int zend, int blocks) {
      const int n = rows_per_block(q.d);
      const unsigned bytes = (unsigned)((is_g ? q.N : q.K) * q.d * 4);
      const int64_t ld = is_g ? p.ldo : p.ldx;
      const float* src = (is_g ? p.g + q.o_off : p.x + q.x_off) + (int64_t)z0 * ld;
      for (int b = 0; b < blocks && ok; ++b, ++it, src += n * ld) {
        const unsigned s = it % kGwRawStages;
        ok = bar_wait(rawempty + s, ((it / kGwRawStages) & 1) ^ 1, p.status);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const int nodes = min(n, zend - (z0 + b * n));
        const unsigned raw = s32(base + kGwRaw + s * 2 * kBlk + (is_g ? kBlk : 0));
        if (lane == 0) bar_expect_tx(rawfull + s, nodes * bytes);
        __syncwarp();
        if (lane < nodes)                                            // one node per lane; at most 32 / d of them
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                       ::"r"(raw + lane * bytes), "l"(src + lane * ld), "r"(bytes), "r"(s32(rawfull + s)) : "memory");
      }
    });
  } else {
    const int tid = threadIdx.x - 160;
    unsigned it = 0;
    bool dead = false;
    for_each_run(p, first, last, rows_per_block, [&](const LPath& q, int, int z0, int zend, int blocks) {
      const int n = rows_per_block(q.d);
      for (int b = 0; b < blocks; ++b, ++it) {
        const unsigned r = it % kGwRawStages, s = it & 1;
        if (!dead) dead = !bar_wait(rawfull + r, (it / kGwRawStages) & 1, p.status);
        if (!dead) dead = !bar_wait(opempty + s, ((it >> 1) & 1) ^ 1, p.status);
        const float* raw = reinterpret_cast<const float*>(base + kGwRaw + r * 2 * kBlk);
        unsigned char* st = base + kGwOps + s * 4 * kBlk;
        const int nodes = min(n, zend - (z0 + b * n));
        if (!dead) {
          LINEAR_DISPATCH(gw_transpose, q.d, p.x_mul_ir, raw, st, q.K, nodes, tid)
          LINEAR_DISPATCH(gw_transpose, q.d, p.o_mul_ir, raw + kBlk / 4, st + 2 * kBlk, q.N, nodes, tid)
        }
        publish(opfull + s, lane);
        if (lane == 0) bar_arrive(rawempty + r);
      }
    });
  }
  tmem_free_all(tmem_base, warp, 4);
}

// The runs of one (path, class) added up in their order and put into the gradient.  Before, every run was added to the
// gradient by red.global.add, and the last bits changed from call to call.
// start[s]: first K block of (path, class) s = path * num_classes + class; the thread block of a K block t is the largest b
// with total * b / blocks <= t.
struct GwStarts { int start[kMaxPaths * kMaxClasses + 1]; };
__global__ void __launch_bounds__(128) linear_gw_sum_kernel(const __grid_constant__ LParams p, const __grid_constant__ GwStarts t, int blocks) {
  const int s = blockIdx.y, cls = s % p.num_classes;
  const LPath& q = p.path[s / p.num_classes];
  const int e = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (e >= q.K * q.N || !status_clean(p.status)) return;
  auto block_of = [&](int64_t item) { return (int)(((item + 1) * blocks + p.total - 1) / p.total) - 1; };
  const int b0 = block_of(t.start[s]), n = t.start[s] == t.start[s + 1] ? 0 : block_of(t.start[s + 1] - 1) - b0 + 1;   // 0: a class without rows
  const float* src = p.parts + (int64_t)(b0 + s) * p.slot + e;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < n; ++k) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(src + k * p.slot));
    v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
  }
  *reinterpret_cast<float4*>(p.out + cls * p.w_class_stride + q.w_off + e) = make_float4(q.c * v.x, q.c * v.y, q.c * v.z, q.c * v.w);
}

// Checks the arguments and fills the kernel parameters; `per_item` = nodes per tile or K block.  Returns the status.
template <class PerItem>
int make_params(const cueq_linear_args* a, PerItem per_item, bool gw, LParams* p) {
  if (!a || !a->x || !a->w || !a->out) return cueq::fail("linear: null operand");
  if (a->struct_bytes != (int)sizeof(cueq_linear_args)) return cueq::fail("linear: the binding declares another argument block");
  if (a->num_paths < 1 || a->num_paths > kMaxPaths) return cueq::fail("linear: between 1 and %d paths", kMaxPaths);
  if (a->num_classes < 1 || a->num_classes > kMaxClasses) return cueq::fail("linear: between 1 and %d classes", kMaxClasses);
  if (!a->bounds) return cueq::fail("linear: null class bounds");
  if ((a->ldx % 4) || (a->ldo % 4) || (((uintptr_t)a->x | (uintptr_t)a->out | (uintptr_t)a->w) & 15) || (a->w_class_stride % 4))
    return cueq::fail("linear: operands and rows must be 16-byte aligned");
  std::memset(p, 0, sizeof(*p));
  p->x = (const float*)a->x;
  p->ldx = a->ldx; p->ldo = a->ldo; p->w_class_stride = a->w_class_stride;
  p->x_mul_ir = a->x_mul_ir; p->o_mul_ir = a->out_mul_ir;
  p->num_paths = a->num_paths; p->num_classes = a->num_classes;
  p->status = (int*)a->status;
  for (int c = 0; c <= a->num_classes; ++c) {
    p->bounds[c] = a->bounds[c];
    if (a->bounds[c] < 0 || (c && a->bounds[c] < a->bounds[c - 1])) return cueq::fail("linear: class bounds must ascend from 0 or above");
  }
  int64_t total = 0;
  for (int k = 0; k < a->num_paths; ++k) {
    const cueq_linear_path& s = a->paths[k];
    if (s.u % 32 || s.v % 32 || s.u < 32 || s.v < 32 || s.u > 128 || s.v > 128) return cueq::fail("linear: multiplicities must be 32, 64, 96 or 128");
    if (s.d != 1 && s.d != 3 && s.d != 5 && s.d != 7) return cueq::fail("linear: irreps of dimension 1, 3, 5 or 7 only");
    if ((s.x_off | s.out_off | s.w_off) % 4 || s.x_off < 0 || s.out_off < 0 || s.w_off < 0) return cueq::fail("linear: offsets must be multiples of 4");
    LPath& q = p->path[k];
    q.d = s.d; q.c = s.c; q.w_off = s.w_off;
    if (a->transposed && !gw) {   // the input gradient: rows of the output irreps in, rows of the input irreps out
      q.K = s.v; q.N = s.u; q.x_off = s.out_off; q.o_off = s.x_off; q.w_sn = s.v; q.w_sk = 1;
    } else {
      q.K = s.u; q.N = s.v; q.x_off = s.x_off; q.o_off = s.out_off; q.w_sn = 1; q.w_sk = s.v;
    }
    for (int c = 0; c < a->num_classes; ++c) total += (a->bounds[c + 1] - a->bounds[c] + per_item(s.d) - 1) / per_item(s.d);
  }
  if (total > 2147483647LL) return cueq::fail("linear: too many rows");
  p->total = (int)total;
  return 0;
}

// every run ends with 64 KB of partial sums, so short inputs use fewer blocks; long ones are cut so that an accumulation
// chain does not grow with the number of rows
int gw_blocks(const LParams& p) {
  int grid = (p.total + 7) / 8;
  grid = grid < 148 ? grid : 148;
  const int most = (p.total + kMaxRunGw - 1) / kMaxRunGw;
  return grid < most ? most : grid;
}
int64_t gw_slot(const LParams& p) {
  int64_t slot = 0;
  for (int k = 0; k < p.num_paths; ++k) slot = (int64_t)p.path[k].K * p.path[k].N > slot ? (int64_t)p.path[k].K * p.path[k].N : slot;
  return slot;
}
int64_t gw_floats(const LParams& p, int grid) { return (int64_t)(grid + p.num_paths * p.num_classes) * gw_slot(p); }

}  // namespace

extern "C" int64_t cueq_b200_linear_gw_floats(const cueq_linear_args* a) {
  LParams p;
  if (make_params(a, rows_per_block, true, &p)) return -1;
  return p.total == 0 ? 0 : gw_floats(p, gw_blocks(p));
}

extern "C" int cueq_b200_linear_map(const cueq_linear_args* a, void* stream) {
  LParams p;
  if (int rc = make_params(a, rows_per_tile, false, &p)) return rc;
  p.w = (const float*)a->w;
  p.out = (float*)a->out;
  if (p.total == 0) return 0;
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(linear_map_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMapSmem));
    configured.set();
  }
  linear_map_kernel<<<p.total < 148 ? p.total : 148, kMapThreads, kMapSmem, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int cueq_b200_linear_gw(const cueq_linear_args* a, void* stream) {
  LParams p;
  if (int rc = make_params(a, rows_per_block, true, &p)) return rc;
  p.g = (const float*)a->w;
  p.out = (float*)a->out;
  if (p.total == 0) return 0;
  const int grid = gw_blocks(p);
  const int64_t need = gw_floats(p, grid);
  if (!a->parts || a->parts_floats < need || ((uintptr_t)a->parts & 15))
    return cueq::fail("linear: the weight gradient needs room for %lld floats of partial sums, 16-byte aligned", (long long)need);
  p.parts = (float*)a->parts;
  p.slot = gw_slot(p);
  GwStarts t;
  int widest = 0;
  for (int k = 0, s = 0, at = 0; k < p.num_paths; ++k) {
    widest = p.path[k].K * p.path[k].N > widest ? p.path[k].K * p.path[k].N : widest;
    const int n = rows_per_block(p.path[k].d);
    for (int c = 0; c < p.num_classes; ++c, ++s) {
      t.start[s] = at;
      at += (p.bounds[c + 1] - p.bounds[c] + n - 1) / n;
      t.start[s + 1] = at;
    }
  }
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(linear_gw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGwSmem));
    configured.set();
  }
  linear_gw_kernel<<<grid, kGwThreads, kGwSmem, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  CUEQ_CUDA_OK(cudaGetLastError());
  linear_gw_sum_kernel<<<dim3((widest / 4 + 127) / 128, p.num_paths * p.num_classes), 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p, t, grid);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}
