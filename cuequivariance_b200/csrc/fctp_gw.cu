// Fully connected tensor product (uvw,iu,jv,kw+ijk, shared weights): weight gradient in float32 accuracy.
//
// With T = sum C[i,j,k] W[u,v,w] x1[i,u] x2[j,v] g[k,w], the gradient of a path is a sum over samples
//
//     gW[x, y, t] += sum_e sum_z H_e[(x, y), z] T[z, e, t],    H_e[(x, y), z] = sum_b S_e[b, x, z] Y[z, b, y],
//     S_e[b, x, z] = sum_a C[a, b, e] X[z, a, x]
//
// where T is the operand with the fewest components (that many passes on the tensor cores) and X, Y the two others.  The
// samples are the K axis, so all operands come transposed ([column][sample], fctp_tri.cu).  H never leaves the chip: sixteen
// warps build its [128 rows x 32 samples] tiles, split into TF32 halves, straight into the K-major operand tiles; the T rows
// arrive split by TMA.  The coupled operand used to be written to memory per path and component of the output and read back
// by a row-reduction GEMM that transposed it: 3.5 + 8.0 ms for 32,768 samples of 64x(0e+1o+2e).
//
// A thread block owns one path, a range of x (all of TMEM: 512 columns of accumulators) and a range of samples.  Its result is
// added to the gradient, with more than kOrdered K blocks by red.global.add, in no fixed order; up to there through partial
// sums that a second kernel adds in their order.  hi*hi and the small terms have accumulators of their own, and the range of samples is cut so that
// a chain stays short (see `launch`).
// What bounds it: shared memory.  Per tile the MMAs read 56 KB (hi of the tile against both halves of T in one instruction),
// the builders 40 KB of S for two rows per thread and write 32 KB.  32,768 samples of 64x(0e+1o+2e): 4.3 ms.
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

using namespace cueq_tc;

constexpr int kMaxPaths = CUEQ_FCTP_TRI_MAX_PATHS;
constexpr int kBuilders = 512;                         // warps 0-15
constexpr int kThreads = kBuilders + 64;               // 16: TMA, 17: MMA issue and TMEM owner
constexpr int kBlk = 128 * 128;                        // 128 rows x 32 float32
// 2,048 samples.  The row-reduction GEMM before had one thread block per weight tile up to there, so that its result repeated
// bit for bit; partial sums for all samples of a large batch would be 50 to 250 copies of the weights.
constexpr int kOrdered = 64;

// item0: first thread block of the path; chunk: K blocks (32 samples) per thread block; mask: bit 5 * e + b
// slot0: first partial sum of the path
struct GwPath { int x_row, na, y_row, nb, t_row, ne, w_off, sx, sy, st, item0, chunk, mask, slot0; float coef[5][5][5]; };   // [e][a][b]
struct GwParams {
  float* gw;
  float* parts;             // partial sums of channels^3 floats each, or null
  int* status;
  int nblocks, num_paths;   // K blocks of all samples
  GwPath path[kMaxPaths];
};

template <int C>
struct Cfg {
  static constexpr int XP = 128 / C;                   // x values per tile
  static constexpr int kRows = XP * C;                 // used rows of a tile (C = 96: 96)
  static constexpr int TPC = C == 32 ? 8 : C == 64 ? 4 : 2;   // tiles per thread block: two accumulators of C columns each
  static constexpr int XR = XP * TPC;                  // x values per thread block
  static constexpr int YH = C == 96 ? 64 : C / 2;      // distance of the two y values of a thread
  static constexpr int kZStages = C == 96 ? 1 : 2;
  static constexpr int kY = 5 * C * 128, kX = (5 * XR * 128 + 1023) / 1024 * 1024;   // bytes per K block
  static constexpr int kS = 5 * XR * 128;
  static constexpr int kT = 2 * C * 128;               // hi, lo
  static constexpr int oT = 4 * kBlk, oZ = oT + 2 * kT, oS = oZ + kZStages * (kY + kX), oBar = oS + 2 * kS;
  static constexpr size_t smem = oBar + 256 + 1024;
};

__device__ __forceinline__ void umma_tf32(unsigned tmem_c, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
               ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
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
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void fma4(float4& d, const float4& a, const float4& b) {
  d.x = fmaf(a.x, b.x, d.x); d.y = fmaf(a.y, b.y, d.y); d.z = fmaf(a.z, b.z, d.z); d.w = fmaf(a.w, b.w, d.w);
}

template <int C>
__global__ void __launch_bounds__(kThreads, 1) fctp_gw_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                                                              const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                                                              const __grid_constant__ GwParams p) {
  using K = Cfg<C>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned long long* zfull = reinterpret_cast<unsigned long long*>(smem + K::oBar);
  unsigned long long* zempty = zfull + 2;
  unsigned long long* tfull = zempty + 2;
  unsigned long long* tempty = tfull + 2;
  unsigned long long* afull = tempty + 2;
  unsigned long long* aempty = afull + 2;
  unsigned long long* done = aempty + 2;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      bar_init(zfull + s, 1); bar_init(zempty + s, kBuilders / 32);
      bar_init(tfull + s, 1); bar_init(tempty + s, 1);
      bar_init(afull + s, kBuilders / 32); bar_init(aempty + s, 1);
    }
    bar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = *tmem_slot;

  int k = 0;
  while (k + 1 < p.num_paths && (int)blockIdx.x >= p.path[k + 1].item0) ++k;
  const GwPath& t = p.path[k];
  const int item = blockIdx.x - t.item0, x0 = item % (C / K::XR) * K::XR;
  const int b0 = item / (C / K::XR) * t.chunk, nblk = min(t.chunk, p.nblocks - b0);

  if (warp == 16) {
    if (lane == 0) {
      unsigned it = 0;
      bool ok = true;
      for (int b = 0; b < nblk && ok; ++b) {
        const int s = b % K::kZStages, z = (b0 + b) * 32;
        ok = bar_wait(zempty + s, ((b / K::kZStages) & 1) ^ 1, p.status);
        if (!ok) break;
        unsigned char* st = smem + K::oZ + s * (K::kY + K::kX);
        bar_expect_tx(zfull + s, t.nb * C * 128 + t.na * K::XR * 128);
        for (int j = 0; j < t.nb; ++j) tma_load_2d(st + j * C * 128, &map_y, z, t.y_row + j * C, zfull + s);
        for (int i = 0; i < t.na; ++i) tma_load_2d(st + K::kY + i * K::XR * 128, &map_x, z, t.x_row + i * C + x0, zfull + s);
        for (int e = 0; e < t.ne && ok; ++e, ++it) {
          const unsigned u = it & 1;
          ok = bar_wait(tempty + u, ((it >> 1) & 1) ^ 1, p.status);
          if (!ok) break;
          bar_expect_tx(tfull + u, K::kT);
          tma_load_2d(smem + K::oT + u * K::kT, &map_hi, z, t.t_row + e * C, tfull + u);
          tma_load_2d(smem + K::oT + u * K::kT + C * 128, &map_lo, z, t.t_row + e * C, tfull + u);
        }
      }
    }
  } else if (warp == 17) {
    if (lane == 0) {
      constexpr unsigned idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(C >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
      constexpr unsigned idesc2 = idesc + ((unsigned)(C >> 3) << 17);   // N = 2 C
      unsigned it = 0, a = 0;
      bool ok = true;
      const int steps = nblk * t.ne;
      for (; (int)it < steps && ok; ++it) {
        const unsigned u = it & 1;
        ok = bar_wait(tfull + u, (it >> 1) & 1, p.status);
        const unsigned char* tb = smem + K::oT + u * K::kT;
        for (int m = 0; m < K::TPC && ok; ++m, ++a) {
          const unsigned s = a & 1;
          ok = bar_wait(afull + s, (a >> 1) & 1, p.status);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const unsigned char* ab = smem + s * 2 * kBlk;
          const unsigned acc = tmem_base + m * 2 * C;
          umma_block(acc, ab, tb, idesc2, it ? 1u : 0u);                 // hi * hi and hi * lo: T's halves are neighbours
          umma_block(acc + C, ab + kBlk, tb, idesc, 1u);                 // lo * hi
          umma_commit(aempty + s);
        }
        if (ok) umma_commit(tempty + u);
      }
      if (ok) umma_commit(done);
    }
  } else {
    // a thread builds samples 4 * z4 .. + 3 of two rows (x, y) and (x, y + YH): one read of S for both
    const int tid = threadIdx.x, z4 = tid & 7, xl = C == 96 ? 0 : (tid >> 3) / K::YH, y0 = (tid >> 3) - xl * K::YH;
    unsigned it = 0, a = 0;
    bool dead = false;
    for (int b = 0; b < nblk; ++b) {
      const int s = b % K::kZStages;
      if (!dead) dead = !bar_wait(zfull + s, (b / K::kZStages) & 1, p.status);
      const float4* ys = reinterpret_cast<const float4*>(smem + K::oZ + s * (K::kY + K::kX));
      const float4* xs = reinterpret_cast<const float4*>(smem + K::oZ + s * (K::kY + K::kX) + K::kY);
      float4 y[2][5];
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (j < t.nb) {
          y[0][j] = ys[(j * C + y0) * 8 + z4];
          y[1][j] = ys[(j * C + min(y0 + K::YH, C - 1)) * 8 + z4];
        }
      for (int e = 0; e < t.ne; ++e, ++it) {
        const unsigned mask = (unsigned)t.mask >> (5 * e);
        float4* S = reinterpret_cast<float4*>(smem + K::oS + (it & 1) * K::kS);
        for (int q = tid; q < t.nb * K::XR * 8; q += kBuilders) {       // S[b][x][z4]
          const int j = q / (K::XR * 8), rest = q % (K::XR * 8);
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int i = 0; i < t.na; ++i) {
            const float c = t.coef[e][i][j];
            fma4(v, make_float4(c, c, c, c), xs[i * K::XR * 8 + rest]);
          }
          S[q] = v;
        }
        asm volatile("bar.sync 1, 512;\n" ::: "memory");
        if (e + 1 == t.ne) {                                            // the raw rows are in registers and in S
          __syncwarp();
          if (lane == 0) bar_arrive(zempty + s);
        }
        for (int m = 0; m < K::TPC; ++m, ++a) {
          const unsigned st = a & 1;
          if (!dead) dead = !bar_wait(aempty + st, ((a >> 1) & 1) ^ 1, p.status);
          unsigned char* hi = smem + st * 2 * kBlk;
          const float4* sx = S + (m * K::XP + xl) * 8 + z4;
          float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
          for (int j = 0; j < 5; ++j)
            if ((mask >> j) & 1u) {
              const float4 f = sx[j * K::XR * 8];
              fma4(v[0], f, y[0][j]);
              fma4(v[1], f, y[1][j]);
            }
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            if (C != 96 || n == 0 || y0 + K::YH < C) {
              const int r = xl * C + y0 + n * K::YH;
              float4 h, l;
              h.x = tf32_hi(v[n].x); h.y = tf32_hi(v[n].y); h.z = tf32_hi(v[n].z); h.w = tf32_hi(v[n].w);
              l.x = tf32_hi(v[n].x - h.x); l.y = tf32_hi(v[n].y - h.y); l.z = tf32_hi(v[n].z - h.z); l.w = tf32_hi(v[n].w - h.w);
              const int off = r * 128 + ((z4 ^ (r & 7)) << 4);
              *reinterpret_cast<float4*>(hi + off) = h;
              *reinterpret_cast<float4*>(hi + kBlk + off) = l;
            }
          }
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          __syncwarp();
          if (lane == 0) bar_arrive(afull + st);
        }
      }
    }
    if (!dead) dead = !bar_wait(done, 0, p.status);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const bool good = !dead && status_clean(p.status);
    const int row = (warp & 3) * 32 + lane;                            // TMEM lane quadrant = warp % 4
    for (int m = warp >> 2; m < K::TPC; m += 4) {
      const int x = x0 + m * K::XP + row / C, yy = row % C;
      float* dst = (p.parts ? p.parts + (int64_t)(t.slot0 + b0 / t.chunk) * (C * C * C) : p.gw + t.w_off) + (int64_t)x * t.sx + (int64_t)yy * t.sy;
      const unsigned col = tmem_base + ((unsigned)((warp & 3) * 32) << 16) + m * 2 * C;
      for (int c = 0; c < C; c += 8) {
        unsigned h[8], l[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                     : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]), "=r"(h[4]), "=r"(h[5]), "=r"(h[6]), "=r"(h[7]) : "r"(col + c));
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                     : "=r"(l[0]), "=r"(l[1]), "=r"(l[2]), "=r"(l[3]), "=r"(l[4]), "=r"(l[5]), "=r"(l[6]), "=r"(l[7]) : "r"(col + C + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (good && row < K::kRows) {
          float v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(h[q]) + __uint_as_float(l[q]);
          if (p.parts && t.st == 1) {
#pragma unroll
            for (int q = 0; q < 8; q += 4) *reinterpret_cast<float4*>(dst + c + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
          } else if (p.parts) {
#pragma unroll
            for (int q = 0; q < 8; ++q) dst[(int64_t)(c + q) * t.st] = v[q];
          } else if (t.st == 1) {
#pragma unroll
            for (int q = 0; q < 8; q += 4)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst + c + q), "f"(v[q]), "f"(v[q + 1]), "f"(v[q + 2]), "f"(v[q + 3]) : "memory");
          } else {                                                      // neighbouring lanes are neighbouring weights
#pragma unroll
            for (int q = 0; q < 8; ++q) asm volatile("red.global.add.f32 [%0], %1;\n" ::"l"(dst + (int64_t)(c + q) * t.st), "f"(v[q]) : "memory");
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 17) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// The partial sums of a path in their order, into the gradient (paths may share weights).
__global__ void __launch_bounds__(256) fctp_gw_sum_kernel(const __grid_constant__ GwParams p, int size) {
  const GwPath& t = p.path[blockIdx.y];
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4, n = (p.nblocks + t.chunk - 1) / t.chunk;
  if (e >= size || !status_clean(p.status)) return;
  const float* src = p.parts + (int64_t)t.slot0 * size + e;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(src + (int64_t)k * size));
    v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
  }
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p.gw + t.w_off + e), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

int make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t zp, int box_rows, bool swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return cueq::fail("fctp gw: cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[2] = {(cuuint64_t)zp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)zp * 4};
  cuuint32_t box[2] = {32u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cueq::fail("fctp gw: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

// K blocks per thread block: a chain has 4 additions at full magnitude per block and component.  80 keep the error below that
// of the GEMM before (chains of up to 192), which had shorter ones where there are few samples: 12 per four blocks.
int chunk_of(int nblocks, int ne) {
  const int chain = nblocks * 3 < 80 ? nblocks * 3 : 80;
  return chain / (4 * ne) > 1 ? chain / (4 * ne) : 1;
}

template <int C>
int launch(const cueq_fctp_gw_args* a, GwParams& p, cudaStream_t st) {
  using K = Cfg<C>;
  int64_t items = 0, slots = 0;
  for (int k = 0; k < p.num_paths; ++k) {
    GwPath& t = p.path[k];
    t.item0 = (int)items;
    t.slot0 = (int)slots;
    t.chunk = chunk_of(p.nblocks, t.ne);
    const int64_t chunks = (p.nblocks + t.chunk - 1) / t.chunk;
    items += (C / K::XR) * chunks;
    slots += chunks;
  }
  if (items > 2147483647LL) return cueq::fail("fctp gw: too many samples");
  CUtensorMap mx, my, mh, ml;
  if (int rc = make_map(&mx, a->t, a->rows, a->zp, K::XR, false)) return rc;
  if (int rc = make_map(&my, a->t, a->rows, a->zp, C, false)) return rc;
  if (int rc = make_map(&mh, a->t_hi, a->rows, a->zp, C, true)) return rc;
  if (int rc = make_map(&ml, a->t_lo, a->rows, a->zp, C, true)) return rc;
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(fctp_gw_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem));
    configured.set();
  }
  fctp_gw_kernel<C><<<(unsigned)items, kThreads, K::smem, st>>>(mx, my, mh, ml, p);
  CUEQ_CUDA_OK(cudaGetLastError());
  if (p.parts) {
    fctp_gw_sum_kernel<<<dim3((C * C * C / 4 + 255) / 256, p.num_paths), 256, 0, st>>>(p, C * C * C);
    CUEQ_CUDA_OK(cudaGetLastError());
  }
  return 0;
}

}  // namespace

extern "C" int64_t cueq_b200_fctp_gw_floats(const cueq_fctp_gw_args* a) {
  if (!a || !a->paths || a->struct_bytes != (int)sizeof(cueq_fctp_gw_args) || a->batch < 0 || a->num_paths < 1 || a->num_paths > kMaxPaths || a->channels < 1) return -1;
  const int64_t nblocks = (a->batch + 31) / 32;
  if (nblocks > kOrdered || nblocks == 0) return 0;
  int64_t slots = 0;
  for (int k = 0; k < a->num_paths; ++k) {
    if (a->paths[k].ne < 1) return -1;
    const int chunk = chunk_of((int)nblocks, a->paths[k].ne);
    slots += (nblocks + chunk - 1) / chunk;
  }
  return slots * a->channels * a->channels * a->channels;
}

extern "C" int cueq_b200_fctp_gw(const cueq_fctp_gw_args* a, void* stream) {
  if (!a || !a->t || !a->t_hi || !a->t_lo || !a->gw || !a->paths) return cueq::fail("fctp gw: null operand");
  if (a->struct_bytes != (int)sizeof(cueq_fctp_gw_args)) return cueq::fail("fctp gw: the binding declares another argument block");
  if (a->num_paths < 1 || a->num_paths > kMaxPaths) return cueq::fail("fctp gw: between 1 and %d paths", kMaxPaths);
  if (a->zp % 128 || a->batch < 0 || a->batch > a->zp || a->zp > 2147483647LL) return cueq::fail("fctp gw: invalid batch or pitch");
  if (((uintptr_t)a->t | (uintptr_t)a->t_hi | (uintptr_t)a->t_lo | (uintptr_t)a->gw | (uintptr_t)a->parts) & 15) return cueq::fail("fctp gw: operands must be 16-byte aligned");
  const int C = a->channels;
  if (C != 32 && C != 64 && C != 96) return cueq::fail("fctp gw: %d channels are not covered", C);
  GwParams p;
  std::memset(&p, 0, sizeof(p));
  p.gw = (float*)a->gw;
  p.status = (int*)a->status;
  p.nblocks = (int)((a->batch + 31) / 32);
  p.num_paths = a->num_paths;
  for (int k = 0; k < a->num_paths; ++k) {
    const cueq_fctp_gw_path& s = a->paths[k];
    GwPath& t = p.path[k];
    auto dim = [](int d) { return d == 1 || d == 3 || d == 5; };
    if (!dim(s.na) || !dim(s.nb) || !dim(s.ne)) return cueq::fail("fctp gw: irreps of dimension 1, 3 or 5 only");
    if (s.x_row < 0 || s.y_row < 0 || s.t_row < 0 || (int64_t)s.x_row + s.na * C > a->rows || (int64_t)s.y_row + s.nb * C > a->rows || (int64_t)s.t_row + s.ne * C > a->rows)
      return cueq::fail("fctp gw: operand rows out of range");
    if (s.w_off < 0 || s.w_off % 4) return cueq::fail("fctp gw: weight offsets must be multiples of 4");
    t.x_row = s.x_row; t.na = s.na; t.y_row = s.y_row; t.nb = s.nb; t.t_row = s.t_row; t.ne = s.ne; t.w_off = s.w_off;
    const int stride[3] = {C * C, C, 1};
    const int ax = s.order / 100, ay = s.order / 10 % 10, at = s.order % 10;
    if (s.order < 0 || ax > 2 || ay > 2 || at > 2 || ax == ay || ay == at || ax == at) return cueq::fail("fctp gw: order must permute the three axes");
    t.sx = stride[ax]; t.sy = stride[ay]; t.st = stride[at];
    for (int e = 0; e < s.ne; ++e)
      for (int i = 0; i < s.na; ++i)
        for (int j = 0; j < s.nb; ++j) {
          t.coef[e][i][j] = s.coef[(e * 5 + i) * 5 + j];
          if (t.coef[e][i][j] != 0.f) t.mask |= 1 << (5 * e + j);
        }
  }
  if (a->batch == 0) return 0;
  const int64_t need = cueq_b200_fctp_gw_floats(a);
  if (need > 0 && (!a->parts || a->parts_floats < need)) return cueq::fail("fctp gw: needs room for %lld floats of partial sums", (long long)need);
  p.parts = need > 0 ? (float*)a->parts : nullptr;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return C == 32 ? launch<32>(a, p, st) : C == 64 ? launch<64>(a, p, st) : launch<96>(a, p, st);
}
