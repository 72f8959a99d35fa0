// Fully connected tensor product (uvw,iu,jv,kw+ijk; reference: the fused_tp call of
// cuequivariance_torch/primitives/segmented_polynomial_fused_tp.py:27-72) with shared weights: the output and the
// gradients of both inputs, one launch per irrep of the result.
//
// With T = sum C[i,j,k] W[u,v,w] x1[i,u] x2[j,v] g[k,w] each of the three is the derivative of T with respect to one of
// (x1, x2, g), so one kernel serves all: R names the operand that is differentiated out, P and Q the two others,
//
//     Y[z, a, (q, r)] = sum_p P[z, a, p] W[p, q, r]                        tensor cores, K = p
//     R[z, c, r]     += sum_q sum_a (sum_b C[a, b, c] Q[z, b, q]) Y[z, a, (q, r)]      CUDA cores, from TMEM
//
// P is the operand with fewer components.  Y never leaves the chip: [128 samples x 128 (q, r)] accumulators, four of
// them in TMEM, are consumed by sixteen warps (lane = sample) that keep R's components in registers over the whole sum.
// The route this replaces wrote the coupled operand Z[z, k, (u, v)] - 18.8 GB for 32,768 samples of 64x(0e+1o+2e) in
// float32 - and read it back, in each of five passes; its MMAs also ran once per component of the result instead of
// once per component of the smaller operand (35 against 27 blocks of 64^3 per sample).
//
// float32: P and W are split into TF32 halves (P on chip, W by fctp_tri_weights), three passes, small terms first, so
// that an accumulation chain has K / 8 <= 8 additions at full magnitude; all further sums are float32 FMAs.
// bf16: one pass; Y stays in float32, where the route before rounded the products of the inputs to bf16.
// What bounds it, per launch set at 32,768 samples of 64x(0e+1o+2e), float32: 3.5 ms.  The MMAs alone need 1.2 ms (27 * 64^3 * 3
// multiply-adds per sample); they wait for the weight blocks, 64 KB per 128 columns, of which two fit beside the operand
// tile, and with five components of the result for the multiply-adds of the consumers.
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

using namespace cueq_tc;

constexpr int kMaxPaths = CUEQ_FCTP_TRI_MAX_PATHS;
constexpr int kConsumers = 512;                        // warps 0-15
constexpr int kThreads = kConsumers + 128;             // 16: TMA, 17: MMA issue and TMEM owner, 18 and 19 fill the warpgroup
constexpr int kBlk = 128 * 128;                        // 128 rows x 128 bytes
// Registers: 20 warps leave 96 per thread at launch; the consumers' components of R alone are up to 80.  The producers'
// warpgroup gives its surplus to the four consumer warpgroups: 640 * 96 = 61440 = 512 * 112 + 128 * 32.  Every kernel of
// this file is compiled to exactly 96 (__launch_bounds__ allows no more, the host checks that it is no less; a build by another
// compiler where it is not says so in cueq_b200_fctp_tri_ready and keeps the routes for other shapes).
constexpr int kLaunchRegs = 96;
#define CONSUMER_REGS() asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n")
#define PRODUCER_REGS() asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n")

struct TriPath { int a_src, a_off, na, q_src, q_off, nb, b_row0, mask; float coef[5][5][5]; };   // mask: bit 5 * a + c
struct TriParams {
  const void* a[2];
  const float* qt[2];
  float* out;
  int64_t lda[2], zp, ldo, part;   // part: distance of the partial results of two divisions of the sum
  int batch, out_off, num_paths, splits;
  int* status;
  TriPath path[kMaxPaths];
};

template <bool BF16, int C>
struct Cfg {
  static constexpr int RT = C <= 64 ? C : C / 2;       // channels of the result per thread block
  static constexpr int RPT = RT / 4;                   // per thread
  static constexpr int NQ = RT == 32 ? 4 : 2;          // q values per accumulator
  static constexpr int NT = NQ * RT;                   // accumulator columns: 128
  static constexpr int KB = BF16 ? 64 : 32;            // elements per 128-byte operand row
  static constexpr int NKB = C / KB;
  static constexpr int kTwin = BF16 ? 1 : 2;           // hi (and lo)
  static constexpr int kStageB = NT * 128 * kTwin;
  static constexpr int kStages = BF16 ? 8 : 4;
  static constexpr int kS = NQ * 5 * 512;              // factors of an accumulator: [q][c][128 samples]
  static constexpr int kA = NKB * kBlk * kTwin;
  static constexpr int EPC = BF16 ? 8 : 4;             // elements per 16 bytes
  static constexpr int AU = 128 * (C / EPC) / kConsumers;
  static constexpr size_t smem = kA + kStages * kStageB + 2 * kS + 256 + 1024;
};

__device__ __forceinline__ void umma_tf32(unsigned tmem_c, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
               ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// the four instructions of one 128-byte-wide K block
template <bool BF16>
__device__ __forceinline__ void umma_block(unsigned tmem_c, const void* a, const void* b, unsigned idesc, unsigned accumulate) {
  const unsigned long long da = smem_desc(a), db = smem_desc(b);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    if constexpr (BF16) umma_bf16(tmem_c, da + 2ull * kk, db + 2ull * kk, idesc, kk ? 1u : accumulate);
    else umma_tf32(tmem_c, da + 2ull * kk, db + 2ull * kk, idesc, kk ? 1u : accumulate);
  }
}
__device__ __forceinline__ float tf32_hi(float v) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void tmem_ld(unsigned t, float (&y)[16]) {
  unsigned v[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(t));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < 16; ++c) y[c] = __uint_as_float(v[c]);
}
__device__ __forceinline__ void tmem_ld(unsigned t, float (&y)[8]) {
  unsigned v[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(t));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < 8; ++c) y[c] = __uint_as_float(v[c]);
}
template <bool BF16, int C, int NC>
__global__ void __launch_bounds__(kThreads, 1) fctp_tri_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                                                               const __grid_constant__ TriParams p) {
  using K = Cfg<BF16, C>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* ring = smem + K::kA;
  unsigned char* factors = ring + K::kStages * K::kStageB;           // of this accumulator and the next
  unsigned long long* full = reinterpret_cast<unsigned long long*>(factors + 2 * K::kS);
  unsigned long long* empty = full + K::kStages;
  unsigned long long* accfull = empty + K::kStages;
  unsigned long long* accempty = accfull + 4;
  unsigned long long* aready = accempty + 4;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(aready + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z0 = blockIdx.x * 128, rpart = blockIdx.y;
  const int qb = (C / p.splits) * blockIdx.z, qe = qb + C / p.splits;     // a multiple of NQ values

  if (threadIdx.x == 0) {
    for (int s = 0; s < K::kStages; ++s) { bar_init(full + s, 1); bar_init(empty + s, 1); }
    for (int b = 0; b < 4; ++b) { bar_init(accfull + b, 1); bar_init(accempty + b, kConsumers / 32); }
    bar_init(aready, kConsumers / 32);
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

  if (warp >= 16) {
    PRODUCER_REGS();
    if (warp == 16 && lane == 0) {
      unsigned it = 0;
      bool ok = true;
      for (int k = 0; k < p.num_paths && ok; ++k)
        for (int a = 0; a < p.path[k].na && ok; ++a)
          for (int q = qb; q < qe && ok; q += K::NQ)
            for (int kb = 0; kb < K::NKB && ok; ++kb, ++it) {
              const unsigned s = it % K::kStages;
              ok = bar_wait(empty + s, ((it / K::kStages) & 1) ^ 1, p.status);
              if (!ok) break;
              unsigned char* st = ring + s * K::kStageB;
              const int row = p.path[k].b_row0 + (rpart * C + q) * K::RT;
              bar_expect_tx(full + s, K::kStageB);
              tma_load_2d(st, &map_hi, kb * K::KB, row, full + s);
              if (!BF16) tma_load_2d(st + K::NT * 128, &map_lo, kb * K::KB, row, full + s);
            }
    } else if (warp == 17 && lane == 0) {
      constexpr unsigned fmt = BF16 ? 1u : 2u;
      constexpr unsigned idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((unsigned)(K::NT >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
      unsigned it = 0, n = 0, step = 0;
      bool ok = true;
      for (int k = 0; k < p.num_paths && ok; ++k)
        for (int a = 0; a < p.path[k].na && ok; ++a, ++step) {
          ok = bar_wait(aready, step & 1, p.status);
          for (int q = qb; q < qe && ok; q += K::NQ, ++n) {
            const unsigned buf = n & 3, acc = tmem_base + buf * 128;
            ok = bar_wait(accempty + buf, ((n >> 2) & 1) ^ 1, p.status);
            if (!BF16) {                                             // small terms of all K blocks first
              for (int kb = 0; kb < K::NKB && ok; ++kb) {
                const unsigned s = (it + kb) % K::kStages;
                ok = bar_wait(full + s, ((it + kb) / K::kStages) & 1, p.status);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const unsigned char* st = ring + s * K::kStageB;
                umma_block<BF16>(acc, smem + (K::NKB + kb) * kBlk, st, idesc, kb ? 1u : 0u);
                umma_block<BF16>(acc, smem + kb * kBlk, st + K::NT * 128, idesc, 1u);
              }
            }
            for (int kb = 0; kb < K::NKB && ok; ++kb, ++it) {
              const unsigned s = it % K::kStages;
              if (BF16) {
                ok = bar_wait(full + s, (it / K::kStages) & 1, p.status);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
              }
              umma_block<BF16>(acc, smem + kb * kBlk, ring + s * K::kStageB, idesc, (BF16 && kb == 0) ? 0u : 1u);
              umma_commit(empty + s);
            }
            if (ok) umma_commit(accfull + buf);
          }
        }
    }
  } else {
    CONSUMER_REGS();
    const int quad = warp & 3, g = warp >> 2;
    const int tid = threadIdx.x, z = z0 + quad * 32 + lane;          // < zp
    // the next operand tile waits in registers while the last accumulator of a step is consumed, where there is room
    constexpr bool kEarlyA = NC < 5;
    uint4 areg[K::AU];
    auto fetch_a = [&](const TriPath& t, int a) {
      const char* base = reinterpret_cast<const char*>(p.a[t.a_src]);
#pragma unroll
      for (int j = 0; j < K::AU; ++j) {
        const int unit = tid + j * kConsumers, zz = z0 + unit / (C / K::EPC), ch = unit % (C / K::EPC) * K::EPC;
        areg[j] = zz < p.batch ? __ldg(reinterpret_cast<const uint4*>(base + (BF16 ? 2 : 4) * ((int64_t)zz * p.lda[t.a_src] + t.a_off + a * C + ch)))
                               : make_uint4(0, 0, 0, 0);
      }
    };
    float acc[NC][K::RPT];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int j = 0; j < K::RPT; ++j) acc[c][j] = 0.f;
    // Factors of the result's components, s[q][c][z] = sum_b C[a, b, c] Q[z, b, q].  The four warps that share their samples
    // divide them: g picks the q value and, where there are two, half of the components.  The Q values of the next
    // accumulator are requested before this one is consumed and turned into factors after it.
    int nk = 0, na = 0, nq = qb;                                      // path, component and q of the next accumulator
    const int d_own = K::NQ == 4 ? g : g & 1;
    const int c_lo = K::NQ == 4 || g < 2 ? 0 : (NC + 1) / 2, c_hi = K::NQ == 4 || g >= 2 ? NC : (NC + 1) / 2;
    float qv[5];
    auto request = [&]() {
      if (nk >= p.num_paths || c_lo >= c_hi) return;
      const TriPath& t = p.path[nk];
      const float* src = p.qt[t.q_src] + (int64_t)(t.q_off + nq + d_own) * p.zp + z;
#pragma unroll
      for (int b = 0; b < 5; ++b) qv[b] = b < t.nb ? __ldg(src + (int64_t)b * C * p.zp) : 0.f;
    };
    auto combine = [&](unsigned slot) {
      if (nk < p.num_paths) {
        const TriPath& t = p.path[nk];
        float* dst = reinterpret_cast<float*>(factors + slot * K::kS) + d_own * 5 * 128 + quad * 32 + lane;
        for (int c = c_lo; c < c_hi; ++c) {
          float s = t.coef[na][0][c] * qv[0];
          if (t.nb > 1) { s = fmaf(t.coef[na][1][c], qv[1], s); s = fmaf(t.coef[na][2][c], qv[2], s); }
          if (t.nb > 3) { s = fmaf(t.coef[na][3][c], qv[3], s); s = fmaf(t.coef[na][4][c], qv[4], s); }
          dst[c * 128] = s;
        }
        if ((nq += K::NQ) >= qe) {
          nq = qb;
          if (++na >= t.na) { na = 0; ++nk; }
        }
      }
      asm volatile("bar.sync %0, 128;\n" ::"r"(quad + 1) : "memory"); // the four warps of these samples
    };
    unsigned n = 0;
    bool dead = false;
    request();
    combine(0);
    if (kEarlyA) fetch_a(p.path[0], 0);
    for (int k = 0; k < p.num_paths; ++k) {
      const TriPath& t = p.path[k];
      for (int a = 0; a < t.na; ++a) {
        if (!kEarlyA) fetch_a(t, a);
        // operand tile of this step; every MMA of the step before has completed (its last accumulator has been waited for)
#pragma unroll
        for (int j = 0; j < K::AU; ++j) {
          const int unit = tid + j * kConsumers, zz = unit / (C / K::EPC), ch = unit % (C / K::EPC) * K::EPC;
          unsigned char* tile = smem + (ch / K::KB) * kBlk + zz * 128 + (((ch % K::KB / K::EPC) ^ (zz & 7)) << 4);
          if (BF16) {
            *reinterpret_cast<uint4*>(tile) = areg[j];
          } else {
            const float v[4] = {__uint_as_float(areg[j].x), __uint_as_float(areg[j].y), __uint_as_float(areg[j].z), __uint_as_float(areg[j].w)};
            float h[4], l[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) { h[c] = tf32_hi(v[c]); l[c] = tf32_hi(v[c] - h[c]); }
            *reinterpret_cast<float4*>(tile) = make_float4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<float4*>(tile + K::NKB * kBlk) = make_float4(l[0], l[1], l[2], l[3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(aready);
        const unsigned mask = (unsigned)t.mask >> (5 * a);
        for (int q = qb; q < qe; q += K::NQ, ++n) {
          if (kEarlyA && q + K::NQ >= qe) {                           // last accumulator of the step: request the next operand tile
            if (a + 1 < t.na) fetch_a(t, a + 1);
            else if (k + 1 < p.num_paths) fetch_a(p.path[k + 1], 0);
          }
          const unsigned buf = n & 3;
          const unsigned col = tmem_base + ((unsigned)(quad * 32) << 16) + buf * 128 + g * K::RPT;
          request();
          if (!dead) dead = !bar_wait(accfull + buf, (n >> 2) & 1, p.status);
          const float* qs = reinterpret_cast<const float*>(factors + (n & 1) * K::kS) + quad * 32 + lane;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int d = 0; d < K::NQ; ++d) {
            float sv[NC], y[K::RPT];
#pragma unroll
            for (int c = 0; c < NC; ++c) sv[c] = qs[(d * 5 + c) * 128];
            tmem_ld(col + d * K::RT, y);
            if (d == K::NQ - 1) {
              asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
              __syncwarp();
              if (lane == 0) bar_arrive(accempty + buf);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              if ((mask >> c) & 1u) {
#pragma unroll
                for (int j = 0; j < K::RPT; ++j) acc[c][j] = fmaf(sv[c], y[j], acc[c][j]);
              }
            }
          }
          combine((n + 1) & 1);
        }
      }
    }
    if (!dead && status_clean(p.status) && z < p.batch) {
      float* row = p.out + blockIdx.z * p.part + (int64_t)z * p.ldo + p.out_off + rpart * K::RT + g * K::RPT;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int j = 0; j < K::RPT; j += 4)
          *reinterpret_cast<float4*>(row + c * C + j) = make_float4(acc[c][j], acc[c][j + 1], acc[c][j + 2], acc[c][j + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 17) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// The divisions of a sum, added in their order: the result does not depend on which thread block was faster.  Bound by memory
// (a read of every partial result).  Added by red.global.add into the result instead, the last bits changed from call to call.
__global__ void __launch_bounds__(256) fctp_tri_sum_kernel(const float4* __restrict__ parts, float4* __restrict__ out, int64_t n, int splits,
                                                           const int* status) {
  if (!status_clean(status)) return;                                  // after a wait that ran out the parts are incomplete
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float4 v = __ldcs(parts + i);
#pragma unroll 4
    for (int s = 1; s < splits; ++s) {
      const float4 a = __ldcs(parts + s * n + i);
      v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
    }
    out[i] = v;
  }
}

// Weights W[u][v][w] of every path -> rows ((channel half, q, r), p), p contiguous: float32 as TF32 halves, or bf16.
struct WParams {
  const void* w;
  void *hi, *lo;
  int w_bf16, C, RT;
  int w_off[kMaxPaths], order[kMaxPaths];   // order: 100 * axis of p + 10 * axis of q + axis of r, axes u = 0, v = 1, w = 2
};
template <bool BF16>
__global__ void __launch_bounds__(256) fctp_tri_weights_kernel(const __grid_constant__ WParams p) {
  __shared__ float tile[32][129];
  const int C = p.C, q = blockIdx.x, k = blockIdx.y;
  const int stride[3] = {C * C, C, 1};
  const int sp = stride[p.order[k] / 100], sq = stride[p.order[k] / 10 % 10], sr = stride[p.order[k] % 10];
  for (int r0 = 0; r0 < C; r0 += 32) {
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * C; e += 256) {
      // neighbouring threads read neighbouring weights where p or r is the contiguous axis
      const int r = sr == 1 ? e & 31 : e / C, pp = sr == 1 ? e >> 5 : e % C;
      const int64_t at = p.w_off[k] + (int64_t)q * sq + (int64_t)(r0 + r) * sr + (int64_t)pp * sp;
      tile[r][pp] = p.w_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.w)[at]) : __ldg(reinterpret_cast<const float*>(p.w) + at);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * C; e += 256) {
      const int r = e / C, pp = e % C, rr = r0 + r;
      const int64_t row = (int64_t)k * C * C + (int64_t)(rr / p.RT * C + q) * p.RT + rr % p.RT;
      const float v = tile[r][pp];
      if (BF16) {
        reinterpret_cast<__nv_bfloat16*>(p.hi)[row * C + pp] = __float2bfloat16(v);
      } else {
        const float h = tf32_hi(v);
        reinterpret_cast<float*>(p.hi)[row * C + pp] = h;
        reinterpret_cast<float*>(p.lo)[row * C + pp] = tf32_hi(v - h);
      }
    }
  }
}

// rows [batch][ld] -> float32 [cols][zp], as they are and / or as TF32 halves; zeros for batch <= z < zp
template <class T>
__global__ void __launch_bounds__(256) fctp_tri_transpose_kernel(const T* __restrict__ x, float* __restrict__ y, float* __restrict__ y_hi,
                                                                 float* __restrict__ y_lo, int batch, int cols, int64_t ld, int64_t zp) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, z0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    const int z = z0 + ty + k, c = c0 + tx;
    tile[ty + k][tx] = z < batch && c < cols ? (float)x[(int64_t)z * ld + c] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 32; k += 8)
    if (c0 + ty + k < cols) {
      const int64_t at = (int64_t)(c0 + ty + k) * zp + z0 + tx;
      const float v = tile[tx][ty + k];
      if (y) y[at] = v;
      if (y_hi) {
        const float h = tf32_hi(v);
        y_hi[at] = h;
        y_lo[at] = tf32_hi(v - h);
      }
    }
}

int make_map(CUtensorMap* map, bool bf16, const void* base, int64_t rows, int C, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return cueq::fail("fctp tri: cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[2] = {(cuuint64_t)C, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)C * (bf16 ? 2 : 4)};
  cuuint32_t box[2] = {bf16 ? 64u : 32u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cueq::fail("fctp tri: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

// setmaxnreg.inc would wait for registers that the block was not launched with
template <bool BF16, int C, int NC>
cudaError_t launch_regs(int* regs) {
  cudaFuncAttributes attr;
  const cudaError_t e = cudaFuncGetAttributes(&attr, fctp_tri_kernel<BF16, C, NC>);
  *regs = e == cudaSuccess ? attr.numRegs : 0;
  return e;
}
template <bool BF16, int C>
int compiled_as_needed() {
  int a = 0, b = 0, c = 0;
  if (launch_regs<BF16, C, 1>(&a) != cudaSuccess || launch_regs<BF16, C, 3>(&b) != cudaSuccess || launch_regs<BF16, C, 5>(&c) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return a == kLaunchRegs && b == kLaunchRegs && c == kLaunchRegs;
}

template <bool BF16, int C, int NC>
int launch_c(const CUtensorMap& hi, const CUtensorMap& lo, const TriParams& p, cudaStream_t st) {
  using K = Cfg<BF16, C>;
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    int regs = 0;
    CUEQ_CUDA_OK((launch_regs<BF16, C, NC>(&regs)));
    if (regs != kLaunchRegs) return cueq::fail("fctp tri: compiled to %d registers per thread, the warpgroups divide %d", regs, kLaunchRegs);
    CUEQ_CUDA_OK(cudaFuncSetAttribute(fctp_tri_kernel<BF16, C, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem));
    configured.set();
  }
  dim3 grid((p.batch + 127) / 128, C / K::RT, p.splits);
  fctp_tri_kernel<BF16, C, NC><<<grid, kThreads, K::smem, st>>>(hi, lo, p);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}
template <bool BF16, int C>
int launch(const cueq_fctp_tri_args* a, TriParams& p, cudaStream_t st) {
  using K = Cfg<BF16, C>;
  if (p.splits < 1 || C % p.splits || (C / p.splits) % K::NQ || p.splits > 16) return cueq::fail("fctp tri: invalid number of splits");
  CUtensorMap hi, lo;
  if (int rc = make_map(&hi, BF16, a->b_hi, a->b_rows, C, K::NT)) return rc;
  if (int rc = make_map(&lo, BF16, BF16 ? a->b_hi : a->b_lo, a->b_rows, C, K::NT)) return rc;
  if (p.splits > 1) {
    if (!a->parts) return cueq::fail("fctp tri: a divided sum needs room for its partial results");
    p.out = (float*)a->parts;
    p.part = p.ldo * p.batch;
  }
  switch (a->nc) {
    case 1: return launch_c<BF16, C, 1>(hi, lo, p, st);
    case 3: return launch_c<BF16, C, 3>(hi, lo, p, st);
    case 5: return launch_c<BF16, C, 5>(hi, lo, p, st);
    default: return cueq::fail("fctp tri: irreps of dimension 1, 3 or 5 only");
  }
}

}  // namespace

extern "C" int cueq_b200_fctp_tri_ready(int dtype, int channels) {
  if (dtype == CUEQ_BF16) return channels == 128 ? compiled_as_needed<true, 128>() : 0;
  if (dtype == CUEQ_F32) return channels == 32 ? compiled_as_needed<false, 32>() : channels == 64 ? compiled_as_needed<false, 64>() : 0;
  return 0;
}

extern "C" int cueq_b200_fctp_tri(const cueq_fctp_tri_args* a, void* stream) {
  if (!a || !a->out || !a->b_hi || !a->paths) return cueq::fail("fctp tri: null operand");
  if (a->struct_bytes != (int)sizeof(cueq_fctp_tri_args)) return cueq::fail("fctp tri: the binding declares another argument block");
  if (a->num_paths < 1 || a->num_paths > kMaxPaths) return cueq::fail("fctp tri: between 1 and %d paths", kMaxPaths);
  if (a->batch < 0 || a->batch > 2147483647LL - 128 || a->zp < (a->batch + 127) / 128 * 128) return cueq::fail("fctp tri: invalid batch or pitch");
  const bool bf16 = a->dtype == CUEQ_BF16;
  if (!bf16 && a->dtype != CUEQ_F32) return cueq::fail("fctp tri: float32 or bf16 operands");
  if (!bf16 && !a->b_lo) return cueq::fail("fctp tri: null operand");
  const int C = a->channels, unit = bf16 ? 8 : 4;
  if ((((uintptr_t)a->out | (uintptr_t)a->parts | (uintptr_t)a->b_hi | (uintptr_t)a->b_lo | (uintptr_t)a->a[0] | (uintptr_t)a->a[1] | (uintptr_t)a->qt[0] | (uintptr_t)a->qt[1]) & 15) || a->ldo % 4 || a->out_off % 4)
    return cueq::fail("fctp tri: operands and rows must be 16-byte aligned");
  TriParams p;
  std::memset(&p, 0, sizeof(p));
  for (int s = 0; s < 2; ++s) {
    p.a[s] = a->a[s]; p.lda[s] = a->lda[s]; p.qt[s] = (const float*)a->qt[s];
  }
  p.out = (float*)a->out;
  p.zp = a->zp; p.ldo = a->ldo; p.batch = (int)a->batch; p.out_off = a->out_off; p.num_paths = a->num_paths; p.splits = a->splits;
  p.status = (int*)a->status;
  for (int k = 0; k < a->num_paths; ++k) {
    const cueq_fctp_tri_path& s = a->paths[k];
    TriPath& t = p.path[k];
    auto dim = [](int d) { return d == 1 || d == 3 || d == 5; };
    if (!dim(s.na) || !dim(s.nb) || (s.a_src & ~1) || (s.q_src & ~1)) return cueq::fail("fctp tri: irreps of dimension 1, 3 or 5 only");
    if (!p.a[s.a_src] || !p.qt[s.q_src]) return cueq::fail("fctp tri: null operand");
    if (p.lda[s.a_src] % unit || s.a_off % unit || s.a_off < 0) return cueq::fail("fctp tri: operands and rows must be 16-byte aligned");
    if (s.q_off < 0 || a->zp % 128) return cueq::fail("fctp tri: invalid transposed operand");
    if (s.b_row0 < 0 || (int64_t)s.b_row0 + C * C > a->b_rows) return cueq::fail("fctp tri: weight rows out of range");
    t.a_src = s.a_src; t.a_off = s.a_off; t.na = s.na; t.q_src = s.q_src; t.q_off = s.q_off; t.nb = s.nb; t.b_row0 = s.b_row0;
    for (int i = 0; i < s.na; ++i)
      for (int j = 0; j < s.nb; ++j)
        for (int c = 0; c < a->nc && c < 5; ++c) {
          t.coef[i][j][c] = s.coef[(i * 5 + j) * 5 + c];
          if (t.coef[i][j][c] != 0.f) t.mask |= 1 << (5 * i + c);
        }
  }
  if (a->batch == 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (bf16) {
    if (C == 128) return launch<true, 128>(a, p, st);
  } else {
    if (C == 32) return launch<false, 32>(a, p, st);
    if (C == 64) return launch<false, 64>(a, p, st);
  }
  return cueq::fail("fctp tri: %d channels are not covered", C);
}

extern "C" int cueq_b200_fctp_tri_sum(const void* parts, void* out, int64_t batch, int64_t ldo, int splits, const void* status, void* stream) {
  if (!parts || !out) return cueq::fail("fctp tri: null operand");
  if (batch < 0 || ldo < 4 || ldo % 4 || splits < 1 || ((uintptr_t)parts | (uintptr_t)out) & 15) return cueq::fail("fctp tri: rows must be 16-byte aligned");
  if (batch == 0) return 0;
  const int64_t n = batch * ldo / 4, blocks = (n + 255) / 256;
  fctp_tri_sum_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const float4*)parts, (float4*)out, n, splits, (const int*)status);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int cueq_b200_fctp_tri_weights(const void* w, int w_dtype, int dtype, int channels, int num_paths, const int32_t* w_off, const int32_t* order,
                                          void* hi, void* lo, void* stream) {
  const bool bf16 = dtype == CUEQ_BF16;
  if (!w || !hi || !w_off || !order || (!bf16 && !lo)) return cueq::fail("fctp tri: null operand");
  if (num_paths < 1 || num_paths > kMaxPaths || channels % 32 || channels < 32 || channels > 128) return cueq::fail("fctp tri: invalid number of paths or channels");
  if (w_dtype != CUEQ_F32 && w_dtype != CUEQ_BF16) return cueq::fail("fctp tri: float32 or bf16 weights");
  WParams p;
  std::memset(&p, 0, sizeof(p));
  p.w = w; p.hi = hi; p.lo = lo; p.w_bf16 = w_dtype == CUEQ_BF16; p.C = channels; p.RT = channels <= 64 ? channels : channels / 2;
  for (int k = 0; k < num_paths; ++k) {
    const int a = order[k] / 100, b = order[k] / 10 % 10, c = order[k] % 10;
    if (a < 0 || a > 2 || b > 2 || c > 2 || a == b || b == c || a == c) return cueq::fail("fctp tri: order must permute the three axes");
    p.w_off[k] = w_off[k]; p.order[k] = order[k];
  }
  const dim3 grid(channels, num_paths);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (bf16) fctp_tri_weights_kernel<true><<<grid, 256, 0, st>>>(p);
  else fctp_tri_weights_kernel<false><<<grid, 256, 0, st>>>(p);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int cueq_b200_fctp_tri_transpose(const void* x, int dtype, int64_t batch, int32_t cols, int64_t ld, float* y, float* y_hi, float* y_lo,
                                            int64_t zp, void* stream) {
  if (!x || (!y && !y_hi) || (!y_hi != !y_lo)) return cueq::fail("fctp tri: null operand");
  if (batch < 1 || cols < 1 || zp % 32 || zp < batch || zp > 2147483647LL - 32 || (cols + 31) / 32 > 65535) return cueq::fail("fctp tri: invalid shape");
  const dim3 grid((unsigned)(zp / 32), (unsigned)((cols + 31) / 32));
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == CUEQ_F32) fctp_tri_transpose_kernel<float><<<grid, 256, 0, st>>>((const float*)x, y, y_hi, y_lo, (int)batch, cols, ld, zp);
  else if (dtype == CUEQ_BF16) fctp_tri_transpose_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)x, y, y_hi, y_lo, (int)batch, cols, ld, zp);
  else return cueq::fail("fctp tri: float32 or bf16 operands");
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}
