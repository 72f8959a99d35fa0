// Channelwise ("uvu") tensor product: fused gather * Clebsch-Gordan multiply-add * receiver
// reduction, forward and backward, one launch per group of paths that read the same irrep of
// the first operand.
//
// These kernels replace the reference's closed uniform-1d kernel on the hot polynomial
// ``uv,iu,jv,kuv+ijk`` (descriptor: cuequivariance/group_theory/descriptors/irreps_tp.py:232-321;
// module: cuequivariance_torch/operations/tp_channel_wise.py:186-258), including the layout
// transpositions the reference performs as separate passes (tp_channel_wise.py:221-222,258).
//
// Work decomposition
//   * edges are addressed through a CSR over receivers (rowptr, optional edge order), so the
//     reduction over the edges of a receiver happens in registers: every output row is
//     written exactly once, without atomics and without a prior memset;
//   * one warp owns one receiver at a time; a lane owns two (or four) consecutive channels (one
//     128-bit access per segment), so a warp covers 128 channels; wider operands use
//     blockIdx.y;
//   * per edge, the channel-independent matrices M[i,k] = sum_j C[i,j,k] x2[j] of all paths of
//     the group are computed once per warp into shared memory (a table-driven loop spread
//     over the lanes) and then read back as broadcasts by the straight-line generated code;
//   * the rows of the next edge (the gathered x1 block and one weight segment per path) are
//     prefetched with cp.async into a per-warp, lane-private double buffer, so HBM latency
//     overlaps the arithmetic of the current edge;
//   * backward: the cotangent row of the receiver is staged once per receiver; the gradient
//     of the gathered operand goes out as vectorised reductions (red.global.add.v4.f32) keyed
//     by sender, the weight gradient is streamed out, the gradient of x2 is reduced over the
//     channels with warp shuffles.
//
// Which polynomials: every one whose paths are a subset of a group's (harmonics or outputs cut at a lower degree).  A
// full group runs the MASKED = false kernels; a subset runs the same code with one warp-uniform test per path, so the
// whole family costs one more instantiation instead of one per combination of degrees.  Against the table-driven kernel
// these polynomials ran on before (40,003 edges, 96 channels, lmax 2, forward + all gradients): 4.46 -> 0.48 ms.
// float64 instantiates the same kernels with two channels (16 bytes) per thread: half the FMA rate and twice the bytes of
// float32; 65,536 edges, 128 channels, lmax 3, forward + all gradients: 41.6 -> 2.36 ms (4.07 GB: 0.63 ms at 6.46 TB/s).
#pragma once
#include <cstdint>
#include <cstring>

#include "common.cuh"
#include "cw_entry.h"
#include "generated/cw_groups.cuh"

namespace {

using namespace cueq::cw;

#ifndef CW_WARPS
#define CW_WARPS 4
#endif
constexpr int kWarps = CW_WARPS;  // warps per CTA
#ifndef CW_MINBLOCKS
#define CW_MINBLOCKS 4
#endif

template <int C, class T> struct VecT;
template <> struct VecT<4, float> { using type = float4; };
template <> struct VecT<2, float> { using type = float2; };
template <> struct VecT<2, double> { using type = double2; };
template <int C, class T = float> using Vec = typename VecT<C, T>::type;

__device__ __forceinline__ void to_array(const float4& v, float (&a)[4]) { a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w; }
__device__ __forceinline__ void to_array(const float2& v, float (&a)[2]) { a[0] = v.x; a[1] = v.y; }
__device__ __forceinline__ void to_array(const double2& v, double (&a)[2]) { a[0] = v.x; a[1] = v.y; }

template <int C, int N, class T>
__device__ __forceinline__ Vec<C, T> make_vec(const T (&f)[N], int t) {
  Vec<C, T> v;
  v.x = f[t]; v.y = f[t + 1];
  if constexpr (C == 4) { v.z = f[t + 2]; v.w = f[t + 3]; }
  return v;
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
// L2 cache policies: per-edge operands are read once (evict first), the gathered node rows
// and the scattered node gradients are revisited by other edges (evict last)
__device__ __forceinline__ unsigned long long policy_evict_first() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long policy_evict_last() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
template <int BYTES>
__device__ __forceinline__ void cp_async_hint(void* smem_dst, const void* gmem_src, unsigned long long policy) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem_src), "l"(policy) : "memory");
  else
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %3, %2;\n" ::"r"(d), "l"(gmem_src), "l"(policy), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void red_add_hint(float* addr, const float (&v)[4], unsigned long long policy) {
  asm volatile("red.global.add.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;\n" ::"l"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "l"(policy) : "memory");
}
__device__ __forceinline__ void red_add_hint(float* addr, const float (&v)[2], unsigned long long policy) {
  asm volatile("red.global.add.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;\n" ::"l"(addr), "f"(v[0]), "f"(v[1]), "l"(policy) : "memory");
}
__device__ __forceinline__ void red_add_hint(double* addr, const double (&v)[2], unsigned long long policy) {
  asm volatile("red.global.add.L2::cache_hint.f64 [%0], %1, %2;\n" ::"l"(addr), "d"(v[0]), "l"(policy) : "memory");
  asm volatile("red.global.add.L2::cache_hint.f64 [%0], %1, %2;\n" ::"l"(addr + 1), "d"(v[1]), "l"(policy) : "memory");
}
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---- bulk-copy (TMA) staging ----------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: gives up after ~2^20 polls (each poll itself blocks for a hardware time slice),
// records the failure and lets the kernel run to its end instead of hanging the GPU.
__device__ __forceinline__ void mbar_wait(unsigned long long* bar, unsigned parity, int* status) {
  for (int spin = 0; spin < (1 << 20); ++spin)
    if (mbar_try_wait(bar, parity)) return;
  if (status) atomicExch(status, 1);
}
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// One bulk reduction (float32 add) of `bytes` contiguous bytes from shared to global memory, issued by one thread
// and tracked by that thread's bulk async-group; both addresses 16-byte aligned, `bytes` a multiple of 16.
__device__ __forceinline__ void bulk_reduce_add(float* gmem_dst, const void* smem_src, unsigned bytes, unsigned long long pol) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.L2::cache_hint.add.f32 [%0], [%1], %2, %3;\n"
               ::"l"(gmem_dst), "r"(smem_u32(smem_src)), "r"(bytes), "l"(pol) : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_reduce_add(double* gmem_dst, const void* smem_src, unsigned bytes, unsigned long long pol) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.L2::cache_hint.add.f64 [%0], [%1], %2, %3;\n"
               ::"l"(gmem_dst), "r"(smem_u32(smem_src)), "r"(bytes), "l"(pol) : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
// the issuing thread waits until its bulk reductions have read their shared-memory source / have completed
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

__device__ __forceinline__ void st_stream(float* addr, const float (&v)[4]) {
  asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ void st_stream(float* addr, const float (&v)[2]) {
  asm volatile("st.global.cs.v2.f32 [%0], {%1, %2};\n" ::"l"(addr), "f"(v[0]), "f"(v[1]) : "memory");
}

__device__ __forceinline__ void st_stream(double* addr, const double (&v)[2]) {
  asm volatile("st.global.cs.v2.f64 [%0], {%1, %2};\n" ::"l"(addr), "d"(v[0]), "d"(v[1]) : "memory");
}

// shared memory carve-up, in elements.  C = channels per lane.  Everything is per warp.
template <class G, int C, class T = float>
struct Smem {
  static constexpr int kM = G::NPAIR_PAD;                                   // per stage
  static constexpr int kX2 = 16;                                            // per stage: x2 row (<= 16 elements)
  static constexpr int kStage = (G::D1 + G::NPATH) * 32 * C;                // per stage: x1 block + weights
  static constexpr int kPerStage = kX2 + kStage;
  static constexpr int kPerWarpFwd = kM + 2 * kPerStage;
  static constexpr int kGrow = G::SUMD3 * 32 * C;                           // cotangent row of the receiver
  static constexpr int kPerWarpBwd = kPerWarpFwd + kGrow;
  static constexpr size_t bytes_fwd() { return sizeof(T) * (kWarps * kPerWarpFwd); }
  static constexpr size_t bytes_bwd() { return sizeof(T) * (kWarps * kPerWarpBwd); }
};

// Block of D contiguous-per-component values of the C channels of this lane, between global
// memory and lane-private staging.  ir_mul: component t of the lane's channels sits at
// base + t*extent + ch;  mul_ir: the lane's C*D values are contiguous at base + ch*D.
template <int D, int C, bool MUL_IR, class T>
__device__ __forceinline__ void stage_block(Vec<C, T>* dst, const T* base, int extent, int ch, int lane) {
#pragma unroll
  for (int t = 0; t < D; ++t) {
    const T* src = MUL_IR ? base + (int64_t)ch * D + C * t : base + (int64_t)t * extent + ch;
    cp_async<(int)sizeof(T) * C>(dst + t * 32 + lane, src);
  }
}
template <int D, int C, bool MUL_IR, class T>
__device__ __forceinline__ void stage_block_hint(Vec<C, T>* dst, const T* base, int extent, int ch, int lane, unsigned long long pol) {
#pragma unroll
  for (int t = 0; t < D; ++t) {
    const T* src = MUL_IR ? base + (int64_t)ch * D + C * t : base + (int64_t)t * extent + ch;
    cp_async_hint<(int)sizeof(T) * C>(dst + t * 32 + lane, src, pol);
  }
}

template <int D, int C, bool MUL_IR, int ROWS, class T>
__device__ __forceinline__ void unstage_block(const Vec<C, T>* src, int lane, T (&X)[ROWS][C]) {
  T f[D * C];
#pragma unroll
  for (int t = 0; t < D; ++t) {
    T a[C];
    to_array(src[t * 32 + lane], a);
#pragma unroll
    for (int c = 0; c < C; ++c) f[C * t + c] = a[c];
  }
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) X[i][c] = MUL_IR ? f[c * D + i] : f[C * i + c];
}

// registers -> global, same two layouts; RED: vector reduction, else streaming store
template <int D, int C, bool MUL_IR, bool RED, int ROWS, class T>
__device__ __forceinline__ void emit_block(T* base, int extent, int ch, const T (&V)[ROWS][C], int row0, unsigned long long pol = 0) {
  if (MUL_IR) {
    T f[D * C];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) f[c * D + i] = V[row0 + i][c];
#pragma unroll
    for (int t = 0; t < D; ++t) {
      T v[C];
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = f[C * t + c];
      if (RED) red_add_hint(base + (int64_t)ch * D + C * t, v, pol); else st_stream(base + (int64_t)ch * D + C * t, v);
    }
  } else {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      if (RED) red_add_hint(base + (int64_t)i * extent + ch, V[row0 + i], pol); else st_stream(base + (int64_t)i * extent + ch, V[row0 + i]);
    }
  }
}

// The channel-independent matrices M of one edge: M[q] = sum_t c[t] * x2[j[t]] for every table
// entry q of the group - one per non-zero (i,k) pair in the backward kernels (N = NPAIR), one per
// distinct value among them in the forward kernels (N = NVAL: many pairs carry the same combination
// of x2 up to sign, and every entry costs a broadcast read per warp and edge).  Lane L owns the
// entries L, L+32, ...; an entry has at most two terms (true for every coupling with l <= 3), whose
// coefficients and x2 positions the lane keeps in registers for the whole kernel, so the per-edge
// work is a handful of shared-memory reads and FMAs without any loop or branch.
template <int N, class T = float>
struct MTerms {
  static constexpr int R = (N + 31) / 32;
  static constexpr int NPAD = (N + 3) / 4 * 4;
  T c[R][2];
  unsigned j[R];  // two 16-bit x2 positions per pair

  __device__ __forceinline__ void load(const CwParamsT<T>& p, int lane) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = lane + 32 * r;
      c[r][0] = c[r][1] = T(0);
      j[r] = 0;
      if (q < N) {
        const int t0 = __ldg(p.tab_start + q), t1 = __ldg(p.tab_start + q + 1);
        if (t1 > t0) { c[r][0] = __ldg(p.tab_c + t0); j[r] = (unsigned)__ldg(p.tab_j + t0); }
        if (t1 > t0 + 1) { c[r][1] = __ldg(p.tab_c + t0 + 1); j[r] |= (unsigned)__ldg(p.tab_j + t0 + 1) << 16; }
      }
    }
  }
  // MASKED: an entry with one term does not read a second one, so that an infinite or undefined component of x2 reaches only
  // the paths that use it, as on the table-driven kernel that takes what these kernels do not.
  template <bool MASKED>
  __device__ __forceinline__ void compute(T* M, const T* x2row, int lane) const {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      T m = c[r][0] * x2row[j[r] & 0xffffu];
      if (!MASKED || c[r][1] != T(0)) m = fma(c[r][1], x2row[j[r] >> 16], m);
      if (N % 32 == 0 || r + 1 < R || lane + 32 * r < NPAD) M[lane + 32 * r] = m;
    }
  }
};

// asynchronous loads of everything edge `pos` needs into the stage at `st`; returns the edge id
// The edge id (through the optional permutation) and the sender of the edge at position `pos`: two dependent
// index loads.  The kernels request them one edge earlier than they issue that edge's copies, so that their
// latency is hidden behind the arithmetic of an edge instead of being waited for in front of the copies.
struct EdgeIds { int eid, snd; };
template <class T>
__device__ __forceinline__ EdgeIds load_ids(const CwParamsT<T>& p, int pos) {
  EdgeIds e;
  e.eid = p.order ? __ldg(p.order + pos) : pos;
  e.snd = p.senders ? __ldg(p.senders + e.eid) : e.eid;
  return e;
}

// Whether path q of the group takes part (a kernel of the full group knows that all do).
template <bool MASKED, class T>
__device__ __forceinline__ bool has_path(const CwParamsT<T>& p, int q) { return !MASKED || ((p.path_mask >> q) & 1u); }

template <class G, int C, bool X1_MUL_IR, bool MASKED, class T>
__device__ __forceinline__ void issue_edge_ids(const CwParamsT<T>& p, T* st, const EdgeIds ids, int ch, int lane, bool active,
                                               unsigned long long pol_stream, unsigned long long pol_keep) {
  T* x2s = st;
  Vec<C, T>* stage = reinterpret_cast<Vec<C, T>*>(x2s + Smem<G, C, T>::kX2);
  if constexpr (MASKED) {   // rows of 1, 4, 9 or 16 components: one element per lane, no alignment asked of the rows
    if (lane < p.nx2) cp_async_hint<(int)sizeof(T)>(x2s + lane, p.x2 + (int64_t)ids.eid * p.x2_stride + lane, pol_stream);
  } else {
    constexpr int V = 16 / (int)sizeof(T);
    if (lane < (G::NX2 + V - 1) / V) cp_async_hint<16>(x2s + V * lane, p.x2 + (int64_t)ids.eid * p.x2_stride + V * lane, pol_stream);
  }
  if (active) {
    stage_block_hint<G::D1, C, X1_MUL_IR>(stage, p.x1 + (int64_t)ids.snd * p.x1_stride + p.x1_off, p.extent, ch, lane, pol_keep);
    const T* wrow = p.w + (int64_t)ids.eid * p.w_stride + ch;
    Vec<C, T>* wst = stage + G::D1 * 32;
#pragma unroll
    for (int q = 0; q < G::NPATH; ++q)
      if (has_path<MASKED>(p, q)) cp_async_hint<(int)sizeof(T) * C>(wst + q * 32 + lane, wrow + p.w_off[q], pol_stream);
  }
  cp_async_commit();
}

template <class G, int C, int P, bool MASKED, class T>
struct FwdPaths {
  __device__ __forceinline__ static void run(const CwParamsT<T>& p, const T (&X)[G::D1][C], const Vec<C, T>* wst, int lane, const T* M,
                                             T (&acc)[G::SUMD3][C]) {
    if (has_path<MASKED>(p, P)) {
      T W[C];
      to_array(wst[P * 32 + lane], W);
      G::template fwd_path<P, C>(X, W, M, acc);
    }
    if constexpr (P + 1 < G::NPATH) FwdPaths<G, C, P + 1, MASKED, T>::run(p, X, wst, lane, M, acc);
  }
};

template <class G, int C, int P, bool OUT_MUL_IR, bool MASKED, class T>
struct StoreOut {
  __device__ __forceinline__ static void run(T* orow, const CwParamsT<T>& p, int ch, const T (&acc)[G::SUMD3][C]) {
    if (has_path<MASKED>(p, P)) emit_block<G::d3(P), C, OUT_MUL_IR, false>(orow + p.out_off[P], p.extent, ch, acc, G::out_offset(P));
    if constexpr (P + 1 < G::NPATH) StoreOut<G, C, P + 1, OUT_MUL_IR, MASKED, T>::run(orow, p, ch, acc);
  }
};

template <class T> constexpr int kFwdMinBlocks = sizeof(T) == 8 ? 2 : CW_MINBLOCKS;

// OVERLAP: part of a chain of overlapping launches (launch_kernel).  The two instructions cost the l >= 1 kernels 5 % - two
// registers at their limit of 128, a spill and 7 % more instructions - so a launch that gains nothing from it goes without.
template <class T, class G, int C, bool MUL_IR, bool MASKED, bool OVERLAP>
__global__ void __launch_bounds__(kWarps * 32, kFwdMinBlocks<T>) cw_fwd_kernel(const __grid_constant__ CwParamsT<T> p) {
  if constexpr (OVERLAP) let_next_start();
  extern __shared__ __align__(16) unsigned char smem_bytes[];
  T* smem = reinterpret_cast<T*>(smem_bytes);
  using S = Smem<G, C, T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* mine = smem + warp * S::kPerWarpFwd;
  const int ch = blockIdx.y * (32 * C) + C * lane;   // first channel of this lane
  const bool active = ch < p.extent;
  MTerms<G::NVAL, T> mt;
  mt.load(p, lane);
  const unsigned long long pol_stream = policy_evict_first(), pol_keep = policy_evict_last();

  const int total_warps = gridDim.x * kWarps;
  for (int n = blockIdx.x * kWarps + warp; n < p.num_receivers; n += total_warps) {
    const int beg = __ldg(p.rowptr + n), end = __ldg(p.rowptr + n + 1);
    T acc[G::SUMD3][C];
#pragma unroll
    for (int a = 0; a < G::SUMD3; ++a)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[a][c] = T(0);
    T* Msm = mine;
    T* stages = mine + S::kM;
    EdgeIds ahead = {0, 0};                                        // ids of the edge whose copies are issued next
    if (beg < end) issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages, load_ids(p, beg), ch, lane, active, pol_stream, pol_keep);
    if (beg + 1 < end) ahead = load_ids(p, beg + 1);
    for (int pos = beg; pos < end; ++pos) {
      T* st = stages + ((pos - beg) & 1) * S::kPerStage;
      if (pos + 1 < end) {
        issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages + ((pos + 1 - beg) & 1) * S::kPerStage, ahead, ch, lane, active, pol_stream, pol_keep);
        if (pos + 2 < end) ahead = load_ids(p, pos + 2);           // used in the next trip
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncwarp();
      mt.template compute<MASKED>(Msm, st, lane);
      __syncwarp();
      if (active) {
        const Vec<C, T>* stage = reinterpret_cast<const Vec<C, T>*>(st + S::kX2);
        T X[G::D1][C];
        unstage_block<G::D1, C, MUL_IR>(stage, lane, X);
        FwdPaths<G, C, 0, MASKED, T>::run(p, X, stage + G::D1 * 32, lane, Msm, acc);
      }
      __syncwarp();
    }
    if (active) StoreOut<G, C, 0, MUL_IR, MASKED, T>::run(p.out + (int64_t)n * p.out_stride, p, ch, acc);
  }
  if constexpr (OVERLAP) wait_for_previous();
}

// ---- forward, staging by bulk copies ----------------------------------------------------------
//
// Same arithmetic as cw_fwd_kernel; the rows of the next edge are fetched by the copy engine
// (cp.async.bulk, one instruction per contiguous piece, issued by one lane) and their arrival
// is signalled on an mbarrier, instead of one cp.async per lane and piece.  The staged data
// keep their global layout: for mul_ir the whole [channel][component] block of the gathered
// row is one contiguous copy.
template <class G, int C>
struct SmemBulk {
  static constexpr int NCH = 32 * C;                                        // channels per warp
  static constexpr int kBar = 4;                                            // two 64-bit barriers
  static constexpr int kM = G::NPAIR_PAD;
  static constexpr int kX2 = 16;
  static constexpr int kPerStage = kX2 + (G::D1 + G::NPATH) * NCH;
  static constexpr int kPerWarp = kBar + kM + 2 * kPerStage;
  static constexpr size_t bytes() { return sizeof(float) * (kWarps * kPerWarp); }
};

template <class G, int C, bool MUL_IR>
__device__ __forceinline__ void bulk_issue_edge(const CwParams& p, float* st, unsigned long long* bar, int pos, int c0, int nch) {
  using S = SmemBulk<G, C>;
  const int eid = p.order ? __ldg(p.order + pos) : pos;
  const int snd = p.senders ? __ldg(p.senders + eid) : eid;
  constexpr unsigned x2_bytes = ((G::NX2 + 3) / 4) * 16;
  const unsigned row_bytes = (unsigned)nch * 4u;
  fence_proxy_async();
  mbar_expect_tx(bar, x2_bytes + row_bytes * (G::D1 + G::NPATH));
  bulk_g2s(st, p.x2 + (int64_t)eid * p.x2_stride, x2_bytes, bar);
  float* xs = st + S::kX2;
  const float* xrow = p.x1 + (int64_t)snd * p.x1_stride + p.x1_off;
  if (MUL_IR) {
    bulk_g2s(xs, xrow + (int64_t)c0 * G::D1, row_bytes * G::D1, bar);
  } else {
#pragma unroll
    for (int i = 0; i < G::D1; ++i) bulk_g2s(xs + i * S::NCH, xrow + (int64_t)i * p.extent + c0, row_bytes, bar);
  }
  float* ws = xs + G::D1 * S::NCH;
  const float* wrow = p.w + (int64_t)eid * p.w_stride + c0;
#pragma unroll
  for (int q = 0; q < G::NPATH; ++q) bulk_g2s(ws + q * S::NCH, wrow + p.w_off[q], row_bytes, bar);
}

template <class G, int C, int P>
struct FwdPathsBulk {
  __device__ __forceinline__ static void run(const float (&X)[G::D1][C], const float* ws, int lane, const float* M,
                                             float (&acc)[G::SUMD3][C]) {
    float W[C];
    to_array(*reinterpret_cast<const Vec<C>*>(ws + P * (32 * C) + C * lane), W);
    G::template fwd_path<P, C>(X, W, M, acc);
    if constexpr (P + 1 < G::NPATH) FwdPathsBulk<G, C, P + 1>::run(X, ws, lane, M, acc);
  }
};

template <class G, int C, bool MUL_IR>
__global__ void __launch_bounds__(kWarps * 32, C == 2 ? CW_MINBLOCKS : 2) cw_fwd_bulk_kernel(const __grid_constant__ CwParams p) {
  extern __shared__ __align__(16) float smem[];
  using S = SmemBulk<G, C>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* mine = smem + warp * S::kPerWarp;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(mine);
  float* Msm = mine + S::kBar;
  float* stages = Msm + S::kM;
  const int c0 = blockIdx.y * S::NCH;
  const int ch = c0 + C * lane;
  const bool active = ch < p.extent;
  const int nch = min(S::NCH, p.extent - c0);
  MTerms<G::NVAL> mt;
  mt.load(p, lane);
  if (lane == 0) {
    mbar_init(bars + 0, 1);
    mbar_init(bars + 1, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  unsigned it = 0;  // edges consumed by this warp so far: stage = it & 1, parity = (it >> 1) & 1

  const int total_warps = gridDim.x * kWarps;
  for (int n = blockIdx.x * kWarps + warp; n < p.num_receivers; n += total_warps) {
    const int beg = __ldg(p.rowptr + n), end = __ldg(p.rowptr + n + 1);
    float acc[G::SUMD3][C];
#pragma unroll
    for (int a = 0; a < G::SUMD3; ++a)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[a][c] = 0.f;
    if (beg < end && lane == 0) bulk_issue_edge<G, C, MUL_IR>(p, stages + (it & 1) * S::kPerStage, bars + (it & 1), beg, c0, nch);
    for (int pos = beg; pos < end; ++pos, ++it) {
      const unsigned s = it & 1;
      float* st = stages + s * S::kPerStage;
      if (pos + 1 < end && lane == 0)
        bulk_issue_edge<G, C, MUL_IR>(p, stages + (s ^ 1) * S::kPerStage, bars + (s ^ 1), pos + 1, c0, nch);
      mbar_wait(bars + s, (it >> 1) & 1, p.status);
      mt.template compute<false>(Msm, st, lane);
      __syncwarp();
      if (active) {
        const float* xs = st + S::kX2;
        float X[G::D1][C];
        if (MUL_IR) {
          float f[G::D1 * C];
          const Vec<C>* src = reinterpret_cast<const Vec<C>*>(xs + (int64_t)C * lane * G::D1);
#pragma unroll
          for (int t = 0; t < G::D1; ++t) {
            float a[C];
            to_array(src[t], a);
#pragma unroll
            for (int c = 0; c < C; ++c) f[C * t + c] = a[c];
          }
#pragma unroll
          for (int i = 0; i < G::D1; ++i)
#pragma unroll
            for (int c = 0; c < C; ++c) X[i][c] = f[c * G::D1 + i];
        } else {
#pragma unroll
          for (int i = 0; i < G::D1; ++i) to_array(*reinterpret_cast<const Vec<C>*>(xs + i * S::NCH + C * lane), X[i]);
        }
        FwdPathsBulk<G, C, 0>::run(X, xs + G::D1 * S::NCH, lane, Msm, acc);
      }
      __syncwarp();
    }
    if (active) StoreOut<G, C, 0, MUL_IR, false, float>::run(p.out + (int64_t)n * p.out_stride, p, ch, acc);
  }
}

// ---- backward ---------------------------------------------------------------------------------
template <class G, int C, int P, bool MUL_IR, bool NEED_R, bool MASKED, class T>
struct BwdPaths {
  __device__ __forceinline__ static void run(const T (&X)[G::D1][C], const Vec<C, T>* wst, const Vec<C, T>* grow, int lane,
                                             const T* M, const CwCoefT<T>& coef, const CwParamsT<T>& p, T* gwrow,
                                             T (&gX)[G::D1][C], T (&r)[16]) {
    if (has_path<MASKED>(p, P)) {
      T W[C];
      to_array(wst[P * 32 + lane], W);
      T Gk[G::MAXD3][C];
      unstage_block<G::d3(P), C, MUL_IR>(grow + G::out_offset(P) * 32, lane, Gk);
      T gw[C];
      G::template bwd_path<P, C, NEED_R>(X, W, M, Gk, coef, gX, gw, r);
      if (p.need_gw) st_stream(gwrow + p.w_off[P], gw);
    }
    if constexpr (P + 1 < G::NPATH) BwdPaths<G, C, P + 1, MUL_IR, NEED_R, MASKED, T>::run(X, wst, grow, lane, M, coef, p, gwrow, gX, r);
  }
};

// cotangent row of a receiver -> lane-private staging; block P holds d3(P) vectors per lane
template <class G, int C, int P, bool MUL_IR, bool MASKED, class T>
struct StageG {
  __device__ __forceinline__ static void run(Vec<C, T>* dst, const T* grow, const CwParamsT<T>& p, int ch, int lane) {
    if (has_path<MASKED>(p, P)) stage_block<G::d3(P), C, MUL_IR>(dst + G::out_offset(P) * 32, grow + p.out_off[P], p.extent, ch, lane);
    if constexpr (P + 1 < G::NPATH) StageG<G, C, P + 1, MUL_IR, MASKED, T>::run(dst, grow, p, ch, lane);
  }
};

// Sum of 16 per-lane values over the warp: on return lane L holds the total of r[L >> 1].
// Each step exchanges half of the remaining values with the partner lane, so the whole
// reduction costs about one shuffle per value instead of five.
template <class T>
__device__ __forceinline__ T reduce16(T (&r)[16], int lane) {
#pragma unroll
  for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int t = 0; t < half; ++t) {
      const T send = up ? r[t] : r[t + half];
      const T keep = up ? r[t + half] : r[t];
      r[t] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
  return r[0] + __shfl_xor_sync(0xffffffffu, r[0], 1);
}

template <class G, int C, bool MUL_IR, bool MASKED>
__global__ void __launch_bounds__(kWarps * 32, CW_MINBLOCKS) cw_bwd_kernel(const __grid_constant__ CwParams p, const __grid_constant__ CwCoef coef) {
  let_next_start();
  extern __shared__ __align__(16) float smem[];
  using S = Smem<G, C>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* mine = smem + warp * S::kPerWarpBwd;
  Vec<C>* grow = reinterpret_cast<Vec<C>*>(mine + S::kPerWarpFwd);
  const int ch = blockIdx.y * (32 * C) + C * lane;
  const bool active = ch < p.extent;
  MTerms<G::NPAIR> mt;
  mt.load(p, lane);
  const unsigned long long pol_stream = policy_evict_first(), pol_keep = policy_evict_last();

  const int total_warps = gridDim.x * kWarps;
  for (int n = blockIdx.x * kWarps + warp; n < p.num_receivers; n += total_warps) {
    const int beg = __ldg(p.rowptr + n), end = __ldg(p.rowptr + n + 1);
    if (beg >= end) continue;
    const int nrow = p.recv_mod ? n % p.recv_mod : n;
    if (active) StageG<G, C, 0, MUL_IR, MASKED, float>::run(grow, p.gout + (int64_t)nrow * p.out_stride, p, ch, lane);
    cp_async_commit();
    float* Msm = mine;
    float* stages = mine + S::kM;
    EdgeIds cur = {0, 0}, next = load_ids(p, beg), ahead = {0, 0};
    issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages, next, ch, lane, active, pol_stream, pol_keep);
    if (beg + 1 < end) ahead = load_ids(p, beg + 1);
    for (int pos = beg; pos < end; ++pos) {
      float* st = stages + ((pos - beg) & 1) * S::kPerStage;
      cur = next;
      if (pos + 1 < end) {
        next = ahead;
        issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages + ((pos + 1 - beg) & 1) * S::kPerStage, next, ch, lane, active, pol_stream, pol_keep);
        if (pos + 2 < end) ahead = load_ids(p, pos + 2);           // used in the next trip
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      const int eid = cur.eid;
      __syncwarp();
      mt.template compute<MASKED>(Msm, st, lane);
      __syncwarp();
      float r[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = 0.f;
      if (active) {
        const Vec<C>* stage = reinterpret_cast<const Vec<C>*>(st + S::kX2);
        float X[G::D1][C], gX[G::D1][C];
        unstage_block<G::D1, C, MUL_IR>(stage, lane, X);
#pragma unroll
        for (int i = 0; i < G::D1; ++i)
#pragma unroll
          for (int c = 0; c < C; ++c) gX[i][c] = 0.f;
        BwdPaths<G, C, 0, MUL_IR, true, MASKED, float>::run(X, stage + G::D1 * 32, grow, lane, Msm, coef, p, p.gw + (int64_t)eid * p.w_stride + ch, gX, r);
        if (p.need_gx1) {
          emit_block<G::D1, C, MUL_IR, true>(p.gx1 + (int64_t)cur.snd * p.x1_stride + p.x1_off, p.extent, ch, gX, 0, pol_keep);
        }
      }
      if (p.need_gx2) {
        const float tot = reduce16(r, lane);
        if (!(lane & 1) && (lane >> 1) < p.nx2) atomicAdd(p.gx2 + (int64_t)eid * p.x2_stride + (lane >> 1), tot);
      }
      __syncwarp();
    }
  }
  wait_for_previous();
}

// ---- backward, one thread block per receiver ---------------------------------------------------
//
// Same arithmetic as cw_bwd_kernel with a different division of the work: the warps of a block
// share one receiver (its cotangent row is staged once per block instead of once per warp, which
// is what makes room in shared memory for four channels per thread at full occupancy) and deal
// the receiver's edges among themselves.  Nothing has to be combined afterwards, because every
// result of the backward pass belongs to an edge (weight gradient, x2 gradient) or is reduced in
// global memory anyway (x1 gradient).  A thread that owns four channels reads each broadcast
// entry of the per-edge matrices, issues each copy and computes each address once for four
// channels instead of two.
template <class G, int C, int P, bool MUL_IR, bool MASKED, class T>
struct StageGSplit {
  // the rows of the cotangent blocks are dealt round-robin to the warps of the block
  __device__ __forceinline__ static void run(Vec<C, T>* dst, const T* grow, const CwParamsT<T>& p, int ch, int lane, int warp) {
    constexpr int D = G::d3(P);
    const T* base = grow + p.out_off[P];
#pragma unroll
    for (int t = 0; t < D; ++t) {
      if (has_path<MASKED>(p, P) && (G::out_offset(P) + t) % kWarps == warp) {
        const T* src = MUL_IR ? base + (int64_t)ch * D + C * t : base + (int64_t)t * p.extent + ch;
        cp_async<(int)sizeof(T) * C>(dst + (G::out_offset(P) + t) * 32 + lane, src);
      }
    }
    if constexpr (P + 1 < G::NPATH) StageGSplit<G, C, P + 1, MUL_IR, MASKED, T>::run(dst, grow, p, ch, lane, warp);
  }
};

template <class T, class G, int C, bool MUL_IR, bool BULK_RED, bool NEED_GX2, bool MASKED>
__global__ void __launch_bounds__(kWarps * 32, sizeof(T) == 8 ? 2 : C == 2 ? 4 : 3) cw_bwd_block_kernel(const __grid_constant__ CwParamsT<T> p, const __grid_constant__ CwCoefT<T> coef) {
  let_next_start();
  // BULK_RED (mul_ir rows only): the x1 gradient of an edge - the 32 lanes' C*D1 values are one contiguous run of
  // the sender's row - leaves as ONE bulk reduction per warp and edge instead of D1 vector reductions per lane.
  // Its shared-memory source is the slot the edge's x1 block was staged in (free once X is in registers); the
  // slot is refilled two trips later, after the issuing lane has waited for the reduction to have read it.
  constexpr bool kBulk = BULK_RED && MUL_IR;
  extern __shared__ __align__(16) unsigned char smem_bytes[];
  T* smem = reinterpret_cast<T*>(smem_bytes);
  using S = Smem<G, C, T>;
  constexpr int kStage = S::kPerStage;
  constexpr int kPerWarp = S::kM + 2 * kStage;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Vec<C, T>* grow = reinterpret_cast<Vec<C, T>*>(smem);                 // shared by the block
  T* mine = smem + S::kGrow + warp * kPerWarp;                // per warp: M, two edge stages
  T* Msm = mine;
  T* stages = mine + S::kM;
  const int ch = blockIdx.y * (32 * C) + C * lane;
  const bool active = ch < p.extent;
  MTerms<G::NPAIR, T> mt;
  mt.load(p, lane);
  const unsigned long long pol_stream = policy_evict_first(), pol_keep = policy_evict_last();

  for (int n = blockIdx.x; n < p.num_receivers; n += gridDim.x) {
    const int beg = __ldg(p.rowptr + n), end = __ldg(p.rowptr + n + 1);
    if (beg >= end) continue;                                      // same decision in every thread of the block
    const int nrow = p.recv_mod ? n % p.recv_mod : n;
    if (kBulk) {                                                   // the last reduction of the previous receiver has left its slot
      if (lane == 0) bulk_wait_read();
      __syncwarp();
    }
    __syncthreads();                                               // everybody is done with the previous cotangent row
    if (active) StageGSplit<G, C, 0, MUL_IR, MASKED, T>::run(grow, p.gout + (int64_t)nrow * p.out_stride, p, ch, lane, warp);
    cp_async_commit();
    int pos = beg + warp;
    EdgeIds cur = {0, 0}, next = {0, 0}, ahead = {0, 0};
    if (pos < end) {
      next = load_ids(p, pos);
      issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages, next, ch, lane, active, pol_stream, pol_keep);
    } else {
      cp_async_commit();
    }
    if (pos + kWarps < end) ahead = load_ids(p, pos + kWarps);
    cp_async_wait<1>();                                            // this thread's share of the cotangent row has landed
    __syncthreads();                                               // ... and everybody else's
    for (int it = 0; pos < end; pos += kWarps, ++it) {
      T* st = stages + (it & 1) * kStage;
      cur = next;
      if (!kBulk) {
        if (pos + kWarps < end) {
          next = ahead;
          issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages + ((it + 1) & 1) * kStage, next, ch, lane, active, pol_stream, pol_keep);
          if (pos + 2 * kWarps < end) ahead = load_ids(p, pos + 2 * kWarps);   // used in the next trip
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
      } else {
        cp_async_wait<0>();                                          // the copies of this edge are the only ones in flight
      }
      const int eid = cur.eid;
      __syncwarp();
      mt.template compute<MASKED>(Msm, st, lane);
      __syncwarp();
      if (kBulk) {
        // the other slot is the source of the previous edge's reduction: refill it only after that has been read
        // (the matrices above were computed in the meantime)
        if (lane == 0) bulk_wait_read();
        __syncwarp();
        if (pos + kWarps < end) {
          next = ahead;
          issue_edge_ids<G, C, MUL_IR, MASKED>(p, stages + ((it + 1) & 1) * kStage, next, ch, lane, active, pol_stream, pol_keep);
          if (pos + 2 * kWarps < end) ahead = load_ids(p, pos + 2 * kWarps);
        }
      }
      T r[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = T(0);
      if (active) {
        const Vec<C, T>* stage = reinterpret_cast<const Vec<C, T>*>(st + S::kX2);
        T X[G::D1][C], gX[G::D1][C];
        unstage_block<G::D1, C, MUL_IR>(stage, lane, X);
#pragma unroll
        for (int i = 0; i < G::D1; ++i)
#pragma unroll
          for (int c = 0; c < C; ++c) gX[i][c] = T(0);
        BwdPaths<G, C, 0, MUL_IR, NEED_GX2, MASKED, T>::run(X, stage + G::D1 * 32, grow, lane, Msm, coef, p, p.gw + (int64_t)eid * p.w_stride + ch, gX, r);
        if (p.need_gx1 && !kBulk) {
          emit_block<G::D1, C, MUL_IR, true>(p.gx1 + (int64_t)cur.snd * p.x1_stride + p.x1_off, p.extent, ch, gX, 0, pol_keep);
        }
        if (p.need_gx1 && kBulk) {
          // the lane's C*D1 values in the order of the global row (channel-major), lane after lane
          T f[G::D1 * C];
#pragma unroll
          for (int i = 0; i < G::D1; ++i)
#pragma unroll
            for (int c = 0; c < C; ++c) f[c * G::D1 + i] = gX[i][c];
          __syncwarp();                                              // every lane has taken its X out of the slot
          Vec<C, T>* slot = reinterpret_cast<Vec<C, T>*>(st + S::kX2);
#pragma unroll
          for (int t = 0; t < G::D1; ++t) slot[lane * G::D1 + t] = make_vec<C>(f, C * t);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0)
            bulk_reduce_add(p.gx1 + (int64_t)cur.snd * p.x1_stride + p.x1_off + (int64_t)(blockIdx.y * 32 * C) * G::D1, slot,
                            (unsigned)(G::D1 * 32 * C * sizeof(T)), pol_keep);
        }
      }
      if (NEED_GX2) {
        const T tot = reduce16(r, lane);
        // a reduction without return value: the warp does not wait for it (a load-add-store would stall on the load)
        if (!(lane & 1) && (lane >> 1) < p.nx2) atomicAdd(p.gx2 + (int64_t)eid * p.x2_stride + (lane >> 1), tot);
      }
      __syncwarp();
    }
  }
  if (kBulk && lane == 0) bulk_wait_all();                           // shared memory stays allocated until the last reduction is done
  wait_for_previous();
}

// ---- launchers ----------------------------------------------------------------------------------
// The groups of one call read the same inputs and write different columns (the x2 gradient adds up), so a group need not
// wait for the one before it: its blocks fill the SMs that the other's last wave leaves idle.  Every kernel lets its
// successor start at once and ends only when its predecessor has, so that the end of the last group is the end of all.
// Only a launch that says so starts early; the first group of a call waits for everything before it as usual.
// 65,536 unsorted edges on 4,096 nodes, 128 channels, forward: 244 -> 220 us; 40,003 edges, 96 channels, lmax 2, forward and
// gradients: 402 -> 340 us.  Which groups of a backward call overlap: cw_kernels.cu, cueq_b200_cw_run.
template <class... Params, class... Args>
int launch_kernel(void (*kernel)(Params...), dim3 grid, size_t smem, cudaStream_t st, int overlap, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap == kFollows ? 1 : 0;
  CUEQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, args...));
  return 0;
}

int grid_x(int num_receivers) {
  const int want = (num_receivers + kWarps - 1) / kWarps;
  const int cap = 148 * 32;
  return want < 1 ? 1 : (want < cap ? want : cap);
}

template <class T, class G, int C, bool A, bool MASKED, bool OVERLAP>
int launch_fwd_o(const CwParamsT<T>& p, cudaStream_t st) {
  const size_t smem = Smem<G, C, T>::bytes_fwd();
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(cw_fwd_kernel<T, G, C, A, MASKED, OVERLAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.set();
  }
  dim3 grid(grid_x(p.num_receivers), (p.extent + 32 * C - 1) / (32 * C));
  return launch_kernel(cw_fwd_kernel<T, G, C, A, MASKED, OVERLAP>, grid, smem, st, p.overlap, p);
}
template <class T, class G, int C, bool A, bool MASKED>
int launch_fwd_t(const CwParamsT<T>& p, cudaStream_t st) {
  return p.overlap == kAlone ? launch_fwd_o<T, G, C, A, MASKED, false>(p, st) : launch_fwd_o<T, G, C, A, MASKED, true>(p, st);
}

template <class G, int C, bool A>
int launch_fwd_bulk_t(const CwParams& p, cudaStream_t st) {
  const size_t smem = SmemBulk<G, C>::bytes();
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(cw_fwd_bulk_kernel<G, C, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.set();
  }
  dim3 grid(grid_x(p.num_receivers), (p.extent + 32 * C - 1) / (32 * C));
  cw_fwd_bulk_kernel<G, C, A><<<grid, kWarps * 32, smem, st>>>(p);
  CUEQ_CUDA_OK(cudaGetLastError());
  return 0;
}

template <class G, bool MASKED>
int launch_fwd_m(const CwParams& p, int mul_ir, int cpl, cudaStream_t st) {
  if (cpl == 2) return mul_ir ? launch_fwd_t<float, G, 2, true, MASKED>(p, st) : launch_fwd_t<float, G, 2, false, MASKED>(p, st);
  return mul_ir ? launch_fwd_t<float, G, 4, true, MASKED>(p, st) : launch_fwd_t<float, G, 4, false, MASKED>(p, st);
}

template <class G>
int launch_fwd(const CwParams& p, int mul_ir, int cpl, bool masked, cudaStream_t st) {
  return masked ? launch_fwd_m<G, true>(p, mul_ir, cpl, st) : launch_fwd_m<G, false>(p, mul_ir, cpl, st);
}

template <class G>
int launch_fwd_bulk(const CwParams& p, int mul_ir, int cpl, cudaStream_t st) {
  if (cpl == 2) return mul_ir ? launch_fwd_bulk_t<G, 2, true>(p, st) : launch_fwd_bulk_t<G, 2, false>(p, st);
  return mul_ir ? launch_fwd_bulk_t<G, 4, true>(p, st) : launch_fwd_bulk_t<G, 4, false>(p, st);
}

template <class G, int C, bool A, bool MASKED>
int launch_bwd_t(const CwParams& p, const CwCoef& coef, cudaStream_t st) {
  const size_t smem = Smem<G, C>::bytes_bwd();
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(cw_bwd_kernel<G, C, A, MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.set();
  }
  dim3 grid(grid_x(p.num_receivers), (p.extent + 32 * C - 1) / (32 * C));
  return launch_kernel(cw_bwd_kernel<G, C, A, MASKED>, grid, smem, st, p.overlap, p, coef);
}

template <class G, bool MASKED>
int launch_bwd_m(const CwParams& p, const CwCoef& coef, int mul_ir, int cpl, cudaStream_t st) {
  if (cpl == 2) return mul_ir ? launch_bwd_t<G, 2, true, MASKED>(p, coef, st) : launch_bwd_t<G, 2, false, MASKED>(p, coef, st);
  return mul_ir ? launch_bwd_t<G, 4, true, MASKED>(p, coef, st) : launch_bwd_t<G, 4, false, MASKED>(p, coef, st);
}

template <class G>
int launch_bwd(const CwParams& p, const CwCoef& coef, int mul_ir, int cpl, bool masked, cudaStream_t st) {
  return masked ? launch_bwd_m<G, true>(p, coef, mul_ir, cpl, st) : launch_bwd_m<G, false>(p, coef, mul_ir, cpl, st);
}

template <class T, class G, int C, bool A, bool BULK, bool GX2, bool MASKED>
int launch_bwd_block_t(const CwParamsT<T>& p, const CwCoefT<T>& coef, cudaStream_t st) {
  using S = Smem<G, C, T>;
  const size_t smem = sizeof(T) * (S::kGrow + kWarps * S::kPerWarpFwd);
  static cueq::PerDeviceFlag configured;
  if (!configured.get()) {
    CUEQ_CUDA_OK(cudaFuncSetAttribute(cw_bwd_block_kernel<T, G, C, A, BULK, GX2, MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.set();
  }
  // blocks walk the receivers with a grid stride; many short-lived blocks (a few receivers each) let the hardware
  // balance the uneven edge counts better than eight waves of long ones (l = 3 launch 3.48 -> 3.40 ms)
  const int cap = 148 * 96;
  dim3 grid(p.num_receivers < cap ? p.num_receivers : cap, (p.extent + 32 * C - 1) / (32 * C));
  return launch_kernel(cw_bwd_block_kernel<T, G, C, A, BULK, GX2, MASKED>, grid, smem, st, p.overlap, p, coef);
}

// bulk: the x1 gradient leaves as one bulk reduction per warp and edge; needs mul_ir rows whose blocks start on
// 16-byte boundaries (checked here: a misaligned bulk operation is an illegal instruction, not an error code)
template <class T, class G, int C, bool MASKED>
int launch_bwd_block_m(const CwParamsT<T>& p, const CwCoefT<T>& coef, int mul_ir, int bulk, cudaStream_t st) {
  constexpr int V = 16 / (int)sizeof(T);
  const bool aligned = (reinterpret_cast<uintptr_t>(p.gx1) % 16 == 0) && (p.x1_stride % V == 0) && (p.x1_off % V == 0) && (p.extent % (32 * C) == 0);
  // the x2-gradient partials are a third of the arithmetic: a launch that does not need them runs without
  if (bulk && mul_ir && p.need_gx1 && aligned)
    return p.need_gx2 ? launch_bwd_block_t<T, G, C, true, true, true, MASKED>(p, coef, st) : launch_bwd_block_t<T, G, C, true, true, false, MASKED>(p, coef, st);
  if (mul_ir) return p.need_gx2 ? launch_bwd_block_t<T, G, C, true, false, true, MASKED>(p, coef, st) : launch_bwd_block_t<T, G, C, true, false, false, MASKED>(p, coef, st);
  return p.need_gx2 ? launch_bwd_block_t<T, G, C, false, false, true, MASKED>(p, coef, st) : launch_bwd_block_t<T, G, C, false, false, false, MASKED>(p, coef, st);
}

template <class G>
int launch_bwd_block(const CwParams& p, const CwCoef& coef, int mul_ir, int cpl, int bulk, bool masked, cudaStream_t st) {
  if (cpl == 2) return masked ? launch_bwd_block_m<float, G, 2, true>(p, coef, mul_ir, bulk, st) : launch_bwd_block_m<float, G, 2, false>(p, coef, mul_ir, bulk, st);
  return masked ? launch_bwd_block_m<float, G, 4, true>(p, coef, mul_ir, bulk, st) : launch_bwd_block_m<float, G, 4, false>(p, coef, mul_ir, bulk, st);
}

// float64: two channels per thread, one form of each kernel (it walks the path mask whether or not all paths are there)
template <class G>
int launch_fwd_f64(const CwParamsT<double>& p, int mul_ir, cudaStream_t st) {
  return mul_ir ? launch_fwd_t<double, G, 2, true, true>(p, st) : launch_fwd_t<double, G, 2, false, true>(p, st);
}
template <class G>
int launch_bwd_f64(const CwParamsT<double>& p, const CwCoefT<double>& coef, int mul_ir, cudaStream_t st) {
  return launch_bwd_block_m<double, G, 2, true>(p, coef, mul_ir, 1, st);
}

}  // namespace

#define CW_DEFINE_GROUP(NAME, G)                                                                                            \
  static_assert(G::NTERM <= cueq::cw::kMaxTerms && G::NPATH <= cueq::cw::kMaxPaths, "group tables");                        \
  namespace cueq { namespace cw {                                                                                           \
  const GroupEntry NAME = {G::signature(), G::D1, G::NPATH, G::NPAIR, G::NTERM, G::SUMD3, G::NX2, G::NVAL, G::NTERM_FWD,     \
                           &launch_fwd<G>, &launch_bwd<G>, &launch_fwd_bulk<G>, &launch_bwd_block<G>};                      \
  } }
#define CW_DEFINE_GROUP_F64(NAME, G)                                                                                        \
  namespace cueq { namespace cw {                                                                                           \
  const GroupEntry64 NAME = {&launch_fwd_f64<G>, &launch_bwd_f64<G>};                                                       \
  } }
