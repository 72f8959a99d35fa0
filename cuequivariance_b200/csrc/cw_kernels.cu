// Channelwise ("uvu") tensor product: the C entry points (argument checks, dispatch between the kernels of
// cw_kernels.cuh, which each group of paths instantiates in a file of its own).
#include <cstdint>
#include <cstring>

#include "common.cuh"
#include "cw_entry.h"

namespace {

using namespace cueq::cw;

const GroupEntry* const kGroups[] = {&kGroupL0, &kGroupL1, &kGroupL2, &kGroupL3};
const GroupEntry64* const kGroups64[] = {&kGroupL0F64, &kGroupL1F64, &kGroupL2F64, &kGroupL3F64};
constexpr int kNumGroups = sizeof(kGroups) / sizeof(kGroups[0]);

// Channels per thread of the kernels with a warp per receiver.  Four hold up to 132 accumulators per thread and spill; with
// two a warp has 64 channels, which is all there are where this matters.  Path subsets take two: 40,000 edges, 4 channels,
// lmax 2, forward, 20 edges per receiver 152 -> 83 us (117 us on the table-driven kernel they came from), one edge 171 -> 84
// us (258).  Whole groups of fewer than 64 channels keep four.
int pick_cpl(const cueq_cw_args* a, bool masked) {
  if (a->channels_per_lane == 2 || a->channels_per_lane == 4) return a->channels_per_lane;
  return masked || a->extent >= 64 ? 2 : 4;
}

// A polynomial with all paths of the group and 16-element x2 rows takes the kernels that know so at compile time and copy a
// row 16 bytes at a time; rows at another pitch (harmonics beyond l = 3 that no path reads) go element by element as well.
template <class T>
bool is_masked(const CwParamsT<T>& p, const GroupEntry& g) { return p.path_mask != (1u << g.npath) - 1u || p.nx2 != g.nx2 || (p.x2_stride & 3); }

template <class T>
int fill_params(const cueq_cw_args* a, const cueq_cw_options& o, const GroupEntry& g, CwParamsT<T>& p, int expected_terms) {
  constexpr int V = 16 / (int)sizeof(T);   // elements per 16-byte access
  if (!a) return cueq::fail("channelwise: null arguments");
  if (a->extent < V || a->extent % V) return cueq::fail("channelwise: extent %d must be a positive multiple of %d", a->extent, V);
  if (a->x1_mul_ir != a->out_mul_ir) return cueq::fail("channelwise: x1 and out must use the same layout");
  if (a->staging != 0 && a->staging != 1) return cueq::fail("channelwise: staging must be 0 (cp.async) or 1 (bulk copy)");
  if (a->channels_per_lane != 0 && a->channels_per_lane != 2 && a->channels_per_lane != 4)
    return cueq::fail("channelwise: channels_per_lane must be 0 (auto), 2 or 4");
  if (a->num_paths != g.npath) return cueq::fail("channelwise: group has %d paths, got %d", g.npath, a->num_paths);
  if (a->num_terms != expected_terms) return cueq::fail("channelwise: this call's table has %d terms, got %d", expected_terms, a->num_terms);
  if (!a->rowptr || !a->tab_start || !a->tab_j || !a->tab_c) return cueq::fail("channelwise: null table or rowptr");
  if (a->num_receivers < 0) return cueq::fail("channelwise: negative receiver count");
  std::memset(&p, 0, sizeof(p));
  p.w = (const T*)a->w; p.x1 = (const T*)a->x1; p.x2 = (const T*)a->x2; p.out = (T*)a->out;
  p.gout = (const T*)a->gout; p.gw = (T*)a->gw; p.gx1 = (T*)a->gx1; p.gx2 = (T*)a->gx2;
  p.senders = a->senders; p.order = a->order; p.rowptr = a->rowptr;
  p.tab_start = a->tab_start; p.tab_j = a->tab_j; p.tab_c = (const T*)a->tab_c;
  p.w_stride = a->w_stride; p.x1_stride = a->x1_stride; p.x2_stride = a->x2_stride; p.out_stride = a->out_stride;
  p.num_receivers = (int)a->num_receivers; p.extent = a->extent; p.x1_off = a->x1_offset;
  for (int q = 0; q < g.npath; ++q) {
    p.w_off[q] = a->w_offset[q];
    p.out_off[q] = a->out_offset[q];
    if ((p.w_off[q] | p.out_off[q]) & (V - 1)) return cueq::fail("channelwise: segment offsets must be multiples of %d elements", V);
  }
  if (p.x1_off & (V - 1)) return cueq::fail("channelwise: x1 offset must be a multiple of %d elements", V);
  if ((p.w_stride | p.x1_stride | p.out_stride) & (V - 1)) return cueq::fail("channelwise: row strides must be multiples of %d elements", V);
  const uintptr_t ptrs = (uintptr_t)a->w | (uintptr_t)a->x1 | (uintptr_t)a->x2 | (uintptr_t)a->out | (uintptr_t)a->gout | (uintptr_t)a->gw | (uintptr_t)a->gx1;
  const unsigned all = (1u << g.npath) - 1u;
  p.path_mask = o.path_mask ? (unsigned)o.path_mask : all;
  p.nx2 = o.x2_width ? o.x2_width : g.nx2;
  if ((p.path_mask & ~all) || p.nx2 < 1 || p.nx2 > g.nx2) return cueq::fail("channelwise: path mask or x2 width outside the group");
  if (ptrs & 15) return cueq::fail("channelwise: tensors must be 16-byte aligned");
  p.need_gw = a->gw != nullptr; p.need_gx1 = a->gx1 != nullptr; p.need_gx2 = a->gx2 != nullptr;
  return 0;
}

}  // namespace

extern "C" int cueq_b200_cw_num_groups(void) { return kNumGroups; }

extern "C" const char* cueq_b200_cw_group_signature(int g) { return (g >= 0 && g < kNumGroups) ? kGroups[g]->signature : nullptr; }

extern "C" int cueq_b200_cw_group_info(int g, int32_t* d1, int32_t* npath, int32_t* npair, int32_t* nterm) {
  if (g < 0 || g >= kNumGroups) return cueq::fail("channelwise: group %d out of range", g);
  if (d1) *d1 = kGroups[g]->d1;
  if (npath) *npath = kGroups[g]->npath;
  if (npair) *npair = kGroups[g]->npair;
  if (nterm) *nterm = kGroups[g]->nterm;
  return 0;
}

namespace {

int take_options(const cueq_cw_options* options, cueq_cw_options& o) {
  std::memset(&o, 0, sizeof(o));
  if (!options) return 0;
  if (options->struct_bytes != (int)sizeof(o)) return cueq::fail("channelwise: the binding declares another options block");
  o = *options;
  return 0;
}

int run_forward(int g, const cueq_cw_args* a, const cueq_cw_options& o, int overlap, void* stream) {
  if (g < 0 || g >= kNumGroups) return cueq::fail("channelwise: group %d out of range", g);
  if (o.dtype == CUEQ_F64) {
    CwParamsT<double> p;
    if (int rc = fill_params(a, o, *kGroups[g], p, kGroups[g]->nterm_fwd)) return rc;
    p.overlap = overlap;
    if (!p.w || !p.x1 || !p.x2 || !p.out) return cueq::fail("channelwise forward: null tensor");
    return p.num_receivers == 0 ? 0 : kGroups64[g]->fwd(p, a->x1_mul_ir, reinterpret_cast<cudaStream_t>(stream));
  }
  if (o.dtype != CUEQ_F32) return cueq::fail("channelwise: float32 or float64 operands");
  CwParams p;
  if (int rc = fill_params(a, o, *kGroups[g], p, kGroups[g]->nterm_fwd)) return rc;
  p.overlap = overlap;
  if (!p.w || !p.x1 || !p.x2 || !p.out) return cueq::fail("channelwise forward: null tensor");
  if (p.num_receivers == 0) return 0;
  p.status = reinterpret_cast<int*>(a->status);
  if (a->variant < 0 || a->variant > 2) return cueq::fail("channelwise: variant must be 0 (automatic), 1 or 2");
  const bool masked = is_masked(p, *kGroups[g]);
  if (a->staging == 1 && !masked) return kGroups[g]->fwd_bulk(p, a->x1_mul_ir, pick_cpl(a, false), reinterpret_cast<cudaStream_t>(stream));
  return kGroups[g]->fwd(p, a->x1_mul_ir, pick_cpl(a, masked), masked, reinterpret_cast<cudaStream_t>(stream));
}

int run_backward(int g, const cueq_cw_args* a, const cueq_cw_options& o, int overlap, void* stream) {
  if (g < 0 || g >= kNumGroups) return cueq::fail("channelwise: group %d out of range", g);
  if (o.dtype == CUEQ_F64) {
    CwParamsT<double> p;
    if (int rc = fill_params(a, o, *kGroups[g], p, kGroups[g]->nterm)) return rc;
    p.overlap = overlap;
    if (!p.w || !p.x1 || !p.x2 || !p.gout) return cueq::fail("channelwise backward: null tensor");
    if (!a->bwd_coef) return cueq::fail("channelwise backward: null coefficient table");
    p.recv_mod = a->recv_mod;
    CwCoefT<double> coef = {};
    for (int t = 0; t < kGroups[g]->nterm; ++t) coef.c[t] = static_cast<const double*>(a->bwd_coef)[t];
    return p.num_receivers == 0 ? 0 : kGroups64[g]->bwd(p, coef, a->x1_mul_ir, reinterpret_cast<cudaStream_t>(stream));
  }
  if (o.dtype != CUEQ_F32) return cueq::fail("channelwise: float32 or float64 operands");
  CwParams p;
  if (int rc = fill_params(a, o, *kGroups[g], p, kGroups[g]->nterm)) return rc;
  p.overlap = overlap;
  if (!p.w || !p.x1 || !p.x2 || !p.gout) return cueq::fail("channelwise backward: null tensor");
  if (!a->bwd_coef) return cueq::fail("channelwise backward: null coefficient table");
  if (p.num_receivers == 0) return 0;
  p.recv_mod = a->recv_mod;
  CwCoef coef;
  std::memset(&coef, 0, sizeof(coef));
  for (int t = 0; t < kGroups[g]->nterm; ++t) coef.c[t] = static_cast<const float*>(a->bwd_coef)[t];
  if (a->variant < 0 || a->variant > 3) return cueq::fail("channelwise backward: variant must be 0 (automatic), 1, 2 or 3");
  // One thread block per receiver, four channels per thread where a warp's 128 channels are all in use, else two.  With two
  // and few edges per receiver the cotangent row is staged by a block for too little work; 100,000 edges, lmax 3, one warp
  // against one block per receiver: 64 channels, 20 edges 680 / 536 us, 5 edges 720 / 757 us; 32 channels, 5 edges
  // 1371 / 687 us; 2,000 edges on 100 receivers, 64 channels: 153 / 51 us.
  // Up to 32 channels the same holds for receivers of one edge (calls without a receiver index among them) only; 50,000 edges,
  // lmax 2 x 3 -> 3, warp against block: 32 channels, one edge 804 / 972 us, two 645 / 644 us, four 568 / 479 us; 4 channels,
  // one edge 675 / 853 us.
  const bool few = o.mean_degree > 0 && o.mean_degree < (a->extent > 32 ? 8 : 2) && a->extent % 128;
  const bool masked = is_masked(p, *kGroups[g]);
  const bool block_per_receiver = a->variant >= 2 || (a->variant == 0 && a->channels_per_lane != 2 && !few);
  if (a->variant == 3 && a->extent % 128) return cueq::fail("channelwise backward: variant 3 needs a multiple of 128 channels");
  // bulk reductions pay from three components per channel on (one 1.5 KB operation instead of three vector
  // reductions per lane); for the scalar block (512 bytes per edge) the vector reductions are faster
  const bool bulk = a->variant == 3 || (a->variant == 0 && kGroups[g]->d1 >= 3);
  if (block_per_receiver)
    return kGroups[g]->bwd_block(p, coef, a->x1_mul_ir, a->variant >= 2 || a->extent % 128 == 0 ? 4 : 2, bulk, masked, reinterpret_cast<cudaStream_t>(stream));
  return kGroups[g]->bwd(p, coef, a->x1_mul_ir, pick_cpl(a, masked), masked, reinterpret_cast<cudaStream_t>(stream));
}

}  // namespace

extern "C" int cueq_b200_cw_forward_opt(int g, const cueq_cw_args* a, const cueq_cw_options* options, void* stream) {
  cueq_cw_options o;
  if (int rc = take_options(options, o)) return rc;
  return run_forward(g, a, o, kAlone, stream);
}
extern "C" int cueq_b200_cw_backward_opt(int g, const cueq_cw_args* a, const cueq_cw_options* options, void* stream) {
  cueq_cw_options o;
  if (int rc = take_options(options, o)) return rc;
  return run_backward(g, a, o, kAlone, stream);
}
extern "C" int cueq_b200_cw_forward(int g, const cueq_cw_args* a, void* stream) { return cueq_b200_cw_forward_opt(g, a, nullptr, stream); }
extern "C" int cueq_b200_cw_backward(int g, const cueq_cw_args* a, void* stream) { return cueq_b200_cw_backward_opt(g, a, nullptr, stream); }

// All groups of a polynomial by one call: the constant part of each group's arguments comes from `templates`, which the
// caller keeps, tensors and sizes from `call`.  Every group but the first may start before the one in front of it has
// ended (cw_kernels.cuh, launch_kernel), unless that would leave the x2 gradient's sum in no fixed order: where one block of
// channels holds them all, a group adds one value to a component, the first two in either order (0 + a + b), the others
// each after the groups before.  Several blocks of channels add in no fixed order anyway.  Forward calls overlap up to
// kOverlapBytes of weights: beyond, what the tails of the groups give is less than the 5 % that the kernels cost for it.
// 128 channels, lmax 3, forward, without / with overlap: 65,536 edges 334 / 300 us, 262,144 1070 / 1061 us, 1,048,576 3977 / 4128 us.
constexpr long long kOverlapBytes = 3500000000LL;
extern "C" int cueq_b200_cw_run(int backward, int num_groups, const int32_t* groups, const cueq_cw_args* templates, const cueq_cw_options* options,
                                const cueq_cw_args* call, int32_t mean_degree, void* stream) {
  if (num_groups < 0 || (num_groups && (!groups || !templates || !options || !call))) return cueq::fail("channelwise: null argument");
  for (int i = 0; i < num_groups; ++i) {
    cueq_cw_args a = templates[i];
    cueq_cw_options o;
    if (int rc = take_options(options + i, o)) return rc;
    o.mean_degree = mean_degree;
    a.w = call->w; a.x1 = call->x1; a.x2 = call->x2; a.out = call->out;
    a.gout = call->gout; a.gw = call->gw; a.gx1 = call->gx1; a.gx2 = call->gx2;
    a.senders = call->senders; a.order = call->order; a.rowptr = call->rowptr;
    a.num_receivers = call->num_receivers; a.recv_mod = call->recv_mod;
    a.x1_mul_ir = call->x1_mul_ir; a.out_mul_ir = call->out_mul_ir;
    const bool chain = backward || (call->num_receivers * (mean_degree + 1LL)) * a.w_stride * (o.dtype == CUEQ_F64 ? 8 : 4) <= kOverlapBytes;
    const bool one_block = a.extent <= (o.dtype == CUEQ_F32 && a.extent % 128 == 0 ? 128 : 64);
    const int overlap = !chain ? kAlone : i > 0 && !(backward && a.gx2 && one_block && i > 1) ? kFollows : kStarts;
    if (int rc = backward ? run_backward(groups[i], &a, o, overlap, stream) : run_forward(groups[i], &a, o, overlap, stream)) return rc;
  }
  return 0;
}

// ---- forward without caller-provided scratch ----------------------------------------------------
//
// cueq_b200_cw_forward needs two pieces of device memory besides its inputs and outputs: the
// CSR row pointers over receivers and the term tables.  Some hosts of this library cannot
// provide them: code that runs where device allocation is forbidden or owned by someone else
// (an inference-engine plugin whose enqueue call gets only its input and output bindings, a
// callback running inside a memory pool it must not grow, a real-time loop that may not call
// the allocator).  For those there is one entry point whose scratch lives in a fixed array
// inside the library image.  The array exists once per GPU that loads the library, for the
// life of the process, and every call reuses it.
namespace {

constexpr int kNoAllocMaxReceivers = 262144;   // row pointers: (N + 1) * 4 bytes = 1 MiB
constexpr int kNoAllocMaxPairs = 256;
constexpr int kNoAllocMaxTerms = 256;
constexpr size_t kScratchRowptr = 0;
constexpr size_t kScratchTabStart = ((size_t)(kNoAllocMaxReceivers + 1) * 4 + 255) & ~size_t(255);
constexpr size_t kScratchTabJ = kScratchTabStart + ((kNoAllocMaxPairs + 1) * 4 + 255) / 256 * 256;
constexpr size_t kScratchTabC = kScratchTabJ + (kNoAllocMaxTerms * 4 + 255) / 256 * 256;
constexpr size_t kScratchBytes = kScratchTabC + (kNoAllocMaxTerms * 4 + 255) / 256 * 256;

// Host code may only use this name with cudaGetSymbolAddress: as a plain expression it is the
// host-side shadow of the symbol, not a device address.
static __device__ __align__(256) unsigned char g_cw_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
void* g_scratch_ptr[kMaxDevices] = {nullptr};

struct NoAllocTables {
  int start[kNoAllocMaxPairs + 1];
  int j[kNoAllocMaxTerms];
  float c[kNoAllocMaxTerms];
};

// rowptr[r] = first position whose receiver is >= r (receivers sorted ascending); also copies
// the term tables from the kernel parameters into the scratch array
__global__ void cw_noalloc_prepare(const int* __restrict__ receivers, int num_edges, int num_receivers, int* __restrict__ rowptr,
                                   const __grid_constant__ NoAllocTables t, int npair, int nterm, int* tab_start, int* tab_j,
                                   float* tab_c) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  for (int r = gid; r <= num_receivers; r += gridDim.x * blockDim.x) {
    int lo = 0, hi = num_edges;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(receivers + mid) < r) lo = mid + 1; else hi = mid;
    }
    rowptr[r] = lo;
  }
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i <= npair; i += blockDim.x) tab_start[i] = t.start[i];
    for (int i = threadIdx.x; i < nterm; i += blockDim.x) { tab_j[i] = t.j[i]; tab_c[i] = t.c[i]; }
  }
}

}  // namespace

extern "C" int cueq_b200_cw_forward_noalloc(int g, const cueq_cw_noalloc_args* a, void* stream) {
  if (g < 0 || g >= kNumGroups) return cueq::fail("channelwise (no-alloc): group %d out of range", g);
  if (!a) return cueq::fail("channelwise (no-alloc): null arguments");
  const GroupEntry& ge = *kGroups[g];
  if (a->num_receivers > kNoAllocMaxReceivers)
    return cueq::fail("channelwise (no-alloc): %lld receivers exceed the built-in scratch (max %d); use cueq_b200_cw_forward",
                      (long long)a->num_receivers, kNoAllocMaxReceivers);
  if (ge.nval > kNoAllocMaxPairs || ge.nterm_fwd > kNoAllocMaxTerms)
    return cueq::fail("channelwise (no-alloc): group tables exceed the built-in scratch");
  if (a->num_edges < 0 || a->num_edges > 2147483647LL) return cueq::fail("channelwise (no-alloc): invalid edge count");
  if (!a->receivers && a->num_edges > 0) return cueq::fail("channelwise (no-alloc): null receivers");
  if (!a->tab_start_host || !a->tab_j_host || !a->tab_c_host) return cueq::fail("channelwise (no-alloc): null host table");

  int dev = 0;
  CUEQ_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return cueq::fail("channelwise (no-alloc): device ordinal %d not supported", dev);
  if (!g_scratch_ptr[dev]) {  // set-up, once per device, with that device current
    void* ptr = nullptr;
    CUEQ_CUDA_OK(cudaGetSymbolAddress(&ptr, g_cw_scratch));
    g_scratch_ptr[dev] = ptr;
  }
  unsigned char* scratch = static_cast<unsigned char*>(g_scratch_ptr[dev]);
  int* rowptr = reinterpret_cast<int*>(scratch + kScratchRowptr);
  int* tab_start = reinterpret_cast<int*>(scratch + kScratchTabStart);
  int* tab_j = reinterpret_cast<int*>(scratch + kScratchTabJ);
  float* tab_c = reinterpret_cast<float*>(scratch + kScratchTabC);

  cueq_cw_args full;
  std::memset(&full, 0, sizeof(full));
  full.w = a->w; full.x1 = a->x1; full.x2 = a->x2; full.out = a->out;
  full.senders = a->senders; full.order = nullptr; full.rowptr = rowptr;
  full.tab_start = tab_start; full.tab_j = tab_j; full.tab_c = tab_c;
  full.w_stride = a->w_stride; full.x1_stride = a->x1_stride; full.x2_stride = a->x2_stride; full.out_stride = a->out_stride;
  full.num_receivers = a->num_receivers; full.extent = a->extent; full.x1_offset = a->x1_offset;
  full.num_paths = a->num_paths; full.num_terms = a->num_terms;
  for (int q = 0; q < 8; ++q) { full.w_offset[q] = a->w_offset[q]; full.out_offset[q] = a->out_offset[q]; }
  full.x1_mul_ir = a->mul_ir; full.out_mul_ir = a->mul_ir; full.channels_per_lane = 0;
  const cueq_cw_options whole = {};
  CwParams p;
  if (int rc = fill_params(&full, whole, ge, p, ge.nterm_fwd)) return rc;
  if (!p.w || !p.x1 || !p.x2 || !p.out) return cueq::fail("channelwise (no-alloc): null tensor");
  if (p.num_receivers == 0) return 0;

  NoAllocTables t;
  std::memset(&t, 0, sizeof(t));
  for (int i = 0; i <= ge.nval; ++i) t.start[i] = a->tab_start_host[i];
  for (int i = 0; i < ge.nterm_fwd; ++i) { t.j[i] = a->tab_j_host[i]; t.c[i] = a->tab_c_host[i]; }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int blocks = (int)((a->num_receivers + 1 + 255) / 256);
  cw_noalloc_prepare<<<blocks < 1 ? 1 : blocks, 256, 0, st>>>(a->receivers, (int)a->num_edges, (int)a->num_receivers, rowptr, t, ge.nval,
                                                              ge.nterm_fwd, tab_start, tab_j, tab_c);
  CUEQ_CUDA_OK(cudaGetLastError());
  return ge.fwd(p, a->mul_ir, pick_cpl(&full, is_masked(p, ge)), is_masked(p, ge), st);
}
