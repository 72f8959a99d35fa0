// What the translation units of the channelwise kernels share: the launch parameters and the table of launchers
// (one entry per group of paths; each group is instantiated in a file of its own).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cueq {
namespace cw {

constexpr int kMaxPaths = 8;
constexpr int kMaxTerms = 160;

// A launch by itself; the first of a chain of groups that overlap, or one that waits for all before it; one that may start
// while the group before it, in the chain too, still runs.
enum { kAlone = 0, kStarts = 1, kFollows = 2 };

template <class T>
struct CwCoefT {
  T c[kMaxTerms];
};
using CwCoef = CwCoefT<float>;

template <class T>
struct CwParamsT {
  const T* w;
  const T* x1;
  const T* x2;
  T* out;          // forward output / unused in backward
  const T* gout;   // backward: cotangent of out
  T* gw;
  T* gx1;
  T* gx2;
  const int* senders;  // [E] row of x1 for each edge (edge ids, not CSR positions); null: edge id
  const int* order;    // [E] CSR position -> edge id; null: identity
  const int* rowptr;   // [num_receivers + 1]
  const int* tab_start;  // [NPAIR + 1] term range of every (i,k) pair
  const int* tab_j;      // [NTERM] x2 element of the term
  const T* tab_c;        // [NTERM] coefficient of the term
  int64_t w_stride, x1_stride, x2_stride, out_stride;
  int num_receivers;
  int extent;
  int x1_off;               // element offset of the group's irrep block inside an x1 row
  int w_off[kMaxPaths];     // element offset of each path's weight segment inside a w row
  int out_off[kMaxPaths];   // element offset of each path's output block inside an out row
  int need_gw, need_gx1, need_gx2;
  int* status;              // nullable: set to 1 if a bounded wait on a bulk copy ran out
  int recv_mod;             // backward: CSR rows are (pass, receiver) pairs; the cotangent row is row % recv_mod (0: off)
  unsigned path_mask;       // bit q: path q of the group belongs to the polynomial (MASKED kernels)
  int nx2;                  // components of an x2 row (MASKED kernels; 16 otherwise)
  int overlap;              // launch: kAlone, kStarts or kFollows
};
using CwParams = CwParamsT<float>;

// Launchers of one group.  `masked`: the polynomial has only the paths of `path_mask` or x2 rows narrower than 16.
struct GroupEntry {
  const char* signature;
  int d1, npath, npair, nterm, sumd3, nx2, nval, nterm_fwd;
  int (*fwd)(const CwParams&, int mul_ir, int cpl, bool masked, cudaStream_t);
  int (*bwd)(const CwParams&, const CwCoef&, int mul_ir, int cpl, bool masked, cudaStream_t);
  int (*fwd_bulk)(const CwParams&, int mul_ir, int cpl, cudaStream_t);
  int (*bwd_block)(const CwParams&, const CwCoef&, int mul_ir, int cpl, int bulk, bool masked, cudaStream_t);
};
struct GroupEntry64 {
  int (*fwd)(const CwParamsT<double>&, int mul_ir, cudaStream_t);
  int (*bwd)(const CwParamsT<double>&, const CwCoefT<double>&, int mul_ir, cudaStream_t);
};

extern const GroupEntry kGroupL0, kGroupL1, kGroupL2, kGroupL3;
extern const GroupEntry64 kGroupL0F64, kGroupL1F64, kGroupL2F64, kGroupL3F64;

}  // namespace cw
}  // namespace cueq
