// Launch description of the row kernels (vm_row.cu): the two normalisation shapes of a vector stage that run as straight-line
// kernels instead of through the vector interpreter.
#ifndef DVM_B200_VM_ROW_H_
#define DVM_B200_VM_ROW_H_

#include <cstdint>

#include "isa.h"

namespace dvmb {

constexpr int kRowMaxStreams = 7;     // tensors walked element by element
constexpr int kRowMaxScalars = 8;     // group scalars in memory (inputs and results of the scalar sections)
constexpr uint32_t kRowNone = 0xffu;
constexpr uint32_t kRowRmsMaxElems = 8192;   // longest row of ROW_RMS_GATE: it stays in a CTA's registers

enum RowForm : uint32_t {
  ROW_OFF = 0,
  // sums of d = x - s and of d * d over a group of runs, then ((x - s0) * s1) * s2 + s3 stored in x's type
  ROW_STATS_AFFINE,
  // sum of (a + b)^2 over a row, then ((a + b) * s) * w stored; beside it ((sigmoid(g)) * g) * u stored
  ROW_RMS_GATE
};

struct RowStream {
  uint64_t ptr;
  uint32_t kstride[kMaxKept];   // element strides along the group's coordinates
  uint32_t slot;                // tensor slot of the stage it was matched from
};

struct RowParam {
  uint32_t form;
  uint32_t dtype;               // of every stream (16-bit)
  uint32_t groups, kept_size[kMaxKept];
  uint32_t runs, run_len, run_stride;   // a group is `runs` runs of `run_len` elements, `run_stride` elements apart
  // set by the launcher
  uint32_t slots_per_run;       // 16-byte units a run touches (at most)
  uint32_t cluster, per_cta;    // CTAs per group and units per CTA
  uint32_t buffers, buffer_bytes;      // shared-memory copies of a CTA's share: this group's and the next one's
  uint32_t tg;                  // ROW_RMS_GATE: threads per row
  // ROW_STATS_AFFINE: streams 0 = x, 1 = result.  ROW_RMS_GATE: a, b, w, result 1, g, u, result 2
  RowStream stream[kRowMaxStreams];
  uint32_t have_b, have_w, have_gate;
  // the scalar sections in closed form (row_match.cc follows the words symbolically)
  //   ROW_STATS_AFFINE: m = T i1 + s, v = (Q - T (T i1)) i2, x' = ((x - m) / sqrt(v + eps)) * gamma + beta, m and v stored
  //   ROW_RMS_GATE: scale = 1 / sqrt(S i1 + eps)
  float i1, i2, eps;
  uint32_t at_shift, at_gamma, at_beta, at_mean, at_var;   // entries of scalar[] (kRowNone: absent)
  TensorDesc scalar[kRowMaxScalars];
  uint8_t scalar_of[kMaxTensors];       // tensor slot -> entry of scalar[]
  uint32_t n_scalars;
};
static_assert(sizeof(RowParam) <= 4000, "RowParam is a kernel parameter");

// True when the addresses now in `p` allow the row kernels: the streams of a group lie alike relative to 16 bytes.
bool RowAddressesOk(const RowParam &p);
// True when the row kernel is estimated to be faster than the interpreter, which works on chunks of `chunk_elems` elements.
bool RowKernelPays(const RowParam &p, uint32_t chunk_elems);
unsigned int ReadRowStatus();
// Enqueue.  Returns the cudaError_t of the launch.
int LaunchRow(const RowParam &p, void *stream);

}  // namespace dvmb

#endif  // DVM_B200_VM_ROW_H_
