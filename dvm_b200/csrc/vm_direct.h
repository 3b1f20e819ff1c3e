// Launch description of the direct kernel (vm_direct.cu): reduce-free programs over dense tensors, run without staging.
#ifndef DVM_B200_VM_DIRECT_H_
#define DVM_B200_VM_DIRECT_H_

#include <cstdint>

#include "isa.h"

namespace dvmb {

constexpr int kDirectTensors = 6;   // inputs and results together
constexpr int kDirectInputs = 4;
constexpr int kDirectTemps = 2;
constexpr int kDirectCode = 48;

struct DirectParam {
  uint32_t elems;               // 0: the stage is not one of this kernel's
  uint32_t n_in, n_tensors;     // inputs come first
  uint8_t dtype[8];
  uint64_t ptr[kDirectTensors];
  uint8_t slot[8];              // tensor slots of the stage they were matched from
  uint64_t code[kDirectCode];   // instruction words (isa.h), tensors renumbered, ending with OP_END
};

int LaunchDirect(const DirectParam &p, void *stream);

}  // namespace dvmb

#endif  // DVM_B200_VM_DIRECT_H_
