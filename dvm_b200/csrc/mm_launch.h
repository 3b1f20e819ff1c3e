// Host-callable entry points of the tensor-core kernels (MatMul with fused post-ops, fused attention).
#ifndef DVM_B200_MM_LAUNCH_H_
#define DVM_B200_MM_LAUNCH_H_

#include <cuda.h>

#include <cstdint>

#include "isa.h"

namespace dvmb {

constexpr int kMmMaxEpilogueWords = 96;
constexpr int kMmMaxEpiTensors = 8;

// A tensor the post-fusion program reads or writes, addressed by (batch0, batch1, row, column) of the
// MatMul result.  A stride of 0 broadcasts along that coordinate.
struct EpiTensor {
  uint64_t ptr;
  int64_t sb0, sb1;   // element strides along the two batch coordinates
  int64_t sm;         // element stride along rows
  int32_t sn;         // element stride along columns (0 or 1 for the vector paths)
  uint32_t dtype;
};

// One batched MatMul  C[b0,b1] = op(A[..]) * op(B[..]) (+ bias), rounded to the operand type, followed by the
// fused post-ops.  Batch coordinates: b = b0 * batch1 + b1; an operand's batch slice is
// z = b0 * mul0 + b1 * mul1 (multipliers 0 broadcast the operand).
struct MmParam {
  uint32_t M, N, K;
  uint32_t batch0, batch1;
  uint32_t a_mmajor;        // 1: A is stored [K, M] (trans_a), 0: A is stored [M, K]
  uint32_t b_kmajor;        // 1: B is stored [N, K] (trans_b), 0: B is stored [K, N]
  uint32_t in_dtype;        // T_F16 or T_BF16: operand type and the type the product is rounded to
  uint32_t bias_dtype;      // element type of bias (ignored when bias_ptr == 0)
  uint32_t a_mul0, a_mul1, a_batches;   // batch-slice multipliers and slice count of A
  uint32_t b_mul0, b_mul1, b_batches;
  uint64_t a_ptr, b_ptr, bias_ptr;
  // Optional: memory of MmPackBytes() bytes each, for a copy of an operand in rows of whole 16-byte units; and the pitch of
  // such rows in elements, set by the launcher (0: the rows are as long as their contents)
  uint64_t a_pack, b_pack;
  uint32_t a_pitch, b_pitch;
  // post-fusion program: instruction words (isa.h Insn) over 16 consecutive columns of one row, ending with
  // OP_END; operand kind K_TENSOR with index `mma_slot` names the rounded product itself
  uint32_t n_tensors;
  uint32_t mma_slot;
  uint32_t num_temps;
  uint32_t group_m;         // row blocks swept together over all column blocks (L2 reuse of the A panel); set by the launcher
  // Set by the launcher: what the post-fusion program does (EpiMode), and the tensor it stores to when it is one of the forms
  // that leave through shared memory in the operand type.  EPI_GATE is  y = x / (c2 + exp(c1 * (x + c0 * x^3)))  of the rounded
  // product x (tanh-GeLU written through the exponential, c0 = 0.044715, c1 = -2 sqrt(2/pi), c2 = 1), computed in registers with
  // the interpreter's operations in the interpreter's order instead of eleven interpreted words per strip.
  uint32_t epi_mode, out_slot;
  uint32_t gate_c[3];
  uint32_t tma_out;         // set by the launcher: the copy engine can address the result (16-byte base and strides)
  uint32_t leave_sms;       // set by the planner: SMs this launch leaves free (a collective runs beside it); 0 = none
  EpiTensor tensor[kMmMaxEpiTensors];
  uint64_t epilogue[kMmMaxEpilogueWords];
};

enum EpiMode : uint32_t {
  EPI_PROGRAM = 0,   // interpreted, strip by strip
  EPI_WIDEN = 1,     // one store of the product widened to fp32 (a partial product that another launch finishes)
  EPI_STORE = 2,     // one store of the product in the operand type
  EPI_GATE = 3,      // the gated form, stored in the operand type
};

// Enqueue the MatMul.  Returns 0, a cudaError_t (> 0), or a negative code for an unsupported shape.
int LaunchMatMul(const MmParam &p, void *stream);
// True when the copy engine cannot address an operand (rows of `inner` 16-bit elements, batch slices of `slice`): base, row
// pitch or slice not a multiple of 16 bytes.  Its tiles are then loaded by the tile kernel's work warps.
bool MmOperandNeedsGather(uint64_t ptr, uint64_t pitch, uint64_t slice, uint32_t batches);
inline uint32_t MmInnerA(const MmParam &p) { return p.a_mmajor ? p.M : p.K; }
inline uint32_t MmInnerB(const MmParam &p) { return p.b_kmajor ? p.K : p.N; }
inline uint32_t MmRowsA(const MmParam &p) { return p.a_mmajor ? p.K : p.M; }
inline uint32_t MmRowsB(const MmParam &p) { return p.b_kmajor ? p.N : p.K; }
inline uint32_t MmPitchA(const MmParam &p) { return p.a_pitch != 0 ? p.a_pitch : MmInnerA(p); }
inline uint32_t MmPitchB(const MmParam &p) { return p.b_pitch != 0 ? p.b_pitch : MmInnerB(p); }
inline bool MmGatherA(const MmParam &p) {
  return MmOperandNeedsGather(p.a_ptr, MmPitchA(p), static_cast<uint64_t>(MmPitchA(p)) * MmRowsA(p), p.a_batches);
}
inline bool MmGatherB(const MmParam &p) {
  return MmOperandNeedsGather(p.b_ptr, MmPitchB(p), static_cast<uint64_t>(MmPitchB(p)) * MmRowsB(p), p.b_batches);
}
inline bool MmNeedsGather(const MmParam &p) { return MmGatherA(p) || MmGatherB(p); }
// Bytes of memory for repacked operands that make this product faster (0: none; see the rule there).
void MmPackBytes(const MmParam &p, uint64_t *a_bytes, uint64_t *b_bytes);
// Copies the operands that the copy engine cannot address into a_pack / b_pack, and makes `p` read them there.
int LaunchMmPack(MmParam *p, void *stream);
// Tensor map over the result of a staged mode (EPI_STORE, EPI_GATE): boxes of 32 x 32, 64-byte swizzle; false if the copy
// engine cannot address it.
bool EncodeMmResult(CUtensorMap *map, const MmParam &p);
// The tile kernel (mm_tile.cu): 128 x bn tiles (bn 64 or 128), K cut into `split` (1, 2, 4, 8) parts.
int LaunchMmTile(const MmParam &p, uint32_t bn, uint32_t split, void *stream);
unsigned int ReadMmTileStatus();
// 3-d tensor map over a [batches, rows, inner] 16-bit operand (`pitch` elements from row to row): boxes of box_rows rows of 64 elements, 128-byte swizzle.
int EncodeMmOperand(CUtensorMap *map, uint64_t ptr, uint64_t inner, uint64_t pitch, uint64_t rows, uint64_t batches, uint32_t box_rows);
unsigned int ReadMatMulStatus();

// Fused attention  O[b,h] = softmax(scale * Q[b,h] K[b,h]^T) V[b,h]  (non-causal), bf16 or fp16 operands,
// fp32 softmax, result in the operand type.  Q [B0,B1,Sq,D], K and V [B0,B1,Skv,D], all contiguous.
struct AttnParam {
  uint32_t batch;           // B0 * B1
  uint32_t sq, skv, d;      // d is 64 or 128
  uint32_t dtype;           // T_F16 or T_BF16
  uint32_t scale_bits;      // scale in the operand type's register form (fp32 bits)
  uint32_t scale_first;     // 1: the score is rounded to the operand type, scaled, rounded again (the graph's order)
  uint32_t q_tiles, units;  // set by the launcher: tiles of 128 query rows per unit (1 or 2), units of work
  uint64_t q_ptr, k_ptr, v_ptr, o_ptr;
};
int LaunchAttention(const AttnParam &p, void *stream);
constexpr uint32_t kDecodeMaxRows = 16;
int LaunchAttentionDecode(const AttnParam &p, void *stream);   // at most kDecodeMaxRows query rows (attn_decode.cu)
bool AttentionSupported(const AttnParam &p);
unsigned int ReadAttentionStatus();

}  // namespace dvmb

#endif  // DVM_B200_MM_LAUNCH_H_
