// Lookup of the executor instantiation for a (dtype, op) pair.
#include "exec.cuh"

namespace piccl {
extern ExecKernelFn exec_table_I8[4], exec_table_U8[4], exec_table_I32[4], exec_table_U32[4], exec_table_I64[4], exec_table_U64[4],
    exec_table_F16[4], exec_table_F32[4], exec_table_F64[4], exec_table_BF16[4];

ExecKernelFn exec_kernel_for(int dtype, int op) {
  if (op < 0 || op > 3) return nullptr;
  switch (dtype) {
    case DT_I8: return exec_table_I8[op];
    case DT_U8: return exec_table_U8[op];
    case DT_I32: return exec_table_I32[op];
    case DT_U32: return exec_table_U32[op];
    case DT_I64: return exec_table_I64[op];
    case DT_U64: return exec_table_U64[op];
    case DT_F16: return exec_table_F16[op];
    case DT_F32: return exec_table_F32[op];
    case DT_F64: return exec_table_F64[op];
    case DT_BF16: return exec_table_BF16[op];
    default: return nullptr;
  }
}
extern ExecKernelFn exec_shift_table_I8[4], exec_shift_table_U8[4], exec_shift_table_I32[4], exec_shift_table_U32[4], exec_shift_table_I64[4], exec_shift_table_U64[4],
    exec_shift_table_F16[4], exec_shift_table_F32[4], exec_shift_table_F64[4], exec_shift_table_BF16[4];
// The variant for operands that are not 16-byte aligned (exec_impl.cuh).
ExecKernelFn exec_shift_kernel_for(int dtype, int op) {
  if (op < 0 || op > 3) return nullptr;
  switch (dtype) {
    case DT_I8: return exec_shift_table_I8[op];
    case DT_U8: return exec_shift_table_U8[op];
    case DT_I32: return exec_shift_table_I32[op];
    case DT_U32: return exec_shift_table_U32[op];
    case DT_I64: return exec_shift_table_I64[op];
    case DT_U64: return exec_shift_table_U64[op];
    case DT_F16: return exec_shift_table_F16[op];
    case DT_F32: return exec_shift_table_F32[op];
    case DT_F64: return exec_shift_table_F64[op];
    case DT_BF16: return exec_shift_table_BF16[op];
    default: return nullptr;
  }
}
extern ExecKernelFn exec_ll_table_I8[4], exec_ll_table_U8[4], exec_ll_table_I32[4], exec_ll_table_U32[4], exec_ll_table_I64[4], exec_ll_table_U64[4],
    exec_ll_table_F16[4], exec_ll_table_F32[4], exec_ll_table_F64[4], exec_ll_table_BF16[4];
ExecKernelFn exec_ll_kernel_for(int dtype, int op) {
  if (op < 0 || op > 3) return nullptr;
  switch (dtype) {
    case DT_I8: return exec_ll_table_I8[op];
    case DT_U8: return exec_ll_table_U8[op];
    case DT_I32: return exec_ll_table_I32[op];
    case DT_U32: return exec_ll_table_U32[op];
    case DT_I64: return exec_ll_table_I64[op];
    case DT_U64: return exec_ll_table_U64[op];
    case DT_F16: return exec_ll_table_F16[op];
    case DT_F32: return exec_ll_table_F32[op];
    case DT_F64: return exec_ll_table_F64[op];
    case DT_BF16: return exec_ll_table_BF16[op];
    default: return nullptr;
  }
}
extern FlowKernelFn exec_flow_table_I8[8], exec_flow_table_U8[8], exec_flow_table_I32[8], exec_flow_table_U32[8], exec_flow_table_I64[8], exec_flow_table_U64[8], exec_flow_table_F16[8], exec_flow_table_F32[8], exec_flow_table_F64[8], exec_flow_table_BF16[8];
// All ranks in one launch on one GPU (exec_flow.cuh); shift: operands that are not 16-byte aligned.
FlowKernelFn exec_flow_kernel_for(int dtype, int op, bool shift) {
  if (op < 0 || op > 3) return nullptr;
  if (shift) op += 4;
  switch (dtype) {
    case DT_I8: return exec_flow_table_I8[op];
    case DT_U8: return exec_flow_table_U8[op];
    case DT_I32: return exec_flow_table_I32[op];
    case DT_U32: return exec_flow_table_U32[op];
    case DT_I64: return exec_flow_table_I64[op];
    case DT_U64: return exec_flow_table_U64[op];
    case DT_F16: return exec_flow_table_F16[op];
    case DT_F32: return exec_flow_table_F32[op];
    case DT_F64: return exec_flow_table_F64[op];
    case DT_BF16: return exec_flow_table_BF16[op];
    default: return nullptr;
  }
}
extern FlowKernelFn exec_flow_copy_table[2];
FlowKernelFn exec_flow_copy_kernel(bool shift) { return exec_flow_copy_table[shift]; }
ExecKernelFn exec_ll_copy_kernel() { return exec_ll_table_U8[0]; }
// Byte-wise instantiations used by the collectives that only move data.
extern ExecKernelFn exec_copy_table[2];
ExecKernelFn exec_copy_kernel() { return exec_copy_table[0]; }
ExecKernelFn exec_shift_copy_kernel() { return exec_copy_table[1]; }
}  // namespace piccl
