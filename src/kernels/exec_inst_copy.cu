// Executor instantiations of the collectives that only move data: aligned operands, any operands.
#include "exec_impl.cuh"
namespace piccl {
ExecKernelFn exec_copy_table[2] = {exec_kernel<uint8_t, OP_COPY, false>, exec_kernel<uint8_t, OP_COPY, true>};
}  // namespace piccl
