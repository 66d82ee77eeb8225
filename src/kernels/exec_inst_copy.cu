// Executor instantiations of the collectives that only move data: aligned operands, any operands.
#include "exec_flow.cuh"
namespace piccl {
FlowKernelFn exec_flow_copy_table[2] = {exec_flow_kernel<uint8_t, OP_COPY, false>, exec_flow_kernel<uint8_t, OP_COPY, true>};
ExecKernelFn exec_copy_table[2] = {exec_kernel<uint8_t, OP_COPY, false>, exec_kernel<uint8_t, OP_COPY, true>};
}  // namespace piccl
