// Translation unit of the matrix products (SIMT and tensor-core tiles).
#include "kvm_ops_mm.cuh"
#include "kvm_gemm_tc.cuh"
#include "kvm_dispatch.cuh"

__device__ __noinline__ void kvm_unit_mm(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 8: kvm_op_matmul(c, a); break;
    case 34: kvm_op_matmul_tile(c, a); break;
    case 114: kvm_op_matmul_tile_bf16(c, a); break;
    case 122: kvm_op_matmul_mma_bf16(c, a, aux); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
