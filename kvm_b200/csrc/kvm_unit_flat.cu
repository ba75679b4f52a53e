// Translation unit of the elementwise ops over flat ranges.
#include "kvm_ops_flat.cuh"
#include "kvm_dispatch.cuh"

__device__ __noinline__ void kvm_unit_flat(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 1: kvm_op_copy(c, a); break;
    case 2: kvm_op_add(c, a); break;
    case 3: kvm_op_scale(c, a); break;
    case 4: kvm_op_relu(c, a); break;
    case 5: kvm_op_sgd(c, a); break;
    case 6: kvm_op_predict(c, a); break;
    case 7: kvm_op_mse_grad(c, a); break;
    case 9: kvm_op_fill(c, a); break;
    case 10: kvm_op_spin(c, a); break;
    case 40: kvm_op_gelu_fwd(c, a); break;
    case 41: kvm_op_gelu_bwd(c, a); break;
    case 42: kvm_op_residual_add(c, a); break;
    case 59: kvm_op_zero_buf(c, a); break;
    case 60: kvm_op_counter_inc(c, a); break;
    case 62: kvm_op_select_window(c, a); break;
    case 96: kvm_op_act_fwd(c, a); break;
    case 97: kvm_op_act_bwd(c, a); break;
    case 98: kvm_op_silu_mul_fwd(c, a); break;
    case 113: kvm_op_round_bf16(c, a); break;
    case 117: kvm_op_scale_flat(c, a); break;
    case 123: kvm_op_sgd_range(c, a); break;
    case 126: kvm_op_round_tf32(c, a); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
