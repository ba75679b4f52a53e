// Translation unit of the causal attention of the training graphs.
#include "kvm_ops_attn.cuh"
#include "kvm_attn_tc.cuh"
#include "kvm_dispatch.cuh"

__device__ __noinline__ void kvm_unit_attn(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 45: if ((aux.x & 255) == 2 && !(c.cfg_flags & KVM_CFG_NO_TENSOR_CORES)) kvm_attn_fwd_tc(c, a, aux); else kvm_op_attn_fwd(c, a); break;
    case 46: kvm_op_attn_bwd_delta(c, a); break;
    case 47: if ((aux.x & 255) == 2 && !(c.cfg_flags & KVM_CFG_NO_TENSOR_CORES)) kvm_attn_dq_tc(c, a, aux); else kvm_op_attn_bwd_dq(c, a); break;
    case 48: if ((aux.x & 255) == 2 && !(c.cfg_flags & KVM_CFG_NO_TENSOR_CORES)) kvm_attn_dkv_tc(c, a, aux); else kvm_op_attn_bwd_dkv(c, a); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
