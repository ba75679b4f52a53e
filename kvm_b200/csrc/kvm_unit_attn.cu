// Translation unit of the causal attention of the training graphs.
#include "kvm_ops_attn.cuh"
#include "kvm_attn_tc.cuh"
#include "kvm_dispatch.cuh"

// For the static kernel; the ready-queue kernel takes a tcgen05 task before it dispatches.
KVM_OP_FN bool kvm_attn_tc_call(const KvmCtx& c, int op, const int32_t* a, const int4& aux) { return kvm_attn_tc(c, op, a, aux); }

__device__ __noinline__ void kvm_unit_attn(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  if (kvm_attn_tc_call(c, op, a, aux)) return;
  switch (op) {
    case 45: kvm_op_attn_fwd(c, a); break;
    case 46: kvm_op_attn_bwd_delta(c, a); break;
    case 47: kvm_op_attn_bwd_dq(c, a); break;
    case 48: kvm_op_attn_bwd_dkv(c, a); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
