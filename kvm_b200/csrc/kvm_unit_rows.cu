// Translation unit of the row-structured ops (norms, embeddings, cross-entropy, optimizer, reductions).
#include "kvm_ops_rows.cuh"
#include "kvm_dispatch.cuh"

__device__ __noinline__ void kvm_unit_rows(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 32: kvm_op_embedding_fwd(c, a); break;
    case 33: kvm_op_embedding_bwd(c, a); break;
    case 35: kvm_op_layernorm_fwd(c, a); break;
    case 36: kvm_op_rmsnorm_fwd(c, a); break;
    case 37: kvm_op_layernorm_bwd_dx(c, a); break;
    case 38: kvm_op_rmsnorm_bwd_dx(c, a); break;
    case 39: kvm_op_norm_bwd_params(c, a); break;
    case 43: kvm_op_rope_fwd(c, a); break;
    case 44: kvm_op_rope_bwd(c, a); break;
    case 51: kvm_op_softmax_ce_fwd(c, a); break;
    case 52: kvm_op_softmax_ce_reduce(c, a); break;
    case 53: kvm_op_softmax_ce_bwd(c, a); break;
    case 54: kvm_op_adamw(c, a); break;
    case 55: kvm_op_gradnorm_partial(c, a); break;
    case 56: kvm_op_gradnorm_finish(c, a); break;
    case 58: kvm_op_argmax(c, a); break;
    case 61: kvm_op_colsum(c, a); break;
    case 63: kvm_op_gather_rows(c, a); break;
    case 115: kvm_op_adamw_lr(c, a); break;
    case 116: kvm_op_lr_schedule(c, a); break;
    case 118: kvm_op_add_rowtile(c, a); break;
    case 127: kvm_op_softmax_ce_fused(c, a); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
