// Translation unit of the decode and peer-exchange ops.
#include "kvm_ops_decode.cuh"
#include "kvm_ops_peer.cuh"
#include "kvm_dispatch.cuh"

__device__ __noinline__ void kvm_unit_decode(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 49: kvm_op_kv_append(c, a); break;
    case 50: kvm_op_attn_decode(c, a); break;
    case 57: kvm_op_sample(c, a); break;
    case 134: kvm_op_gemv_bf16(c, a); break;
    case 135: kvm_op_attn_decode_part(c, a); break;
    case 136: kvm_op_attn_decode_merge(c, a); break;
    case 300: kvm_op_attn_decode_part_qkn(c, a); break;
    case 301: kvm_op_gemv_bf16_rows(c, a); break;
    case 302: kvm_op_peer_put_signal(c, a); break;
    case 303: kvm_op_peer_wait_sum(c, a); break;
    case 304: kvm_op_peer_wait(c, a); break;
    default: c.fail(KVM_ERR_BAD_OP, op); break;
  }
}
