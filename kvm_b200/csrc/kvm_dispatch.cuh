// The op dispatcher.  Op bodies are functions of their own (KVM_OP_FN), grouped by family into translation units (kvm_unit_*.cu) that
// both executor kernels call: each body gets registers of its own (all of them inlined into one kernel left the compiler spilling
// kilobytes per thread) and is compiled once, side by side with the others.
#pragma once
#include "kvm_dev.cuh"

__device__ void kvm_unit_flat(const KvmCtx& c, int op, const int32_t* a, const int4& aux);      // elementwise ops over flat ranges
__device__ void kvm_unit_rows(const KvmCtx& c, int op, const int32_t* a, const int4& aux);      // row-structured ops (norms, embeddings, cross-entropy, optimizer, reductions)
__device__ void kvm_unit_mm(const KvmCtx& c, int op, const int32_t* a, const int4& aux);      // matrix products (SIMT and tensor-core tiles)
__device__ void kvm_unit_attn(const KvmCtx& c, int op, const int32_t* a, const int4& aux);      // causal attention of the training graphs
__device__ void kvm_unit_decode(const KvmCtx& c, int op, const int32_t* a, const int4& aux);      // decode and peer-exchange ops

static __device__ __forceinline__ void kvm_dispatch(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 8: case 34: case 114: case 122:
      kvm_unit_mm(c, op, a, aux); break;
    case 45: case 46: case 47: case 48:
      kvm_unit_attn(c, op, a, aux); break;
    case 49: case 50: case 57: case 134: case 135: case 136: case 300: case 301: case 302: case 303: case 304:
      kvm_unit_decode(c, op, a, aux); break;
    case 1: case 2: case 3: case 4: case 5: case 6: case 7: case 9: case 10: case 40: case 41: case 42: case 59: case 60: case 62: case 96: case 97: case 98: case 113: case 117: case 123: case 126:
      kvm_unit_flat(c, op, a, aux); break;
    default: kvm_unit_rows(c, op, a, aux); break;      // unknown ids end there with KVM_ERR_BAD_OP
  }
}
