// The static-schedule path: the resident program runs as per-worker task lists planned on the host (kvm_static_host.inl), with
// no ready queue, no dependency counters and no atomics on the task path.  What it implements of the reference: the static path
// of include/mvm_static.h:1-17,43-51 (list schedule -> per-worker records, cross-worker watermark waits) and its worker loop
// include/mvm_static.cuh:161-229 (fetch the next record ahead, poll the watermarks, dispatch, publish own progress).
//
// One CTA per SM as in the dynamic kernel: 16 compute warps, a FRONT warp and a STREAM warp.  The front warp walks the worker's list
// ahead of the compute group: it fetches task records into a four-slot shared-memory ring, polls the task's dependencies (pairs of
// (worker, tasks that worker must have finished), lanes in parallel over the pairs), and marks the slot ready.  A worker's
// progress word is one release store per finished task; nothing else is written to global memory for scheduling.
//
// Because a worker knows its next tasks, the stream warp STREAMS AHEAD: for decode GEMVs and split decode attention it issues the
// bulk copies of the task's weight rows / cache rows into a shared-memory stage ring as soon as stages are free, BEFORE the task's
// dependencies are resolved (weights and old cache rows do not change during a launch; the host marks a task whose streamed operand
// is written by some task of the batch, and its copies then wait for the dependencies like everything else).  The dependency wait
// then only gates the prologue and the arithmetic, so HBM keeps streaming across phase boundaries.
//
// Every wait is bounded (time limit); on expiry KVM_ERR_TIMEOUT is recorded, every CTA leaves, copies in flight are awaited.
#pragma once
#include "kvm_attn_tc.cuh"
#include "kvm_dispatch.cuh"
#include "kvm_ring_attn.cuh"
#include "kvm_ops_decode.cuh"
#include "kvm_static_api.h"

#define KVM_ST_SLOTS 4                 // record ring depth (tasks fetched ahead)
#define KVM_ST_HDR 3072                // header bytes: slots, control words, barriers
#define KVM_ST_WAITED 4                // stamp[0] end of the prologue, [1] of the stage loop, [2] start of the task, [4] waits for stages so far (ns)
#define KVM_ST_ARRIVALS 16             // arrivals that free a stage: every compute warp, once it is done with the stage (or has nothing to do with it)

struct KvmStSlot {
  int task;
  int state;                  // 0 free, 1 fetched, 2 ready, 3 leave
  int pos;                    // position in the worker's list of the record the slot holds
  int go;
  int kind;                   // 0 generic op, 1 streamed gemv (one activation row, SIMT consumer), 2 streamed split attention, 3 streamed gemv on tensor cores (rows)
  int nchunks;                // stage uses of this task
  int R;                      // gemv: weight rows per stage (kind 3 keeps its chunk columns / row groups / k-chunks in j0 / j1 / newrow)
  int wait_off, wait_cnt;
  int32_t desc[16];
  int32_t args[KVM_MAX_ARGS];
  int4 aux;
  int prefetch;               // 1: copies may be issued before the dependencies are met
  int j0, j1, newrow;         // attention: key range of the split, index of the appended key inside it (-1 none)
  KvmBuf lb[7];               // streamed tasks: the buffer-table entries of the task's buffer arguments (argument j -> lb[j]), looked up once by the front warp
};
#define KVM_ST_CTX_BYTES 192            // the compute group's KvmCtx, in front of the rope cache
static_assert(sizeof(KvmCtx) <= KVM_ST_CTX_BYTES, "context grew");
static_assert(sizeof(KvmStSlot) * KVM_ST_SLOTS + 128 * 4 + KVM_ST_CTX_BYTES + 288 + 128 <= KVM_ST_HDR, "static header too small");      // slots | control words | ... | rope cache (288) | ring barriers (128)

__device__ __forceinline__ bool kvm_mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}

struct KvmRing {
  uint32_t bar0;              // full[s] at bar0 + 8 s, empty[s] at bar0 + 64 + 8 s
  unsigned char* base;        // stage s at base + s * KVM_ST_STAGE
  uint32_t base_addr;
  unsigned ns;                // stages: 3 (32 KB of op scratch beside them) or, for programs with gemv_bf16_rows, 2 (96 KB of scratch: the activations of eight rows)
};
__device__ __forceinline__ unsigned kvm_ring_slot(const KvmRing& r, unsigned it) { return r.ns == 2 ? (it & 1u) : it % 3u; }
__device__ __forceinline__ uint32_t kvm_ring_full(const KvmRing& r, unsigned it) { return r.bar0 + 8 * kvm_ring_slot(r, it); }
__device__ __forceinline__ uint32_t kvm_ring_empty(const KvmRing& r, unsigned it) { return r.bar0 + 64 + 8 * kvm_ring_slot(r, it); }
__device__ __forceinline__ uint32_t kvm_ring_parity(const KvmRing& r, unsigned it) { return (r.ns == 2 ? (it >> 1) : it / 3u) & 1u; }
__device__ __forceinline__ unsigned char* kvm_ring_stage(const KvmRing& r, unsigned it) { return r.base + kvm_ring_slot(r, it) * KVM_ST_STAGE; }

// Buffer argument j of a streamed task from the slot's own copy of the table entries (same checks as kvm_buf).
__device__ __forceinline__ bool kvm_buf_local(const KvmCtx& c, const KvmBuf* lb, const int32_t* a, int j, int mask, KvmBuf& out, bool optional = false) {
  const int idx = a[j];
  if (idx == -1 && optional) { out.p = nullptr; out.rows = out.cols = out.ld = 0; out.dtype = 0; return true; }
  if (idx < 0 || idx >= c.nbufs) { c.fail(KVM_OPE_BUF, idx); return false; }
  out = lb[j];
  if (out.p == nullptr || !((1 << out.dtype) & mask)) { c.fail(KVM_OPE_DTYPE, idx, out.dtype); return false; }
  return true;
}
__device__ __forceinline__ int kvm_ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Wait for stage use `it` to land (bounded by the launch deadline and by an error recorded elsewhere); the verdict is the same for the
// whole warp.  All 32 lanes poll: with one lane polling and a shuffle behind it the compiler kept that lane's path apart from the
// others' through the arithmetic that follows, and the warp went through it twice (a GEMV phase took 57 us instead of 36).
__device__ __forceinline__ bool kvm_ring_wait_warp(const KvmRing& ring, unsigned it, unsigned long long deadline, const KvmErrRec* err) {
  const uint32_t bar = kvm_ring_full(ring, it), par = kvm_ring_parity(ring, it);
  bool ok = true;
  unsigned spins = 0;
  while (!kvm_mbar_test(bar, par))
    if ((++spins & 1023u) == 0 && (kvm_globaltimer() > deadline || *(volatile const int*)&err->code != 0)) { ok = false; break; }      // an error elsewhere: the copies may never come
  return __all_sync(0xffffffffu, ok);
}

// ---- streamed GEMV, consumer side --------------------------------------------------------------------------------------------
// Stage use `cit + ci` holds rows n0 + ci*R .. of the weight matrix in full (R*K*2 bytes).  All sixteen warps consume: warp = (row group,
// part of K), KP parts of 256 columns or more, 16 / KP row groups of up to eight rows a stage.  A thread owns J pieces of eight columns
// of the activation row v = bf16(prologue(x)): it computes them itself and keeps them over the task (as float32, or as bf16 from four
// pieces on), so the prologue has one barrier at most (the sum of squares).  The eight rows' sums leave a warp through one transposing
// reduction (nine shuffles for eight rows).
// What bounds it: a 64 KB stage is 1.5 us of an SM's share of HBM and about 700 issue cycles here; every value of the loop has to stay
// in registers, since a spilled one costs an L2 round trip per stage (the stages leave 28 KB of L1 for 512 threads' local memory).
// Partial sums are added in pairs.  Semantics as kvm_op_gemv_bf16 (runtime/ref_extra.py:398-415).  Always consumes its nchunks
// stage uses, also after an error.
__device__ __forceinline__ unsigned long long kvm_pack2(float lo, float hi) { unsigned long long r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void kvm_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint4 kvm_pack_bf16x8(const float (&v)[8]) {
  uint4 pk;
  __nv_bfloat162* hh = (__nv_bfloat162*)&pk;
#pragma unroll
  for (int j = 0; j < 4; ++j) hh[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
  return pk;
}
// acc += eight bf16 weights * eight float32 activations
__device__ __forceinline__ void kvm_gv_dot8(unsigned long long& acc, const uint4& w, const unsigned long long (&x)[4]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) kvm_fma2(acc, kvm_pack2(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u)), x[i]);
}
// v = bf16(pro(x)) to shared memory, any storage types and alignments.
static __device__ __noinline__ void kvm_gemv_stage_x(const KvmBuf* lb, __nv_bfloat16* vs, float* red, int K, int pro, float eps) {
  const KvmBuf x = lb[0], x2 = lb[1];
  const int tid = threadIdx.x;
  float rs = 1.0f;
  if (pro == 1) {
    float q = 0.0f;
    for (int k = tid; k < K; k += KVM_NT) { const float t = kvm_ld(x, k); q += t * t; }
    q = kvm_block_sum(q, red);
    rs = 1.0f / sqrtf(q / K + eps);
  }
  for (int k = tid; k < K; k += KVM_NT) {
    const float p = kvm_ld(x, k);
    vs[k] = __float2bfloat16_rn(pro == 1 ? p * rs * ((const float*)lb[2].p)[k] : pro == 2 ? kvm_silu(p) * kvm_ld(x2, k) : p);
  }
}
// Warps a row is split over (a power of two: what is left of the sixteen takes other rows) and rows a stage holds; the front warp and
// the consumers compute the same.
__device__ __forceinline__ int kvm_gv_parts(int K) { return K > 2048 ? 16 : K > 1024 ? 8 : K > 512 ? 4 : K > 256 ? 2 : 1; }
__device__ __forceinline__ int kvm_gv_rows(int K) { return (KVM_NWARPS / kvm_gv_parts(K)) * min(8, KVM_ST_STAGE / (K * 2 * (KVM_NWARPS / kvm_gv_parts(K)))); }
#define KVM_GV_RED 256                                     // scratch: reduction words | partial sums [KP][rows]

// Sums over the warp's lanes of eight values per lane: lane 4 r + (0..3) ends with the total of value r.
__device__ __forceinline__ float kvm_gv_reduce8(float (&s)[8], int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {                            // lanes with bit 4 keep values 4..7
    const float keep = lane & 16 ? s[i + 4] : s[i], give = lane & 16 ? s[i] : s[i + 4];
    s[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float keep = lane & 8 ? s[i + 2] : s[i], give = lane & 8 ? s[i] : s[i + 2];
    s[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
  }
  const float keep = lane & 4 ? s[1] : s[0], give = lane & 4 ? s[0] : s[1];
  float t = keep + __shfl_xor_sync(0xffffffffu, give, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  return t + __shfl_xor_sync(0xffffffffu, t, 1);
}

// The checks of kvm_op_gemv_bf16 on the slot's table entries, one entry at a time.
__device__ __forceinline__ bool kvm_gv_args_ok(const KvmCtx& c, const int32_t* a, const KvmBuf* lb) {
  const int K = a[8], n1 = a[7], pro = a[9];
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    KvmBuf b;
    ok = ok && kvm_buf_local(c, lb, a, j, j == 3 ? KVM_M_BF16 : j == 2 ? KVM_M_F32 : KVM_M_FLT, b, j == 1 || j == 2 || j == 5);
    if (ok && ((j == 1 && pro == 2 && !b.p) || (j == 2 && pro == 1 && !b.p) || pro < 0 || pro > 2)) { c.fail(KVM_OPE_SHAPE, K, pro); ok = false; }
    if (ok && j != 3) ok = j == 2 ? kvm_flat_ok(c, b, K) : kvm_mat_ok(c, b, 1, j >= 4 ? n1 : K);
  }
  return ok;
}

// Reciprocal RMS of a row from the threads' sums of squares (one barrier).
__device__ __forceinline__ float kvm_gv_rms(const KvmCtx& c, float q, int rg, int KP, int K, float eps) {
  float* red = (float*)c.smem;
  q = kvm_warp_sum(q);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
  kvm_sync();
  q = 0.0f;
  for (int i = 0; i < KP; ++i) q += red[rg * KP + i];
  return 1.0f / sqrtf(q / K + eps);
}

template <int J, bool TR>      // TR: notes its times in `stamp` (KVM_ST_WAITED)
__device__ __forceinline__ void kvm_gemv_ring(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, const KvmRing ring, unsigned cit, int R, int NC, int* stamp) {
  const int K = a[8], rows = a[7] - a[6], KP = kvm_gv_parts(K);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = warp & (KP - 1), rg = warp / KP, m = R * KP / KVM_NWARPS;      // rows rg*m .. of a stage
  const int k0 = (part * 32 + lane) * 8, kstep = KP * 256;
  float* parts = (float*)(c.smem + KVM_GV_RED);            // [KP][rows]
  bool ok;
  constexpr bool PACK = J > 3;                             // activations kept as bf16 pairs
  unsigned long long xs[PACK ? 1 : J][4];
  uint4 xp[PACK ? J : 1];
  float rv = 0.0f;                                         // this thread's residual value, on its way while the weights stream
  {
    const int pro = a[9];
    auto put = [&](int j, const float (&t)[8]) {
      if (PACK) xp[PACK ? j : 0] = kvm_pack_bf16x8(t);
      else
#pragma unroll
        for (int i = 0; i < 4; ++i) xs[PACK ? 0 : j][i] = kvm_pack2(t[2 * i], t[2 * i + 1]);
    };
    ok = kvm_gv_args_ok(c, a, lb);
    if (ok && a[5] >= 0 && (lane & 15) == 0 && tid / 16 < rows) rv = kvm_ld(lb[5], a[6] + tid / 16);
    const KvmBuf x = lb[0];
    bool f32 = x.dtype == KVM_F32 && kvm_vec_ok(x);
    const float* up = nullptr;                             // the prologue's second operand: gamma or the up projection
    if (pro == 1) { up = (const float*)lb[2].p; f32 = f32 && kvm_vec_ok(lb[2]); }
    else if (pro == 2) { up = (const float*)lb[1].p; f32 = f32 && lb[1].dtype == KVM_F32 && kvm_vec_ok(lb[1]); }
    if (J > 1 && ok && f32) {
      // piece after piece (the next one's loads in flight), the results through shared memory: with a thread's 8 J evaluations of silu
      // unrolled their code does not stay in the instruction cache between tasks (a token of the 8B shape: 5.63 ms unrolled, 5.56 as a
      // loop), and all the loads of three pieces at once leave the kernel no registers
      uint4* mine = (uint4*)(c.smem + ((KVM_GV_RED + rows * KP * 4 + 15) & ~15));
      const float* xp = (const float*)x.p;
      const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float rs = 1.0f;
      float4 a0, a1, b0 = zero, b1 = zero;
      auto load = [&](int k, bool both) {
        a0 = k < K ? *(const float4*)(xp + k) : zero; a1 = k < K ? *(const float4*)(xp + k + 4) : zero;
        if (both) { b0 = k < K ? *(const float4*)(up + k) : zero; b1 = k < K ? *(const float4*)(up + k + 4) : zero; }
      };
      if (pro == 1) {
        float q = 0.0f;
        load(k0, false);
#pragma unroll 1
        for (int k = k0; k < K; k += kstep) {
          const float4 p0 = a0, p1 = a1;
          load(k + kstep, false);
          q += p0.x * p0.x; q += p0.y * p0.y; q += p0.z * p0.z; q += p0.w * p0.w; q += p1.x * p1.x; q += p1.y * p1.y; q += p1.z * p1.z; q += p1.w * p1.w;
        }
        rs = kvm_gv_rms(c, q, rg, KP, K, kvm_bits_f32(a[10]));
      }
      load(k0, pro != 0);
#pragma unroll 1
      for (int k = k0; k < K; k += kstep) {
        const float4 p0 = a0, p1 = a1, q0 = b0, q1 = b1;
        load(k + kstep, pro != 0);
        const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w}, q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        float t[8];
        if (pro == 2)
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = kvm_silu(p[i]) * q[i];
        else
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = pro == 1 ? p[i] * rs * q[i] : p[i];
        mine[k / 8] = kvm_pack_bf16x8(t);
      }
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const uint4 w = k0 + j * kstep < K ? mine[(k0 + j * kstep) / 8] : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
        float t[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) { t[2 * i] = __uint_as_float(u[i] << 16); t[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
        put(j, t);
      }
    } else if (ok && f32) {
      // one piece per thread, float32: all loads in flight together
      float v[8], u[8];
      const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        const float4 t = k0 < K ? *(const float4*)((const float*)x.p + k0 + i) : zero, g = k0 < K && pro ? *(const float4*)(up + k0 + i) : zero;
        v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
        u[i] = g.x; u[i + 1] = g.y; u[i + 2] = g.z; u[i + 3] = g.w;
      }
      float rs = 1.0f;
      if (pro == 1) {
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) q += v[i] * v[i];
        rs = kvm_gv_rms(c, q, rg, KP, K, kvm_bits_f32(a[10]));
      }
      float t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = kvm_bf16_round(pro == 1 ? v[i] * rs * u[i] : pro == 2 ? kvm_silu(v[i]) * u[i] : v[i]);
      put(0, t);
    } else {
      // anything else is staged through shared memory (behind the partial sums)
      __nv_bfloat16* vs = (__nv_bfloat16*)(c.smem + ((KVM_GV_RED + rows * KP * 4 + 15) & ~15));
      if (ok) kvm_gemv_stage_x(lb, vs, (float*)c.smem, K, pro, kvm_bits_f32(a[10]));
      kvm_sync();
#pragma unroll
      for (int j = 0; j < J; ++j) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = ok && k0 + j * kstep < K ? __bfloat162float(vs[k0 + j * kstep + i]) : 0.0f;
        put(j, t);
      }
    }
  }
  if (TR && tid == 0) stamp[0] = (int)kvm_globaltimer();
  bool waited = true;
  constexpr int RB = J <= 1 ? 4 : 1;          // rows whose loads are in flight together
#pragma unroll 1
  for (int ci = 0; ci < NC; ++ci) {
    const int t0 = TR ? (int)kvm_globaltimer() : 0;
    if (!kvm_ring_wait_warp(ring, cit + ci, c.deadline, c.err)) { waited = false; break; }      // warp-uniform
    if (TR && tid == 0) stamp[KVM_ST_WAITED] += (int)kvm_globaltimer() - t0;
    const unsigned char* st = kvm_ring_stage(ring, cit + ci) + (size_t)(rg * m) * (K * 2);
    const int left = min(m, rows - ci * R - rg * m);
    float s[8];
#pragma unroll
    for (int h = 0; h < 8; h += RB) {
#pragma unroll
      for (int r = 0; r < RB; ++r) s[h + r] = 0.0f;
      if (h < left) {
        uint4 w[RB][J];
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
          for (int j = 0; j < J; ++j) w[r][j] = h + r < left && k0 + j * kstep < K ? *(const uint4*)(st + ((h + r) * K + k0 + j * kstep) * 2) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          unsigned long long acc = 0ull;
#pragma unroll
          for (int j = 0; j < J; ++j) {
            if (PACK) {
              const uint32_t p[4] = {xp[PACK ? j : 0].x, xp[PACK ? j : 0].y, xp[PACK ? j : 0].z, xp[PACK ? j : 0].w};
              unsigned long long xx[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) xx[i] = kvm_pack2(__uint_as_float(p[i] << 16), __uint_as_float(p[i] & 0xffff0000u));
              kvm_gv_dot8(acc, w[r][j], xx);
            } else kvm_gv_dot8(acc, w[r][j], xs[PACK ? 0 : j]);
          }
          const float2 f = *(float2*)&acc;
          s[h + r] = f.x + f.y;
        }
      }
    }
    const float t = kvm_gv_reduce8(s, lane);
    __syncwarp();                                          // (the shuffles have met already; this orders the lanes' reads before the release)
    if (lane == 0) kvm_mbar_arrive(kvm_ring_empty(ring, cit + ci));
    if ((lane & 3) == 0 && (lane >> 2) < left) parts[part * rows + ci * R + rg * m + (lane >> 2)] = t;
  }
  if (!waited && *(volatile int*)&c.err->code == 0) kvm_stream_timeout(c, 1134);
  if (TR && tid == 0) stamp[1] = (int)kvm_globaltimer();
  kvm_sync();
  if (ok && waited) {
    const KvmBuf out = lb[4];
    // sixteen lanes per row (KP of them hold a part), added in pairs
    for (int base = warp * 2; base < rows; base += 2 * KVM_NWARPS) {
      const int i = base + (lane >> 4);
      float sum = i < rows && (lane & 15) < KP ? parts[(lane & 15) * rows + i] : 0.0f;
#pragma unroll
      for (int o = 1; o < 16; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if ((lane & 15) == 0 && i < rows) {
        if (a[5] >= 0) sum = __fadd_rn(sum, base == warp * 2 ? rv : kvm_ld(lb[5], a[6] + i));
        kvm_st(out, a[6] + i, sum);
      }
    }
  }
}
// rows of more than 12288 columns (their staging bounds them to 16 Ki): the activations beside the loop do not fit the kernel's registers, a function of its own
KVM_OP_FN void kvm_gemv_ring_wide(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, const KvmRing ring, unsigned cit, int R, int NC) { kvm_gemv_ring<4, false>(c, a, lb, ring, cit, R, NC, nullptr); }
// Pieces of eight columns per thread.
__device__ __forceinline__ int kvm_gv_pieces(int K) { return (K + 256 * kvm_gv_parts(K) - 1) / (256 * kvm_gv_parts(K)); }
// A traced task: a copy of its own, called, so that tracing costs an untraced program nothing (tests of a switch inside the loops cost
// three users' decode step 1.83 -> 1.88 ms, a small model's 0.59 -> 0.62).
KVM_OP_FN void kvm_gemv_ring_traced(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, const KvmRing ring, unsigned cit, int R, int NC, int* stamp) {
  const int J = kvm_gv_pieces(a[8]);
  if (J == 1) kvm_gemv_ring<1, true>(c, a, lb, ring, cit, R, NC, stamp);
  else if (J <= 3) kvm_gemv_ring<3, true>(c, a, lb, ring, cit, R, NC, stamp);
  else kvm_gemv_ring<4, true>(c, a, lb, ring, cit, R, NC, stamp);
}

// ---- streamed GEMV on tensor cores (gemv_bf16 with one activation row, gemv_bf16_rows with up to eight), consumer side --------------
// D[16 x 8] += A[16 x 16] B[16 x 8] (mma.sync m16n8k16, bf16 operands, float32 accumulate) with A = activations (rows = activation
// rows, at most eight of the sixteen used), B = the weight rows of a stage (columns).  A dot product does not care in which order k
// is visited, so both operands are read 16 bytes per thread from row-major [row][k] arrays at the SAME k offsets (thread t of a quad
// takes k = 8t .. 8t+7 of a 32-wide step, for two MMAs) instead of in the instruction's interleaved k layout.  Steps are taken in
// pairs: weight rows sit a multiple of 128 bytes apart, so an odd row reads the pair's steps in the other order (and swaps the
// registers back before the MMAs): the eight lanes of a quarter warp (two rows, four quads) then read eight different 16-byte
// bank groups.  The activations are staged as bf16 with a row pitch of 64 bytes mod 128 for the same reason.
//
// Two stage layouts, chosen by kvm_gemv_mma_layout from the shapes alone (the front warp and the consumers compute the same):
//   whole rows   a stage holds R <= 8 weight rows in full (KC = K, R*K*2 <= 64 KB, one bulk copy); every stage is a row group of
//                its own, its sums leave the registers when the stage is done; needs all of the M activation rows staged at once;
//   k chunks     a stage holds 8 weight rows x KC columns (KC < K, eight copies); stages run k-chunk outer, row group inner, the
//                accumulators of up to eight row groups stay in registers over the whole task, the activations are staged per k-chunk.
// All sixteen warps multiply (pairs of steps are dealt round robin); their partial sums are added in warp order at the end.
// Semantics per activation row as gemv_bf16 (runtime/ref_extra.py:398-415).  Always consumes its nchunks stage uses, also after an error.
#define KVM_MMA_PARTS_OFF 512
struct KvmMmaLayout {
  int R, KC, nkc, ng;       // weight rows and columns per stage, k-chunks, row groups
  int full_x;               // all k of the activations staged once
  int pitch;                // bytes per staged activation row
  int parts_off;            // byte offset of the partial sums [16 warps][ng][M][R] in the scratch
  int nchunks;
  bool ok;
};
__device__ __forceinline__ KvmMmaLayout kvm_gemv_mma_layout(int rows, int K, int M, int scratch_bytes) {
  KvmMmaLayout L;
  L.ok = false;
  const int row_pitch = K * 2 + 64;
  // whole rows
  L.R = K * 2 * 8 <= KVM_ST_STAGE ? 8 : KVM_ST_STAGE / (K * 2);
  if (L.R >= 1) {
    L.KC = K; L.nkc = 1; L.ng = (rows + L.R - 1) / L.R; L.full_x = 1; L.pitch = row_pitch;
    L.parts_off = M * row_pitch + KVM_MMA_PARTS_OFF;
    if (L.parts_off + 16 * L.ng * M * L.R * 4 <= scratch_bytes) { L.nchunks = L.ng; L.ok = true; return L; }
  }
  // k chunks
  L.R = 8; L.KC = 4096;
  while (L.KC > 0 && K % L.KC) L.KC -= 256;
  if (L.KC <= 0 || L.KC >= K) return L;
  L.nkc = K / L.KC; L.ng = (rows + 7) / 8;
  if (L.ng > 8) return L;
  L.full_x = M * row_pitch + KVM_MMA_PARTS_OFF + 16 * L.ng * M * 8 * 4 <= scratch_bytes;
  L.pitch = L.full_x ? row_pitch : L.KC * 2 + 64;
  L.parts_off = M * L.pitch + KVM_MMA_PARTS_OFF;
  if (L.parts_off + 16 * L.ng * M * 8 * 4 > scratch_bytes) return L;
  L.nchunks = L.nkc * L.ng; L.ok = true;
  return L;
}
__device__ __forceinline__ void kvm_mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}
// v[j] = prologue value of 8 consecutive activations starting at column k of row u
__device__ __forceinline__ void kvm_mma_pro8(int pro, float (&v)[8], const float (&v2)[8], float rs) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = pro == 1 ? v[j] * rs * v2[j] : pro == 2 ? kvm_silu(v[j]) * v2[j] : v[j];
}
// Staging of the activations v = bf16(pro(x)) for the tensor-core consumer, functions of their own (registers of their own).
struct KvmStageX {
  KvmBuf x, x2, gm;
  unsigned char* xs;        // [M][pitch] bytes
  float* rsq;               // [8] reciprocal RMS per row, from [64] on reduction scratch
  int r0, M, K, pro, pitch;
  float eps;
};
// One activation row whose prologue loads all fit into registers: every load in flight at once, one pass.  false = not taken.
KVM_OP_FN bool kvm_stage_one_row(const KvmStageX& s) {
  const KvmBuf x = s.x, x2 = s.x2, gm = s.gm;
  const int K = s.K, pro = s.pro, tid = threadIdx.x;
  if (K > 3 * 8 * KVM_NT || (x.ld & 7) || !kvm_vec_ok(x) || (pro == 2 && ((x2.ld & 7) || !kvm_vec_ok(x2))) || (pro == 1 && !kvm_vec_ok(gm))) return false;
  float v[3][8], v2[3][8];
  const size_t xo = (size_t)s.r0 * x.ld, x2o = x2.p ? (size_t)s.r0 * x2.ld : 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = (tid + j * KVM_NT) * 8;
    if (k < K) {
      kvm_ld8(x, xo + k, v[j]);
      if (pro == 2) kvm_ld8(x2, x2o + k, v2[j]);
      else if (pro == 1) { *(float4*)v2[j] = *(const float4*)((const float*)gm.p + k); *(float4*)(v2[j] + 4) = *(const float4*)((const float*)gm.p + k + 4); }
    }
  }
  float rs = 0.0f;
  if (pro == 1) {
    float q = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j) if ((tid + j * KVM_NT) * 8 < K)
#pragma unroll
      for (int u = 0; u < 8; ++u) q += v[j][u] * v[j][u];
    q = kvm_block_sum(q, s.rsq + 64);
    rs = 1.0f / sqrtf(q / K + s.eps);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = (tid + j * KVM_NT) * 8;
    if (k < K) { kvm_mma_pro8(pro, v[j], v2[j], rs); *(uint4*)(s.xs + (size_t)k * 2) = kvm_pack_bf16x8(v[j]); }
  }
  return true;
}
// RMS statistics of up to eight rows: two warps per activation row.  Whole compute group.
KVM_OP_FN void kvm_stage_rms(const KvmStageX& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, u = warp >> 1, hf = warp & 1, K = s.K;
  float q = 0.0f;
  if (u < s.M) for (int k = hf * (K / 2) + lane; k < (hf + 1) * (K / 2); k += 32) { const float v = kvm_ld(s.x, (size_t)(s.r0 + u) * s.x.ld + k); q += v * v; }
  q = kvm_warp_sum(q);
  if (lane == 0) s.rsq[64 + warp] = q;
  kvm_sync();
  if (tid < 8) s.rsq[tid] = tid < s.M ? 1.0f / sqrtf((s.rsq[64 + 2 * tid] + s.rsq[64 + 2 * tid + 1]) / K + s.eps) : 0.0f;
  kvm_sync();
}
// Columns [kb, kb + kn) of the M rows to column offset 0 of the staged rows (all 16 warps).
KVM_OP_FN void kvm_stage_rows(const KvmStageX& s, int kb, int kn) {
  const KvmBuf x = s.x, x2 = s.x2, gm = s.gm;
  const int pro = s.pro, r0 = s.r0;
  const bool vec_x = (x.ld & 7) == 0 && kvm_vec_ok(x), vec_x2 = x2.p && (x2.ld & 7) == 0 && kvm_vec_ok(x2), vec_g = gm.p && kvm_vec_ok(gm);
  for (int e = threadIdx.x; e < s.M * (kn / 8); e += KVM_NT) {
    const int u = e / (kn / 8), k0 = (e % (kn / 8)) * 8, k = kb + k0;
    float v[8], v2[8];
    if (vec_x) kvm_ld8(x, (size_t)(r0 + u) * x.ld + k, v);
    else for (int j = 0; j < 8; ++j) v[j] = kvm_ld(x, (size_t)(r0 + u) * x.ld + k + j);
    if (pro == 2) {
      if (vec_x2) kvm_ld8(x2, (size_t)(r0 + u) * x2.ld + k, v2);
      else for (int j = 0; j < 8; ++j) v2[j] = kvm_ld(x2, (size_t)(r0 + u) * x2.ld + k + j);
    } else if (pro == 1) {
      if (vec_g) { *(float4*)v2 = *(const float4*)((const float*)gm.p + k); *(float4*)(v2 + 4) = *(const float4*)((const float*)gm.p + k + 4); }
      else for (int j = 0; j < 8; ++j) v2[j] = ((const float*)gm.p)[k + j];
    }
    kvm_mma_pro8(pro, v, v2, pro == 1 ? s.rsq[u] : 0.0f);
    *(uint4*)(s.xs + (size_t)u * s.pitch + (size_t)k0 * 2) = kvm_pack_bf16x8(v);
  }
}
template <bool CHUNKED>      // the k-chunk layout (accumulators of eight row groups live over the task) or the whole-row layout, a function each
KVM_OP_FN void kvm_gemv_mma_ring_t(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool has_rows, const KvmRing ring, unsigned cit, int* stamp) {
  KvmBuf x, x2, gm, w, out, res;
  const int n0 = a[6], n1 = a[7], K = a[8], pro = a[9], r0 = has_rows ? a[11] : 0, r1 = has_rows ? a[12] : 1;
  const float eps = kvm_bits_f32(a[10]);
  bool ok = kvm_buf_local(c, lb, a, 0, KVM_M_FLT, x) && kvm_buf_local(c, lb, a, 1, KVM_M_FLT, x2, true) && kvm_buf_local(c, lb, a, 2, KVM_M_F32, gm, true) &&
            kvm_buf_local(c, lb, a, 3, KVM_M_BF16, w) && kvm_buf_local(c, lb, a, 4, KVM_M_FLT, out) && kvm_buf_local(c, lb, a, 5, KVM_M_FLT, res, true);
  const int rows = n1 - n0, M = r1 - r0;
  const KvmMmaLayout L = kvm_gemv_mma_layout(rows, K, M, c.smem_bytes);       // the front warp accepted the same layout
  const int R = L.R, KC = L.KC, ng = L.ng, nkc = L.nkc, pitch = L.pitch;
  if (ok && (pro < 0 || pro > 2 || (pro == 1 && !gm.p) || (pro == 2 && !x2.p) || !L.ok || CHUNKED != (L.nkc > 1))) { c.fail(KVM_OPE_SHAPE, K, pro); ok = false; }
  if (ok) ok = kvm_mat_ok(c, x, r1, K) && kvm_mat_ok(c, x2, r1, K) && kvm_flat_ok(c, gm, K) && kvm_mat_ok(c, out, r1, n1) && kvm_mat_ok(c, res, r1, n1);
  unsigned char* xs = c.smem;                              // [M][pitch]
  float* rsq = (float*)(c.smem + M * pitch);               // [8] reciprocal RMS per activation row, from [64] on reduction scratch
  float* parts = (float*)(c.smem + L.parts_off);           // [16 warps][ng][M][R]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  kvm_sync();                                              // the previous task is done with the scratch
  struct KvmStageX sx;
  sx.x = x; sx.x2 = x2; sx.gm = gm; sx.xs = xs; sx.rsq = rsq; sx.r0 = r0; sx.M = M; sx.K = K; sx.pro = pro; sx.pitch = pitch; sx.eps = eps;
  bool staged = false;
  if (ok && M == 1 && L.full_x) staged = kvm_stage_one_row(sx);
  if (ok && !staged && pro == 1) kvm_stage_rms(sx);
  if (ok && !staged && L.full_x) kvm_stage_rows(sx, 0, K);
  kvm_sync();
  if (stamp && tid == 0) stamp[0] = (int)kvm_globaltimer();
  bool waited = true;
  const int npairs = KC / 64;
  // one stage use: wait for it, multiply it into acc (x columns from xk0 of the staged rows), release it
  auto consume = [&](unsigned it, float (&acc)[4], int xk0) {
    const int t0 = stamp && tid == 0 ? (int)kvm_globaltimer() : 0;
    if (waited && !kvm_ring_wait_warp(ring, it, c.deadline, c.err)) waited = false;
    if (stamp && tid == 0) stamp[KVM_ST_WAITED] += (int)kvm_globaltimer() - t0;
    if (!waited) return;                                   // warp-uniform; the warp still takes part in every barrier of the task
    if (ok) {
      const unsigned char* wrow = kvm_ring_stage(ring, it) + (size_t)g * KC * 2 + t * 16;
      const unsigned char* xrow = xs + (size_t)g * pitch + (size_t)xk0 * 2 + t * 16;
      const int odd = g & 1;
      float acc2[4] = {0.0f, 0.0f, 0.0f, 0.0f};                  // the two steps of a pair accumulate side by side
#pragma unroll 2
      for (int p = warp; p < npairs; p += KVM_NT / 32) {
        uint4 b0 = make_uint4(0, 0, 0, 0), b1 = b0, a0 = b0, a1 = b0;
        if (g < R) { b0 = *(const uint4*)(wrow + (2 * p + odd) * 64); b1 = *(const uint4*)(wrow + (2 * p + 1 - odd) * 64); }
        if (g < M) { a0 = *(const uint4*)(xrow + (2 * p) * 64); a1 = *(const uint4*)(xrow + (2 * p + 1) * 64); }
        const uint4 e0 = odd ? b1 : b0, e1 = odd ? b0 : b1;       // weights of step 2p and of step 2p + 1
        kvm_mma_bf16_16816(acc, a0.x, a0.y, e0.x, e0.y);
        kvm_mma_bf16_16816(acc2, a1.x, a1.y, e1.x, e1.y);
        kvm_mma_bf16_16816(acc, a0.z, a0.w, e0.z, e0.w);
        kvm_mma_bf16_16816(acc2, a1.z, a1.w, e1.z, e1.w);
      }
      acc[0] += acc2[0]; acc[1] += acc2[1]; acc[2] += acc2[2]; acc[3] += acc2[3];
    }
    __syncwarp();
    if (lane == 0) kvm_mbar_arrive(kvm_ring_empty(ring, it));
  };
  // thread (g, t) holds D[activation row g][weight rows 2t, 2t + 1]
  auto put_parts = [&](int rg, const float (&acc)[4]) {
    if (g < M) {
      float* pp = parts + (((size_t)warp * ng + rg) * M + g) * R;
      if (2 * t < R) pp[2 * t] = acc[0];
      if (2 * t + 1 < R) pp[2 * t + 1] = acc[1];
    }
  };
  if (!CHUNKED) {
    for (int rg = 0; rg < ng; ++rg) {
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      consume(cit + (unsigned)rg, acc, 0);
      put_parts(rg, acc);
    }
  } else {
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    for (int kc = 0; kc < nkc; ++kc) {
      if (!L.full_x) {
        if (kc) kvm_sync();                                // the consumers are done with the previous chunk's activations
        if (ok) kvm_stage_rows(sx, kc * KC, KC);
        kvm_sync();
      }
#pragma unroll
      for (int rg = 0; rg < 8; ++rg) if (rg < ng) consume(cit + (unsigned)(kc * ng + rg), acc[rg], L.full_x ? kc * KC : 0);
    }
#pragma unroll
    for (int rg = 0; rg < 8; ++rg) if (rg < ng) put_parts(rg, acc[rg]);
  }
  __syncwarp();
  if (stamp && tid == 0) stamp[1] = (int)kvm_globaltimer();
  if (!waited && *(volatile int*)&c.err->code == 0) kvm_stream_timeout(c, 1301);
  kvm_sync();
  if (ok && *(volatile int*)&c.err->code == 0)            // a warp that gave up has recorded the timeout before the barrier
    for (int e = tid; e < ng * M * R; e += KVM_NT) {
      const int rg = e / (M * R), u = (e / R) % M, nn = e % R, n = n0 + rg * R + nn;
      if (n >= n1) continue;
      float sum = 0.0f;
#pragma unroll
      for (int wv = 0; wv < KVM_NT / 32; ++wv) sum += parts[(((size_t)wv * ng + rg) * M + u) * R + nn];
      const size_t o = (size_t)(r0 + u) * out.ld + n;
      kvm_st(out, o, res.p ? __fadd_rn(sum, kvm_ld(res, (size_t)(r0 + u) * res.ld + n)) : sum);
    }
}

__device__ __forceinline__ void kvm_gemv_mma_ring(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool has_rows, const KvmRing ring, unsigned cit, int nkc, int* stamp) {
  if (nkc > 1) kvm_gemv_mma_ring_t<true>(c, a, lb, has_rows, ring, cit, stamp);
  else kvm_gemv_mma_ring_t<false>(c, a, lb, has_rows, ring, cit, stamp);
}

// ---- streamed split attention, consumer side (kvm_ring_attn.cuh) --------------------------------------------------------------------
// Stage use `cit` holds the split's keys, `cit + 1` its values (the appended row left out).  The front warp has validated the geometry
// of the caches before it issued the copies; the other arguments are checked here.
template <int HD, int GT, bool TR>      // head dimension, query heads per key head at most, traced
KVM_OP_FN void kvm_attn_part_ring_t(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool qkn, const KvmRing ring, unsigned cit, int j0, int j1, int newrow, int* stamp) {
  KvmPartArgs P;
  const int bb = a[7], S = a[10], H = a[11], Hkv = a[12], hd = a[13];
  bool ok;
  {
    KvmBuf q, kc, vc, lens, part, kn, vn, gam;
    ok = kvm_buf_local(c, lb, a, 0, KVM_M_FLT, q) && kvm_buf_local(c, lb, a, 1, KVM_M_BF16, kc) && kvm_buf_local(c, lb, a, 2, KVM_M_BF16, vc) &&
         kvm_buf_local(c, lb, a, 3, KVM_M_I32, lens) && kvm_buf_local(c, lb, a, 4, KVM_M_F32, part) && kvm_buf_local(c, lb, a, 5, KVM_M_FLT, kn, true) &&
         kvm_buf_local(c, lb, a, 6, KVM_M_FLT, vn, true);
    gam.p = c.smem; gam.ld = 0;
    if (ok && qkn) ok = kvm_buf(c, a[18], KVM_M_F32, gam) && kvm_mat_ok(c, gam, 2, hd);
    if (ok) ok = kvm_mat_ok(c, q, bb + 1, H * hd) && kvm_mat_ok(c, part, (long long)(bb + 1) * S * H, hd + 2) && kvm_mat_ok(c, kn, bb + 1, Hkv * hd) && kvm_mat_ok(c, vn, bb + 1, Hkv * hd);
    if (ok && (!kn.p || !vn.p)) { c.fail(KVM_OPE_SHAPE, hd, a[17]); ok = false; }
    P.lb = lb; P.a = a; P.qkn = qkn; P.gam = (const float*)gam.p; P.gam_ld = gam.ld; P.G = H / Hkv; P.nk = max(j1 - j0, 0); P.newrow = newrow;
    P.p0 = ok ? ((const int*)lens.p)[bb] : 0;
  }
  const float theta = kvm_bits_f32(a[16]);
  unsigned char* Ks = kvm_ring_stage(ring, cit);
  unsigned char* Vs = kvm_ring_stage(ring, cit + 1);
  bool waited = true;
  auto wait = [&](unsigned it) {
    const int t0 = TR ? (int)kvm_globaltimer() : 0;
    const bool landed = kvm_ring_wait_warp(ring, it, c.deadline, c.err);
    if (TR && threadIdx.x == 0) {
      if (it == cit) stamp[0] = t0;                        // the prologue ends where the wait for the keys begins
      stamp[KVM_ST_WAITED] += (int)kvm_globaltimer() - t0;
    }
    return landed;
  };
  auto wk = [&]() { return wait(cit); };
  auto wv = [&]() { return wait(cit + 1); };
  if (ok) {
    // theta^(-2i/hd) is a double-precision pow per frequency: computed once per (theta, head dimension) and launch, not per task
    float* rc = c.rope_cache;
    if (__float_as_int(rc[0]) != __float_as_int(theta) || __float_as_int(rc[1]) != hd) {
      kvm_sync();                                          // every thread has looked at the key before anyone replaces it
      for (int i = threadIdx.x; i < hd / 2; i += KVM_NT) rc[2 + i] = kvm_rope_inv(theta, i, hd);
      if (threadIdx.x == 0) { rc[0] = theta; rc[1] = __int_as_float(hd); }
      kvm_sync();
    }
    P.inv = rc + 2;
    waited = kvm_ra_part<HD, GT>(P, c.smem, Ks, Vs, wk, wv);
  } else {
    waited = wk() && wv();
  }
  if (!waited && *(volatile int*)&c.err->code == 0) kvm_stream_timeout(c, 1135);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the stages were written by threads; the next copies into them come after it
  __syncwarp();
  if (waited && (threadIdx.x & 31) == 0) { kvm_mbar_arrive(kvm_ring_empty(ring, cit)); kvm_mbar_arrive(kvm_ring_empty(ring, cit + 1)); }
}

template <bool TR>
__device__ __forceinline__ void kvm_attn_part_ring(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool qkn, const KvmRing ring, unsigned cit, int j0, int j1, int newrow, int* stamp) {
  const int hd = a[13];
  const bool few = a[11] <= 4 * a[12];
  if (hd == 128) { if (few) kvm_attn_part_ring_t<128, 4, TR>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp); else kvm_attn_part_ring_t<128, 8, TR>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp); }
  else if (hd == 64) { if (few) kvm_attn_part_ring_t<64, 4, TR>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp); else kvm_attn_part_ring_t<64, 8, TR>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp); }
  else kvm_attn_part_ring_t<32, 8, TR>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp);
}
// Traced splits: called from a function of their own, so that the kernel's task loop does not grow by them.
KVM_OP_FN void kvm_attn_part_ring_traced(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool qkn, const KvmRing ring, unsigned cit, int j0, int j1, int newrow, int* stamp) {
  kvm_attn_part_ring<true>(c, a, lb, qkn, ring, cit, j0, j1, newrow, stamp);
}

// Splits that the warp form (kvm_ring_attn.cuh) does not take, from the same two stages: queries in float32 (flags 0 and 1), head dimension
// 16.  One softmax over the split by all warps (kvm_attn_part_core); one, two or four query heads per key
// head (eight need more scratch than the three stages leave).
KVM_OP_FN void kvm_attn_part_ring_any(const KvmCtx& c, const int32_t* a, const KvmBuf* lb, bool qkn, const KvmRing ring, unsigned cit, int j0, int j1, int newrow, int* stamp) {
  KvmBuf q, kc, vc, lens, part, kn, vn, gam{};
  bool ok = kvm_buf_local(c, lb, a, 0, KVM_M_FLT, q) && kvm_buf_local(c, lb, a, 1, KVM_M_BF16, kc) && kvm_buf_local(c, lb, a, 2, KVM_M_BF16, vc) &&
            kvm_buf_local(c, lb, a, 3, KVM_M_I32, lens) && kvm_buf_local(c, lb, a, 4, KVM_M_F32, part) && kvm_buf_local(c, lb, a, 5, KVM_M_FLT, kn, true) &&
            kvm_buf_local(c, lb, a, 6, KVM_M_FLT, vn, true);
  const int b = a[7], kvh = a[8], S = a[10], H = a[11], Hkv = a[12], hd = a[13], fl = a[17], G = H / Hkv, nk = max(j1 - j0, 0);
  if (ok && qkn) ok = kvm_buf(c, a[18], KVM_M_F32, gam) && kvm_mat_ok(c, gam, 2, hd);
  if (ok) ok = kvm_mat_ok(c, q, b + 1, H * hd) && kvm_mat_ok(c, part, (long long)(b + 1) * S * H, hd + 2) && kvm_mat_ok(c, kn, b + 1, Hkv * hd) && kvm_mat_ok(c, vn, b + 1, Hkv * hd);
  if (ok && (fl & 1) && (!kn.p || !vn.p)) { c.fail(KVM_OPE_SHAPE, hd, fl); ok = false; }
  auto wait = [&](unsigned it) {
    const int t0 = stamp ? (int)kvm_globaltimer() : 0;
    const bool landed = kvm_ring_wait_warp(ring, it, c.deadline, c.err);
    if (stamp && threadIdx.x == 0) {
      if (it == cit) stamp[0] = t0;
      stamp[KVM_ST_WAITED] += (int)kvm_globaltimer() - t0;
    }
    return landed;
  };
  auto wk = [&]() { return wait(cit); };
  auto wv = [&]() { return wait(cit + 1); };
  kvm_sync();                                              // the previous task is done with the scratch
  bool waited;
  if (ok) {
    unsigned char* sm = c.smem;
    KvmPartPro P;
    P.q = q; P.kc = kc; P.vc = vc; P.kn = kn; P.vn = vn; P.gam = gam;
    P.b = b; P.kvh = kvh; P.G = G; P.hd = hd; P.fl = fl; P.p0 = ((const int*)lens.p)[b]; P.base = (size_t)(b * Hkv + kvh) * a[14]; P.theta = kvm_bits_f32(a[16]);
    P.eps = qkn ? kvm_bits_f32(a[19]) : 0.0f; P.appends = newrow >= 0; P.rope_cache = c.rope_cache;
    P.qs = (float*)(sm + KVM_AS_OFF_QS); P.inv = (float*)(sm + KVM_AS_OFF_INV); P.kns = (float*)(sm + KVM_AS_OFF_KNEW); P.vns = (float*)(sm + KVM_AS_OFF_VNEW);
    P.rsq = (float*)(sm + KVM_AS_OFF_ML);
    auto prologue = [&]() { kvm_part_prologue(P); };
    auto emit = [&](int g, int cc, float M, float L, float A) {
      float* row = (float*)part.p + ((size_t)(b * S + a[9]) * H + kvh * G + g) * part.ld;
      row[cc] = L > 0.0f ? A : 0.0f;
      if (cc == 0) { row[hd] = L > 0.0f ? M : KVM_ATTN_EMPTY_M_STREAM; row[hd + 1] = L; }
    };
    unsigned char* Ks = kvm_ring_stage(ring, cit);
    unsigned char* Vs = kvm_ring_stage(ring, cit + 1);
    const float sc = kvm_bits_f32(a[15]);
    if (G <= 1) waited = kvm_attn_part_core<1>(sm, Ks, Vs, nk, newrow, G, hd, sc, prologue, wk, wv, emit);
    else if (G <= 2) waited = kvm_attn_part_core<2>(sm, Ks, Vs, nk, newrow, G, hd, sc, prologue, wk, wv, emit);
    else if (G <= 4) waited = kvm_attn_part_core<4>(sm, Ks, Vs, nk, newrow, G, hd, sc, prologue, wk, wv, emit);
    else waited = kvm_attn_part_core<8>(sm, Ks, Vs, nk, newrow, G, hd, sc, prologue, wk, wv, emit);
  } else {
    waited = wk() && wv();
  }
  if (!waited && *(volatile int*)&c.err->code == 0) kvm_stream_timeout(c, 1135);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the appended row was written by threads; the next copies into these stages come after it
  kvm_sync();
  if (waited && (threadIdx.x & 31) == 0) { kvm_mbar_arrive(kvm_ring_empty(ring, cit)); kvm_mbar_arrive(kvm_ring_empty(ring, cit + 1)); }
}
__device__ __forceinline__ bool kvm_ra_takes(int hd, int flags) { return flags == 3 && hd != 16; }      // the warp form

// ---- front warp: stream geometry of a fetched task (lane 0) ---------------------------------------------------------------------
// Decides whether the task streams through the ring and with which chunking; every bound the copies rely on is checked here,
// a task that fails one runs as a generic op (whose own checks then report the error).
static __device__ void kvm_static_geometry(const KvmDevState& S, KvmStSlot& sl, int scratch_bytes) {
  sl.kind = 0; sl.nchunks = 0; sl.R = 1; sl.j0 = sl.j1 = 0; sl.newrow = -1;
  const int op = sl.desc[0];
  const int32_t* a = sl.args;
  if (op == 134 || op == 301) {
    const int wi = a[3], n0 = a[6], n1 = a[7], K = a[8], r0 = op == 301 ? a[11] : 0, r1 = op == 301 ? a[12] : 1;
    if (wi < 0 || wi >= S.nbufs || n0 < 0 || n1 <= n0 || K <= 0 || (K & 7) || r0 < 0 || r1 <= r0 || r1 - r0 > 8) return;
    const KvmBuf w = sl.lb[3];
    if (!w.p || w.dtype != KVM_BF16 || (w.ld & 7) || ((uintptr_t)w.p & 15) || n1 > w.rows || K > w.cols) return;
    // one activation row: the SIMT consumer over stages of whole rows (measured faster than mma.sync fragments at one row: the
    // legacy tensor path of this part issues an m16n8k16 every few hundred cycles per warp); several rows: the tensor-core consumer
    if (op == 134 && K * 2 <= KVM_ST_STAGE) {
      const int RG = KVM_NWARPS / kvm_gv_parts(K), R = min(kvm_gv_rows(K), (n1 - n0 + RG - 1) / RG * RG);
      if (KVM_GV_RED + (n1 - n0) * kvm_gv_parts(K) * 4 + 16 + K * 2 <= scratch_bytes) { sl.kind = 1; sl.R = R; sl.nchunks = (n1 - n0 + R - 1) / R; return; }
    }
    if (K & 255) return;
    const KvmMmaLayout L = kvm_gemv_mma_layout(n1 - n0, K, r1 - r0, scratch_bytes);
    if (L.ok) { sl.kind = 3; sl.R = L.R; sl.j0 = L.KC; sl.j1 = L.ng; sl.newrow = L.nkc; sl.nchunks = L.nchunks; }      // j0 / j1 / newrow double as KC / row groups / k-chunks
  } else if (op == 135 || op == 300) {
    const int kci = a[1], vci = a[2], li = a[3], b = a[7], kvh = a[8], s = a[9], Sp = a[10], H = a[11], Hkv = a[12], hd = a[13], Tmax = a[14], fl = a[17];
    if (kci < 0 || kci >= S.nbufs || vci < 0 || vci >= S.nbufs || li < 0 || li >= S.nbufs) return;
    if (b < 0 || Hkv <= 0 || H <= 0 || H % Hkv || kvh < 0 || kvh >= Hkv || s < 0 || Sp <= 0 || s >= Sp || Tmax <= 0 || !(fl == 0 || fl == 1 || fl == 3)) return;
    const int G = H / Hkv;
    const bool warp_form = kvm_ra_takes(hd, fl);
    if (G > 8 || !(hd == 16 || hd == 32 || hd == 64 || hd == 128) || (!warp_form && (G & (G - 1)))) return;
    const KvmBuf kc = sl.lb[1], vc = sl.lb[2], lens = sl.lb[3];
    if (!kc.p || !vc.p || !lens.p || kc.dtype != KVM_BF16 || vc.dtype != KVM_BF16 || lens.dtype != KVM_I32 || kc.ld != hd || vc.ld != hd || ((uintptr_t)kc.p & 15) || ((uintptr_t)vc.p & 15)) return;
    if ((long long)(b + 1) * Hkv * Tmax > kc.rows || (long long)(b + 1) * Hkv * Tmax > vc.rows || hd > kc.cols || hd > vc.cols || lens.ld != lens.cols || b >= lens.rows * lens.cols) return;
    const int p0 = ((const int*)lens.p)[b], n = p0 + 1;
    if (p0 < 0 || n > Tmax) return;
    const int chunk = (n + Sp - 1) / Sp, j0 = s * chunk, j1 = min(n, s * chunk + chunk), nk = max(j1 - j0, 0);
    if (nk * hd * 2 > KVM_ST_STAGE || (warp_form ? KVM_RA_BYTES : kvm_attn_part_scratch(nk, G, hd)) > scratch_bytes) return;
    sl.kind = 2; sl.nchunks = 2; sl.j0 = j0; sl.j1 = j1;
    sl.newrow = ((fl & 1) && j0 <= n - 1 && n - 1 < j1) ? n - 1 - j0 : -1;
  }
}

// Issue the copies of chunk `ci` of the task in `sl` as stage use `it` (stream warp, lane 0; the stage is known to be free).
static __device__ void kvm_static_issue(const KvmDevState& S, const KvmStSlot& sl, const KvmRing& ring, unsigned it, int ci) {
  const uint32_t full = kvm_ring_full(ring, it), dst = ring.base_addr + kvm_ring_slot(ring, it) * KVM_ST_STAGE;
  const int32_t* a = sl.args;
  if (sl.kind == 3) {
    // stage = R weight rows x KC columns; chunk ci = (k-chunk, row group), row group inner
    const KvmBuf w = sl.lb[3];
    const int n0 = a[6], n1 = a[7], K = a[8], R = sl.R, KC = sl.j0, ng = sl.j1;
    const int kc = ci / ng, rg = ci % ng, r0 = n0 + rg * R, nr = min(R, n1 - r0);
    const __nv_bfloat16* wp = (const __nv_bfloat16*)w.p + (size_t)kc * KC;
    kvm_mbar_expect_tx(full, (uint32_t)(nr * KC * 2));
    if (KC == K && w.ld == K) kvm_bulk_g2s(dst, wp + (size_t)r0 * w.ld, (uint32_t)(nr * K * 2), full);
    else for (int r = 0; r < nr; ++r) kvm_bulk_g2s(dst + r * KC * 2, wp + (size_t)(r0 + r) * w.ld, (uint32_t)(KC * 2), full);
  } else if (sl.kind == 1) {
    const KvmBuf w = sl.lb[3];
    const int n0 = a[6], n1 = a[7], K = a[8], R = sl.R;
    const int r0 = n0 + ci * R, nr = min(R, n1 - r0);
    const __nv_bfloat16* wp = (const __nv_bfloat16*)w.p;
    kvm_mbar_expect_tx(full, (uint32_t)(nr * K * 2));
    if (w.ld == K) kvm_bulk_g2s(dst, wp + (size_t)r0 * w.ld, (uint32_t)(nr * K * 2), full);
    else for (int r = 0; r < nr; ++r) kvm_bulk_g2s(dst + r * K * 2, wp + (size_t)(r0 + r) * w.ld, (uint32_t)(K * 2), full);
  } else {
    const KvmBuf cb = sl.lb[ci == 0 ? 1 : 2];
    const int b = a[7], kvh = a[8], Hkv = a[12], hd = a[13], Tmax = a[14];
    const size_t base = (size_t)(b * Hkv + kvh) * Tmax;
    const int nk = max(sl.j1 - sl.j0, 0), ncopy = sl.newrow >= 0 ? nk - 1 : nk;
    const uint32_t bytes = (uint32_t)(ncopy * hd * 2);
    kvm_mbar_expect_tx(full, bytes);
    if (bytes) kvm_bulk_g2s(dst, (const __nv_bfloat16*)cb.p + (base + sl.j0) * cb.ld, bytes, full);
  }
}

__global__ void __launch_bounds__(KVM_ST_THREADS, 1) kvm_static_kernel(KvmStaticState T) {
  extern __shared__ __align__(1024) unsigned char kvm_smem[];
  const KvmDevState& S = T.D;
  KvmStSlot* slots = (KvmStSlot*)kvm_smem;
  int* ctl = (int*)(kvm_smem + KVM_ST_SLOTS * sizeof(KvmStSlot));          // as in the dynamic kernel: ctl[0] = TMEM base, tensor-core barriers from ctl[8]
  int* sctl = ctl + 96;                                                     // static path's own words: [0] consumer stage-use count, [1] tasks finished, [2] producer stage-use count, [3..5] and [7] trace, [6] leave
  const uint32_t sbar = kvm_smem_addr(kvm_smem + KVM_ST_HDR - 128);         // stream ring barriers: full[3] | empty[3]
  const int tid = threadIdx.x;
  const int w = blockIdx.x;
  unsigned dyn;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
  if (tid < KVM_ST_SLOTS) { slots[tid].state = 0; slots[tid].task = -1; slots[tid].pos = -1; }
  if (tid == 0) { sctl[0] = 0; sctl[1] = 0; sctl[6] = 0; ((int*)(kvm_smem + KVM_ST_HDR - 128 - 288))[0] = 0; ((int*)(kvm_smem + KVM_ST_HDR - 128 - 288))[1] = 0; }
  kvm_tc_init(ctl, kvm_smem);
  const unsigned ring_ns = T.ring == 2 ? 2u : 3u;
  const int ring_bytes = (int)ring_ns * KVM_ST_STAGE;
  const bool use_ring = T.ring && dyn >= KVM_ST_HDR + ring_bytes + 32768;
  if (tid == 64 && use_ring) {
    for (int s = 0; s < 3; ++s) { kvm_mbar_init(sbar + 8 * s, 1); kvm_mbar_init(sbar + 64 + 8 * s, KVM_ST_ARRIVALS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  const int cache_bytes = (int)(((size_t)S.nbufs * sizeof(KvmBuf) + 1023) & ~(size_t)1023);
  const bool buf_cache = !use_ring && S.buf_cache && cache_bytes <= KVM_BUFCACHE_BYTES && dyn >= KVM_ST_HDR + KVM_BUFCACHE_BYTES + 192 * 1024;
  if (buf_cache) {
    const uint4* src = (const uint4*)S.bufs;
    uint4* dst = (uint4*)(kvm_smem + KVM_ST_HDR);
    for (int i = tid; i < S.nbufs * 2; i += KVM_ST_THREADS) dst[i] = src[i];
  }
  __syncthreads();
  const unsigned long long t_begin = kvm_globaltimer();
  const unsigned long long deadline = t_begin + S.timeout_ns;
  KvmRing ring;
  ring.bar0 = sbar;
  ring.ns = ring_ns;
  ring.base = kvm_smem + (use_ring ? dyn - ring_bytes : 0);
  ring.base_addr = kvm_smem_addr(ring.base);
  const int p_lo = T.prog_off[w], n = T.prog_off[w + 1] - p_lo;

  if (tid >= KVM_NT + 32) {
    // ---- stream warp: issues the copies of the fetched tasks in list order, as soon as there are free stages.  It does nothing else:
    // behind the dependency polls (an L2 round trip each, several microseconds when the copies saturate the memory system) a freed
    // stage waited for its next copy, and the weights arrived at half the HBM rate.
    if ((tid & 31) == 0) {
      unsigned pit = 0, idle = 0;                // stage uses issued
      bool leave = false;
      // an error may leave stages unconsumed, and the front warp may have finished its list by then: watched here too
      auto quit = [&]() { return (++idle & 1023u) == 0 && (kvm_ld_volatile_shared(&sctl[6]) || *(volatile int*)&S.err->code != 0 || kvm_globaltimer() > deadline); };
      for (int ii = 0; ii < n && !leave; ++ii) {
        KvmStSlot& sl = slots[ii % KVM_ST_SLOTS];
        // The record may have come and gone if the task does not stream (its slot is refilled once it has finished); one that streams
        // stays until its copies are issued here, so a kind read between two looks at the same position belongs to it.
        int kind = 0;
        while (true) {
          const int seen = kvm_ld_volatile_shared(&sl.pos);
          if (seen == ii) {
            kind = kvm_ld_volatile_shared(&sl.kind);
            if (kvm_ld_volatile_shared(&sl.pos) != ii) kind = 0;
            break;
          }
          if (seen > ii) break;
          if (quit()) { leave = true; break; }
        }
        if (leave || kind == 0) continue;
        __threadfence_block();
        const bool pre = sl.prefetch & 1;
        // constants may run ahead; anything else waits until the task is ready
        while (!pre && kvm_ld_volatile_shared(&sl.state) < 2) if (quit()) { leave = true; break; }
        if (!pre) asm volatile("fence.proxy.async;" ::: "memory");      // data other workers wrote with plain stores, read here by bulk copies
        const int nch = sl.nchunks;
        for (int ci = 0; ci < nch && !leave; ++ci) {
          while (pit >= ring.ns && !kvm_mbar_test(kvm_ring_empty(ring, pit), kvm_ring_parity(ring, pit) ^ 1u))
            if (quit()) { leave = true; break; }
          if (leave) break;
          kvm_static_issue(S, sl, ring, pit, ci);
          ++pit;
        }
      }
      sctl[2] = (int)pit;
    }
  } else if (tid >= KVM_NT) {
    // ---- front warp: fetches the records of the next tasks and finds them ready
    const int lane = tid & 31;
    int fi = 0, ri = 0;                        // next position to fetch / to mark ready
    int dep[5] = {-1, -1, -1, -1, -1}, dep_pos = -1;     // dependency entries of the task at `ri`
    bool stop = false;
    unsigned idle = 0;
    while (!stop && ri < n) {
      bool progressed = false;
      // 1. fetch the next record into a free slot
      if (fi < n && __shfl_sync(0xffffffffu, lane == 0 ? kvm_ld_volatile_shared(&slots[fi % KVM_ST_SLOTS].state) : 0, 0) == 0) {      // the warp decides as one
        KvmStSlot& sl = slots[fi % KVM_ST_SLOTS];
        const int task = T.prog[p_lo + fi];
        if (lane == 0) { *(volatile int*)&sl.pos = -1; __threadfence_block(); }      // see the stream warp
        const int32_t* rec = S.recs + (size_t)task * KVM_REC_WORDS;
        const int32_t w0 = rec[lane], w1 = lane < 16 ? rec[32 + lane] : 0;
        if (lane < 16) sl.desc[lane] = w0; else sl.args[lane - 16] = w0;
        if (lane < 4) sl.args[16 + lane] = w1; else if (lane < 8) ((int32_t*)&sl.aux)[lane - 4] = w1;
        if (lane == 8) sl.wait_off = w1;
        if (lane == 9) sl.wait_cnt = w1;
        if (lane == 10) sl.prefetch = w1 & 1;
        if (lane == 31) sl.task = task;
        __syncwarp();
        if (use_ring) {                                      // table entries of the buffer arguments of a streaming op, lanes in parallel
          const int op = sl.desc[0], nb = (op == 134 || op == 301) ? 6 : (op == 135 || op == 300) ? 7 : 0;
          if (lane < nb) {
            const int idx = sl.args[lane];
            KvmBuf e; e.p = nullptr; e.rows = e.cols = e.ld = 0; e.dtype = 0; e.reserved[0] = e.reserved[1] = 0;
            if (idx >= 0 && idx < S.nbufs) e = S.bufs[idx];
            sl.lb[lane] = e;
          }
          __syncwarp();
        }
        if (lane == 0) {
          if (use_ring) kvm_static_geometry(S, sl, (int)dyn - KVM_ST_HDR - ring_bytes); else { sl.kind = 0; sl.nchunks = 0; }
          __threadfence_block();
          *(volatile int*)&sl.state = 1;
          *(volatile int*)&sl.pos = fi;
        }
        __syncwarp();
        ++fi; progressed = true;
      }
      // 2. dependencies of the next task to become ready: its entries are held in registers (up to five per lane) and polled with
      //    plain loads, all in flight together; one acquire fence once they are all met
      if (ri < fi) {
        KvmStSlot& sl = slots[ri % KVM_ST_SLOTS];
        if (dep_pos != ri) {
          const int off = sl.wait_off, cnt = sl.wait_cnt;
#pragma unroll
          for (int j = 0; j < 5; ++j) dep[j] = lane + 32 * j < cnt ? T.waits[off + lane + 32 * j] : -1;
          dep_pos = ri;
        }
        int seen[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) seen[j] = dep[j] >= 0 ? kvm_ld_relaxed(&T.progress[dep[j] >> KVM_ST_WAIT_BITS]) : 0;
        bool met = true;
#pragma unroll
        for (int j = 0; j < 5; ++j) if (dep[j] >= 0 && seen[j] < (dep[j] & ((1 << KVM_ST_WAIT_BITS) - 1))) met = false;
        if (__all_sync(0xffffffffu, met)) {
          __threadfence();                                   // acquire: what the finished predecessors wrote is visible to this CTA's compute group
          if (lane == 0) { S.indeg[sl.task] = 0; sl.state = 2; }     // every predecessor's completion was observed
          __syncwarp();
          ++ri; progressed = true;
        }
      }
      // 3. failure / stall
      if (!progressed) {
        if ((++idle & 63u) == 0) {
          int e = 0;
          if (lane == 0) e = *(volatile int*)&S.err->code;
          e = __shfl_sync(0xffffffffu, e, 0);
          if (e != 0) stop = true;
          else if (kvm_globaltimer() > deadline) {
            if (lane == 0) kvm_dev_fail(S, KVM_ERR_TIMEOUT, ri < n ? T.prog[p_lo + ri] : -1, ri, fi);
            stop = true;
          }
        }
      } else idle = 0;
    }
    // leave: the compute group takes slots in order; the first one that is not ready tells it to go
    if (stop) {
      if (lane == 0) {
        sctl[6] = 1;
        for (int k = 0; k < KVM_ST_SLOTS; ++k) {
          KvmStSlot& sl = slots[(ri + k) % KVM_ST_SLOTS];
          if (kvm_ld_volatile_shared(&sl.state) != 2) { sl.state = 3; break; }
        }
      }
    }
  } else {
    KvmCtx& c = *(KvmCtx*)(kvm_smem + KVM_ST_HDR - 128 - 288 - KVM_ST_CTX_BYTES);      // in shared memory (see kvm_sched.cuh)
    if (tid == 0) {
      c.nbufs = S.nbufs; c.err = S.err; c.cfg_flags = S.cfg_flags; c.ctl = ctl; c.tmaps = S.tmaps; c.pair = -1; c.engine = 0; c.gemm_seq = 0;
      c.rope_cache = (float*)(kvm_smem + KVM_ST_HDR - 128 - 288);
      c.yield_word = nullptr; c.yield_count = nullptr; c.q_head = c.q_tail = nullptr;      // program order: a waiting task waits in place
      c.deadline = deadline - S.timeout_ns / 8;      // a task's own wait gives up (and names itself) before the launch's stall limit does
      c.bufs = buf_cache ? (const KvmBuf*)(kvm_smem + KVM_ST_HDR) : S.bufs;
      const int used = KVM_ST_HDR + (buf_cache ? cache_bytes : 0);
      c.smem = kvm_smem + used;
      c.smem_bytes = (int)dyn - used - (use_ring ? ring_bytes : 0);
    }
    unsigned cit = 0;
    int i = 0;
    for (; i < n; ++i) {
      KvmStSlot& sl = slots[i % KVM_ST_SLOTS];
      if (tid == 0) {
        unsigned polls = 0;
        int st;
        while ((st = kvm_ld_volatile_shared(&sl.state)) < 2) {
          if ((++polls & 1023u) == 0 && kvm_globaltimer() > c.deadline + 2 * S.timeout_ns) { st = 3; break; }      // the front warp always answers first
        }
        sl.go = st == 3 ? 0 : (*(volatile int*)&S.err->code == 0 ? 1 : 2);
        c.task = sl.task;
      }
      kvm_sync();
      const int go = kvm_ld_volatile_shared(&sl.go);
      if (go == 0) break;
      const int task = sl.task;
      if (tid == 0 && S.trace) { const unsigned long long t_task = kvm_globaltimer(); S.t_start[task] = t_task; sctl[3] = sctl[4] = sctl[3 + KVM_ST_WAITED] = 0; sctl[5] = (int)t_task; }
      const int op = sl.desc[0], kind = sl.kind, nch = sl.nchunks;
      if (kind == 1) {
        const int J = kvm_gv_pieces(sl.args[8]);
        if (S.trace) kvm_gemv_ring_traced(c, sl.args, sl.lb, ring, cit, sl.R, nch, sctl + 3);
        else if (J == 1) kvm_gemv_ring<1, false>(c, sl.args, sl.lb, ring, cit, sl.R, nch, nullptr);
        else if (J <= 3) kvm_gemv_ring<3, false>(c, sl.args, sl.lb, ring, cit, sl.R, nch, nullptr);
        else kvm_gemv_ring_wide(c, sl.args, sl.lb, ring, cit, sl.R, nch);
      }
      else if (kind == 3) kvm_gemv_mma_ring(c, sl.args, sl.lb, op == 301, ring, cit, sl.newrow, S.trace ? sctl + 3 : nullptr);
      else if (kind == 2) {
        if (!kvm_ra_takes(sl.args[13], sl.args[17])) kvm_attn_part_ring_any(c, sl.args, sl.lb, op == 300, ring, cit, sl.j0, sl.j1, sl.newrow, S.trace ? sctl + 3 : nullptr);
        else if (S.trace) kvm_attn_part_ring_traced(c, sl.args, sl.lb, op == 300, ring, cit, sl.j0, sl.j1, sl.newrow, sctl + 3);
        else kvm_attn_part_ring<false>(c, sl.args, sl.lb, op == 300, ring, cit, sl.j0, sl.j1, sl.newrow, nullptr);
      }
      else if (op != 0 && go == 1 && !(op == 136 && kvm_hot_merge(c, sl.args))) kvm_dispatch(c, op, sl.args, sl.aux);
      cit += (unsigned)nch;
      // Results that a later bulk copy or TMA load may read (cache rows appended by an attention split, operands of tensor-core ops)
      // need the writer's generic-to-async proxy fence.  A streamed GEMV writes activations only, which every consumer reads with
      // plain loads: it skips the fence (it waits for the task's global stores, about a microsecond per task).
      if (kind != 1 && kind != 3) asm volatile("fence.proxy.async;" ::: "memory");
      kvm_sync();
      if (tid == 0) {
        if (S.trace) {                                       // bits 8.. : detail of a streamed task (kvm_trace_detail)
          const int pro = sctl[3] ? sctl[3] - sctl[5] : 0, waits = sctl[3 + KVM_ST_WAITED];
          const int detail = kind == 1 || kind == 3 ? min(255, pro / 200) | min(255, (sctl[4] - sctl[3]) / 200) << 8 | min(255, waits / 200) << 16
                           : kind == 2 ? min(255, pro / 100) | min(255, waits / 100) << 8 : 0;
          S.t_end[task] = kvm_globaltimer(); S.t_smid[task] = (int)kvm_smid() | (detail << 8);
        }
        atomicAdd(&S.exec_count[task], 1);                   // no result needed: nothing waits for the old value
        const int pv = sl.desc[10];
        if (pv >= 0) {                                       // publish (include/mvm_task_abi.h:20-23): old + 1, else VERSION_GAP
          if (pv >= S.nvars) kvm_dev_fail(S, KVM_ERR_BAD_VAR, task, pv);
          else {
            __threadfence();                                 // the task's writes before its version
            const int ver = sl.desc[11] + S.ver_off[pv];
            if (atomicCAS(&S.versions[pv], ver - 1, ver) != ver - 1) kvm_dev_fail(S, KVM_ERR_VERSION_GAP, task, pv, ver);
          }
        }
        kvm_st_release(&T.progress[w], i + 1);               // release at gpu scope: the CTA's writes (ordered before this thread by the barrier) come first
        sctl[0] = (int)cit;
        sl.state = 0;
      }
    }
    if (tid == 0) { sctl[1] = i; atomicAdd(S.done, i); }
  }
  __syncthreads();
  // copies issued but never consumed (an early exit): wait for them, bounded, before the shared memory goes away
  if (use_ring && tid == KVM_NT + 32) {
    const unsigned pit = (unsigned)sctl[2], cit = (unsigned)sctl[0];
    for (unsigned it = cit; it < pit; ++it) {
      const uint32_t bar = kvm_ring_full(ring, it), par = kvm_ring_parity(ring, it);
      const unsigned long long t0 = kvm_globaltimer();
      unsigned spins = 0;
      while (!kvm_mbar_test(bar, par)) if ((++spins & 63u) == 0 && kvm_globaltimer() - t0 > 50000000ull) break;      // 50 ms: a bulk copy lands in microseconds
    }
  }
  __syncthreads();
  kvm_tc_fini(ctl);
}

// Arm kernel of the static path: progress words and witnesses cleared, version offsets taken.
__global__ void kvm_static_arm_kernel(KvmStaticState T, int workers) {
  const KvmDevState& S = T.D;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < S.nt) { S.indeg[i] = S.tasks[i].indegree; S.exec_count[i] = 0; }
  if (i < workers) T.progress[i] = 0;
  if (i < S.nvars) S.ver_off[i] = S.versions[i] - S.ver_base[i];
}
