// Typed bodies of the memory-bound ops that make up most of the tasks of a training program, inlined into the executor kernels (a
// call would save and restore some fifty registers per thread through local memory, which the little L1 beside 227 KB of shared
// memory cannot hold: 2-4 us per task).  Each takes the common storage types and alignments and returns false for anything else,
// argument errors included: the op's general body (kvm_ops_rows.cuh, kvm_ops_flat.cuh, kvm_ops_attn.cuh) then does the task or
// reports the error.  Storage types are template arguments, so that the loads of a batch are issued back to back.
// One SM's share of HBM is 44 KB/us at a loaded latency of 1.5 us: 66 KB in flight keep it busy.  The streaming loops have 64 to 128.
#pragma once
#include "kvm_attn_tc.cuh"
#include "kvm_decode_stream.cuh"
#include "kvm_dev.cuh"
#include "kvm_ops_flat.cuh"
#include "kvm_ops_rows.cuh"

__device__ __forceinline__ bool kvm_hot_buf(const KvmCtx& c, int idx, int dtype, KvmBuf& out) {
  if (idx < 0 || idx >= c.nbufs) return false;
  out = c.bufs[idx];
  return out.p != nullptr && out.dtype == dtype && ((uintptr_t)out.p & 15) == 0;
}
__device__ __forceinline__ bool kvm_hot_float(const KvmCtx& c, int idx, KvmBuf& out) {
  if (idx < 0 || idx >= c.nbufs) return false;
  out = c.bufs[idx];
  return out.p != nullptr && out.dtype != KVM_I32 && ((uintptr_t)out.p & 15) == 0;
}
__device__ __forceinline__ bool kvm_hot_mat(const KvmBuf& b, int rows, int cols) { return rows <= b.rows && cols <= b.cols && (b.ld & 3) == 0; }
__device__ __forceinline__ bool kvm_hot_flat(const KvmBuf& b, long long n) { return b.ld == b.cols && n <= (long long)b.rows * b.cols; }
__device__ __forceinline__ float4 kvm_bf16x4(uint2 u) { return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u)); }
__device__ __forceinline__ uint2 kvm_to_bf16x4(float4 v) {
  uint2 u;
  ((__nv_bfloat162*)&u)[0] = __floats2bfloat162_rn(v.x, v.y);
  ((__nv_bfloat162*)&u)[1] = __floats2bfloat162_rn(v.z, v.w);
  return u;
}
__device__ __forceinline__ void kvm_st4(const KvmBuf& b, size_t i, float4 v) {
  if (b.dtype == KVM_BF16) *(uint2*)((__nv_bfloat16*)b.p + i) = kvm_to_bf16x4(v);
  else *(float4*)((float*)b.p + i) = v;
}

// ---- layernorm forward, float32 rows -------------------------------------------------------------------------------------------
// A warp per row, NV float4 per lane (pairs of them make up eight neighbouring columns: the general body's order of summation, for rows of
// a multiple of eight columns); gamma and beta wait in shared memory, the next row is in flight while this one is reduced.
__device__ __forceinline__ int kvm_hot_ln_col(int t) { return (threadIdx.x & 31) * 8 + (t >> 1) * 256 + (t & 1) * 4; }      // first column of a lane's piece t
template <int NV>
__device__ __forceinline__ void kvm_hot_ln_fwd_t(const KvmBuf& x, const KvmBuf& out, float* mean, float* rstd, const float* gs, int r0, int r1, int d, float eps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* xp = (const float*)x.p;
  constexpr bool AHEAD = NV <= 6;                     // 1024-wide rows leave no registers for a second one
  float4 nx[NV];
  auto load = [&](int r) {
#pragma unroll
    for (int t = 0; t < NV; ++t) { const int k = kvm_hot_ln_col(t); nx[t] = (r < r1 && k < d) ? *(const float4*)(xp + (size_t)r * x.ld + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
  };
  if (AHEAD) load(r0 + warp);
#pragma unroll 1
  for (int r = r0 + warp; r < r1; r += KVM_NWARPS) {
    float4 v[NV];
    float s = 0.0f, q = 0.0f;
    if (!AHEAD) load(r);
#pragma unroll
    for (int t = 0; t < NV; ++t) { v[t] = nx[t]; s += v[t].x; s += v[t].y; s += v[t].z; s += v[t].w; }
    if (AHEAD) load(r + KVM_NWARPS);
    const float mu = kvm_warp_sum(s) / d;
#pragma unroll
    for (int t = 0; t < NV; ++t) if (kvm_hot_ln_col(t) < d) {
      v[t].x -= mu; v[t].y -= mu; v[t].z -= mu; v[t].w -= mu;
      q += v[t].x * v[t].x; q += v[t].y * v[t].y; q += v[t].z * v[t].z; q += v[t].w * v[t].w;
    }
    const float rs = 1.0f / sqrtf(kvm_warp_sum(q) / d + eps);
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const int k = kvm_hot_ln_col(t);
      if (k < d) {
        const float4 g = *(const float4*)(gs + k), b = *(const float4*)(gs + 1024 + k);
        kvm_st4(out, (size_t)r * out.ld + k, make_float4(v[t].x * rs * g.x + b.x, v[t].y * rs * g.y + b.y, v[t].z * rs * g.z + b.z, v[t].w * rs * g.w + b.w));
      }
    }
    if (lane == 0) { rstd[r] = rs; mean[r] = mu; }
  }
}
__device__ __forceinline__ bool kvm_hot_ln_fwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, g, be, out, mean, rstd;
  const int r0 = a[6], r1 = a[7], d = a[8];
  const float eps = kvm_bits_f32(a[9]);
  if (!kvm_hot_buf(c, a[0], KVM_F32, x) || !kvm_hot_buf(c, a[1], KVM_F32, g) || !kvm_hot_buf(c, a[2], KVM_F32, be) || !kvm_hot_float(c, a[3], out) || !kvm_hot_buf(c, a[4], KVM_F32, mean) ||
      !kvm_hot_buf(c, a[5], KVM_F32, rstd)) return false;
  if (r0 < 0 || r1 < r0 || d <= 0 || d > 1024 || ((d | x.ld | out.ld) & 7) || !kvm_hot_mat(x, r1, d) || !kvm_hot_mat(out, r1, d) || !kvm_hot_flat(g, d) || !kvm_hot_flat(be, d) || !kvm_hot_flat(mean, r1) ||
      !kvm_hot_flat(rstd, r1)) return false;
  float* gs = (float*)c.smem;                     // gamma, beta
  kvm_sync();
  if (threadIdx.x * 4 < d) { *(float4*)(gs + threadIdx.x * 4) = *(const float4*)((const float*)g.p + threadIdx.x * 4); *(float4*)(gs + 1024 + threadIdx.x * 4) = *(const float4*)((const float*)be.p + threadIdx.x * 4); }
  kvm_sync();
  float* mp = (float*)mean.p; float* rp = (float*)rstd.p;
  if (d <= 256) kvm_hot_ln_fwd_t<2>(x, out, mp, rp, gs, r0, r1, d, eps);
  else if (d <= 768) kvm_hot_ln_fwd_t<6>(x, out, mp, rp, gs, r0, r1, d, eps);
  else kvm_hot_ln_fwd_t<8>(x, out, mp, rp, gs, r0, r1, d, eps);
  return true;
}

// ---- layernorm backward (dx), float32 x / dx, dy float32 or bf16 ------------------------------------------------------------------------
template <int NV, bool YB>
__device__ __forceinline__ void kvm_hot_ln_bwd_t(const KvmBuf& x, const KvmBuf& dy, const KvmBuf& dx, const float* mean, const float* rstd, const float* gs, int r0, int r1, int d, int acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
  for (int r = r0 + warp; r < r1; r += KVM_NWARPS) {
    float4 xv[NV], yf[YB ? 1 : NV];
    uint2 yb[YB ? NV : 1];
    const float* xp = (const float*)x.p + (size_t)r * x.ld;
    float* op = (float*)dx.p + (size_t)r * dx.ld;
#pragma unroll
    for (int t = 0; t < NV; ++t) { const int k = kvm_hot_ln_col(t); xv[t] = k < d ? *(const float4*)(xp + k) : zero; }
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const int k = kvm_hot_ln_col(t);
      if (YB) yb[t] = k < d ? *(const uint2*)((const __nv_bfloat16*)dy.p + (size_t)r * dy.ld + k) : make_uint2(0u, 0u);
      else yf[t] = k < d ? *(const float4*)((const float*)dy.p + (size_t)r * dy.ld + k) : zero;
    }
    const float mu = mean[r], rs = rstd[r];
    auto grad = [&](int t) {                       // dy * gamma of this lane's piece t
      const int k = kvm_hot_ln_col(t);
      const float4 y = YB ? kvm_bf16x4(yb[YB ? t : 0]) : yf[YB ? 0 : t];
      if (k >= d) return zero;
      const float4 g = *(const float4*)(gs + k);
      return make_float4(y.x * g.x, y.y * g.y, y.z * g.z, y.w * g.w);
    };
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const float4 g = grad(t);
      xv[t] = make_float4((xv[t].x - mu) * rs, (xv[t].y - mu) * rs, (xv[t].z - mu) * rs, (xv[t].w - mu) * rs);
      s1 += g.x; s2 += g.x * xv[t].x; s1 += g.y; s2 += g.y * xv[t].y;
      s1 += g.z; s2 += g.z * xv[t].z; s1 += g.w; s2 += g.w * xv[t].w;
    }
    s1 = kvm_warp_sum(s1) / d;
    s2 = kvm_warp_sum(s2) / d;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const int k = kvm_hot_ln_col(t);
      if (k < d) {
        const float4 g = grad(t);
        const float4 o = acc ? *(const float4*)(op + k) : zero;
        float4 v = make_float4(rs * (g.x - s1 - xv[t].x * s2), rs * (g.y - s1 - xv[t].y * s2), rs * (g.z - s1 - xv[t].z * s2), rs * (g.w - s1 - xv[t].w * s2));
        if (acc) v = make_float4(__fadd_rn(o.x, v.x), __fadd_rn(o.y, v.y), __fadd_rn(o.z, v.z), __fadd_rn(o.w, v.w));
        *(float4*)(op + k) = v;
      }
    }
  }
}
__device__ __forceinline__ bool kvm_hot_ln_bwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, dy, g, mean, rstd, dx;
  const int r0 = a[6], r1 = a[7], d = a[8], acc = a[9];
  if (!kvm_hot_buf(c, a[0], KVM_F32, x) || !kvm_hot_float(c, a[1], dy) || !kvm_hot_buf(c, a[2], KVM_F32, g) || !kvm_hot_buf(c, a[3], KVM_F32, mean) || !kvm_hot_buf(c, a[4], KVM_F32, rstd) ||
      !kvm_hot_buf(c, a[5], KVM_F32, dx)) return false;
  if (r0 < 0 || r1 < r0 || d <= 0 || d > 1024 || ((d | x.ld | dy.ld | dx.ld) & 7) || !kvm_hot_mat(x, r1, d) || !kvm_hot_mat(dy, r1, d) || !kvm_hot_mat(dx, r1, d) || !kvm_hot_flat(g, d) || !kvm_hot_flat(mean, r1) ||
      !kvm_hot_flat(rstd, r1)) return false;
  float* gs = (float*)c.smem;
  kvm_sync();
  if (threadIdx.x * 4 < d) *(float4*)(gs + threadIdx.x * 4) = *(const float4*)((const float*)g.p + threadIdx.x * 4);
  kvm_sync();
  const float* mp = (const float*)mean.p; const float* rp = (const float*)rstd.p;
  const bool yb = dy.dtype == KVM_BF16;
  if (d <= 256) { if (yb) kvm_hot_ln_bwd_t<2, true>(x, dy, dx, mp, rp, gs, r0, r1, d, acc); else kvm_hot_ln_bwd_t<2, false>(x, dy, dx, mp, rp, gs, r0, r1, d, acc); }
  else if (!yb) return false;                      // wide float32 rows: the general body
  else if (d <= 768) kvm_hot_ln_bwd_t<6, true>(x, dy, dx, mp, rp, gs, r0, r1, d, acc);
  else kvm_hot_ln_bwd_t<8, true>(x, dy, dx, mp, rp, gs, r0, r1, d, acc);
  return true;
}

// ---- column sums (and the parameter gradients of a norm) -------------------------------------------------------------------------------
// 64 columns at a time.  Rows come through shared memory, copied sixteen bytes at a time, 72 to 112 KB in flight (one column per thread
// straight from global memory left the loop at 10 KB/us); they are added from there by eight row groups of a thread per column, in the
// general body's order.  Bound by HBM: 8192 rows of 64 columns take 43 us for a column sum of bf16 rows and 111 us for the parameter
// gradients of a norm in the 162M step (94 and 301 in the general body).
__device__ __forceinline__ void kvm_cp_async(uint32_t dst, const void* src, int bytes) {      // 16 or 4
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
template <int MODE, bool XB, bool YB> struct KvmColStage {
  static constexpr int S = MODE == 0 && XB ? 128 : 64, DEPTH = MODE == 0 ? 8 : 4;      // rows of a stage, stages (of 16 KB, 24 or 32 KB for two operands)
  static constexpr int XR = XB ? 128 : 256, YR = MODE == 0 ? 0 : YB ? 128 : 256;      // bytes of a staged row
  static constexpr int OFF_Y = S * XR, OFF_M = OFF_Y + S * YR, BYTES = OFF_M + (MODE == 1 ? S * 8 : 0);      // x | dy | mean | rstd
  static constexpr int SCRATCH = DEPTH * BYTES + KVM_NT * 8;           // and the row groups' sums
};
template <int MODE, bool XB, bool YB>
__device__ __forceinline__ bool kvm_hot_colreduce_t(const KvmCtx& c, const KvmBuf& x, const KvmBuf& dy, const float* mean, const float* rstd, float* o1, float* o2, int R, int c0, int c1, int acc) {
  typedef KvmColStage<MODE, XB, YB> G;
  if (c.smem_bytes < G::SCRATCH) return false;
  const int tid = threadIdx.x, col = tid & 63, rg = tid >> 6, ns = (R + G::S - 1) / G::S;
  const uint32_t base = kvm_smem_addr(c.smem);
  float* red = (float*)(c.smem + G::DEPTH * G::BYTES);
#pragma unroll 1
  for (int cb = c0; cb < c1; cb += 64) {
    const int w = min(64, c1 - cb);
    auto issue = [&](int st) {                         // one group of copies, empty past the last stage
      if (st < ns) {
        const int r0 = st * G::S;
        const uint32_t dst = base + (st & (G::DEPTH - 1)) * G::BYTES;
#pragma unroll
        for (int i = tid; i < G::S * G::XR / 16; i += KVM_NT) {
          const int r = i / (G::XR / 16), k = i % (G::XR / 16) * (XB ? 8 : 4);
          if (r0 + r < R && k < w) kvm_cp_async(dst + r * G::XR + k * (XB ? 2 : 4), (const char*)x.p + ((size_t)(r0 + r) * x.ld + cb + k) * (XB ? 2 : 4), 16);
        }
        if (MODE == 1)
#pragma unroll
          for (int i = tid; i < G::S * G::YR / 16; i += KVM_NT) {
            const int r = i / (MODE == 1 ? G::YR / 16 : 1), k = i % (MODE == 1 ? G::YR / 16 : 1) * (YB ? 8 : 4);
            if (r0 + r < R && k < w) kvm_cp_async(dst + G::OFF_Y + r * G::YR + k * (YB ? 2 : 4), (const char*)dy.p + ((size_t)(r0 + r) * dy.ld + cb + k) * (YB ? 2 : 4), 16);
          }
        if (MODE == 1 && tid < 2 * G::S && r0 + (tid & (G::S - 1)) < R) kvm_cp_async(dst + G::OFF_M + tid * 4, (tid < G::S ? mean : rstd) + r0 + (tid & (G::S - 1)), 4);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    kvm_sync();                                        // the scratch is free
#pragma unroll
    for (int st = 0; st < G::DEPTH - 1; ++st) issue(st);
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll 1
    for (int st = 0; st < ns; ++st) {
      asm volatile("cp.async.wait_group %0;" ::"n"(G::DEPTH - 2) : "memory");
      kvm_sync();                                      // the stage has landed for everyone, and everyone is done with the one before
      issue(st + G::DEPTH - 1);
      const unsigned char* sm = c.smem + (st & (G::DEPTH - 1)) * G::BYTES;
      const int left = R - st * G::S;
      auto ldx = [&](int r) { return XB ? __bfloat162float(*(const __nv_bfloat16*)(sm + r * G::XR + col * 2)) : *(const float*)(sm + r * G::XR + col * 4); };
      auto ldy = [&](int r) { return YB ? __bfloat162float(*(const __nv_bfloat16*)(sm + G::OFF_Y + r * G::YR + col * 2)) : *(const float*)(sm + G::OFF_Y + r * G::YR + col * 4); };
      const float* mu = (const float*)(sm + G::OFF_M);
      auto add = [&](float xv, float gv, float m, float rs) { if (MODE == 0) s1 += xv; else { s1 += gv * (xv - m) * rs; s2 += gv; } };
      if (col < w) {
        if (left >= G::S) {                            // a whole stage: eight rows' values before the first of them is added
#pragma unroll
          for (int b = 0; b < G::S; b += 64) {
            float xv[8], gv[8], mv[8], rv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int r = b + u * 8 + rg;
              xv[u] = ldx(r);
              gv[u] = MODE == 1 ? ldy(r) : 0.0f; mv[u] = MODE == 1 ? mu[r] : 0.0f; rv[u] = MODE == 1 ? mu[G::S + r] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) add(xv[u], gv[u], mv[u], rv[u]);
          }
        } else {
#pragma unroll 1
          for (int r = rg; r < left; r += 8) add(ldx(r), MODE == 1 ? ldy(r) : 0.0f, MODE == 1 ? mu[r] : 0.0f, MODE == 1 ? mu[G::S + r] : 0.0f);
        }
      }
    }
    red[tid] = s1;
    if (MODE == 1) red[KVM_NT + tid] = s2;
    kvm_sync();
    if (tid < (MODE == 1 ? 128 : 64)) {
      const int k = tid & 63, m = tid >> 6, cc = cb + k;
      float t = 0.0f;
#pragma unroll
      for (int g = 0; g < 8; ++g) t += red[m * KVM_NT + g * 64 + k];
      float* o = m ? o2 : o1;
      if (cc < c1) o[cc] = acc ? __fadd_rn(o[cc], t) : t;
    }
  }
  return true;
}
// columns [c0, c1) in pieces of sixteen bytes
__device__ __forceinline__ bool kvm_hot_cols(const KvmBuf& b, int c0, int c1) { return ((c0 | c1 | b.ld) & (b.dtype == KVM_BF16 ? 7 : 3)) == 0; }
__device__ __forceinline__ bool kvm_hot_colsum(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, out;
  const int R = a[2], c0 = a[3], c1 = a[4];
  if (!kvm_hot_float(c, a[0], x) || !kvm_hot_buf(c, a[1], KVM_F32, out)) return false;
  if (R < 0 || c0 < 0 || c1 < c0 || !kvm_hot_cols(x, c0, c1) || !kvm_hot_mat(x, R, c1) || !kvm_hot_flat(out, c1)) return false;
  KvmBuf none{};
  if (x.dtype == KVM_BF16) return kvm_hot_colreduce_t<0, true, false>(c, x, none, nullptr, nullptr, (float*)out.p, nullptr, R, c0, c1, a[5]);
  return kvm_hot_colreduce_t<0, false, false>(c, x, none, nullptr, nullptr, (float*)out.p, nullptr, R, c0, c1, a[5]);
}
__device__ __forceinline__ bool kvm_hot_norm_params(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, dy, mean, rstd, dg, db;
  const int R = a[6], d = a[7], c0 = a[8], c1 = a[9];
  if (!kvm_hot_float(c, a[0], x) || !kvm_hot_float(c, a[1], dy) || !kvm_hot_buf(c, a[2], KVM_F32, mean) || !kvm_hot_buf(c, a[3], KVM_F32, rstd) || !kvm_hot_buf(c, a[4], KVM_F32, dg) ||
      !kvm_hot_buf(c, a[5], KVM_F32, db)) return false;
  if (R < 0 || c0 < 0 || c1 < c0 || c1 > d || !kvm_hot_cols(x, c0, c1) || !kvm_hot_cols(dy, c0, c1) || !kvm_hot_mat(x, R, d) || !kvm_hot_mat(dy, R, d) || !kvm_hot_flat(mean, R) || !kvm_hot_flat(rstd, R) || !kvm_hot_flat(dg, d) ||
      !kvm_hot_flat(db, d)) return false;
  if (x.dtype == KVM_BF16) {
    if (dy.dtype == KVM_BF16) return kvm_hot_colreduce_t<1, true, true>(c, x, dy, (const float*)mean.p, (const float*)rstd.p, (float*)dg.p, (float*)db.p, R, c0, c1, a[10]);
    return false;                                  // bf16 x with a float32 gradient: the general body
  }
  if (dy.dtype == KVM_BF16) return kvm_hot_colreduce_t<1, false, true>(c, x, dy, (const float*)mean.p, (const float*)rstd.p, (float*)dg.p, (float*)db.p, R, c0, c1, a[10]);
  return kvm_hot_colreduce_t<1, false, false>(c, x, dy, (const float*)mean.p, (const float*)rstd.p, (float*)dg.p, (float*)db.p, R, c0, c1, a[10]);
}

// ---- attention delta: sum over a head's columns of o * dO -----------------------------------------------------------------------------
// An item is 8 neighbouring columns (hd / 8 neighbouring lanes make a head), four items per thread in flight.
template <bool B>
__device__ __forceinline__ void kvm_hot_delta_t(const KvmBuf& o, const KvmBuf& dO, float* delta, int r0, int r1, int T, int H, int hd) {
  constexpr int U = B ? 4 : 2, P = B ? 1 : 2;          // items in flight, 16-byte pieces of an item
  const int cpr = H * hd / 8, lph = hd / 8, lane = threadIdx.x & 31;
  const int dr = KVM_NT / cpr, dq = KVM_NT % cpr;      // KVM_NT items further on
  int r = r0 + threadIdx.x / cpr, q = threadIdx.x % cpr;
#pragma unroll 1
  while (__any_sync(0xffffffffu, r < r1)) {
    uint4 ov[U][P], dv[U][P];
    int rr = r, qq = q;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (rr < r1) {
        const uint4* op = (const uint4*)((const char*)o.p + ((size_t)rr * o.ld + qq * 8) * (B ? 2 : 4));
        const uint4* dp = (const uint4*)((const char*)dO.p + ((size_t)rr * dO.ld + qq * 8) * (B ? 2 : 4));
#pragma unroll
        for (int i = 0; i < P; ++i) { ov[u][i] = op[i]; dv[u][i] = dp[i]; }
      }
      rr += dr; qq += dq;
      if (qq >= cpr) { qq -= cpr; ++rr; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float s = 0.0f;
      if (r < r1) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          const uint32_t x[4] = {ov[u][i].x, ov[u][i].y, ov[u][i].z, ov[u][i].w}, y[4] = {dv[u][i].x, dv[u][i].y, dv[u][i].z, dv[u][i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (B) { s += __uint_as_float(x[j] << 16) * __uint_as_float(y[j] << 16); s += __uint_as_float(x[j] & 0xffff0000u) * __uint_as_float(y[j] & 0xffff0000u); }
            else s += __uint_as_float(x[j]) * __uint_as_float(y[j]);
          }
        }
      }
      for (int w = lph >> 1; w; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);      // KVM_NT and cpr are multiples of hd / 8: a head never straddles warps or steps
      if (r < r1 && (lane % lph) == 0) delta[(size_t)((r / T) * H + q / lph) * T + r % T] = s;
      r += dr; q += dq;
      if (q >= cpr) { q -= cpr; ++r; }
    }
  }
}
__device__ __forceinline__ bool kvm_hot_delta(const KvmCtx& c, const int32_t* a) {
  KvmBuf o, dO, delta;
  const int r0 = a[3], r1 = a[4], T = a[5], H = a[6], hd = a[7];
  if (!kvm_hot_float(c, a[0], o) || !kvm_hot_float(c, a[1], dO) || !kvm_hot_buf(c, a[2], KVM_F32, delta)) return false;
  if (o.dtype != dO.dtype || !(hd == 32 || hd == 64 || hd == 128) || r0 < 0 || r1 < r0 || T <= 0 || H <= 0 || !kvm_hot_mat(o, r1, H * hd) || !kvm_hot_mat(dO, r1, H * hd) ||
      ((o.ld | dO.ld) & 7) || !kvm_hot_flat(delta, (long long)((r1 + T - 1) / T) * H * T) || (long long)(r1 - r0) * H * hd >= (1LL << 30)) return false;
  if (o.dtype == KVM_BF16) kvm_hot_delta_t<true>(o, dO, (float*)delta.p, r0, r1, T, H, hd);
  else kvm_hot_delta_t<false>(o, dO, (float*)delta.p, r0, r1, T, H, hd);
  return true;
}

// ---- cross entropy of long bf16 rows (forward and gradient in one op) -------------------------------------------------------------------
// A row is fetched once, by a bulk copy into shared memory that runs while the row before it is worked on (two row buffers; with
// room for one only, the next copy starts when the row is done), and read from there twice: maximum and sum, gradient.  Maximum
// and sum take one barrier each.  Bound by HBM (read + write, 4 bytes per logit: 4.6 us for 50304 of them at an SM's share) with
// the exponentials (two per logit, 16 a cycle: 3.2 us) beside it; the loop it replaces read the row twice from HBM, 19 us a row.
__device__ __forceinline__ bool kvm_hot_ce_fused(const KvmCtx& c, const int32_t* a) {
  KvmBuf lg, tg, rl, ls, dl;
  const int r0 = a[5], r1 = a[6], V = a[7];
  if (!kvm_hot_buf(c, a[0], KVM_BF16, lg) || !kvm_hot_buf(c, a[1], KVM_I32, tg) || !kvm_hot_buf(c, a[2], KVM_F32, rl) || !kvm_hot_buf(c, a[3], KVM_F32, ls) || !kvm_hot_buf(c, a[4], KVM_BF16, dl)) return false;
  if (a[8] != -1 || a[9] <= 0 || r0 < 0 || r1 <= r0 || V <= 1024 || (V & 7) || ((lg.ld | dl.ld) & 7) || !kvm_hot_mat(lg, r1, V) || !kvm_hot_mat(dl, r1, V) || !kvm_hot_flat(tg, r1) ||
      !kvm_hot_flat(rl, r1) || !kvm_hot_flat(ls, r1) || c.smem_bytes < 1024 + V * 2) return false;
  const int* tp = (const int*)tg.p;
  for (int r = r0; r < r1; ++r) if (tp[r] < 0 || tp[r] >= V) return false;      // ignored rows and bad tokens: the general body
  const float f = __fmul_rn((float)(1.0 / (double)a[9]), kvm_bits_f32(a[10]));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, pitch = (V * 2 + 127) & ~127;
  const bool two = c.smem_bytes >= 1024 + 2 * pitch;
  float* red = (float*)c.smem;                         // [2][16] maxima, [2][16] sums of the warps
  int* cnt = c.ctl + KVM_CTL_ACNT + 7;
  const uint32_t bar = kvm_bar_addr(c.ctl, KVM_CTL_ABAR + 7), dst = kvm_smem_addr(c.smem + 1024);
  const __nv_bfloat16* src = (const __nv_bfloat16*)lg.p;
  const int phase0 = *cnt;
  auto fetch = [&](int r) {                            // thread 0
    kvm_mbar_expect_tx(bar, (uint32_t)V * 2);
    kvm_bulk_g2s(dst + (two ? ((r - r0) & 1) * pitch : 0), src + (size_t)r * lg.ld, (uint32_t)V * 2, bar);
  };
  kvm_sync();                                          // the scratch is free, and everyone has read the phase count
  if (tid == 0) { asm volatile("fence.proxy.async;" ::: "memory"); fetch(r0); }      // logits written by other tasks' plain stores
  bool ok = true;
#pragma unroll 1
  for (int r = r0; r < r1; ++r) {
    const unsigned char* row = c.smem + 1024 + (two ? ((r - r0) & 1) * pitch : 0);
    const int t = tp[r];
    if (!kvm_mbar_wait(bar, (phase0 + r - r0) & 1)) ok = false;
    if (two && tid == 0 && r + 1 < r1) fetch(r + 1);   // the other buffer was last read before the barrier at the end of the previous row
    float m = -INFINITY, s = 0.0f;                     // online (max, sum) per thread, as the general body
#pragma unroll 2
    for (int k = tid * 8; k < V; k += KVM_NT * 8) {
      const uint4 v = *(const uint4*)(row + k * 2);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      float x[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) { x[2 * i] = __uint_as_float(w[i] << 16); x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
      float mm = x[0];
#pragma unroll
      for (int j = 1; j < 8; ++j) mm = fmaxf(mm, x[j]);
      if (mm > m) { s *= __expf(m - mm); m = mm; }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += __expf(x[j] - m);
    }
    float* rr = red + ((r - r0) & 1) * 32;
    float M = kvm_warp_max(m);
    if (lane == 0) rr[warp] = M;
    kvm_sync();
    M = rr[0];
#pragma unroll
    for (int w = 1; w < KVM_NWARPS; ++w) M = fmaxf(M, rr[w]);
    s = m == -INFINITY ? 0.0f : s * __expf(m - M);
    s = kvm_warp_sum(s);
    if (lane == 0) rr[16 + warp] = s;
    kvm_sync();
    s = 0.0f;
#pragma unroll
    for (int w = 0; w < KVM_NWARPS; ++w) s += rr[16 + w];
    const float lse = M + logf(s);
    if (tid == 0) { ((float*)ls.p)[r] = lse; ((float*)rl.p)[r] = lse - __bfloat162float(*(const __nv_bfloat16*)(row + t * 2)); }
    __nv_bfloat16* out = (__nv_bfloat16*)dl.p + (size_t)r * dl.ld;
#pragma unroll 2
    for (int k = tid * 8; k < V; k += KVM_NT * 8) {
      const uint4 v = *(const uint4*)(row + k * 2);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      uint4 o;
      uint32_t* ow = (uint32_t*)&o;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float p = __expf(__uint_as_float(w[i] << 16) - lse), q = __expf(__uint_as_float(w[i] & 0xffff0000u) - lse);
        if (k + 2 * i == t) p -= 1.0f;
        if (k + 2 * i + 1 == t) q -= 1.0f;
        const __nv_bfloat162 h = __floats2bfloat162_rn(p * f, q * f);
        ow[i] = *(const uint32_t*)&h;
      }
      *(uint4*)(out + k) = o;
    }
    kvm_sync();                                        // everyone is done with the row
    if (!two && tid == 0 && r + 1 < r1) fetch(r + 1);
  }
  if (!ok) kvm_att_fail(c, 127);
  if (tid == 0) *cnt = phase0 + (r1 - r0);
  return true;
}

// ---- flat ranges --------------------------------------------------------------------------------------------------------------------------
// NI inputs of a flat range come through shared memory: bulk copies of SE elements per input, four stages deep (96-128 KB in flight,
// none of it in registers), every thread works on its part of the stage that has landed and stores its results from registers.
// With the same bytes in flight in registers the loops spilled, and the spills' traffic cost more than the loads.
// body(stage, i, n): stage = the inputs' parts of the stage (shared memory), elements [i, i + n) of the range.  false, with nothing done, where
// the stages do not fit the scratch.
#define KVM_STREAM_DEPTH 4
#define KVM_STREAM_BAR 8                               // barriers KVM_CTL_ABAR + 8 .. + 11 and their completed-phase counts
template <int NI, int SE, class Body>
__device__ __forceinline__ bool kvm_stream(const KvmCtx& c, const char* const (&in)[NI], const int (&eb)[NI], int e0, int e1, Body body) {
  int off[NI], bytes = 0;
#pragma unroll
  for (int n = 0; n < NI; ++n) { off[n] = bytes; bytes += SE * eb[n]; }
  if (c.smem_bytes < 1024 + KVM_STREAM_DEPTH * bytes) return false;
  const int ns = (e1 - e0 + SE - 1) / SE;
  int* cnt = c.ctl + KVM_CTL_ACNT + KVM_STREAM_BAR;
  auto bar = [&](int s) { return kvm_bar_addr(c.ctl, KVM_CTL_ABAR + KVM_STREAM_BAR + (s & (KVM_STREAM_DEPTH - 1))); };
  auto issue = [&](int s) {                            // thread 0
    const int i = e0 + s * SE, n = min(SE, e1 - i);
    uint32_t tx = 0;
#pragma unroll
    for (int k = 0; k < NI; ++k) tx += (uint32_t)(n * eb[k]);
    kvm_mbar_expect_tx(bar(s), tx);
    const uint32_t dst = kvm_smem_addr(c.smem + 1024) + (uint32_t)((s & (KVM_STREAM_DEPTH - 1)) * bytes);
#pragma unroll
    for (int k = 0; k < NI; ++k) kvm_bulk_g2s(dst + off[k], in[k] + (size_t)i * eb[k], (uint32_t)(n * eb[k]), bar(s));
  };
  uint32_t ph[KVM_STREAM_DEPTH];
#pragma unroll
  for (int s = 0; s < KVM_STREAM_DEPTH; ++s) ph[s] = (uint32_t)cnt[s];
  kvm_sync();                                          // the scratch is free, the counts have been read
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async;" ::: "memory");   // inputs written by other tasks' plain stores
    for (int s = 0; s < min(ns, KVM_STREAM_DEPTH); ++s) issue(s);
  }
  uint32_t par = 0;
#pragma unroll
  for (int s = 0; s < KVM_STREAM_DEPTH; ++s) par |= (ph[s] & 1u) << s;
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < ns; ++s) {
    const int d = s & (KVM_STREAM_DEPTH - 1);
    if (!kvm_mbar_wait(bar(s), (par >> d) & 1u)) ok = false;
    par ^= 1u << d;
    const char* st = (const char*)c.smem + 1024 + d * bytes;
    const char* part[NI];
#pragma unroll
    for (int n = 0; n < NI; ++n) part[n] = st + off[n];
    const int i = e0 + s * SE;
    body(part, i, min(SE, e1 - i));
    kvm_sync();                                        // the stage has been read
    if (threadIdx.x == 0 && s + KVM_STREAM_DEPTH < ns) issue(s + KVM_STREAM_DEPTH);
  }
  if (!ok) kvm_att_fail(c, 2000);
  if (threadIdx.x < KVM_STREAM_DEPTH) cnt[threadIdx.x] += (ns - (int)threadIdx.x + KVM_STREAM_DEPTH - 1) / KVM_STREAM_DEPTH;
  return true;
}
__device__ __forceinline__ bool kvm_hot_range(int e0, int e1, int align) { return e0 >= 0 && e1 > e0 && ((e0 | e1) & (align - 1)) == 0; }

// Elementwise map of two inputs and an output of one storage type: 8 KB of each input per stage, 16 bytes per thread.  The output may be one
// of the inputs: an element is written after its stage has landed, by the thread that reads it, and later stages are other elements.
template <bool B, class F>
__device__ __forceinline__ bool kvm_hot_map2(const KvmCtx& c, int i0, int i1, int o, int e0, int e1, F f) {
  constexpr int E = B ? 8 : 4, EB = B ? 2 : 4;
  KvmBuf x, y, z;
  const int dt = B ? KVM_BF16 : KVM_F32;
  if (!kvm_hot_range(e0, e1, E) || !kvm_hot_buf(c, i0, dt, x) || !kvm_hot_buf(c, i1, dt, y) || !kvm_hot_buf(c, o, dt, z) || !kvm_hot_flat(x, e1) || !kvm_hot_flat(y, e1) || !kvm_hot_flat(z, e1)) return false;
  const char* const in[2] = {(const char*)x.p, (const char*)y.p};
  const int eb[2] = {EB, EB};
  return kvm_stream<2, KVM_NT * E>(c, in, eb, e0, e1, [&](const char* const (&part)[2], int i, int n) {
    const int k = (int)threadIdx.x * E;
    if (k >= n) return;
    const uint4 u = *(const uint4*)(part[0] + k * EB), v = *(const uint4*)(part[1] + k * EB);
    const uint32_t p[4] = {u.x, u.y, u.z, u.w}, q[4] = {v.x, v.y, v.z, v.w};
    uint4 w;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (B) ((__nv_bfloat162*)&w)[j] = __floats2bfloat162_rn(f(__uint_as_float(p[j] << 16), __uint_as_float(q[j] << 16)), f(__uint_as_float(p[j] & 0xffff0000u), __uint_as_float(q[j] & 0xffff0000u)));
      else ((uint32_t*)&w)[j] = __float_as_uint(f(__uint_as_float(p[j]), __uint_as_float(q[j])));
    }
    *(uint4*)((char*)z.p + (size_t)(i + k) * EB) = w;
  });
}
// f32 -> bf16
__device__ __forceinline__ bool kvm_hot_round_bf16(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, o;
  const int e0 = a[2], e1 = a[3];
  if (!kvm_hot_buf(c, a[0], KVM_F32, x) || !kvm_hot_buf(c, a[1], KVM_BF16, o) || !kvm_hot_range(e0, e1, 4) || !kvm_hot_flat(x, e1) || !kvm_hot_flat(o, e1)) return false;
  const char* const in[1] = {(const char*)x.p};
  const int eb[1] = {4};
  return kvm_stream<1, 4 * KVM_NT * 4>(c, in, eb, e0, e1, [&](const char* const (&part)[1], int i, int n) {
#pragma unroll
    for (int u = 0; u < 4; ++u) { const int k = (u * KVM_NT + (int)threadIdx.x) * 4; if (k < n) *(uint2*)((__nv_bfloat16*)o.p + i + k) = kvm_to_bf16x4(*(const float4*)(part[0] + k * 4)); }
  });
}
// AdamW, float32 state
__device__ __forceinline__ bool kvm_hot_adamw(const KvmCtx& c, const int32_t* a) {
  KvmBuf p, g, m, v, gs, st;
  const int e0 = a[6], e1 = a[7];
  if (!kvm_hot_buf(c, a[0], KVM_F32, p) || !kvm_hot_buf(c, a[1], KVM_F32, g) || !kvm_hot_buf(c, a[2], KVM_F32, m) || !kvm_hot_buf(c, a[3], KVM_F32, v) || a[4] < 0 || a[4] >= c.nbufs ||
      a[5] < 0 || a[5] >= c.nbufs) return false;
  gs = c.bufs[a[4]]; st = c.bufs[a[5]];
  if (!gs.p || gs.dtype != KVM_F32 || !st.p || st.dtype != KVM_I32 || !kvm_hot_range(e0, e1, 4) || !kvm_hot_flat(p, e1) || !kvm_hot_flat(g, e1) || !kvm_hot_flat(m, e1) || !kvm_hot_flat(v, e1)) return false;
  const int t = ((const int*)st.p)[0];
  if (t < 1) return false;
  const KvmAdamK k = kvm_adamw_consts(c, t, kvm_bits_f32(a[8]), kvm_bits_f32(a[9]), kvm_bits_f32(a[10]), kvm_bits_f32(a[11]), kvm_bits_f32(a[12]), ((const float*)gs.p)[0]);
  const char* const in[4] = {(const char*)p.p, (const char*)g.p, (const char*)m.p, (const char*)v.p};
  const int eb[4] = {4, 4, 4, 4};
  float* pp = (float*)p.p; float* mp = (float*)m.p; float* vp = (float*)v.p;
  return kvm_stream<4, KVM_NT * 4>(c, in, eb, e0, e1, [&](const char* const (&part)[4], int i, int n) {
    const int q = (int)threadIdx.x * 4;
    if (q >= n) return;
    float4 P = *(const float4*)(part[0] + q * 4), M = *(const float4*)(part[2] + q * 4), W = *(const float4*)(part[3] + q * 4);
    const float4 G = *(const float4*)(part[1] + q * 4);
    kvm_adamw_step(k, G.x, P.x, M.x, W.x); kvm_adamw_step(k, G.y, P.y, M.y, W.y); kvm_adamw_step(k, G.z, P.z, M.z, W.z); kvm_adamw_step(k, G.w, P.w, M.w, W.w);
    *(float4*)(pp + i + q) = P; *(float4*)(mp + i + q) = M; *(float4*)(vp + i + q) = W;
  });
}
__device__ __forceinline__ bool kvm_hot_gradnorm(const KvmCtx& c, const int32_t* a) {
  KvmBuf g, part;
  const int slot = a[2], e0 = a[3], e1 = a[4];
  if (!kvm_hot_buf(c, a[0], KVM_F32, g) || !kvm_hot_buf(c, a[1], KVM_F32, part) || slot < 0 || !kvm_hot_range(e0, e1, 8) || !kvm_hot_flat(g, e1) || !kvm_hot_flat(part, slot + 1)) return false;
  double s = 0.0;
  const char* const in[1] = {(const char*)g.p};
  const int eb[1] = {4};
  const bool taken = kvm_stream<1, 2 * KVM_NT * 8>(c, in, eb, e0, e1, [&](const char* const (&st)[1], int, int n) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {                      // eight squares in sequence, as the general body
      const int k = (u * KVM_NT + (int)threadIdx.x) * 8;
      if (k < n) {
        const float4 v = *(const float4*)(st[0] + k * 4), w = *(const float4*)(st[0] + k * 4 + 16);
        float q = 0.0f;
        q += v.x * v.x; q += v.y * v.y; q += v.z * v.z; q += v.w * v.w;
        q += w.x * w.x; q += w.y * w.y; q += w.z * w.z; q += w.w * w.w;
        s += q;
      }
    }
  });
  if (!taken) return false;
  s = kvm_block_sum(s, (double*)c.smem);
  if (threadIdx.x == 0) ((float*)part.p)[slot] = (float)s;
  return true;
}

// The inlined form of op `op`, if there is one for this task: tcgen05 attention where the host planned it, a typed form where the buffers
// allow it.
__device__ __forceinline__ bool kvm_hot(const KvmCtx& c, int op, const int32_t* a, const int4& aux) {
  switch (op) {
    case 35: return kvm_hot_ln_fwd(c, a);
    case 37: return kvm_hot_ln_bwd(c, a);
    case 39: return kvm_hot_norm_params(c, a);
    case 41: return !a[5] && kvm_hot_map2<true>(c, a[0], a[1], a[2], a[3], a[4], [](float x, float dy) { return __fmul_rn(dy, kvm_gelu_grad(x)); });
    case 42: return kvm_hot_map2<false>(c, a[0], a[1], a[2], a[3], a[4], [](float x, float y) { return __fadd_rn(x, y); });
    case 45: case 47: case 48: return kvm_attn_tc(c, op, a, aux);
    case 46: return kvm_hot_delta(c, a);
    case 54: return kvm_hot_adamw(c, a);
    case 55: return kvm_hot_gradnorm(c, a);
    case 61: return kvm_hot_colsum(c, a);
    case 113: return kvm_hot_round_bf16(c, a);
    case 127: return kvm_hot_ce_fused(c, a);
    default: return false;
  }
}
