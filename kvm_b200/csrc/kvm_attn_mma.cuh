// Causal attention (training) forward / backward for every shape and storage type that the tcgen05 form (kvm_attn_tc.cuh: bf16, head
// dimension 64, whole 128-row blocks) does not take.  Reference semantics: runtime/ref_gpt.py:279-364 (128 rows per task, natural-log
// lse at (b*H+h)*T+t, GQA kv head = h/(H/Hkv), dk/dv summed over the whole group).
//
// Products run on mma.sync m16n8k16 (bf16 operands, float32 sums) at float32 precision: a float32 operand is split into three bf16
// terms of eight bits each and the products of terms whose orders sum to less than three are added (the rest is below 2^-24); a bf16
// operand is its own single term.  Scores of bf16 inputs are therefore exact products, and the probabilities keep float32 precision.
// The matrix unit truncates where it adds to the accumulator, so a running sum in it drifts towards zero with every instruction: sixteen
// products of the leading terms are added from zero, those of all other terms (2^-8 of them) in an accumulator of their own, and the two
// and the running sums meet in float32 adds.
//
// A warp owns sixteen rows of the task's block from the scores to the output (flash form, 32 keys at a time, nothing but operands in
// shared memory).  Warps left over share the other side: KG groups of warps take every KG-th key tile and are added up at the end in
// group order.  Registers bound the tile: scores, their gradient and at most 64 output columns (CG column groups above that).
// What bounds it: a task is one (sequence, head, 128 rows), a few tens of them on 148 SMs, so a task's own length counts: loads, two
// barriers per key block, and the chain of products.  (One warp per row with dot products from global memory, the form before: 63 us
// forward, 65 us dq and 160 us dk/dv at 64 tokens of dimension 32; 9 of the 11 ms of a step with 200 tokens of dimension 128.)
#pragma once
#include "kvm_dev.cuh"

#define KVM_ATTN_ROWS 128

static __device__ bool kvm_attn_geom(const KvmCtx& c, int b, int h, int r0, int T, int H, int Hkv, int hd) {
  if (!(hd == 16 || hd == 32 || hd == 64 || hd == 128) || T <= 0 || H <= 0 || Hkv <= 0 || H % Hkv || b < 0 || r0 < 0 || r0 >= T || h < 0) {
    c.fail(KVM_OPE_SHAPE, hd, r0); return false; }
  return true;
}

template <int HD> struct KvmAm {                  // HD: head dimension rounded up to 32 / 64 / 128 (columns beyond hd are zero)
  static constexpr int PITCH = HD + 8;            // elements per staged row: an odd number of 16-byte groups, so ldmatrix rows hit different banks
  static constexpr int CG = HD > 64 ? 2 : 1;      // column groups of the output
  static constexpr int NCOL = HD / CG;
};

__device__ __forceinline__ void kvm_am_ldm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void kvm_am_ldm4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void kvm_am_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = its first bf16 term; the remainder stays in x
__device__ __forceinline__ __nv_bfloat16 kvm_am_term(float& x) { const __nv_bfloat16 h = __float2bfloat16_rn(x); x -= __bfloat162float(h); return h; }
__device__ __forceinline__ uint32_t kvm_am_term2(float& x, float& y) {
  const __nv_bfloat162 h = __halves2bfloat162(kvm_am_term(x), kvm_am_term(y));
  return *(const uint32_t*)&h;
}

// Rows row0 .. of `b` (columns col0 .. col0 + hd) as NT planes [rows][PITCH] of bf16 terms; rows from `valid` on are zero.  Whole group.
template <int HD, int NT>
__device__ __forceinline__ void kvm_am_load(const KvmBuf b, size_t row0, int valid, int rows, int col0, int hd, __nv_bfloat16* dst) {
  constexpr int P = KvmAm<HD>::PITCH, C8 = HD / 8, U = NT == 1 ? 4 : 2;
  const bool vec = (b.ld & 7) == 0 && kvm_vec_ok(b);
  for (int e0 = threadIdx.x; e0 < rows * C8; e0 += U * KVM_NT) {
    if (NT == 1 && vec) {                         // bf16 as it is
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * KVM_NT, r = e / C8, k = (e % C8) * 8;
        v[u] = e < rows * C8 && r < valid && k < hd ? *(const uint4*)((const __nv_bfloat16*)b.p + (row0 + r) * b.ld + col0 + k) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) { const int e = e0 + u * KVM_NT; if (e < rows * C8) *(uint4*)(dst + (e / C8) * P + (e % C8) * 8) = v[u]; }
      continue;
    }
    float v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * KVM_NT, r = e / C8, k = (e % C8) * 8;
      const bool in = e < rows * C8 && r < valid && k < hd;
      const size_t o = (row0 + r) * b.ld + col0 + k;
      if (in && vec) kvm_ld8(b, o, v[u]);
      else
#pragma unroll
        for (int j = 0; j < 8; ++j) v[u][j] = in ? kvm_ld(b, o + j) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * KVM_NT;
      if (e >= rows * C8) break;
#pragma unroll
      for (int t = 0; t < NT; ++t)
        *(uint4*)(dst + ((size_t)t * rows + e / C8) * P + (e % C8) * 8) =
            make_uint4(kvm_am_term2(v[u][0], v[u][1]), kvm_am_term2(v[u][2], v[u][3]), kvm_am_term2(v[u][4], v[u][5]), kvm_am_term2(v[u][6], v[u][7]));
    }
  }
}

// s[16 x 32] = A rows ra.. times (B rows nb..)^T over the head dimension; planes of arows / brows rows.  Accumulator layout: s[nt][e] is
// row lane/4 (+8 for e >= 2), column nt*8 + 2*(lane%4) + (e&1).
template <int HD, int NT>
__device__ __forceinline__ void kvm_am_scores(float (&s)[4][4], const __nv_bfloat16* A, int arows, int ra, const __nv_bfloat16* B, int brows, int nb) {
  constexpr int P = KvmAm<HD>::PITCH;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.0f;
  const __nv_bfloat16* ap = A + (ra + (lane & 15)) * P + (lane >> 4) * 8;
  const __nv_bfloat16* bp = B + (nb + (lane & 7) + ((lane >> 4) << 3)) * P + ((lane >> 3) & 1) * 8;
#pragma unroll(HD >= 128 && NT > 1 ? 1 : 2)
  for (int ks = 0; ks < HD / 16; ++ks) {
    float d[4][4], lo[NT > 1 ? 4 : 1][4];      // products of the leading terms | of all others
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0.0f;
      if (NT > 1) lo[NT > 1 ? n : 0][0] = lo[NT > 1 ? n : 0][1] = lo[NT > 1 ? n : 0][2] = lo[NT > 1 ? n : 0][3] = 0.0f;
    }
#pragma unroll
    for (int i = NT - 1; i >= 0; --i) {
      uint32_t a[4];
      kvm_am_ldm4(a, ap + (size_t)i * arows * P + ks * 16);
#pragma unroll
      for (int j = NT - 1 - i; j >= 0; --j)
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t b[4];
          kvm_am_ldm4(b, bp + (size_t)j * brows * P + np * 16 * P + ks * 16);
          if (i + j == 0) { kvm_am_mma(d[2 * np], a, b[0], b[1]); kvm_am_mma(d[2 * np + 1], a, b[2], b[3]); }
          else { kvm_am_mma(lo[NT > 1 ? 2 * np : 0], a, b[0], b[1]); kvm_am_mma(lo[NT > 1 ? 2 * np + 1 : 0], a, b[2], b[3]); }
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] += NT > 1 ? d[n][e] + lo[NT > 1 ? n : 0][e] : d[n][e];
  }
}
// acc[16 x NCOL] += p[16 x 32] times B rows kb.. (32 of them), columns n0..
template <int HD, int NT>
__device__ __forceinline__ void kvm_am_accum(float (&acc)[KvmAm<HD>::NCOL / 8][4], float (&p)[4][4], const __nv_bfloat16* B, int brows, int kb, int n0) {
  constexpr int P = KvmAm<HD>::PITCH;
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* bp = B + (kb + (lane & 7) + ((lane >> 3) & 1) * 8) * P + n0 + (lane >> 4) * 8;
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    uint32_t a[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      a[i][0] = kvm_am_term2(p[2 * kk][0], p[2 * kk][1]); a[i][1] = kvm_am_term2(p[2 * kk][2], p[2 * kk][3]);
      a[i][2] = kvm_am_term2(p[2 * kk + 1][0], p[2 * kk + 1][1]); a[i][3] = kvm_am_term2(p[2 * kk + 1][2], p[2 * kk + 1][3]);
    }
#pragma unroll
    for (int np = 0; np < KvmAm<HD>::NCOL / 16; ++np) {
      float d[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}}, lo[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
      for (int j = NT - 1; j >= 0; --j) {
        uint32_t b[4];
        kvm_am_ldm4t(b, bp + (size_t)j * brows * P + kk * 16 * P + np * 16);
#pragma unroll
        for (int i = 2 - j; i >= 0; --i) {
          if (i + j == 0) { kvm_am_mma(d[0], a[i], b[0], b[1]); kvm_am_mma(d[1], a[i], b[2], b[3]); }
          else { kvm_am_mma(lo[0], a[i], b[0], b[1]); kvm_am_mma(lo[1], a[i], b[2], b[3]); }
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) { acc[2 * np][e] += d[0][e] + lo[0][e]; acc[2 * np + 1][e] += d[1][e] + lo[1][e]; }
    }
  }
}
// Output rows of a warp: row lane/4 (+8) of the block at global row r0, columns col0 + ...; rows from `valid` on and columns from hd on are padding.
template <int HD>
__device__ __forceinline__ void kvm_am_store(const KvmBuf& o, size_t r0, int valid, int col0, int n0, int hd, const float (&acc)[KvmAm<HD>::NCOL / 8][4], float f0, float f1) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < KvmAm<HD>::NCOL / 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = g + (e >> 1) * 8, k = n0 + n * 8 + 2 * t + (e & 1);
      if (r < valid && k < hd) kvm_st(o, (r0 + r) * o.ld + col0 + k, acc[n][e] * (e >> 1 ? f1 : f0));
    }
}
// Rows of a chunk, warps' shares and rows of a block of the other side.
struct KvmAmPlan { int rc, kb; };
template <int HD, int NT>
__device__ __forceinline__ KvmAmPlan kvm_am_plan(int smem, int rows, int other, int a_ops, int max_rc) {
  constexpr int RB = KvmAm<HD>::PITCH * 2 * NT;   // bytes of a staged row of one operand
  KvmAmPlan p;
  p.rc = min((rows + 15) & ~15, max_rc);
  while (p.rc > 16 && a_ops * p.rc * RB > smem / 2) p.rc -= 16;
  p.kb = min((other + 31) & ~31, ((smem - a_ops * p.rc * RB) / (2 * RB + 8)) & ~31);      // 8: lse and delta of a query
  return p;
}
__device__ __forceinline__ int kvm_am_groups(int items, int tiles) { int kg = 1; while (2 * kg * items <= KVM_NWARPS && 2 * kg <= tiles) kg *= 2; return kg; }

template <int HD, int NT>
KVM_OP_FN void kvm_am_fwd(const KvmCtx& c, const int32_t* a, const KvmBuf* B) {
  typedef KvmAm<HD> G;
  const int b = a[5], h = a[6], q0 = a[7], T = a[8], H = a[9], hd = a[11], kvh = h / (H / a[10]);
  const float sc = kvm_bits_f32(a[12]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, q1 = min(q0 + KVM_ATTN_ROWS, T);
  const KvmAmPlan pl = kvm_am_plan<HD, NT>(c.smem_bytes, q1 - q0, q1, 1, KVM_ATTN_ROWS);
  if (pl.kb < 32) { c.fail(KVM_OPE_SMEM, hd, c.smem_bytes); return; }
  for (int r0 = q0; r0 < q1; r0 += pl.rc) {
    const int r1 = min(r0 + pl.rc, q1), RG = (r1 - r0 + 15) / 16, items = RG * G::CG, KG = kvm_am_groups(items, (r1 + 31) / 32);
    const int item = warp % items, kg = warp / items, rg = item % RG, n0 = item / RG * G::NCOL;
    __nv_bfloat16* qs = (__nv_bfloat16*)c.smem;
    __nv_bfloat16* ks = qs + (size_t)NT * RG * 16 * G::PITCH;
    __nv_bfloat16* vs = ks + (size_t)NT * pl.kb * G::PITCH;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f}, acc[G::NCOL / 8][4];
#pragma unroll
    for (int n = 0; n < G::NCOL / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    for (int kb = 0; kb < r1; kb += pl.kb) {
      kvm_sync();                                          // the previous block's operands have been read
      if (kb == 0) kvm_am_load<HD, NT>(B[0], (size_t)b * T + r0, r1 - r0, RG * 16, h * hd, hd, qs);
      kvm_am_load<HD, NT>(B[1], (size_t)b * T + kb, T - kb, pl.kb, kvh * hd, hd, ks);
      kvm_am_load<HD, NT>(B[2], (size_t)b * T + kb, T - kb, pl.kb, kvh * hd, hd, vs);
      kvm_sync();
      const int first = r0 + rg * 16;                      // the warp's rows are first .. first + 15
      if (warp < items * KG)
        for (int k0 = kb + kg * 32; k0 < kb + pl.kb && k0 <= first + 15; k0 += 32 * KG) {
          float s[4][4];
          kvm_am_scores<HD, NT>(s, qs, RG * 16, rg * 16, ks, pl.kb, k0 - kb);
#pragma unroll
          for (int e = 0; e < 2; ++e) {                    // rows g and g + 8
            const int row = first + g + 8 * e;
            float mx = -INFINITY;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                float& x = s[n][2 * e + i];
                x = k0 + n * 8 + 2 * t + i <= row ? x * sc : -INFINITY;
                mx = fmaxf(mx, x);
              }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float mn = fmaxf(m[e], mx), base = mn == -INFINITY ? 0.0f : mn, corr = __expf(m[e] - base);
            float sum = 0.0f;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
              for (int i = 0; i < 2; ++i) { float& x = s[n][2 * e + i]; x = __expf(x - base); sum += x; }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[e] = l[e] * corr + sum; m[e] = mn;
#pragma unroll
            for (int n = 0; n < G::NCOL / 8; ++n) { acc[n][2 * e] *= corr; acc[n][2 * e + 1] *= corr; }
          }
          kvm_am_accum<HD, NT>(acc, s, vs, pl.kb, k0 - kb, n0);
        }
    }
    if (KG > 1) {                                          // the key groups of an item, in order
      kvm_sync();
      constexpr int N = G::NCOL / 2 + 4;
      float* part = (float*)c.smem + (size_t)warp * N * 32 + lane;
      if (warp < items * KG && kg > 0) {
#pragma unroll
        for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) part[(n * 4 + e) * 32] = acc[n][e];
        part[(N - 4) * 32] = m[0]; part[(N - 3) * 32] = m[1]; part[(N - 2) * 32] = l[0]; part[(N - 1) * 32] = l[1];
      }
      kvm_sync();
      if (warp < items)
        for (int k = 1; k < KG; ++k) {
          const float* o = (const float*)c.smem + (size_t)(warp + k * items) * N * 32 + lane;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float mo = o[(N - 4 + e) * 32], mn = fmaxf(m[e], mo), base = mn == -INFINITY ? 0.0f : mn, ca = __expf(m[e] - base), cb = __expf(mo - base);
            l[e] = l[e] * ca + o[(N - 2 + e) * 32] * cb; m[e] = mn;
#pragma unroll
            for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
              for (int i = 0; i < 2; ++i) acc[n][2 * e + i] = acc[n][2 * e + i] * ca + o[(n * 4 + 2 * e + i) * 32] * cb;
          }
        }
    }
    if (warp < items) {
      kvm_am_store<HD>(B[3], (size_t)b * T + r0 + rg * 16, r1 - r0 - rg * 16, h * hd, n0, hd, acc, 1.0f / l[0], 1.0f / l[1]);
      float* lse = (float*)B[4].p + (size_t)(b * H + h) * T + r0 + rg * 16;
      if (n0 == 0 && t == 0) {
        if (g < r1 - r0 - rg * 16) lse[g] = m[0] + logf(l[0]);
        if (g + 8 < r1 - r0 - rg * 16) lse[g + 8] = m[1] + logf(l[1]);
      }
    }
  }
}

template <int HD, int NT>
KVM_OP_FN void kvm_am_dq(const KvmCtx& c, const int32_t* a, const KvmBuf* B) {
  typedef KvmAm<HD> G;
  const int b = a[7], h = a[8], q0 = a[9], T = a[10], H = a[11], hd = a[13], kvh = h / (H / a[12]);
  const float sc = kvm_bits_f32(a[14]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, q1 = min(q0 + KVM_ATTN_ROWS, T);
  const KvmAmPlan pl = kvm_am_plan<HD, NT>(c.smem_bytes, q1 - q0, q1, 2, KVM_ATTN_ROWS);
  if (pl.kb < 32) { c.fail(KVM_OPE_SMEM, hd, c.smem_bytes); return; }
  for (int r0 = q0; r0 < q1; r0 += pl.rc) {
    const int r1 = min(r0 + pl.rc, q1), RG = (r1 - r0 + 15) / 16, items = RG * G::CG, KG = kvm_am_groups(items, (r1 + 31) / 32);
    const int item = warp % items, kg = warp / items, rg = item % RG, n0 = item / RG * G::NCOL;
    __nv_bfloat16* qs = (__nv_bfloat16*)c.smem;
    __nv_bfloat16* os = qs + (size_t)NT * RG * 16 * G::PITCH;
    __nv_bfloat16* ks = os + (size_t)NT * RG * 16 * G::PITCH;
    __nv_bfloat16* vs = ks + (size_t)NT * pl.kb * G::PITCH;
    float acc[G::NCOL / 8][4], li[2], di[2];
#pragma unroll
    for (int n = 0; n < G::NCOL / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = min(r0 + rg * 16 + g + 8 * e, T - 1);  // a padded row's gradient is not stored
      li[e] = ((const float*)B[4].p)[(size_t)(b * H + h) * T + r]; di[e] = ((const float*)B[5].p)[(size_t)(b * H + h) * T + r];
    }
    for (int kb = 0; kb < r1; kb += pl.kb) {
      kvm_sync();
      if (kb == 0) {
        kvm_am_load<HD, NT>(B[0], (size_t)b * T + r0, r1 - r0, RG * 16, h * hd, hd, qs);
        kvm_am_load<HD, NT>(B[3], (size_t)b * T + r0, r1 - r0, RG * 16, h * hd, hd, os);
      }
      kvm_am_load<HD, NT>(B[1], (size_t)b * T + kb, T - kb, pl.kb, kvh * hd, hd, ks);
      kvm_am_load<HD, NT>(B[2], (size_t)b * T + kb, T - kb, pl.kb, kvh * hd, hd, vs);
      kvm_sync();
      const int first = r0 + rg * 16;
      if (warp < items * KG)
        for (int k0 = kb + kg * 32; k0 < kb + pl.kb && k0 <= first + 15; k0 += 32 * KG) {
          float s[4][4], dp[4][4];
          kvm_am_scores<HD, NT>(s, qs, RG * 16, rg * 16, ks, pl.kb, k0 - kb);
          kvm_am_scores<HD, NT>(dp, os, RG * 16, rg * 16, vs, pl.kb, k0 - kb);
#pragma unroll
          for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              s[n][e] = k0 + n * 8 + 2 * t + (e & 1) <= first + g + 8 * (e >> 1) ? __expf(s[n][e] * sc - li[e >> 1]) * (dp[n][e] - di[e >> 1]) : 0.0f;
          kvm_am_accum<HD, NT>(acc, s, ks, pl.kb, k0 - kb, n0);
        }
    }
    if (KG > 1) {
      kvm_sync();
      constexpr int N = G::NCOL / 2;
      if (warp < items * KG && kg > 0)
#pragma unroll
        for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) ((float*)c.smem)[((size_t)warp * N + n * 4 + e) * 32 + lane] = acc[n][e];
      kvm_sync();
      if (warp < items)
        for (int k = 1; k < KG; ++k)
#pragma unroll
          for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += ((const float*)c.smem)[((size_t)(warp + k * items) * N + n * 4 + e) * 32 + lane];
    }
    if (warp < items) kvm_am_store<HD>(B[6], (size_t)b * T + r0 + rg * 16, r1 - r0 - rg * 16, h * hd, n0, hd, acc, sc, sc);
  }
}

// Rows are keys here, the other side queries; a warp makes columns of dv (from the probabilities alone) or of dk.
template <int HD, int NT>
KVM_OP_FN void kvm_am_dkv(const KvmCtx& c, const int32_t* a, const KvmBuf* B) {
  typedef KvmAm<HD> G;
  const int b = a[8], kvh = a[9], k0 = a[10], T = a[11], H = a[12], hd = a[13], GR = H / (B[1].cols / hd);
  const float sc = kvm_bits_f32(a[14]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, k1 = min(k0 + KVM_ATTN_ROWS, T);
  const KvmAmPlan pl = kvm_am_plan<HD, NT>(c.smem_bytes, k1 - k0, T - k0 + 31, 2, KVM_NWARPS / (2 * G::CG) * 16);      // an item per warp at most
  if (pl.kb < 32) { c.fail(KVM_OPE_SMEM, hd, c.smem_bytes); return; }
  for (int r0 = k0; r0 < k1; r0 += pl.rc) {
    const int qa = r0 & ~31, r1 = min(r0 + pl.rc, k1), RG = (r1 - r0 + 15) / 16, items = RG * 2 * G::CG, KG = kvm_am_groups(items, (T - qa + 31) / 32);
    const int item = warp % items, kg = warp / items, rg = item % RG, n0 = item / RG % G::CG * G::NCOL;
    const bool dk = item / RG >= G::CG;
    __nv_bfloat16* ks = (__nv_bfloat16*)c.smem;
    __nv_bfloat16* vs = ks + (size_t)NT * RG * 16 * G::PITCH;
    __nv_bfloat16* qs = vs + (size_t)NT * RG * 16 * G::PITCH;
    __nv_bfloat16* os = qs + (size_t)NT * pl.kb * G::PITCH;
    float* ls = (float*)(os + (size_t)NT * pl.kb * G::PITCH);          // lse | delta of the query block
    float acc[G::NCOL / 8][4];
#pragma unroll
    for (int n = 0; n < G::NCOL / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    for (int h = kvh * GR; h < (kvh + 1) * GR; ++h)
      for (int qb = qa; qb < T; qb += pl.kb) {
        kvm_sync();
        if (h == kvh * GR && qb == qa) {
          kvm_am_load<HD, NT>(B[1], (size_t)b * T + r0, r1 - r0, RG * 16, kvh * hd, hd, ks);
          kvm_am_load<HD, NT>(B[2], (size_t)b * T + r0, r1 - r0, RG * 16, kvh * hd, hd, vs);
        }
        kvm_am_load<HD, NT>(B[0], (size_t)b * T + qb, T - qb, pl.kb, h * hd, hd, qs);
        kvm_am_load<HD, NT>(B[3], (size_t)b * T + qb, T - qb, pl.kb, h * hd, hd, os);
        for (int i = threadIdx.x; i < pl.kb; i += KVM_NT) {
          const size_t r = (size_t)(b * H + h) * T + min(qb + i, T - 1);
          ls[i] = ((const float*)B[4].p)[r]; ls[pl.kb + i] = ((const float*)B[5].p)[r];
        }
        kvm_sync();
        const int first = r0 + rg * 16;
        if (warp < items * KG)
          for (int q = qb + kg * 32; q < qb + pl.kb && q < T; q += 32 * KG) {
            if (q + 31 < first) continue;                  // every query of the tile comes before the keys
            float s[4][4];
            kvm_am_scores<HD, NT>(s, ks, RG * 16, rg * 16, qs, pl.kb, q - qb);
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int j = q + n * 8 + 2 * t + (e & 1);
                s[n][e] = j < T && j >= first + g + 8 * (e >> 1) ? __expf(s[n][e] * sc - ls[j - qb]) : 0.0f;
              }
            if (dk) {
              float dp[4][4];
              kvm_am_scores<HD, NT>(dp, vs, RG * 16, rg * 16, os, pl.kb, q - qb);
#pragma unroll
              for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] *= dp[n][e] - ls[pl.kb + q - qb + n * 8 + 2 * t + (e & 1)];
            }
            kvm_am_accum<HD, NT>(acc, s, dk ? qs : os, pl.kb, q - qb, n0);
          }
      }
    if (KG > 1) {
      kvm_sync();
      constexpr int N = G::NCOL / 2;
      if (warp < items * KG && kg > 0)
#pragma unroll
        for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) ((float*)c.smem)[((size_t)warp * N + n * 4 + e) * 32 + lane] = acc[n][e];
      kvm_sync();
      if (warp < items)
        for (int k = 1; k < KG; ++k)
#pragma unroll
          for (int n = 0; n < G::NCOL / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += ((const float*)c.smem)[((size_t)(warp + k * items) * N + n * 4 + e) * 32 + lane];
    }
    if (warp < items) kvm_am_store<HD>(B[dk ? 6 : 7], (size_t)b * T + r0 + rg * 16, r1 - r0 - rg * 16, kvh * hd, n0, hd, acc, dk ? sc : 1.0f, dk ? sc : 1.0f);
  }
}

#define KVM_AM_PICK(fn)                                                                                             \
  do {                                                                                                             \
    const bool bf = B[0].dtype == KVM_BF16 && B[1].dtype == KVM_BF16 && B[2].dtype == KVM_BF16 && (nbf < 4 || B[3].dtype == KVM_BF16); \
    if (hd <= 32) { if (bf) fn<32, 1>(c, a, B); else fn<32, 3>(c, a, B); }                                          \
    else if (hd == 64) { if (bf) fn<64, 1>(c, a, B); else fn<64, 3>(c, a, B); }                                     \
    else { if (bf) fn<128, 1>(c, a, B); else fn<128, 3>(c, a, B); }                                                 \
  } while (0)

KVM_OP_FN void kvm_op_attn_fwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf B[5];
  for (int i = 0; i < 5; ++i) if (!kvm_buf(c, a[i], i == 4 ? KVM_M_F32 : KVM_M_FLT, B[i])) return;
  const int b = a[5], h = a[6], q0 = a[7], T = a[8], H = a[9], Hkv = a[10], hd = a[11], nbf = 3;
  if (!kvm_attn_geom(c, b, h, q0, T, H, Hkv, hd) || h >= H) { c.fail(KVM_OPE_SHAPE, h, H); return; }
  const long long R = (long long)(b + 1) * T;
  if (!kvm_mat_ok(c, B[0], R, H * hd) || !kvm_mat_ok(c, B[1], R, Hkv * hd) || !kvm_mat_ok(c, B[2], R, Hkv * hd) || !kvm_mat_ok(c, B[3], R, H * hd) || !kvm_flat_ok(c, B[4], R * H)) return;
  KVM_AM_PICK(kvm_am_fwd);
}
KVM_OP_FN void kvm_op_attn_bwd_dq(const KvmCtx& c, const int32_t* a) {
  KvmBuf B[7];
  for (int i = 0; i < 7; ++i) if (!kvm_buf(c, a[i], i == 4 || i == 5 ? KVM_M_F32 : KVM_M_FLT, B[i])) return;
  const int b = a[7], h = a[8], q0 = a[9], T = a[10], H = a[11], Hkv = a[12], hd = a[13], nbf = 4;
  if (!kvm_attn_geom(c, b, h, q0, T, H, Hkv, hd) || h >= H) { c.fail(KVM_OPE_SHAPE, h, H); return; }
  const long long R = (long long)(b + 1) * T;
  if (!kvm_mat_ok(c, B[0], R, H * hd) || !kvm_mat_ok(c, B[1], R, Hkv * hd) || !kvm_mat_ok(c, B[2], R, Hkv * hd) || !kvm_mat_ok(c, B[3], R, H * hd) ||
      !kvm_mat_ok(c, B[6], R, H * hd) || !kvm_flat_ok(c, B[4], R * H) || !kvm_flat_ok(c, B[5], R * H)) return;
  KVM_AM_PICK(kvm_am_dq);
}
KVM_OP_FN void kvm_op_attn_bwd_dkv(const KvmCtx& c, const int32_t* a) {
  KvmBuf B[8];
  for (int i = 0; i < 8; ++i) if (!kvm_buf(c, a[i], i == 4 || i == 5 ? KVM_M_F32 : KVM_M_FLT, B[i])) return;
  const int b = a[8], kvh = a[9], k0 = a[10], T = a[11], H = a[12], hd = a[13], nbf = 4;
  if (hd <= 0 || B[1].cols % hd) { c.fail(KVM_OPE_SHAPE, hd, B[1].cols); return; }
  const int Hkv = B[1].cols / hd;
  if (!kvm_attn_geom(c, b, kvh, k0, T, H, Hkv, hd) || kvh >= Hkv) { c.fail(KVM_OPE_SHAPE, kvh, Hkv); return; }
  const long long R = (long long)(b + 1) * T;
  if (!kvm_mat_ok(c, B[0], R, H * hd) || !kvm_mat_ok(c, B[1], R, (kvh + 1) * hd) || !kvm_mat_ok(c, B[2], R, (kvh + 1) * hd) || !kvm_mat_ok(c, B[3], R, H * hd) ||
      !kvm_mat_ok(c, B[6], R, (kvh + 1) * hd) || !kvm_mat_ok(c, B[7], R, (kvh + 1) * hd) || !kvm_flat_ok(c, B[4], R * H) || !kvm_flat_ok(c, B[5], R * H)) return;
  KVM_AM_PICK(kvm_am_dkv);
}
