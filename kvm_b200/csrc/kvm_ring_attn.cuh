// Split decode attention of the static path from the stage ring (attn_decode_part / _qkn with rounded queries, flags 3), and the merge
// of the splits.  Semantics: runtime/ref_extra.py:421-498 of the reference.
//
// A split is a few microseconds of HBM time, so what bounds it is the length of its dependency chain.  One warp owns sixteen keys from
// the scores to the weighted sum of the values; warps meet at three barriers only:
//   prologue   warp g rotates (and normalises) query head g into a bf16 tile, warp 8 the appended key, warp 9 the appended value
//   scores     mma.sync m16n8k16 with the query heads as rows (queries and keys are bf16: the products are exact, summed sixteen at a time);
//              both operands are read 16 bytes per lane at the same k offsets (a dot product does not care about the order of k)
//   softmax    over the warp's sixteen keys by two shuffles; probabilities stay float32
//   values     lane = HD / 32 columns for all heads, probabilities broadcast from shared memory
//   merge      each warp scales its sums by exp(own maximum - split's maximum) and parks them in the keys' stage; one pass adds the
//              sixteen warps up in pairs
// (The form it replaces, one softmax over the split by all warps with ten barriers, took 18-24 us a task, eight of them in the prologue.)
#pragma once
#include "kvm_decode_stream.cuh"
#include "kvm_dev.cuh"
#include "kvm_ops_rows.cuh"

// What a task needs over its whole length; buffers are looked up in the slot where they are used (registers are short here).
struct KvmPartArgs {
  const KvmBuf* lb;                   // q, kc, vc, lens, part, knew, vnew
  const int32_t* a;
  const float* gam;                   // rows (query, key) of the QK norm's weights; without the norm any readable HD floats (the compiler loads them ahead of the test)
  bool qkn;
  int gam_ld, G, p0, nk, newrow;
  const float* inv;                   // hd / 2 inverse frequencies
};
// scratch: q tile [8][HD] bf16 | probabilities [16 warps][16 keys][8] | (m, l) [16 warps][8]
#define KVM_RA_PS 2048
#define KVM_RA_ML (KVM_RA_PS + 8192)
#define KVM_RA_BYTES (KVM_RA_ML + 1024)

// d = rows g (0..7) of A[16 x 16] B[16 x 8], columns 2t and 2t + 1; rows 8 to 15 of A are zero.
__device__ __forceinline__ void kvm_ra_mma(float (&d)[2], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float pad0, pad1;
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(pad0), "=f"(pad1) : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.0f));
}

// Rotated row of one head: lane handles the pairs (i, i + HD/2), i = lane, lane + 32, ...  put(column, value).
template <int HD, class Put>
__device__ __forceinline__ void kvm_ra_rotate(const KvmBuf& x, size_t off, bool qkn, const float* gam, float eps, const float* inv, float pos, Put put) {
  constexpr int N = HD >= 64 ? HD / 64 : 1;
  const int lane = threadIdx.x & 31;
  float x1[N], x2[N], ss = 0.0f;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int i = lane + 32 * j;
    const bool in = i < HD / 2;
    x1[j] = in ? kvm_ld(x, off + i) : 0.0f; x2[j] = in ? kvm_ld(x, off + i + HD / 2) : 0.0f;
    ss += x1[j] * x1[j] + x2[j] * x2[j];
  }
  if (qkn) {
    const float rs = 1.0f / sqrtf(kvm_warp_sum(ss) / HD + eps);
#pragma unroll
    for (int j = 0; j < N; ++j) { const int i = lane + 32 * j; if (i < HD / 2) { x1[j] = x1[j] * rs * gam[i]; x2[j] = x2[j] * rs * gam[i + HD / 2]; } }
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int i = lane + 32 * j;
    if (i < HD / 2) {
      float sn, co;
      sincosf(__fmul_rn(pos, inv[i]), &sn, &co);
      put(i, x1[j] * co - x2[j] * sn);
      put(i + HD / 2, x1[j] * sn + x2[j] * co);
    }
  }
}

// Whole compute group.  Ks / Vs: the staged keys and values [nk][HD] bf16; waitK / waitV as in kvm_attn_part_core.
template <int HD, int GT, class WaitK, class WaitV>
__device__ __forceinline__ bool kvm_ra_part(const KvmPartArgs& P, unsigned char* sm, unsigned char* Ks, unsigned char* Vs, WaitK waitK, WaitV waitV) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = P.G, nk = P.nk;
  __nv_bfloat16* qt = (__nv_bfloat16*)sm;
  float* ps = (float*)(sm + KVM_RA_PS) + warp * 128;
  float2* ml = (float2*)(sm + KVM_RA_ML);
  const float pos = (float)P.p0;
  const int b = P.a[7], kvh = P.a[8];
  const float eps = P.qkn ? kvm_bits_f32(P.a[19]) : 0.0f;
  if (warp < 8) {
    if (warp < G) {
      const KvmBuf q = P.lb[0];
      kvm_ra_rotate<HD>(q, (size_t)b * q.ld + (kvh * G + warp) * HD, P.qkn, P.gam, eps, P.inv, pos,
                        [&](int k, float v) { qt[warp * HD + k] = __float2bfloat16_rn(v); });
    } else {
      for (int k = lane; k < HD; k += 32) qt[warp * HD + k] = __float2bfloat16_rn(0.0f);
    }
  } else if (warp == 8 && P.newrow >= 0) {
    const KvmBuf kn = P.lb[5];
    __nv_bfloat16* dst = (__nv_bfloat16*)P.lb[1].p + ((size_t)(b * P.a[12] + kvh) * P.a[14] + P.p0) * HD;      // cache rows are contiguous
    kvm_ra_rotate<HD>(kn, (size_t)b * kn.ld + kvh * HD, P.qkn, P.gam + P.gam_ld, eps, P.inv, pos, [&](int k, float v) {
      const __nv_bfloat16 h = __float2bfloat16_rn(v);
      ((__nv_bfloat16*)Ks)[(size_t)P.newrow * HD + k] = h;
      dst[k] = h;
    });
  } else if (warp == 9 && P.newrow >= 0) {
    const KvmBuf vn = P.lb[6];
    __nv_bfloat16* dst = (__nv_bfloat16*)P.lb[2].p + ((size_t)(b * P.a[12] + kvh) * P.a[14] + P.p0) * HD;
    for (int k = lane; k < HD; k += 32) {
      const __nv_bfloat16 h = __float2bfloat16_rn(kvm_ld(vn, (size_t)b * vn.ld + kvh * HD + k));
      ((__nv_bfloat16*)Vs)[(size_t)P.newrow * HD + k] = h;
      dst[k] = h;
    }
  }
  bool ok = waitK();
  kvm_sync();                                          // queries and the appended row are in place
  const int g = lane >> 2, t = lane & 3;
  uint4 qf[HD / 32];
#pragma unroll
  for (int ch = 0; ch < HD / 32; ++ch) qf[ch] = *(const uint4*)((const unsigned char*)qt + g * HD * 2 + ch * 64 + t * 16);
  constexpr int NCOL = HD >= 32 ? HD / 32 : 1;
  float m = KVM_ATTN_EMPTY_M_STREAM, l = 0.0f, acc[GT][NCOL];
#pragma unroll
  for (int h = 0; h < GT; ++h)
#pragma unroll
    for (int j = 0; j < NCOL; ++j) acc[h][j] = 0.0f;
  bool vok = false;
  const float sc = kvm_bits_f32(P.a[15]);
#pragma unroll 1
  for (int k0 = warp * 16; k0 < nk; k0 += 256) {
    float s[2][2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      // sixteen products from zero, float32 adds in pairs between them: the matrix unit truncates where it adds to an accumulator, so a
      // sum kept there over a whole row drifts towards zero (the tile's rows 8 to 15 hold no head)
      const unsigned char* kr = Ks + (size_t)(k0 + nt * 8 + g) * HD * 2 + t * 16;
      float d[HD / 16][2];
#pragma unroll
      for (int ch = 0; ch < HD / 32; ++ch) {
        const uint4 kf = *(const uint4*)(kr + ch * 64);
        kvm_ra_mma(d[2 * ch], qf[ch].x, qf[ch].y, kf.x, kf.y);
        kvm_ra_mma(d[2 * ch + 1], qf[ch].z, qf[ch].w, kf.z, kf.w);
      }
#pragma unroll
      for (int w = 1; w < HD / 16; w *= 2)
#pragma unroll
        for (int i = 0; i < HD / 16; i += 2 * w) { d[i][0] += d[i + w][0]; d[i][1] += d[i + w][1]; }
      s[nt][0] = d[0][0]; s[nt][1] = d[0][1];
    }
    // lane (g, t): scores of head g for the keys k0 + 2t, + 1 and k0 + 8 + 2t, + 1
    float mx = KVM_ATTN_EMPTY_M_STREAM;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[nt][e] = k0 + nt * 8 + 2 * t + e < nk ? s[nt][e] * sc : -INFINITY;
        mx = fmaxf(mx, s[nt][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx), corr = __expf(m - mn);
    float sum = 0.0f;
    __syncwarp();                                      // the previous block's probabilities have been read
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) { const float p = __expf(s[nt][e] - mn); sum += p; ps[(nt * 8 + 2 * t + e) * 8 + g] = p; }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    l = l * corr + sum;
    m = mn;
    if (k0 >= 256) {
#pragma unroll
      for (int h = 0; h < GT; ++h) { const float cf = __shfl_sync(0xffffffffu, corr, h * 4);
#pragma unroll
        for (int j = 0; j < NCOL; ++j) acc[h][j] *= cf; }
    }
    __syncwarp();
    if (!vok) { if (!waitV()) ok = false; vok = true; }
    const int n = min(16, nk - k0);
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      float v[NCOL], p[GT];
      const unsigned char* vr = Vs + (size_t)(k0 + k) * HD * 2;
      if (NCOL == 4) { const uint2 u = *(const uint2*)(vr + lane * 8); v[0] = kvm_bf16lo(u.x); v[NCOL > 1 ? 1 : 0] = kvm_bf16hi(u.x); v[NCOL > 2 ? 2 : 0] = kvm_bf16lo(u.y); v[NCOL > 3 ? 3 : 0] = kvm_bf16hi(u.y); }
      else if (NCOL == 2) { const uint32_t u = *(const uint32_t*)(vr + lane * 4); v[0] = kvm_bf16lo(u); v[NCOL > 1 ? 1 : 0] = kvm_bf16hi(u); }
      else v[0] = __bfloat162float(*(const __nv_bfloat16*)(vr + lane * 2));
      *(float4*)p = *(const float4*)(ps + k * 8);
      if (GT > 4) *(float4*)(p + (GT > 4 ? 4 : 0)) = *(const float4*)(ps + k * 8 + 4);
#pragma unroll
      for (int h = 0; h < GT; ++h)
#pragma unroll
        for (int j = 0; j < NCOL; ++j) acc[h][j] = fmaf(p[h], v[j], acc[h][j]);
    }
  }
  if (!vok && !waitV()) ok = false;
  if (t == 0) ml[warp * 8 + g] = make_float2(m, l);
  kvm_sync();                                          // every warp is done with the keys and the values
  float* red = (float*)Ks;                             // [16 warps][G][HD]
  float M = KVM_ATTN_EMPTY_M_STREAM;
#pragma unroll
  for (int w = 0; w < KVM_NWARPS; ++w) M = fmaxf(M, ml[w * 8 + (lane & 7)].x);
  const float mine = __expf(ml[warp * 8 + (lane & 7)].x - M);      // lane h < 8: this warp's scale for head h
#pragma unroll
  for (int h = 0; h < GT; ++h) {
    const float f = __shfl_sync(0xffffffffu, mine, h);
    if (h < G) {
      float* d = red + ((size_t)warp * G + h) * HD + lane * NCOL;
      if (NCOL == 4) *(float4*)d = make_float4(acc[h][0] * f, acc[h][NCOL > 1 ? 1 : 0] * f, acc[h][NCOL > 2 ? 2 : 0] * f, acc[h][NCOL > 3 ? 3 : 0] * f);
      else if (NCOL == 2) *(float2*)d = make_float2(acc[h][0] * f, acc[h][NCOL > 1 ? 1 : 0] * f);
      else d[0] = acc[h][0] * f;
    }
  }
  kvm_sync();
  const KvmBuf part = P.lb[4];
  for (int e = threadIdx.x; e < G * HD; e += KVM_NT) {
    const int h = e / HD, cc = e % HD;
    float A[KVM_NWARPS];
#pragma unroll
    for (int w = 0; w < KVM_NWARPS; ++w) A[w] = red[((size_t)w * G + h) * HD + cc];
#pragma unroll
    for (int n = 1; n < KVM_NWARPS; n *= 2)
#pragma unroll
      for (int w = 0; w < KVM_NWARPS; w += 2 * n) A[w] += A[w + n];
    float* row = (float*)part.p + ((size_t)(b * P.a[10] + P.a[9]) * P.a[11] + kvh * G + h) * part.ld;
    row[cc] = A[0];
    if (cc == 0) {
      float Mh = KVM_ATTN_EMPTY_M_STREAM, L = 0.0f;
      for (int w = 0; w < KVM_NWARPS; ++w) Mh = fmaxf(Mh, ml[w * 8 + h].x);
      for (int w = 0; w < KVM_NWARPS; ++w) L += ml[w * 8 + h].y * __expf(ml[w * 8 + h].x - Mh);
      row[HD] = Mh; row[HD + 1] = L;
    }
  }
  return ok;
}

// Merge of the splits: thread = (head, column), all splits' partials of a thread in flight together (S <= 20).  false: not taken.
KVM_OP_FN bool kvm_hot_merge(const KvmCtx& c, const int32_t* a) {
  if (a[0] < 0 || a[0] >= c.nbufs || a[1] < 0 || a[1] >= c.nbufs) return false;
  const KvmBuf part = c.bufs[a[0]], o = c.bufs[a[1]];
  const int b = a[2], h0 = a[3], h1 = a[4], S = a[5], H = a[6], hd = a[7];
  if (!part.p || part.dtype != KVM_F32 || !o.p || o.dtype == KVM_I32 || b < 0 || h0 < 0 || h1 <= h0 || h1 > H || S <= 0 || S > 20 || hd <= 0 || (long long)(b + 1) * S * H > part.rows ||
      hd + 2 > part.cols || b + 1 > o.rows || H * hd > o.cols) return false;
  const float* pp = (const float*)part.p;
  for (int e = threadIdx.x; e < (h1 - h0) * hd; e += KVM_NT) {
    const int h = h0 + e / hd, cc = e % hd;
    const float* r = pp + ((size_t)b * S * H + h) * part.ld;
    const size_t step = (size_t)H * part.ld;
    float ms[20], ls[20], as[20];
#pragma unroll
    for (int s = 0; s < 20; ++s) {
      ms[s] = s < S ? r[s * step + hd] : KVM_ATTN_EMPTY_M_STREAM; ls[s] = s < S ? r[s * step + hd + 1] : 0.0f; as[s] = s < S ? r[s * step + cc] : 0.0f;
    }
    float M = KVM_ATTN_EMPTY_M_STREAM, L = 0.0f, A = 0.0f;
#pragma unroll
    for (int s = 0; s < 20; ++s) if (ls[s] > 0.0f) M = fmaxf(M, ms[s]);
#pragma unroll
    for (int s = 0; s < 20; ++s) if (ls[s] > 0.0f) { const float f = __expf(ms[s] - M); L += ls[s] * f; A += as[s] * f; }      // split order
    kvm_st(o, (size_t)b * o.ld + h * hd + cc, A / L);
  }
  return true;
}
