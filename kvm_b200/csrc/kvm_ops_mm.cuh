// GEMM tile ops, SIMT form: the bit-exact float32 path (matmul, matmul_tile) and the fallback of the bf16 tile ops for
// operands the tensor-core path cannot take (unaligned ld / base, f32 operands).  Accumulation is k-ascending with one
// rounded multiply and one rounded add per step, which is the reference's golden for every matmul flavour
// (runtime/ref_gpt.py:69-103, runtime/ref_extra.py:312-331), so results equal its CPU model bit for bit.
// The epilogue (shared with the tcgen05 path in kvm_gemm_tc.cuh) follows the reference order:
//   v = alpha*acc; + bias[n]; (flag 512: * gelu'(pre)) else (pre = v; flag 8: gelu); + res; (flag 4: out += v).
#pragma once
#include "kvm_dev.cuh"
#include "kvm_ops_flat.cuh"

struct KvmMmArgs {
  KvmBuf a, b, out, bias, res, pre;
  int m0, n0, M, N, K, flags;
  float alpha;
  int tm, tn;            // tile extent
  bool round_ops;        // operands rounded to bf16 on load
};

__device__ __forceinline__ float kvm_mm_epilogue(const KvmMmArgs& g, float acc, int m, int n) {
  float v = __fmul_rn(acc, g.alpha);
  if (g.bias.p) v = __fadd_rn(v, ((const float*)g.bias.p)[n]);
  if (g.flags & 512) v = v * kvm_gelu_grad(kvm_ld(g.pre, (size_t)m * g.pre.ld + n));
  else {
    if (g.pre.p) kvm_st(g.pre, (size_t)m * g.pre.ld + n, v);
    if (g.flags & 8) v = kvm_gelu(v);
  }
  if (g.res.p) v = __fadd_rn(v, kvm_ld(g.res, (size_t)m * g.res.ld + n));
  if (g.flags & 4) v = __fadd_rn(kvm_ld(g.out, (size_t)m * g.out.ld + n), v);
  return v;
}

// Four neighbouring columns of a row.  With float32 buffers on 16-byte boundaries everything the epilogue reads is loaded as vectors
// before the first use; otherwise column by column.
template <bool VEC>
__device__ __forceinline__ void kvm_mm_epilogue4(const KvmMmArgs& g, const float (&acc)[4], int m, int n, int n_end) {
  const bool simple = VEC && n + 4 <= n_end && !(g.flags & (4 | 512)) && g.out.dtype == KVM_F32 && (g.out.ld & 3) == 0 && kvm_vec_ok(g.out) && (!g.bias.p || kvm_vec_ok(g.bias)) &&
                      (!g.res.p || (g.res.dtype == KVM_F32 && (g.res.ld & 3) == 0 && kvm_vec_ok(g.res))) &&
                      (!g.pre.p || (g.pre.dtype == KVM_F32 && (g.pre.ld & 3) == 0 && kvm_vec_ok(g.pre)));
  if (!simple) {
#pragma unroll
    for (int j = 0; j < 4; ++j) if (n + j < n_end) kvm_st(g.out, (size_t)m * g.out.ld + n + j, kvm_mm_epilogue(g, acc[j], m, n + j));
    return;
  }
  float v[4] = {acc[0], acc[1], acc[2], acc[3]}, bi[4] = {0, 0, 0, 0}, re[4] = {0, 0, 0, 0};
  if (g.bias.p) *(float4*)bi = *(const float4*)((const float*)g.bias.p + n);
  if (g.res.p) *(float4*)re = *(const float4*)((const float*)g.res.p + (size_t)m * g.res.ld + n);
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[j] = __fmul_rn(v[j], g.alpha); if (g.bias.p) v[j] = __fadd_rn(v[j], bi[j]); }
  if (g.pre.p) *(float4*)((float*)g.pre.p + (size_t)m * g.pre.ld + n) = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
  for (int j = 0; j < 4; ++j) { if (g.flags & 8) v[j] = kvm_gelu(v[j]); if (g.res.p) v[j] = __fadd_rn(v[j], re[j]); }
  *(float4*)((float*)g.out.p + (size_t)m * g.out.ld + n) = make_float4(v[0], v[1], v[2], v[3]);
}

// Decode and check the 13 argument words shared by matmul_tile / matmul_tile_bf16 / matmul_mma_bf16.
static __device__ bool kvm_mm_args(const KvmCtx& c, const int32_t* a, int kind /*0 f32 tile, 1 bf16 tile, 2 mma 128x256*/, KvmMmArgs& g) {
  const int opmask = kind == 0 ? KVM_M_F32 : KVM_M_FLT, omask = kind == 0 ? KVM_M_F32 : KVM_M_FLT;
  if (!kvm_buf(c, a[0], opmask, g.a) || !kvm_buf(c, a[1], opmask, g.b) || !kvm_buf(c, a[2], omask, g.out) || !kvm_buf(c, a[3], KVM_M_F32, g.bias, true) ||
      !kvm_buf(c, a[4], omask, g.res, true) || !kvm_buf(c, a[5], omask, g.pre, true)) return false;
  g.m0 = a[6]; g.n0 = a[7]; g.M = a[8]; g.N = a[9]; g.K = a[10]; g.flags = a[11]; g.alpha = kvm_bits_f32(a[12]);
  const int fl = g.flags;
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.m0 < 0 || g.m0 >= g.M || g.n0 < 0 || g.n0 >= g.N) { c.fail(KVM_OPE_RANGE, g.m0, g.n0); return false; }
  const int allowed = kind == 2 ? (1 | 2 | 4 | 8) : (127 | 256 | 512 | 1024);
  if ((fl & ~allowed) || ((fl & 32) && (fl & 64)) || ((fl & 256) && (fl & 1024)) ||
      ((fl & 512) && (!g.pre.p || g.bias.p || g.res.p || (fl & (4 | 8 | 128))))) { c.fail(KVM_OPE_SHAPE, fl); return false; }
  if (kind == 2) { g.tm = 128; g.tn = 256; }
  else if (fl & 64) { g.tm = 256; g.tn = 128; }
  else if (fl & 32) { g.tm = 128; g.tn = 128; }
  else { g.tm = 64; g.tn = 64; }
  g.round_ops = kind != 0 || (fl & 128);
  const bool ta = fl & 1, tb = fl & 2;
  if (!kvm_mat_ok(c, g.a, ta ? g.K : g.M, ta ? g.M : g.K) || !kvm_mat_ok(c, g.b, tb ? g.N : g.K, tb ? g.K : g.N) || !kvm_mat_ok(c, g.out, g.M, g.N) ||
      !kvm_mat_ok(c, g.res, g.M, g.N) || !kvm_mat_ok(c, g.pre, g.M, g.N) || !kvm_flat_ok(c, g.bias, g.N)) return false;
  return true;
}

// ---- SIMT tile ----------------------------------------------------------------------------------------------------------------
// 64x64 sub-tiles, K staged through shared memory 32 at a time.  The first eight warps multiply, a thread owns 4 rows x 4 columns:
// per k two LDS.128 for 16 products.  The exact multiply-then-add (two roundings per step, no fused multiply-add) needs 64 issue
// cycles per k and SM, the two loads 64 cycles of shared-memory bandwidth; the form before (one row x 8 columns per thread, all
// sixteen warps) asked shared memory for 3 loads per 8 products.  Packed FMAs (the 32x32 form below) do not help here: 66-72 ns per k
// against 69, shared memory and issue overlap no better with two multiplying warps per scheduler.
// All sixteen warps stage: chunk i+2 is in flight from global memory (registers) while chunk i is multiplied, chunk i+1 is in the
// other shared buffer: one barrier per chunk.  Both arrays are stored [k][.] with their 16-byte units XOR-swizzled by (k / 4) & 7, so
// that the transposing stores (k contiguous in global memory) spread over the banks as well as the loads do.
// A warp whose rows or columns lie outside the tile (10-column logits) skips the arithmetic.
#define KVM_SM_A_BYTES (32 * 64 * 4)
#define KVM_SM_STAGE (2 * KVM_SM_A_BYTES)

// Four consecutive elements along the contiguous axis of an operand: row `r` (outer index), columns c..c+3, zero outside [rows, cols).
template <bool VEC>
__device__ __forceinline__ void kvm_sm_fetch(const KvmBuf& b, bool round_ops, int r, int c, int rows, int cols, float (&v)[4]) {
  if (r < rows && c + 4 <= cols && VEC) {
    const float4 f = *(const float4*)((const float*)b.p + (size_t)r * b.ld + c);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (r < rows && c + j < cols) ? (VEC ? ((const float*)b.p)[(size_t)r * b.ld + c + j] : kvm_ld(b, (size_t)r * b.ld + c + j)) : 0.0f;
  }
  if (!VEC && round_ops) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = kvm_bf16_round(v[j]);
  }
}
template <bool VEC>
static __device__ __noinline__ void kvm_mm_simt_t(const KvmCtx& c, const KvmMmArgs& g) {
  const bool ta = g.flags & 1, tb = g.flags & 2, two = c.smem_bytes >= 2 * KVM_SM_STAGE;
  const int m_end = min(g.m0 + g.tm, g.M), n_end = min(g.n0 + g.tn, g.N);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = (warp & 1) * 8 + (lane & 7), cg = (warp >> 1) * 4 + (lane >> 3);      // warps 0..7: rows 4 rg .., columns 4 cg ..
  // this thread's share of a chunk: A element (am, ak .. ak+3) or, transposed, (am .. am+3, ak); B likewise
  const int am = ta ? (tid & 15) * 4 : tid >> 3, ak = ta ? tid >> 4 : (tid & 7) * 4;
  const int bn = tb ? tid >> 3 : (tid & 15) * 4, bk = tb ? (tid & 7) * 4 : tid >> 4;
  for (int mb = g.m0; mb < m_end; mb += 64)
    for (int nb = g.n0; nb < n_end; nb += 64) {
      const bool active = warp < 8 && mb + (warp & 1) * 32 < m_end && nb + (warp >> 1) * 16 < n_end;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
      float xa[2][4], xb[2][4];
      auto fetch = [&](int k0, float (&va)[4], float (&vb)[4]) {
        if (ta) kvm_sm_fetch<VEC>(g.a, g.round_ops, k0 + ak, mb + am, g.K, m_end, va);
        else kvm_sm_fetch<VEC>(g.a, g.round_ops, mb + am, k0 + ak, m_end, g.K, va);
        if (tb) kvm_sm_fetch<VEC>(g.b, g.round_ops, nb + bn, k0 + bk, n_end, g.K, vb);
        else kvm_sm_fetch<VEC>(g.b, g.round_ops, k0 + bk, nb + bn, g.K, n_end, vb);
      };
      auto put1 = [&](unsigned char* st, int o, int k, bool along_k, const float (&v)[4]) {      // element (o, k) of a [k][64] array, four along k or along o
        const int q = (k >> 2) & 7;
        if (along_k) {
          const int at = (((o >> 2) ^ q) << 4) + (o & 3) * 4;
#pragma unroll
          for (int j = 0; j < 4; ++j) *(float*)(st + (k + j) * 256 + at) = v[j];
        } else *(float4*)(st + k * 256 + (((o >> 2) ^ q) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
      };
      auto put = [&](unsigned char* st, const float (&va)[4], const float (&vb)[4]) { put1(st, am, ak, !ta, va); put1(st + KVM_SM_A_BYTES, bn, bk, tb, vb); };
      const int nch = (g.K + 31) / 32;
      fetch(0, xa[0], xb[0]);
      if (nch > 1) fetch(32, xa[1], xb[1]);
      kvm_sync();                                           // whatever used the scratch before is done with it
      put(c.smem, xa[0], xb[0]);
      for (int i = 0; i < nch; ++i) {
        kvm_sync();                                         // chunk i is in its buffer
        unsigned char* st = c.smem + (two ? (i & 1) * KVM_SM_STAGE : 0);
        if (i + 2 < nch) fetch((i + 2) * 32, xa[0], xb[0]);
        if (two && i + 1 < nch) put(c.smem + ((i + 1) & 1) * KVM_SM_STAGE, xa[1], xb[1]);
        if (active) {
          const int kmax = min(32, g.K - i * 32);
          auto step = [&](int k, int q) {
            const float4 x = *(const float4*)(st + k * 256 + ((rg ^ q) << 4)), y = *(const float4*)(st + KVM_SM_A_BYTES + k * 256 + ((cg ^ q) << 4));
            const float xr[4] = {x.x, x.y, x.z, x.w}, yc[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[r][j] = __fadd_rn(acc[r][j], __fmul_rn(xr[r], yc[j]));
          };
          if (kmax == 32) {
#pragma unroll
            for (int k = 0; k < 32; ++k) step(k, (k >> 2) & 7);
          } else
            for (int k = 0; k < kmax; ++k) step(k, (k >> 2) & 7);
        }
        if (!two && i + 1 < nch) { kvm_sync(); put(c.smem, xa[1], xb[1]); }
#pragma unroll
        for (int j = 0; j < 4; ++j) { xa[1][j] = xa[0][j]; xb[1][j] = xb[0][j]; }
      }
      if (active) {
        const int n = nb + cg * 4;
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) {
          const int m = mb + rg * 4 + rr;
          if (m < m_end) kvm_mm_epilogue4<VEC>(g, acc[rr], m, n, n_end);
        }
      }
    }
}
// Tiles of 32x32 at most (what the training graphs cut a product into that would occupy few SMs, so that its length counts and not its
// rate).  Eight warps multiply, a thread owns 2 rows x 2 columns; the other eight stage, two chunks ahead in registers.  The product is
// rounded before it is added; packed FMAs do both with one rounding each, x * y + (-0) and the sum.  The constant comes from constant
// memory, since the compiler contracts a packed multiply and add into one FMA when it sees them.
// What bounds it: shared memory delivers 128 bytes a cycle, 32 cycles per k for the eight warps' two 8-byte loads; the 64x64 form
// above takes four times its share of latency per k at this size.  At K = 512 a tile takes 19 us, of which
// 5 are the call and the first loads (64x64 form: 27-30 us for such a tile, 39 us for a whole one).
static __constant__ unsigned long long kvm_mm_nzero2 = 0x8000000080000000ull;      // (-0, -0)
template <bool VEC>
static __device__ __noinline__ void kvm_mm_simt_32(const KvmCtx& c, const KvmMmArgs& g) {
  extern __shared__ __align__(1024) unsigned char kvm_smem[];
  unsigned char* sm = kvm_smem + (uint32_t)(c.smem - kvm_smem);      // the compiler sees shared memory (through the context's pointer every access is a generic one)
  const bool ta = g.flags & 1, tb = g.flags & 2;
  const int mb = g.m0, nb = g.n0, m_end = min(mb + g.tm, g.M), n_end = min(nb + g.tn, g.N), K = g.K, nch = (K + 31) / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  kvm_sync();                                               // whatever used the scratch before is done with it
  if (tid >= 256) {
    const int t = tid & 255, am = ta ? (t & 7) * 4 : t >> 3, ak = ta ? t >> 3 : (t & 7) * 4, bn = tb ? t >> 3 : (t & 7) * 4, bk = tb ? (t & 7) * 4 : t >> 3;
    const KvmBuf ga = g.a, gb = g.b;
    const bool ro = g.round_ops;
    float xa[4][4], xb[4][4];
    auto fetch = [&](int i, float (&va)[4], float (&vb)[4]) {
      if (i >= nch) return;
      const int k0 = i * 32;
      if (ta) kvm_sm_fetch<VEC>(ga, ro, k0 + ak, mb + am, K, m_end, va); else kvm_sm_fetch<VEC>(ga, ro, mb + am, k0 + ak, m_end, K, va);
      if (tb) kvm_sm_fetch<VEC>(gb, ro, nb + bn, k0 + bk, n_end, K, vb); else kvm_sm_fetch<VEC>(gb, ro, k0 + bk, nb + bn, K, n_end, vb);
    };
    auto put1 = [&](unsigned char* st, int o, int k, bool along_k, const float (&v)[4]) {      // element (o, k) of a [k][32] array, four along k or along o
      const int q = (k >> 2) & 7;
      if (along_k) {
        const int at = (((o >> 2) ^ q) << 4) + (o & 3) * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) *(float*)(st + (k + j) * 128 + at) = v[j];
      } else *(float4*)(st + k * 128 + (((o >> 2) ^ q) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
    };
    auto put = [&](int i, const float (&va)[4], const float (&vb)[4]) {
      if (i >= nch) return;
      unsigned char* st = sm + (i & 1) * 8192;
      put1(st, am, ak, !ta, va); put1(st + 4096, bn, bk, tb, vb);
    };
#pragma unroll
    for (int u = 0; u < 4; ++u) fetch(u, xa[u], xb[u]);
    put(0, xa[0], xb[0]);
    fetch(4, xa[0], xb[0]);
#pragma unroll 1
    for (int i = 0; i < nch; i += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i + u >= nch) break;
        kvm_sync();                                         // chunk i + u is in its buffer
        put(i + u + 1, xa[(u + 1) & 3], xb[(u + 1) & 3]);
        fetch(i + u + 5, xa[(u + 1) & 3], xb[(u + 1) & 3]);
      }
    return;
  }
  const int rg = (warp & 1) * 8 + (lane & 7), cg = (warp >> 1) * 4 + (lane >> 3);      // rows 2 rg, + 1; columns 2 cg, + 1
  const bool active = mb + (warp & 1) * 16 < m_end && nb + (warp >> 1) * 8 < n_end;
  const unsigned long long nzero = kvm_mm_nzero2;
  unsigned long long acc0 = 0ull, acc1 = 0ull;
#pragma unroll 1
  for (int i = 0; i < nch; ++i) {
    kvm_sync();                                             // chunk i is in its buffer
    if (!active) continue;
    const unsigned char* st = sm + (i & 1) * 8192;
    const unsigned char* xp = st + (rg & 1) * 8;
    const unsigned char* yp = st + 4096 + (cg & 1) * 8;
    const int kmax = min(32, K - i * 32);
    auto step = [&](int k, int q) {
      const float2 x = *(const float2*)(xp + k * 128 + (((rg >> 1) ^ q) << 4));
      const unsigned long long y = *(const unsigned long long*)(yp + k * 128 + (((cg >> 1) ^ q) << 4));
      unsigned long long x0, x1, p0, p1;
      asm("mov.b64 %0, {%1, %1};" : "=l"(x0) : "f"(x.x));
      asm("mov.b64 %0, {%1, %1};" : "=l"(x1) : "f"(x.y));
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p0) : "l"(x0), "l"(y), "l"(nzero));
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p1) : "l"(x1), "l"(y), "l"(nzero));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(acc0) : "l"(p0), "l"(acc0));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(acc1) : "l"(p1), "l"(acc1));
    };
    if (kmax == 32) {
#pragma unroll 1
      for (int k4 = 0; k4 < 32; k4 += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) step(k4 + k, ((k4 + k) >> 2) & 7);
    } else
      for (int k = 0; k < kmax; ++k) step(k, (k >> 2) & 7);
  }
  if (!active) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float2 v = r ? *(float2*)&acc1 : *(float2*)&acc0;
    const int m = mb + 2 * rg + r, n = nb + 2 * cg;
    if (m < m_end && n < n_end) kvm_st(g.out, (size_t)m * g.out.ld + n, kvm_mm_epilogue(g, v.x, m, n));
    if (m < m_end && n + 1 < n_end) kvm_st(g.out, (size_t)m * g.out.ld + n + 1, kvm_mm_epilogue(g, v.y, m, n + 1));
  }
}
static __device__ void kvm_mm_simt(const KvmCtx& c, const KvmMmArgs& g) {
  // vector loads: float32 operands as they are (no rounding), rows and tile origin on 16-byte boundaries
  const bool vec = !g.round_ops && g.a.dtype == KVM_F32 && g.b.dtype == KVM_F32 && ((g.a.ld | g.b.ld | g.m0 | g.n0) & 3) == 0 && kvm_vec_ok(g.a) && kvm_vec_ok(g.b);
  if (min(g.tm, g.M - g.m0) <= 32 && min(g.tn, g.N - g.n0) <= 32) { if (vec) kvm_mm_simt_32<true>(c, g); else kvm_mm_simt_32<false>(c, g); }
  else if (vec) kvm_mm_simt_t<true>(c, g); else kvm_mm_simt_t<false>(c, g);
}

KVM_OP_FN void kvm_op_matmul_tile(const KvmCtx& c, const int32_t* a) {
  KvmMmArgs g;
  if (kvm_mm_args(c, a, 0, g)) kvm_mm_simt(c, g);
}
KVM_OP_FN void kvm_op_matmul_tile_bf16(const KvmCtx& c, const int32_t* a) {
  KvmMmArgs g;
  if (kvm_mm_args(c, a, 1, g)) kvm_mm_simt(c, g);
}
// out[m,n] = a[m,k] @ b[k,n] from element 0, contiguous (include/mvm_ops.def:14; runtime/ref_ops.py:55-64).
KVM_OP_FN void kvm_op_matmul(const KvmCtx& c, const int32_t* a) {
  KvmMmArgs g{};
  if (!kvm_buf(c, a[0], KVM_M_F32, g.a) || !kvm_buf(c, a[1], KVM_M_F32, g.b) || !kvm_buf(c, a[2], KVM_M_F32, g.out)) return;
  const int m = a[3], n = a[4], k = a[5];
  if (m < 1 || n < 1 || k < 1 || !kvm_flat_ok(c, g.a, (long long)m * k) || !kvm_flat_ok(c, g.b, (long long)k * n) || !kvm_flat_ok(c, g.out, (long long)m * n)) {
    c.fail(KVM_OPE_RANGE, m, n); return; }
  g.a.ld = k; g.b.ld = n; g.out.ld = n;
  g.M = m; g.N = n; g.K = k; g.m0 = 0; g.n0 = 0; g.tm = m; g.tn = n; g.alpha = 1.0f; g.flags = 0; g.round_ops = false;
  kvm_mm_simt(c, g);
}
