// Row-structured memory-bound ops: embeddings, normalisation forward/backward, column sums, rotary embedding,
// cross-entropy, AdamW, gradient norm, argmax.  Reference semantics: runtime/ref_gpt.py:44-66,107-193,250-275,414-482,
// runtime/ref_extra.py:333-360.  Sums run in float32 warp/block trees of fixed shape (deterministic per launch geometry);
// the reference's CPU model sums in double, so these agree to its documented 1e-5 relative tolerance, not bitwise.
#pragma once
#include "kvm_dev.cuh"

// ---- embeddings --------------------------------------------------------------------------------------------------------------
KVM_OP_FN void kvm_op_embedding_fwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf ids, wte, wpe, out;
  if (!kvm_buf(c, a[0], KVM_M_I32, ids) || !kvm_buf(c, a[1], KVM_M_FLT, wte) || !kvm_buf(c, a[2], KVM_M_FLT, wpe, true) ||
      !kvm_buf(c, a[3], KVM_M_FLT, out)) return;
  int r0 = a[4], r1 = a[5], T = a[6], d = a[7];
  if (r0 < 0 || r1 < r0 || T <= 0 || d <= 0 || !kvm_flat_ok(c, ids, r1) || !kvm_mat_ok(c, out, r1, d) || !kvm_mat_ok(c, wte, 0, d) ||
      !kvm_mat_ok(c, wpe, T, d)) { c.fail(KVM_OPE_RANGE, r0, r1); return; }
  const int* id = (const int*)ids.p;
  if (wte.dtype == KVM_F32 && out.dtype == KVM_F32 && (!wpe.p || (wpe.dtype == KVM_F32 && (wpe.ld & 3) == 0 && kvm_vec_ok(wpe))) && ((d | wte.ld | out.ld) & 3) == 0 && kvm_vec_ok(wte) &&
      kvm_vec_ok(out)) {
    // float32 tables: four 16-byte pieces per thread and table in flight (the scalar loop below has one element in flight, and each
    // waits for its token id: 300 us for 256 rows of 768 values, 20 us here for the same rows)
    const int cpr = d / 4, items = (r1 - r0) * cpr;
    for (int i0 = 0; i0 < items; i0 += 4 * KVM_NT) {
      int tok[4];
      float4 x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) { const int it = i0 + u * KVM_NT + threadIdx.x; tok[u] = it < items ? id[r0 + it / cpr] : -1; }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int it = i0 + u * KVM_NT + threadIdx.x;
        x[u] = y[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (it < items) {
          const int r = r0 + it / cpr, col = (it % cpr) * 4;
          if (tok[u] < 0 || tok[u] >= wte.rows) c.fail_any(KVM_OPE_TOKEN, tok[u], r);
          else {
            x[u] = *(const float4*)((const float*)wte.p + (size_t)tok[u] * wte.ld + col);
            if (wpe.p) y[u] = *(const float4*)((const float*)wpe.p + (size_t)(r % T) * wpe.ld + col);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int it = i0 + u * KVM_NT + threadIdx.x;
        if (it < items) {
          if (wpe.p) { x[u].x = __fadd_rn(x[u].x, y[u].x); x[u].y = __fadd_rn(x[u].y, y[u].y); x[u].z = __fadd_rn(x[u].z, y[u].z); x[u].w = __fadd_rn(x[u].w, y[u].w); }
          *(float4*)((float*)out.p + (size_t)(r0 + it / cpr) * out.ld + (it % cpr) * 4) = x[u];
        }
      }
    }
    return;
  }
  long long n = (long long)(r1 - r0) * d;
  for (long long e = threadIdx.x; e < n; e += KVM_NT) {
    int r = r0 + (int)(e / d), col = (int)(e % d), tok = id[r];
    float v = 0.0f;
    if (tok < 0 || tok >= wte.rows) c.fail_any(KVM_OPE_TOKEN, tok, r);
    else {
      v = kvm_ld(wte, (size_t)tok * wte.ld + col);
      if (wpe.p) v = __fadd_rn(v, kvm_ld(wpe, (size_t)(r % T) * wpe.ld + col));
    }
    kvm_st(out, (size_t)r * out.ld + col, v);
  }
}

// One task owns keys [v0,v1): rows with a key in range are compacted in ascending order into shared memory (block-wide
// ordered scan) together with their key; a warp then adds the rows of its keys (key mod 16) one after the other, its lanes over the
// columns, so every element sums its rows in ascending order with one float32 add each (runtime/ref_gpt.py:55-66) while sixteen
// keys go on side by side.  (The whole block on one row at a time was a serial chain of read-modify-writes over all hits of the
// task: 183 us for 512 rows of 128 columns.)
KVM_OP_FN void kvm_op_embedding_bwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf ids, dout, dt;
  if (!kvm_buf(c, a[0], KVM_M_I32, ids, true) || !kvm_buf(c, a[1], KVM_M_FLT, dout) || !kvm_buf(c, a[2], KVM_M_F32, dt)) return;
  int N = a[3], mod = a[4], v0 = a[5], v1 = a[6], d = a[7], acc = a[8];
  if (N < 0 || v0 < 0 || v1 < v0 || d <= 0 || (!ids.p && mod <= 0) || !kvm_mat_ok(c, dout, N, d) || !kvm_mat_ok(c, dt, v1, d) ||
      !kvm_flat_ok(c, ids, N)) { c.fail(KVM_OPE_RANGE, v0, v1); return; }
  float* tab = (float*)dt.p;
  const bool vec = dout.dtype == KVM_F32 && ((d | dout.ld | dt.ld) & 3) == 0 && kvm_vec_ok(dout) && kvm_vec_ok(dt);
  const int cpr = vec ? d / 4 : d;
  if (!ids.p) {
    // positional table: key k collects rows k, k+mod, k+2*mod, ... in that (ascending) order; thread = (key, column or four columns),
    // eight rows' loads in flight
    for (long long e = threadIdx.x; e < (long long)(v1 - v0) * cpr; e += KVM_NT) {
      const int key = v0 + (int)(e / cpr), col = (int)(e % cpr) * (vec ? 4 : 1);
      const size_t o = (size_t)key * dt.ld + col;
      if (vec) {
        float4 sum = acc ? *(const float4*)(tab + o) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (key < mod)
          for (int r = key; r < N; r += 8 * mod) {
            float4 x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) if (r + (long long)u * mod < N) x[u] = *(const float4*)((const float*)dout.p + (size_t)(r + u * mod) * dout.ld + col);
#pragma unroll
            for (int u = 0; u < 8; ++u) if (r + (long long)u * mod < N) {
              sum.x = __fadd_rn(sum.x, x[u].x); sum.y = __fadd_rn(sum.y, x[u].y); sum.z = __fadd_rn(sum.z, x[u].z); sum.w = __fadd_rn(sum.w, x[u].w);
            }
          }
        *(float4*)(tab + o) = sum;
        continue;
      }
      float sum = acc ? tab[o] : 0.0f;
      if (key < mod) for (int r = key; r < N; r += mod) sum = __fadd_rn(sum, kvm_ld(dout, (size_t)r * dout.ld + col));
      tab[o] = sum;
    }
    return;
  }
  if (!acc) {
    for (long long e = threadIdx.x; e < (long long)(v1 - v0) * cpr; e += KVM_NT) {
      float* o = tab + (size_t)(v0 + e / cpr) * dt.ld + (e % cpr) * (vec ? 4 : 1);
      if (vec) *(float4*)o = make_float4(0.0f, 0.0f, 0.0f, 0.0f); else *o = 0.0f;
    }
  }
  int2* list = (int2*)c.smem;                     // [cap] (row, key), then KVM_NWARPS counters
  const int cap = (c.smem_bytes - 256) / 8;
  int* wcnt = (int*)(list + cap);
  const int* id = (const int*)ids.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  kvm_sync();
  for (int base = 0; base < N;) {
    // fill the list with up to cap matching rows starting at `base`
    int filled = 0, next = base;
    while (next < N && filled + 4 * KVM_NT <= cap) {
      // four rows per thread and pass (a thread's rows are neighbours, so ascending order is thread order)
      const int r = next + threadIdx.x * 4;
      int key[4], n = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) key[u] = r + u < N ? id[r + u] : -1;
#pragma unroll
      for (int u = 0; u < 4; ++u) { if (key[u] < v0 || key[u] >= v1) key[u] = -1; n += key[u] >= 0; }
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
      if (lane == 31) wcnt[warp] = incl;
      kvm_sync();
      int off = filled + incl - n, tot = 0;
      for (int w = 0; w < KVM_NWARPS; ++w) { if (w < warp) off += wcnt[w]; tot += wcnt[w]; }
#pragma unroll
      for (int u = 0; u < 4; ++u) if (key[u] >= 0) list[off++] = make_int2(r + u, key[u]);
      kvm_sync();
      filled += tot; next += 4 * KVM_NT;
    }
    for (int i0 = 0; i0 < filled; i0 += 32) {
      const int2 e = i0 + lane < filled ? list[i0 + lane] : make_int2(0, -1);
      unsigned mine = __ballot_sync(0xffffffffu, e.y >= 0 && (e.y & (KVM_NWARPS - 1)) == warp);
      while (mine) {
        const int src = __ffs(mine) - 1;
        mine &= mine - 1;
        const int r = __shfl_sync(0xffffffffu, e.x, src), key = __shfl_sync(0xffffffffu, e.y, src);
        float* o = tab + (size_t)key * dt.ld;
        if (vec) {
          for (int k = lane * 4; k < d; k += 512) {        // four pieces of the row in flight
            float4 x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) if (k + u * 128 < d) { x[u] = *(const float4*)((const float*)dout.p + (size_t)r * dout.ld + k + u * 128); y[u] = *(const float4*)(o + k + u * 128); }
#pragma unroll
            for (int u = 0; u < 4; ++u) if (k + u * 128 < d)
              *(float4*)(o + k + u * 128) = make_float4(__fadd_rn(y[u].x, x[u].x), __fadd_rn(y[u].y, x[u].y), __fadd_rn(y[u].z, x[u].z), __fadd_rn(y[u].w, x[u].w));
          }
        } else for (int k = lane; k < d; k += 32) o[k] = __fadd_rn(o[k], kvm_ld(dout, (size_t)r * dout.ld + k));
      }
    }
    kvm_sync();
    base = next;
  }
}

KVM_OP_FN void kvm_op_add_rowtile(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, pos, out;
  if (!kvm_buf(c, a[0], KVM_M_FLT, x) || !kvm_buf(c, a[1], KVM_M_FLT, pos) || !kvm_buf(c, a[2], KVM_M_FLT, out)) return;
  int r0 = a[3], r1 = a[4], T = a[5], d = a[6];
  if (r0 < 0 || r1 < r0 || T <= 0 || d <= 0 || !kvm_mat_ok(c, x, r1, d) || !kvm_mat_ok(c, out, r1, d) || !kvm_mat_ok(c, pos, T, d)) {
    c.fail(KVM_OPE_RANGE, r0, r1); return; }
  for (long long e = threadIdx.x; e < (long long)(r1 - r0) * d; e += KVM_NT) {
    int r = r0 + (int)(e / d), col = (int)(e % d);
    kvm_st(out, (size_t)r * out.ld + col, __fadd_rn(kvm_ld(x, (size_t)r * x.ld + col), kvm_ld(pos, (size_t)(r % T) * pos.ld + col)));
  }
}

KVM_OP_FN void kvm_op_gather_rows(const KvmCtx& c, const int32_t* a) {
  KvmBuf src, idx, dst;
  if (!kvm_buf(c, a[0], KVM_M_FLT, src) || !kvm_buf(c, a[1], KVM_M_I32, idx) || !kvm_buf(c, a[2], KVM_M_FLT, dst)) return;
  int r0 = a[3], r1 = a[4], d = a[5];
  if (r0 < 0 || r1 < r0 || d <= 0 || !kvm_flat_ok(c, idx, r1) || !kvm_mat_ok(c, dst, r1, d) || !kvm_mat_ok(c, src, 0, d)) {
    c.fail(KVM_OPE_RANGE, r0, r1); return; }
  if (src.dtype == KVM_BF16 && dst.dtype == KVM_F32 && ((d | src.ld | dst.ld) & 7) == 0 && kvm_vec_ok(src) && kvm_vec_ok(dst)) {      // a decode step's embedding rows: 8 values per access
    const int cpr = d / 8;
#pragma unroll 2
    for (int it = threadIdx.x; it < (r1 - r0) * cpr; it += KVM_NT) {
      const int r = r0 + it / cpr, col = (it % cpr) * 8, i = ((const int*)idx.p)[r];
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (i < 0 || i >= src.rows) c.fail_any(KVM_OPE_TOKEN, i, r);
      else kvm_ld8t<true>(src.p, (size_t)i * src.ld + col, v);
      kvm_st8t<false>(dst.p, (size_t)r * dst.ld + col, v);
    }
    return;
  }
  for (long long e = threadIdx.x; e < (long long)(r1 - r0) * d; e += KVM_NT) {
    int r = r0 + (int)(e / d), col = (int)(e % d), i = ((const int*)idx.p)[r];
    float v = 0.0f;
    if (i < 0 || i >= src.rows) c.fail_any(KVM_OPE_TOKEN, i, r);
    else v = kvm_ld(src, (size_t)i * src.ld + col);
    kvm_st(dst, (size_t)r * dst.ld + col, v);
  }
}

// ---- normalisation: one warp per row -----------------------------------------------------------------------------------------
template <bool RMS>
static __device__ void kvm_norm_fwd(const KvmCtx& c, int xi, int gi, int bi, int oi, int mi, int ri, int r0, int r1, int d, float eps) {
  KvmBuf x, g, be, out, mean, rstd;
  if (!kvm_buf(c, xi, KVM_M_FLT, x) || !kvm_buf(c, gi, KVM_M_F32, g) || !kvm_buf(c, bi, KVM_M_F32, be, RMS) || !kvm_buf(c, oi, KVM_M_FLT, out) ||
      !kvm_buf(c, mi, KVM_M_F32, mean, RMS) || !kvm_buf(c, ri, KVM_M_F32, rstd)) return;
  if (r0 < 0 || r1 < r0 || d <= 0 || !kvm_mat_ok(c, x, r1, d) || !kvm_mat_ok(c, out, r1, d) || !kvm_flat_ok(c, g, d) || !kvm_flat_ok(c, be, d) ||
      !kvm_flat_ok(c, mean, r1) || !kvm_flat_ok(c, rstd, r1)) { c.fail(KVM_OPE_RANGE, r0, r1); return; }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* gp = (const float*)g.p;
  const float* bp = (const float*)be.p;
  const bool vec = (d & 7) == 0 && (x.ld & 7) == 0 && (out.ld & 7) == 0 && kvm_vec_ok(x) && kvm_vec_ok(out) && kvm_vec_ok(g) && (RMS || kvm_vec_ok(be));
  if (vec && d <= 1024) {
    // the row (up to four 8-element vectors per lane) is fetched once and stays in registers over the two reductions (gamma and
    // beta come from L1 as vectors); same per-lane summation order as the loops below
    for (int r = r0 + warp; r < r1; r += KVM_NWARPS) {
      const size_t xo = (size_t)r * x.ld, oo = (size_t)r * out.ld;
      float xv[4][8], s = 0.0f, q = 0.0f;
#pragma unroll
      for (int t = 0; t < 4; ++t) { const int k = lane * 8 + t * 256; if (k < d) kvm_ld8(x, xo + k, xv[t]); }
      if (!RMS) {
#pragma unroll
        for (int t = 0; t < 4; ++t) if (lane * 8 + t * 256 < d) {
#pragma unroll
          for (int j = 0; j < 8; ++j) s += xv[t][j];
        }
        s = kvm_warp_sum(s);
      }
      const float mu = RMS ? 0.0f : s / d;
#pragma unroll
      for (int t = 0; t < 4; ++t) if (lane * 8 + t * 256 < d) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float tt = xv[t][j] - mu; q += tt * tt; }
      }
      q = kvm_warp_sum(q);
      const float rs = 1.0f / sqrtf(q / d + eps);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int k = lane * 8 + t * 256;
        if (k < d) {
          float ov[8], gv[8], bv[8];
          kvm_ld8(g, k, gv);
          if (!RMS) kvm_ld8(be, k, bv);
#pragma unroll
          for (int j = 0; j < 8; ++j) ov[j] = (xv[t][j] - mu) * rs * gv[j] + (RMS ? 0.0f : bv[j]);
          kvm_st8(out, oo + k, ov);
        }
      }
      if (lane == 0) { ((float*)rstd.p)[r] = rs; if (!RMS) ((float*)mean.p)[r] = mu; }
    }
    return;
  }
  for (int r = r0 + warp; r < r1; r += KVM_NWARPS) {
    const size_t xo = (size_t)r * x.ld, oo = (size_t)r * out.ld;
    float s = 0.0f;
    if (!RMS) {
      if (vec) for (int k = lane * 8; k < d; k += 256) { float v[8]; kvm_ld8(x, xo + k, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j]; }
      else for (int k = lane; k < d; k += 32) s += kvm_ld(x, xo + k);
      s = kvm_warp_sum(s);
    }
    const float mu = RMS ? 0.0f : s / d;
    float q = 0.0f;
    if (vec) for (int k = lane * 8; k < d; k += 256) { float v[8]; kvm_ld8(x, xo + k, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) { float t = v[j] - mu; q += t * t; } }
    else for (int k = lane; k < d; k += 32) { float t = kvm_ld(x, xo + k) - mu; q += t * t; }
    q = kvm_warp_sum(q);
    const float rs = 1.0f / sqrtf(q / d + eps);
    if (vec) for (int k = lane * 8; k < d; k += 256) {
      float v[8], o[8]; kvm_ld8(x, xo + k, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (v[j] - mu) * rs * gp[k + j] + (RMS ? 0.0f : bp[k + j]);
      kvm_st8(out, oo + k, o);
    } else for (int k = lane; k < d; k += 32) kvm_st(out, oo + k, (kvm_ld(x, xo + k) - mu) * rs * gp[k] + (RMS ? 0.0f : bp[k]));
    if (lane == 0) { ((float*)rstd.p)[r] = rs; if (!RMS) ((float*)mean.p)[r] = mu; }
  }
}
KVM_OP_FN void kvm_op_layernorm_fwd(const KvmCtx& c, const int32_t* a) {
  kvm_norm_fwd<false>(c, a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], kvm_bits_f32(a[9]));
}
KVM_OP_FN void kvm_op_rmsnorm_fwd(const KvmCtx& c, const int32_t* a) {
  kvm_norm_fwd<true>(c, a[0], a[1], -1, a[2], -1, a[3], a[4], a[5], a[6], kvm_bits_f32(a[7]));
}

template <bool RMS>
static __device__ void kvm_norm_bwd_dx(const KvmCtx& c, int xi, int dyi, int gi, int mi, int ri, int dxi, int r0, int r1, int d, int acc) {
  KvmBuf x, dy, g, mean, rstd, dx;
  if (!kvm_buf(c, xi, KVM_M_FLT, x) || !kvm_buf(c, dyi, KVM_M_FLT, dy) || !kvm_buf(c, gi, KVM_M_F32, g) || !kvm_buf(c, mi, KVM_M_F32, mean, RMS) ||
      !kvm_buf(c, ri, KVM_M_F32, rstd) || !kvm_buf(c, dxi, KVM_M_FLT, dx)) return;
  if (r0 < 0 || r1 < r0 || d <= 0 || !kvm_mat_ok(c, x, r1, d) || !kvm_mat_ok(c, dy, r1, d) || !kvm_mat_ok(c, dx, r1, d) || !kvm_flat_ok(c, g, d) ||
      !kvm_flat_ok(c, mean, r1) || !kvm_flat_ok(c, rstd, r1)) { c.fail(KVM_OPE_RANGE, r0, r1); return; }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* gp = (const float*)g.p;
  const bool vec = (d & 7) == 0 && d <= 1024 && (x.ld & 7) == 0 && (dy.ld & 7) == 0 && (dx.ld & 7) == 0 && kvm_vec_ok(x) && kvm_vec_ok(dy) && kvm_vec_ok(dx) && kvm_vec_ok(g);
  for (int r = r0 + warp; r < r1; r += KVM_NWARPS) {
    const float mu = RMS ? 0.0f : ((const float*)mean.p)[r], rs = ((const float*)rstd.p)[r];
    const size_t xo = (size_t)r * x.ld, yo = (size_t)r * dy.ld, oo = (size_t)r * dx.ld;
    float s1 = 0.0f, s2 = 0.0f;
    if (vec) {      // the row stays in registers between the two passes: up to four 8-element vectors of x and dy per lane
      float xv[4][8], gv[4][8];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int k = lane * 8 + t * 256;
        if (k < d) {
          float yv[8], gm[8];
          kvm_ld8(x, xo + k, xv[t]); kvm_ld8(dy, yo + k, yv); kvm_ld8(g, k, gm);
#pragma unroll
          for (int j = 0; j < 8; ++j) { gv[t][j] = yv[j] * gm[j]; xv[t][j] = (xv[t][j] - mu) * rs; s1 += gv[t][j]; s2 += gv[t][j] * xv[t][j]; }
        }
      }
      s1 = RMS ? 0.0f : kvm_warp_sum(s1) / d;
      s2 = kvm_warp_sum(s2) / d;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int k = lane * 8 + t * 256;
        if (k < d) {
          float o[8];
          if (acc) kvm_ld8(dx, oo + k, o);
#pragma unroll
          for (int j = 0; j < 8; ++j) { const float v = rs * (gv[t][j] - s1 - xv[t][j] * s2); o[j] = acc ? __fadd_rn(o[j], v) : v; }
          kvm_st8(dx, oo + k, o);
        }
      }
      continue;
    }
    for (int k = lane; k < d; k += 32) {
      float gs = kvm_ld(dy, yo + k) * gp[k], xh = (kvm_ld(x, xo + k) - mu) * rs;
      s1 += gs; s2 += gs * xh;
    }
    s1 = RMS ? 0.0f : kvm_warp_sum(s1) / d;
    s2 = kvm_warp_sum(s2) / d;
    for (int k = lane; k < d; k += 32) {
      float gs = kvm_ld(dy, yo + k) * gp[k], xh = (kvm_ld(x, xo + k) - mu) * rs;
      float v = rs * (gs - s1 - xh * s2);
      kvm_st(dx, oo + k, acc ? __fadd_rn(kvm_ld(dx, oo + k), v) : v);
    }
  }
}
KVM_OP_FN void kvm_op_layernorm_bwd_dx(const KvmCtx& c, const int32_t* a) { kvm_norm_bwd_dx<false>(c, a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9]); }
KVM_OP_FN void kvm_op_rmsnorm_bwd_dx(const KvmCtx& c, const int32_t* a) { kvm_norm_bwd_dx<true>(c, a[0], a[1], a[2], -1, a[3], a[4], a[5], a[6], a[7], a[8]); }

// Column sums over R rows for columns [c0,c1): thread = (row group, column), row groups reduced in fixed order through
// shared memory.  MODE 0: colsum of x; MODE 1: dgamma / dbeta of a norm layer.
template <int MODE, bool XB, bool YB>
static __device__ void kvm_colreduce_t(const KvmCtx& c, const KvmBuf& x, const KvmBuf& dy, const KvmBuf& mean, const KvmBuf& rstd, float* o1, float* o2,
                                       int R, int c0, int c1, int acc) {
  float* red = (float*)c.smem;                    // [2][KVM_NT]
  const void* xp = x.p;
  const void* yp = dy.p;
  const float* mp = (const float*)mean.p;
  const float* rp = (const float*)rstd.p;
  const size_t xld = x.ld, yld = MODE == 1 ? dy.ld : 0;
  for (int cb = c0; cb < c1; cb += 64) {
    const int w = min(64, c1 - cb), col = threadIdx.x & 63, rg = threadIdx.x >> 6, ngroups = KVM_NT / 64;
    float s1 = 0.0f, s2 = 0.0f;
    if (col < w) {
      // latency-bound (one short load per row): eight rows' loads are issued before the first is used; the sums run in row order
      int r = rg;
      for (; r + 7 * ngroups < R; r += 8 * ngroups) {
        float xv[8], gv[8], mu[8], rs[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int rr = r + u * ngroups;
          xv[u] = kvm_ldt<XB>(xp, (size_t)rr * xld + cb + col);
          if (MODE == 1) {
            gv[u] = kvm_ldt<YB>(yp, (size_t)rr * yld + cb + col);
            mu[u] = mp ? mp[rr] : 0.0f;
            rs[u] = rp[rr];
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (MODE == 0) s1 += xv[u];
          else { s1 += gv[u] * (xv[u] - mu[u]) * rs[u]; s2 += gv[u]; }
        }
      }
      for (; r < R; r += ngroups) {
        if (MODE == 0) s1 += kvm_ldt<XB>(xp, (size_t)r * xld + cb + col);
        else {
          const float g = kvm_ldt<YB>(yp, (size_t)r * yld + cb + col);
          const float mu = mp ? mp[r] : 0.0f;
          s1 += g * (kvm_ldt<XB>(xp, (size_t)r * xld + cb + col) - mu) * rp[r];
          s2 += g;
        }
      }
    }
    kvm_sync();
    red[threadIdx.x] = s1; red[KVM_NT + threadIdx.x] = s2;
    kvm_sync();
    if (threadIdx.x < w) {
      float t1 = 0.0f, t2 = 0.0f;
      for (int g = 0; g < ngroups; ++g) { t1 += red[g * 64 + threadIdx.x]; t2 += red[KVM_NT + g * 64 + threadIdx.x]; }
      const int cc = cb + threadIdx.x;
      o1[cc] = acc ? __fadd_rn(o1[cc], t1) : t1;
      if (MODE == 1 && o2) o2[cc] = acc ? __fadd_rn(o2[cc], t2) : t2;
    }
  }
}
// Column sums over R rows for columns [c0,c1): thread = (row group, column), row groups reduced in fixed order through
// shared memory.  MODE 0: colsum of x; MODE 1: dgamma / dbeta of a norm layer.  One instance per storage type of x (and dy).
template <int MODE>
static __device__ void kvm_colreduce(const KvmCtx& c, const KvmBuf& x, const KvmBuf& dy, const KvmBuf& mean, const KvmBuf& rstd, float* o1, float* o2,
                              int R, int c0, int c1, int acc) {
  const bool xb = x.dtype == KVM_BF16, yb = MODE == 1 && dy.dtype == KVM_BF16;
  if (MODE == 0) {
    if (xb) kvm_colreduce_t<MODE, true, false>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
    else kvm_colreduce_t<MODE, false, false>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
  } else if (xb) {
    if (yb) kvm_colreduce_t<MODE, true, true>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
    else kvm_colreduce_t<MODE, true, false>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
  } else {
    if (yb) kvm_colreduce_t<MODE, false, true>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
    else kvm_colreduce_t<MODE, false, false>(c, x, dy, mean, rstd, o1, o2, R, c0, c1, acc);
  }
}
KVM_OP_FN void kvm_op_colsum(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, out, none{};
  if (!kvm_buf(c, a[0], KVM_M_FLT, x) || !kvm_buf(c, a[1], KVM_M_F32, out)) return;
  int R = a[2], c0 = a[3], c1 = a[4];
  if (R < 0 || c0 < 0 || c1 < c0 || !kvm_mat_ok(c, x, R, c1) || !kvm_flat_ok(c, out, c1)) { c.fail(KVM_OPE_RANGE, c0, c1); return; }
  kvm_colreduce<0>(c, x, none, none, none, (float*)out.p, nullptr, R, c0, c1, a[5]);
}
KVM_OP_FN void kvm_op_norm_bwd_params(const KvmCtx& c, const int32_t* a) {
  KvmBuf x, dy, mean, rstd, dg, db;
  if (!kvm_buf(c, a[0], KVM_M_FLT, x) || !kvm_buf(c, a[1], KVM_M_FLT, dy) || !kvm_buf(c, a[2], KVM_M_F32, mean, true) || !kvm_buf(c, a[3], KVM_M_F32, rstd) ||
      !kvm_buf(c, a[4], KVM_M_F32, dg) || !kvm_buf(c, a[5], KVM_M_F32, db, true)) return;
  int R = a[6], d = a[7], c0 = a[8], c1 = a[9];
  if (R < 0 || c0 < 0 || c1 < c0 || c1 > d || !kvm_mat_ok(c, x, R, d) || !kvm_mat_ok(c, dy, R, d) || !kvm_flat_ok(c, mean, R) || !kvm_flat_ok(c, rstd, R) ||
      !kvm_flat_ok(c, dg, d) || !kvm_flat_ok(c, db, d)) { c.fail(KVM_OPE_RANGE, c0, c1); return; }
  kvm_colreduce<1>(c, x, dy, mean, rstd, (float*)dg.p, (float*)db.p, R, c0, c1, a[10]);
}

// ---- rotary embedding (pairs (i, i+hd/2); ang = f32(f32(pos) * f32(theta^(-2i/hd))), runtime/ref_gpt.py:250-262) ------------------
__device__ __forceinline__ float kvm_rope_inv(float theta, int i, int hd) { return (float)pow((double)theta, -(double)(float)(2 * i) / hd); }
static __device__ void kvm_rope(const KvmCtx& c, const int32_t* a, float sign) {
  KvmBuf x, out, pos;
  if (!kvm_buf(c, a[0], KVM_M_FLT, x) || !kvm_buf(c, a[1], KVM_M_FLT, out) || !kvm_buf(c, a[2], KVM_M_I32, pos, true)) return;
  int r0 = a[3], r1 = a[4], T = a[5], H = a[6], hd = a[7];
  float theta = kvm_bits_f32(a[8]);
  if (r0 < 0 || r1 < r0 || T <= 0 || H <= 0 || hd <= 0 || (hd & 1) || hd > 512 || !kvm_mat_ok(c, x, r1, H * hd) || !kvm_mat_ok(c, out, r1, H * hd)) {
    c.fail(KVM_OPE_RANGE, r0, r1); return; }
  const int half = hd / 2, p0 = pos.p ? ((const int*)pos.p)[0] : 0;
  float* inv = (float*)c.smem;
  kvm_sync();
  for (int i = threadIdx.x; i < half; i += KVM_NT) inv[i] = kvm_rope_inv(theta, i, hd);
  kvm_sync();
  long long n = (long long)(r1 - r0) * H * half;
  for (long long e = threadIdx.x; e < n; e += KVM_NT) {
    int i = (int)(e % half), h = (int)((e / half) % H), r = r0 + (int)(e / ((long long)half * H));
    float ang = __fmul_rn((float)((r % T) + p0), inv[i]), s, co;
    sincosf(ang, &s, &co);
    s *= sign;
    size_t o1 = (size_t)r * x.ld + h * hd + i, w1 = (size_t)r * out.ld + h * hd + i;
    float x1 = kvm_ld(x, o1), x2 = kvm_ld(x, o1 + half);
    kvm_st(out, w1, x1 * co - x2 * s);
    kvm_st(out, w1 + half, x1 * s + x2 * co);
  }
}
KVM_OP_FN void kvm_op_rope_fwd(const KvmCtx& c, const int32_t* a) { kvm_rope(c, a, 1.0f); }
KVM_OP_FN void kvm_op_rope_bwd(const KvmCtx& c, const int32_t* a) { kvm_rope(c, a, -1.0f); }

// ---- cross entropy: the block walks rows; per row one pass for (max, sum) and one for the gradient -------------------------------------
// MODE bit 0: forward (rowloss, lse); bit 1: backward (dlogits).
// Short rows (V <= 1024): a warp per row, RP rows of a warp side by side, the row in NV registers per lane over both passes (a block per
// row spends its time in two block reductions: 408 us for 256 rows of 10 classes).
template <int MODE, bool LB, int NV, int RP>
static __device__ void kvm_ce_short_t(const KvmCtx& c, const KvmBuf& lg, const KvmBuf& tg, const KvmBuf& rl, const KvmBuf& ls, const KvmBuf& dl, int r0, int r1, int V, int ignore, float f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int rb = r0 + warp * RP; rb < r1; rb += KVM_NWARPS * RP) {
    int t[RP];
    float v[RP][NV], lse[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) {
      const int r = min(rb + i, r1 - 1);
      t[i] = ((const int*)tg.p)[r];
#pragma unroll
      for (int j = 0; j < NV; ++j) { const int k = lane + 32 * j; v[i][j] = k < V ? kvm_ldt<LB>(lg.p, (size_t)r * lg.ld + k) : -INFINITY; }
      if (!(MODE & 1)) lse[i] = ((const float*)ls.p)[r];
    }
#pragma unroll
    for (int i = 0; i < RP; ++i) {
      const int r = rb + i;
      if (MODE & 1) {
        float m = v[i][0], s = 0.0f;
#pragma unroll
        for (int j = 1; j < NV; ++j) m = fmaxf(m, v[i][j]);
        m = kvm_warp_max(m);
#pragma unroll
        for (int j = 0; j < NV; ++j) s += __expf(v[i][j] - m);
        s = kvm_warp_sum(s);
        lse[i] = t[i] == ignore ? 0.0f : m + logf(s);
      }
      if (r >= r1) continue;
      if (t[i] != ignore && (t[i] < 0 || t[i] >= V)) { if (lane == 0) c.fail_any(KVM_OPE_TOKEN, t[i], r); continue; }
      if ((MODE & 1) && lane == 0) { ((float*)ls.p)[r] = lse[i]; ((float*)rl.p)[r] = t[i] == ignore ? 0.0f : lse[i] - kvm_ldt<LB>(lg.p, (size_t)r * lg.ld + t[i]); }
      if (MODE & 2) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int k = lane + 32 * j;
          if (k < V) kvm_st(dl, (size_t)r * dl.ld + k, t[i] == ignore ? 0.0f : (__expf(v[i][j] - lse[i]) - (k == t[i] ? 1.0f : 0.0f)) * f);
        }
      }
    }
  }
}
template <int MODE, bool LB, bool DB>      // storage types of the logits and of their gradient as template arguments: no type test inside the loops
static __device__ void kvm_ce_t(const KvmCtx& c, const KvmBuf& lg, const KvmBuf& tg, const KvmBuf& rl, const KvmBuf& ls, const KvmBuf& dl, int r0, int r1, int V,
                         int ignore, float f) {
  // a short row in registers while a task has rows for most of the warps, or the row is so short that a block cannot use its threads on it
  if (V <= 32) { kvm_ce_short_t<MODE, LB, 1, 8>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); return; }
  if (V <= 256) { kvm_ce_short_t<MODE, LB, 8, 2>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); return; }
  if (V <= 1024) { kvm_ce_short_t<MODE, LB, 32, 1>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); return; }
  float* red = (float*)c.smem;
  const bool vec = (V & 7) == 0 && (lg.ld & 7) == 0 && kvm_vec_ok(lg) && (!(MODE & 2) || ((dl.ld & 7) == 0 && kvm_vec_ok(dl)));
  for (int r = r0; r < r1; ++r) {
    const int t = ((const int*)tg.p)[r];
    const size_t lo = (size_t)r * lg.ld;
    float lse;
    if (t != ignore && (t < 0 || t >= V)) { c.fail(KVM_OPE_TOKEN, t, r); return; }
    if (MODE & 1) {
      if (t == ignore) { if (threadIdx.x == 0) { ((float*)rl.p)[r] = 0.0f; ((float*)ls.p)[r] = 0.0f; } lse = 0.0f; }
      else {
        float m = -INFINITY, s = 0.0f;            // online (max, sum) per thread
        if (vec) for (int k = threadIdx.x * 8; k < V; k += KVM_NT * 8) {
          float v[8]; kvm_ld8t<LB>(lg.p, lo + k, v);
          float mm = v[0];
#pragma unroll
          for (int j = 1; j < 8; ++j) mm = fmaxf(mm, v[j]);
          if (mm > m) { s *= __expf(m - mm); m = mm; }
#pragma unroll
          for (int j = 0; j < 8; ++j) s += __expf(v[j] - m);
        } else for (int k = threadIdx.x; k < V; k += KVM_NT) {
          float v = kvm_ldt<LB>(lg.p, lo + k);
          if (v > m) { s *= __expf(m - v); m = v; }
          s += __expf(v - m);
        }
        float M = kvm_block_max(m, red);
        s = (m == -INFINITY) ? 0.0f : s * __expf(m - M);
        float S = kvm_block_sum(s, red);
        lse = M + logf(S);
        if (threadIdx.x == 0) { ((float*)ls.p)[r] = lse; ((float*)rl.p)[r] = lse - kvm_ld(lg, lo + t); }
      }
    } else lse = ((const float*)ls.p)[r];
    if (MODE & 2) {
      const size_t dq = (size_t)r * dl.ld;
      if (vec) for (int k = threadIdx.x * 8; k < V; k += KVM_NT * 8) {
        float v[8], o[8]; kvm_ld8t<LB>(lg.p, lo + k, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = t == ignore ? 0.0f : (__expf(v[j] - lse) - (k + j == t ? 1.0f : 0.0f)) * f;
        kvm_st8t<DB>(dl.p, dq + k, o);
      } else for (int k = threadIdx.x; k < V; k += KVM_NT)
        kvm_st(dl, dq + k, t == ignore ? 0.0f : (__expf(kvm_ldt<LB>(lg.p, lo + k) - lse) - (k == t ? 1.0f : 0.0f)) * f);
    }
  }
}
template <int MODE>
static __device__ void kvm_ce(const KvmCtx& c, const KvmBuf& lg, const KvmBuf& tg, const KvmBuf& rl, const KvmBuf& ls, const KvmBuf& dl, int r0, int r1, int V,
                       int ignore, float f) {
  const bool lb = lg.dtype == KVM_BF16, db = (MODE & 2) && dl.dtype == KVM_BF16;
  if (lb) { if (db) kvm_ce_t<MODE, true, true>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); else kvm_ce_t<MODE, true, false>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); }
  else { if (db) kvm_ce_t<MODE, false, true>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); else kvm_ce_t<MODE, false, false>(c, lg, tg, rl, ls, dl, r0, r1, V, ignore, f); }
}
static __device__ bool kvm_ce_args(const KvmCtx& c, const KvmBuf& lg, const KvmBuf& tg, const KvmBuf& rl, const KvmBuf& ls, const KvmBuf& dl, int r0, int r1, int V) {
  if (r0 < 0 || r1 < r0 || V <= 0 || !kvm_mat_ok(c, lg, r1, V) || !kvm_flat_ok(c, tg, r1) || !kvm_flat_ok(c, rl, r1) || !kvm_flat_ok(c, ls, r1) ||
      !kvm_mat_ok(c, dl, r1, V)) { c.fail(KVM_OPE_RANGE, r0, r1); return false; }
  return true;
}
KVM_OP_FN void kvm_op_softmax_ce_fwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf lg, tg, rl, ls, none{};
  if (!kvm_buf(c, a[0], KVM_M_FLT, lg) || !kvm_buf(c, a[1], KVM_M_I32, tg) || !kvm_buf(c, a[2], KVM_M_F32, rl) || !kvm_buf(c, a[3], KVM_M_F32, ls)) return;
  if (!kvm_ce_args(c, lg, tg, rl, ls, none, a[4], a[5], a[6])) return;
  kvm_ce<1>(c, lg, tg, rl, ls, none, a[4], a[5], a[6], a[7], 0.0f);
}
KVM_OP_FN void kvm_op_softmax_ce_bwd(const KvmCtx& c, const int32_t* a) {
  KvmBuf lg, tg, ls, loss, dl, none{};
  if (!kvm_buf(c, a[0], KVM_M_FLT, lg) || !kvm_buf(c, a[1], KVM_M_I32, tg) || !kvm_buf(c, a[2], KVM_M_F32, ls) || !kvm_buf(c, a[3], KVM_M_F32, loss) ||
      !kvm_buf(c, a[4], KVM_M_FLT, dl)) return;
  if (!kvm_ce_args(c, lg, tg, none, ls, dl, a[5], a[6], a[7]) || !kvm_flat_ok(c, loss, 2)) return;
  kvm_ce<2>(c, lg, tg, none, ls, dl, a[5], a[6], a[7], a[8], __fmul_rn(((const float*)loss.p)[1], kvm_bits_f32(a[9])));
}
KVM_OP_FN void kvm_op_softmax_ce_fused(const KvmCtx& c, const int32_t* a) {
  KvmBuf lg, tg, rl, ls, dl;
  if (!kvm_buf(c, a[0], KVM_M_FLT, lg) || !kvm_buf(c, a[1], KVM_M_I32, tg) || !kvm_buf(c, a[2], KVM_M_F32, rl) || !kvm_buf(c, a[3], KVM_M_F32, ls) ||
      !kvm_buf(c, a[4], KVM_M_FLT, dl)) return;
  if (a[8] != -1 || a[9] <= 0) { c.fail(KVM_OPE_RANGE, a[8], a[9]); return; }
  if (!kvm_ce_args(c, lg, tg, rl, ls, dl, a[5], a[6], a[7])) return;
  kvm_ce<3>(c, lg, tg, rl, ls, dl, a[5], a[6], a[7], -1, __fmul_rn((float)(1.0 / (double)a[9]), kvm_bits_f32(a[10])));
}
// loss[0] = mean rowloss over non-ignored rows, loss[1] = 1/count (runtime/ref_gpt.py:430-437); double sums, fixed tree.
KVM_OP_FN void kvm_op_softmax_ce_reduce(const KvmCtx& c, const int32_t* a) {
  KvmBuf rl, tg, loss;
  if (!kvm_buf(c, a[0], KVM_M_F32, rl) || !kvm_buf(c, a[1], KVM_M_I32, tg) || !kvm_buf(c, a[2], KVM_M_F32, loss)) return;
  int N = a[3], ign = a[4];
  if (N < 0 || !kvm_flat_ok(c, rl, N) || !kvm_flat_ok(c, tg, N) || !kvm_flat_ok(c, loss, 2)) { c.fail(KVM_OPE_RANGE, N); return; }
  double s = 0.0, cnt = 0.0;
  for (int r = threadIdx.x; r < N; r += KVM_NT)
    if (((const int*)tg.p)[r] != ign) { s += ((const float*)rl.p)[r]; cnt += 1.0; }
  double* red = (double*)c.smem;
  s = kvm_block_sum(s, red);
  cnt = kvm_block_sum(cnt, red);
  if (threadIdx.x == 0) {
    ((float*)loss.p)[0] = cnt > 0 ? (float)(s / cnt) : 0.0f;
    ((float*)loss.p)[1] = cnt > 0 ? (float)(1.0 / cnt) : 0.0f;
  }
}

// ---- optimiser ---------------------------------------------------------------------------------------------------------------------
// AdamW in the reference's strict float32 step order (runtime/ref_gpt.py:457-471): every operation below is one rounded
// float32 operation with no fused multiply-add, so p, m, v come out bit-identical to the CPU model.
struct KvmAdamK { float lr, b1, b2, eps, bc1, bc2, omb1, omb2, lrwd, gsc; };
// Constants of one task; the two double-precision powers run on two warps side by side.  Whole compute group.
__device__ __forceinline__ KvmAdamK kvm_adamw_consts(const KvmCtx& c, int t, float lr, float b1, float b2, float eps, float wd, float gsc) {
  float* sh = (float*)c.smem;
  kvm_sync();
  if (threadIdx.x == 0) sh[0] = (float)(1.0 - (double)(float)pow((double)b1, (double)t));
  if (threadIdx.x == 32) sh[1] = (float)(1.0 - (double)(float)pow((double)b2, (double)t));
  kvm_sync();
  KvmAdamK k;
  k.lr = lr; k.b1 = b1; k.b2 = b2; k.eps = eps; k.bc1 = sh[0]; k.bc2 = sh[1]; k.omb1 = (float)(1.0 - (double)b1); k.omb2 = (float)(1.0 - (double)b2); k.lrwd = __fmul_rn(lr, wd); k.gsc = gsc;
  return k;
}
__device__ __forceinline__ void kvm_adamw_step(const KvmAdamK& k, float g, float& p, float& m, float& v) {
  const float gi = __fmul_rn(g, k.gsc);
  m = __fadd_rn(__fmul_rn(k.b1, m), __fmul_rn(k.omb1, gi));
  v = __fadd_rn(__fmul_rn(k.b2, v), __fmul_rn(__fmul_rn(k.omb2, gi), gi));
  const float decay = __fmul_rn(k.lrwd, p);
  const float step = __fdiv_rn(__fmul_rn(k.lr, __fdiv_rn(m, k.bc1)), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, k.bc2)), k.eps));
  p = __fsub_rn(__fsub_rn(p, decay), step);
}
static __device__ void kvm_adamw(const KvmCtx& c, const int32_t* a, bool lr_buf) {
  KvmBuf p, g, m, v, gs, st, lrb;
  if (!kvm_buf(c, a[0], KVM_M_F32, p) || !kvm_buf(c, a[1], KVM_M_FLT, g) || !kvm_buf(c, a[2], KVM_M_F32, m) || !kvm_buf(c, a[3], KVM_M_F32, v) ||
      !kvm_buf(c, a[4], KVM_M_F32, gs, true) || !kvm_buf(c, a[5], KVM_M_I32, st)) return;
  if (lr_buf && !kvm_buf(c, a[8], KVM_M_F32, lrb)) return;
  long long e0 = a[6], e1 = a[7];
  if (e0 < 0 || e1 < e0 || !kvm_flat_ok(c, p, e1) || !kvm_flat_ok(c, g, e1) || !kvm_flat_ok(c, m, e1) || !kvm_flat_ok(c, v, e1)) { c.fail(KVM_OPE_RANGE, (int)e0, (int)e1); return; }
  const int t = ((const int*)st.p)[0];
  if (t < 1) { c.fail(KVM_OPE_RANGE, t); return; }
  const float lr = lr_buf ? ((const float*)lrb.p)[0] : kvm_bits_f32(a[8]);
  const KvmAdamK k = kvm_adamw_consts(c, t, lr, kvm_bits_f32(a[9]), kvm_bits_f32(a[10]), kvm_bits_f32(a[11]), kvm_bits_f32(a[12]), gs.p ? ((const float*)gs.p)[0] : 1.0f);
  float* pp = (float*)p.p; float* mp = (float*)m.p; float* vp = (float*)v.p;
  const bool vec = (e0 & 7) == 0 && kvm_vec_ok(p) && kvm_vec_ok(g) && kvm_vec_ok(m) && kvm_vec_ok(v);
  long long body = vec ? ((e1 - e0) & ~7LL) : 0;
  for (long long i = e0 + (long long)threadIdx.x * 8; i + 8 <= e0 + body; i += (long long)KVM_NT * 8) {
    float P[8], G[8], M[8], Vv[8];
    kvm_ld8(p, i, P); kvm_ld8(g, i, G); kvm_ld8(m, i, M); kvm_ld8(v, i, Vv);
#pragma unroll
    for (int j = 0; j < 8; ++j) kvm_adamw_step(k, G[j], P[j], M[j], Vv[j]);
    kvm_st8(p, i, P); kvm_st8(m, i, M); kvm_st8(v, i, Vv);
  }
  for (long long i = e0 + body + threadIdx.x; i < e1; i += KVM_NT) kvm_adamw_step(k, kvm_ld(g, i), pp[i], mp[i], vp[i]);
}
KVM_OP_FN void kvm_op_adamw(const KvmCtx& c, const int32_t* a) { kvm_adamw(c, a, false); }
KVM_OP_FN void kvm_op_adamw_lr(const KvmCtx& c, const int32_t* a) { kvm_adamw(c, a, true); }

KVM_OP_FN void kvm_op_lr_schedule(const KvmCtx& c, const int32_t* a) {
  KvmBuf st, lr;
  if (!kvm_buf(c, a[0], KVM_M_I32, st) || !kvm_buf(c, a[1], KVM_M_F32, lr)) return;
  int kind = a[2], warmup = a[4], total = a[5];
  if (kind < 0 || kind > 2) { c.fail(KVM_OPE_RANGE, kind); return; }
  if (threadIdx.x == 0) {
    double t = ((const int*)st.p)[0], base = kvm_bits_f32(a[3]), mr = kvm_bits_f32(a[6]);
    double warm = (warmup > 0 && t <= warmup) ? t / warmup : 1.0;
    double den = total - warmup > 1 ? total - warmup : 1;
    double prog = fmin(fmax((t - warmup) / den, 0.0), 1.0);
    double f = kind == 0 ? 1.0 : kind == 1 ? mr + (1 - mr) * 0.5 * (1 + cos(3.141592653589793 * prog)) : 1.0 - (1 - mr) * prog;
    ((float*)lr.p)[0] = (float)(base * warm * f);
  }
}

KVM_OP_FN void kvm_op_gradnorm_partial(const KvmCtx& c, const int32_t* a) {
  KvmBuf g, part;
  if (!kvm_buf(c, a[0], KVM_M_FLT, g) || !kvm_buf(c, a[1], KVM_M_F32, part)) return;
  int slot = a[2];
  long long e0 = a[3], e1 = a[4];
  if (slot < 0 || e0 < 0 || e1 < e0 || !kvm_flat_ok(c, g, e1) || !kvm_flat_ok(c, part, slot + 1)) { c.fail(KVM_OPE_RANGE, slot); return; }
  double s = 0.0;
  const bool vec = (e0 & 7) == 0 && kvm_vec_ok(g);
  long long body = vec ? ((e1 - e0) & ~7LL) : 0;
  for (long long i = e0 + (long long)threadIdx.x * 8; i + 8 <= e0 + body; i += (long long)KVM_NT * 8) {
    float v[8]; kvm_ld8(g, i, v);
    float q = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) q += v[j] * v[j];
    s += q;
  }
  for (long long i = e0 + body + threadIdx.x; i < e1; i += KVM_NT) { float v = kvm_ld(g, i); s += (double)v * v; }
  s = kvm_block_sum(s, (double*)c.smem);
  if (threadIdx.x == 0) ((float*)part.p)[slot] = (float)s;
}
KVM_OP_FN void kvm_op_gradnorm_finish(const KvmCtx& c, const int32_t* a) {
  KvmBuf part, out;
  if (!kvm_buf(c, a[0], KVM_M_F32, part) || !kvm_buf(c, a[2], KVM_M_F32, out)) return;
  int ns = a[1];
  float mx = kvm_bits_f32(a[3]);
  if (ns < 0 || !kvm_flat_ok(c, part, ns) || !kvm_flat_ok(c, out, 2)) { c.fail(KVM_OPE_RANGE, ns); return; }
  double s = 0.0;
  for (int i = threadIdx.x; i < ns; i += KVM_NT) s += ((const float*)part.p)[i];
  s = kvm_block_sum(s, (double*)c.smem);
  if (threadIdx.x == 0) {
    float n = (float)sqrt(s);
    ((float*)out.p)[0] = mx > 0 ? fminf(1.0f, __fdiv_rn(mx, __fadd_rn(n, 1e-6f))) : 1.0f;
    ((float*)out.p)[1] = n;
  }
}

// ---- argmax (lowest index on ties, NaN never wins; runtime/ref_gpt.py:508-514) -------------------------------------------------------
static __device__ void kvm_argmax_rows(const KvmCtx& c, const KvmBuf& lg, const KvmBuf& out, int r0, int r1, int V) {
  float* rv = (float*)c.smem;
  int* ri = (int*)(rv + KVM_NWARPS);
  for (int r = r0; r < r1; ++r) {
    float bv = -INFINITY; int bi = 0x7fffffff, k0 = 0;
    if (lg.dtype == KVM_F32 && (lg.ld & 3) == 0 && kvm_vec_ok(lg)) {
      // four 16-byte pieces per thread in flight; each thread meets its columns in ascending order (a scalar column per thread and trip
      // took 92 us for 151,936 logits, one load in flight)
      const float* row = (const float*)lg.p + (size_t)r * lg.ld;
      for (; k0 + 16 * KVM_NT <= V; k0 += 16 * KVM_NT) {
        float4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = *(const float4*)(row + k0 + (u * KVM_NT + threadIdx.x) * 4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + (u * KVM_NT + threadIdx.x) * 4;
          if (x[u].x > bv) { bv = x[u].x; bi = k; }
          if (x[u].y > bv) { bv = x[u].y; bi = k + 1; }
          if (x[u].z > bv) { bv = x[u].z; bi = k + 2; }
          if (x[u].w > bv) { bv = x[u].w; bi = k + 3; }
        }
      }
    }
#pragma unroll 4
    for (int k = k0 + threadIdx.x; k < V; k += KVM_NT) {
      float v = kvm_ld(lg, (size_t)r * lg.ld + k);
      if (v > bv) { bv = v; bi = k; }              // a thread's columns ascend; -inf never wins, a row of nothing else gives column 0
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, o); int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    kvm_sync();
    if ((threadIdx.x & 31) == 0) { rv[threadIdx.x >> 5] = bv; ri[threadIdx.x >> 5] = bi; }
    kvm_sync();
    if (threadIdx.x == 0) {
      for (int w = 1; w < KVM_NWARPS; ++w) if (rv[w] > bv || (rv[w] == bv && ri[w] < bi)) { bv = rv[w]; bi = ri[w]; }
      ((int*)out.p)[r] = bi == 0x7fffffff ? 0 : bi;
    }
  }
}
KVM_OP_FN void kvm_op_argmax(const KvmCtx& c, const int32_t* a) {
  KvmBuf lg, out;
  if (!kvm_buf(c, a[0], KVM_M_FLT, lg) || !kvm_buf(c, a[1], KVM_M_I32, out)) return;
  if (a[2] < 0 || a[3] < a[2] || a[4] <= 0 || !kvm_mat_ok(c, lg, a[3], a[4]) || !kvm_flat_ok(c, out, a[3])) { c.fail(KVM_OPE_RANGE, a[2], a[3]); return; }
  kvm_argmax_rows(c, lg, out, a[2], a[3], a[4]);
}
