// Sequence-mixer kernels, second file (include/qspec_b200_seq.h): token shift with a per-slot previous row, residual sum
// with a layer norm or unit-RMS norm of the sublayer's OUTPUT, latent (low-rank) key/value preparation with a rotary
// part, whole-projection query/key norms, sliding-window softmax attention with a per-head sink over a per-slot ring
// cache (shared by the latent and the grouped-query form), the HGRN2 gated linear recurrence with its state in
// float32, per-head output norm, and the gated per-token side input. Element type of activations and large weights:
// bfloat16 or float32; every norm, score, softmax weight, angle, gate of the recurrence and state is float32.
#include <cstdlib>
#include <cstring>
#include "seq_common.cuh"
#include "../../include/qspec_b200_seq.h"

namespace qspec {

// Pairs of elements per lane where rows allow it (even sizes and strides): 4-byte bfloat16 and 8-byte float32 loads.
template <int VEC> __device__ __forceinline__ void ld_pair(const float* p, float (&o)[2]) {
  if (VEC == 2) { const float2 t = *reinterpret_cast<const float2*>(p); o[0] = t.x; o[1] = t.y; }
  else { o[0] = *p; o[1] = 0.f; }
}
template <int VEC> __device__ __forceinline__ void ld_pair(const __nv_bfloat16* p, float (&o)[2]) {
  if (VEC == 2) { const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); o[0] = t.x; o[1] = t.y; }
  else { o[0] = __bfloat162float(*p); o[1] = 0.f; }
}

// ---- token shift --------------------------------------------------------------------------------------------------
// One CTA per token. The row before a segment's first token is the slot's saved row (buffer `phase`), zero at position
// 0; a segment's last row is saved to the other buffer, so that no CTA reads what another one of the same step writes.
template <typename T>
__global__ void __launch_bounds__(256)
token_shift_kernel(const float* __restrict__ x, const float* __restrict__ shift, float* __restrict__ prev, int slots,
                   T* __restrict__ out, const int* __restrict__ meta, int ntok, int W) {
  pdl_enter();
  const int i = blockIdx.x;
  const TokMeta m = load_meta(meta, ntok, i);
  const float* xr = x + (size_t)i * W;
  const float* pr = nullptr;
  if (i > m.seg_begin) pr = xr - W;
  else if (m.pos > 0) pr = prev + ((size_t)m.phase * slots + m.slot) * W;
  float* keep = (i == m.seg_end - 1) ? prev + ((size_t)(1 - m.phase) * slots + m.slot) * W : nullptr;
  T* orow = out + (size_t)i * W;
  for (int c = threadIdx.x; c < W; c += 256) {
    const float v = xr[c];
    const float p = pr ? pr[c] : 0.f;
    orow[c] = from_f<T>(v + (p - v) * shift[c]);
    if (keep) keep[c] = v;
  }
}

// ---- residual sum with a norm of the sublayer's output ------------------------------------------------------------
// v = sum of the parts of y (weighted); n = (v - mean) / sqrt(var + eps) * w + b (kind 0) or v / sqrt(mean(v^2) + eps) * w
// (kind 1); r = x_in + n. The row lives in shared memory between the passes; the variance is the mean of the squared
// deviations (second pass), not E[v^2] - mean^2.
template <typename T, typename YT>
__global__ void __launch_bounds__(256)
add_norm_kernel(const float* __restrict__ x_in, float* __restrict__ x_out, const YT* __restrict__ y, int y_parts,
                long long y_part_stride, long long y_tok_stride, const float* __restrict__ y_w, const float* __restrict__ w,
                const float* __restrict__ b, int kind, T* __restrict__ out, int W, float eps) {
  pdl_enter();
  extern __shared__ float sm_an[];            // row [W]
  __shared__ float red[8];
  const int i = blockIdx.x, tid = threadIdx.x;
  const YT* yr = y + (size_t)i * y_tok_stride;
  float s = 0.f;
  for (int c = tid; c < W; c += 256) {
    float v;
    if (y_parts == 1 && !y_w) {
      v = to_f(yr[c]);
    } else {
      v = 0.f;
      for (int p = 0; p < y_parts; ++p) v += (y_w ? y_w[(size_t)i * y_parts + p] : 1.0f) * to_f(yr[(size_t)p * y_part_stride + c]);
    }
    sm_an[c] = v;
    s += v;
  }
  const float inv_w = 1.0f / (float)W;
  float mean = 0.f;
  if (kind == 0) mean = block_sum_256(s, red) * inv_w;
  float q = 0.f;
  for (int c = tid; c < W; c += 256) {
    const float d = sm_an[c] - mean;
    q += d * d;
  }
  const float var = block_sum_256(q, red) * inv_w;
  const float r = 1.0f / sqrtf(var + eps);
  for (int c = tid; c < W; c += 256) {
    float v = (sm_an[c] - mean) * r * w[c];
    if (b) v += b[c];
    if (x_in) v += x_in[(size_t)i * W + c];
    if (x_out) x_out[(size_t)i * W + c] = v;
    if (out) out[(size_t)i * W + c] = from_f<T>(v);
  }
}

// ---- latent attention: norms of the low-rank projections, rotary key part, cache write ----------------------------
// Row of d: [q latent (q_rank) | kv latent (kv_rank) | shared rotary key part (rot_dim)]; the last two only when the
// layer owns a cache. One CTA per token. Cache row = position % cap: [normalised kv latent | rotated key part].
template <typename T>
__global__ void __launch_bounds__(256)
latent_prep_kernel(const T* __restrict__ d, int ld, int q_rank, int kv_rank, int rot_dim, const float* __restrict__ qn_w,
                   const float* __restrict__ kvn_w, const float* __restrict__ inv_freq, int rot_dims, int pairing, T* __restrict__ cq,
                   T* __restrict__ cache, int cap, const int* __restrict__ meta, int ntok, float eps) {
  pdl_enter();
  __shared__ float red[8];
  const int i = blockIdx.x, tid = threadIdx.x;
  const T* row = d + (size_t)i * ld;
  float ss = 0.f;
  if (q_rank > 0) {
    for (int c = tid; c < q_rank; c += 256) { const float v = to_f(row[c]); ss += v * v; }
    const float rq = 1.0f / sqrtf(block_sum_256(ss, red) / (float)q_rank + eps);
    for (int c = tid; c < q_rank; c += 256) cq[(size_t)i * q_rank + c] = from_f<T>(to_f(row[c]) * rq * qn_w[c]);
  }
  if (!cache) return;
  const int slot = meta[i], pos = meta[ntok + i];
  T* crow = cache + ((size_t)slot * cap + (pos % cap)) * (kv_rank + rot_dim);
  const T* kv = row + q_rank;
  ss = 0.f;
  for (int c = tid; c < kv_rank; c += 256) { const float v = to_f(kv[c]); ss += v * v; }
  const float rk = 1.0f / sqrtf(block_sum_256(ss, red) / (float)kv_rank + eps);
  for (int c = tid; c < kv_rank; c += 256) crow[c] = from_f<T>(to_f(kv[c]) * rk * kvn_w[c]);
  const T* kr = kv + kv_rank;
  const int half = rot_dims >> 1;
  for (int c = tid; c < half; c += 256) {
    float sn, cs;
    sincosf((float)pos * inv_freq[c], &sn, &cs);
    const int iu = pairing == QSPEC_ROTARY_INTERLEAVED ? 2 * c : c, iv = pairing == QSPEC_ROTARY_INTERLEAVED ? 2 * c + 1 : c + half;
    const float u = to_f(kr[iu]), v = to_f(kr[iv]);
    crow[kv_rank + iu] = from_f<T>(u * cs - v * sn);
    crow[kv_rank + iv] = from_f<T>(v * cs + u * sn);
  }
  for (int c = rot_dims + tid; c < rot_dim; c += 256) crow[kv_rank + c] = kr[c];
}

// Rotary positions on a slice of every head: dst[t, h, 0:n] = rotate(src[t, h, off : off + n]) in float32, the first
// rot_dims entries rotated (entry i paired with i + rot_dims / 2), the rest copied.
template <typename T>
__global__ void __launch_bounds__(128)
rotary_kernel(const T* __restrict__ src, long long src_ts, int src_hs, int off, float* __restrict__ dst, long long dst_ts, int dst_hs,
              int H, int n, int rot_dims, int pairing, const float* __restrict__ inv_freq, const int* __restrict__ meta, int ntok) {
  pdl_enter();
  const int i = blockIdx.x;
  const int pos = meta[ntok + i];
  const int half = rot_dims >> 1, rest = n - rot_dims, per = half + rest;
  for (int k = threadIdx.x; k < H * per; k += 128) {
    const int h = k / per, c = k % per;
    const T* s = src + (size_t)i * src_ts + (size_t)h * src_hs + off;
    float* o = dst + (size_t)i * dst_ts + (size_t)h * dst_hs;
    if (c < half) {
      float sn, cs;
      sincosf((float)pos * inv_freq[c], &sn, &cs);
      const int iu = pairing == QSPEC_ROTARY_INTERLEAVED ? 2 * c : c, iv = pairing == QSPEC_ROTARY_INTERLEAVED ? 2 * c + 1 : c + half;
      const float u = to_f(s[iu]), v = to_f(s[iv]);
      o[iu] = u * cs - v * sn;
      o[iv] = v * cs + u * sn;
    } else {
      o[rot_dims + c - half] = to_f(s[rot_dims + c - half]);
    }
  }
}

// ---- grouped-query attention: norm over the whole query / key projection, cache write -----------------------------
// Row of p: [q (HD) | k (GD) | v (GDV) | ...], biases already added by the projection. q -> float32 buffer, k and v ->
// ring cache rows (position % cap).
template <typename T>
__global__ void __launch_bounds__(256)
qkv_prep_kernel(const T* __restrict__ p, int ld, int HD, int GD, int GDV, const float* __restrict__ qn_w,
                const float* __restrict__ kn_w, float* __restrict__ qout, T* __restrict__ cache_k, T* __restrict__ cache_v, int cap,
                const int* __restrict__ meta, int ntok, float eps) {
  pdl_enter();
  __shared__ float red[8];
  const int i = blockIdx.x, tid = threadIdx.x;
  const T* row = p + (size_t)i * ld;
  const int slot = meta[i], pos = meta[ntok + i];
  float ss = 0.f;
  for (int c = tid; c < HD; c += 256) { const float v = to_f(row[c]); ss += v * v; }
  const float rq = 1.0f / sqrtf(block_sum_256(ss, red) / (float)HD + eps);
  for (int c = tid; c < HD; c += 256) qout[(size_t)i * HD + c] = to_f(row[c]) * rq * qn_w[c];
  const T* k = row + HD;
  ss = 0.f;
  for (int c = tid; c < GD; c += 256) { const float v = to_f(k[c]); ss += v * v; }
  const float rk = 1.0f / sqrtf(block_sum_256(ss, red) / (float)GD + eps);
  const size_t r = (size_t)slot * cap + (pos % cap);
  for (int c = tid; c < GD; c += 256) cache_k[r * GD + c] = from_f<T>(to_f(k[c]) * rk * kn_w[c]);
  const T* v = k + GD;
  for (int c = tid; c < GDV; c += 256) cache_v[r * GDV + c] = v[c];
}

// ---- sliding-window softmax attention with a sink -------------------------------------------------------------------
// One CTA of four warps per (token, query head). Query = two float32 parts (qa against key[0:DA], qb against
// key[DA:DA+DB]); keys and values are rows of a per-slot ring (row = position % cap) that already holds the step's
// own tokens. A warp takes every fourth run of four keys of the window: lanes along the rows for the dot products, an
// online softmax per warp, and the four partial results are merged in shared memory together with the sink term
// exp(sink[h]) of the denominator. Which warp takes which key depends on the token's position only, so a token's result
// does not depend on how its sequence was cut into steps or on its neighbours in the batch.
template <typename T, int NACC, int VEC>
__global__ void __launch_bounds__(128)
window_attn_kernel(const float* __restrict__ qa, long long qa_ts, long long qa_hs, int DA, const float* __restrict__ qb,
                   long long qb_ts, long long qb_hs, int DB, const T* __restrict__ kc, long long k_ss, int k_rs, int k_hs,
                   const T* __restrict__ vc, long long v_ss, int v_rs, int v_hs, int DV, const float* __restrict__ sink,
                   const T* __restrict__ gate, int gate_ld, int gate_per_head, T* __restrict__ out, const int* __restrict__ meta,
                   int ntok, int H, int G, int window, int cap, float scale, int keep, long long out_ts, float out_scale) {
  pdl_enter();
  extern __shared__ float sm_wa[];            // q [DK] | acc [4][DV]
  __shared__ float s_m[4], s_l[4];
  const int i = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int DK = DA + DB;
  float* sq = sm_wa;
  float* sacc = sm_wa + ((DK + 3) & ~3);
  const int slot = meta[i], pos = meta[ntok + i];
  const int g = h / (H / G);
  for (int c = tid; c < DA; c += 128) sq[c] = qa[(size_t)i * qa_ts + (size_t)h * qa_hs + c];
  for (int c = tid; c < DB; c += 128) sq[DA + c] = qb[(size_t)i * qb_ts + (size_t)h * qb_hs + c];
  __syncthreads();
  const T* kbase = kc + (size_t)slot * k_ss + (size_t)g * k_hs;
  const T* vbase = vc + (size_t)slot * v_ss + (size_t)g * v_hs;
  // visible keys in order: the first nk positions (kept ones that the window has left behind), then the window from j0 on
  const int j0 = max(0, pos - window + 1), nk = min(keep, j0), nkeys = nk + pos - j0 + 1;
  float m = -INFINITY, l = 0.f;
  float acc[NACC];
#pragma unroll
  for (int a = 0; a < NACC; ++a) acc[a] = 0.f;
  // a warp takes runs of KU consecutive keys (every fourth run): KU independent rows in flight per iteration
  constexpr int KU = 4;
  for (int j = warp * KU; j < nkeys; j += 4 * KU) {
    const int n = min(KU, nkeys - j);
    const T* kr[KU];
    const T* vr[KU];
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      const int ju = j + (u < n ? u : 0), r = ring_row(ju < nk ? ju : j0 + ju - nk, keep, cap);
      kr[u] = kbase + (size_t)r * k_rs;
      vr[u] = vbase + (size_t)r * v_rs;
    }
    float dot[KU];
#pragma unroll
    for (int u = 0; u < KU; ++u) dot[u] = 0.f;
    for (int c = lane * VEC; c < DK; c += 32 * VEC) {
      const float q0 = sq[c], q1 = VEC == 2 ? sq[c + 1] : 0.f;
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        float kv[2];
        ld_pair<VEC>(kr[u] + c, kv);
        dot[u] += q0 * kv[0];
        if (VEC == 2) dot[u] += q1 * kv[1];
      }
    }
    float mn = m;
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      dot[u] = u < n ? warp_xor_sum(dot[u]) * scale : -INFINITY;
      mn = fmaxf(mn, dot[u]);
    }
    const float corr = expf(m - mn);
    float p[KU], ps = 0.f;
#pragma unroll
    for (int u = 0; u < KU; ++u) { p[u] = expf(dot[u] - mn); ps += p[u]; }
    m = mn;
    l = l * corr + ps;
#pragma unroll
    for (int a = 0; a < NACC; a += VEC) {
      const int c = lane * VEC + 32 * a;
      float s0 = 0.f, s1 = 0.f;
      if (c < DV) {
#pragma unroll
        for (int u = 0; u < KU; ++u) {
          float vv[2];
          ld_pair<VEC>(vr[u] + c, vv);
          s0 += p[u] * vv[0];
          s1 += p[u] * vv[1];
        }
      }
      acc[a] = acc[a] * corr + s0;
      if (VEC == 2) acc[a + 1] = acc[a + 1] * corr + s1;
    }
  }
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
#pragma unroll
  for (int a = 0; a < NACC; a += VEC) {
    const int c = lane * VEC + 32 * a;
    if (c < DV) {
      sacc[warp * DV + c] = acc[a];
      if (VEC == 2) sacc[warp * DV + c + 1] = acc[a + 1];
    }
  }
  __syncthreads();
  float M = sink ? sink[h] : -INFINITY;
#pragma unroll
  for (int w = 0; w < 4; ++w) M = fmaxf(M, s_m[w]);
  float f[4], L = sink ? expf(sink[h] - M) : 0.f;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    f[w] = expf(s_m[w] - M);               // a warp without keys has m = -inf: factor 0
    L += s_l[w] * f[w];
  }
  const float inv = 1.0f / L;
  for (int c = tid; c < DV; c += 128) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) o += sacc[w * DV + c] * f[w];
    o *= inv * out_scale;
    if (gate) o *= 1.0f / (1.0f + expf(-to_f(gate[(size_t)i * gate_ld + (gate_per_head ? (size_t)h : (size_t)h * DV + c)])));
    out[(size_t)i * out_ts + (size_t)h * DV + c] = from_f<T>(o);
  }
}

// ---- HGRN2 gates: q = silu(zq), f = lower + (1 - lower) sigmoid(zf + b), and 1 - f, float32, once per (token, row) -------
// gates [ntok][3][H * D]. 1 - f = (1 - lower) / (1 + e^z) is formed without the cancellation of 1 - f near f = 1.
template <typename T>
__global__ void __launch_bounds__(256)
hgrn2_gates_kernel(const T* __restrict__ p, int ld, const float* __restrict__ f_b, const float* __restrict__ lower,
                   float* __restrict__ gates, int HD, int ntok) {
  pdl_enter();
  // a thread keeps its column (an index divided by HD per element cost as much as the exponentials)
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= HD) return;
  const float b = f_b[c], lo = lower[c];
  for (int t = blockIdx.y; t < ntok; t += gridDim.y) {
    const T* row = p + (size_t)t * ld;
    const float zq = to_f(row[c]), z = to_f(row[HD + c]) + b;
    const float om = 1.0f / (1.0f + expf(z));             // 1 - sigmoid(z)
    float* g = gates + (size_t)t * 3 * HD + c;
    g[0] = zq / (1.0f + expf(-zq));
    g[HD] = lo + (1.0f - lo) * (1.0f - om);
    g[2 * HD] = (1.0f - lo) * om;
  }
}


// ---- scalar-decay linear attention: q = silu(zq), k = silu(zk), float32, once per (token, row); gates [ntok][2][H * D]. vs (or NULL)
// [ntok][H * DV]: silu(zv), for the chunk form, whose passes would compute it once each (64 heads of 64 x 64, 9 x 600
// tokens: 1101 -> 748 us) ----
template <typename T>
__global__ void __launch_bounds__(256)
lightning_gates_kernel(const T* __restrict__ p, int ld, float* __restrict__ gates, int HD, int ntok, float* __restrict__ vs, int HDV) {
  pdl_enter();
  const int c = blockIdx.x * 256 + threadIdx.x;
  const bool qk = c < HD, v = vs && c < HDV;
  for (int t = blockIdx.y; t < ntok; t += gridDim.y) {
    const T* row = p + (size_t)t * ld;
    if (qk) {
      const float zq = to_f(row[c]), zk = to_f(row[HD + c]);
      float* g = gates + (size_t)t * 2 * HD + c;
      g[0] = zq / (1.0f + expf(-zq));
      g[HD] = zk / (1.0f + expf(-zk));
    }
    if (v) {
      const float zv = to_f(row[2 * HD + c]);
      vs[(size_t)t * HDV + c] = zv / (1.0f + expf(-zv));
    }
  }
}

// Unit-RMS norm over a whole row of float32 values with a weight and a sigmoid gate: out = src / rms(src) * w * sigmoid(gate).
// One CTA per row (all heads of a token are normed together).
template <typename T>
__global__ void __launch_bounds__(256)
gated_row_norm_kernel(const float* __restrict__ src, const float* __restrict__ w, const T* __restrict__ gate, int gate_ld,
                      T* __restrict__ out, int N, float eps) {
  pdl_enter();
  __shared__ float red[8];
  const int i = blockIdx.x, tid = threadIdx.x;
  const float* s = src + (size_t)i * N;
  float ss = 0.f;
  for (int c = tid; c < N; c += 256) ss += s[c] * s[c];
  const float rr = 1.0f / sqrtf(block_sum_256(ss, red) / (float)N + eps);
  for (int c = tid; c < N; c += 256) {
    const float z = to_f(gate[(size_t)i * gate_ld + c]);
    out[(size_t)i * N + c] = from_f<T>(s[c] * rr * w[c] * (1.0f / (1.0f + expf(-z))));
  }
}

// ---- residual sum with a multiplier, and the norm of the next sublayer's input ---------------------------------------
// r = x_in + mult * y_scale * (sum of weighted parts of y + weighted y2); out = r / sqrt(mean(r^2) + eps) * (w_offset + w). One CTA per
// token; the row lives in shared memory between the passes. VEC = 4: every thread takes four neighbouring columns with one
// load per operand (rows and strides on 16-byte boundaries); the parts' weights wait in shared memory.
template <typename T, typename YT, int VEC>
__global__ void __launch_bounds__(256)
residual_norm_kernel(const float* __restrict__ x_in, float* __restrict__ x_out, const YT* __restrict__ y, int y_parts,
                     long long y_part_stride, long long y_tok_stride, const float* __restrict__ y_w, const YT* __restrict__ y2,
                     const float* __restrict__ y2_w, int y2_w_stride, float mult, const float* __restrict__ w, float w_offset,
                     T* __restrict__ out, int W, float eps, const float* __restrict__ y_scale) {
  pdl_enter();
  extern __shared__ __align__(16) float sm_rn[];            // row [W]
  __shared__ float red[8];
  __shared__ float s_yw[64];
  const int i = blockIdx.x, tid = threadIdx.x;
  const YT* yr = y ? y + (size_t)i * y_tok_stride : nullptr;
  const YT* y2r = y2 ? y2 + (size_t)i * W : nullptr;
  const float w2 = (y2 && y2_w) ? y2_w[(size_t)i * y2_w_stride] : 1.0f;
  const bool weights_in_smem = y_parts <= 64;
  if (yr && weights_in_smem) {
    if (tid < y_parts) s_yw[tid] = y_w ? y_w[(size_t)i * y_parts + tid] : 1.0f;
    __syncthreads();
  }
  const float* xr = x_in + (size_t)i * W;
  float q = 0.f;
  for (int c = tid * VEC; c < W; c += 256 * VEC) {
    VecF<VEC> v;
#pragma unroll
    for (int e = 0; e < VEC; ++e) v.v[e] = 0.f;
    if (yr) {
#pragma unroll 4
      for (int p = 0; p < y_parts; ++p) {
        const float wp = weights_in_smem ? s_yw[p] : (y_w ? y_w[(size_t)i * y_parts + p] : 1.0f);
        const VecF<VEC> t = ldv<VEC>(yr + (size_t)p * y_part_stride + c);
#pragma unroll
        for (int e = 0; e < VEC; ++e) v.v[e] += wp * t.v[e];
      }
    }
    if (y2r) {
      const VecF<VEC> t = ldv<VEC>(y2r + c);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v.v[e] += w2 * t.v[e];
    }
    if (y_scale) {                                          // one factor per column (a layer scale)
      const VecF<VEC> sc = ldv<VEC>(y_scale + c);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v.v[e] *= sc.v[e];
    }
    VecF<VEC> r = ldv<VEC>(xr + c);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      r.v[e] += mult * v.v[e];
      q += r.v[e] * r.v[e];
    }
    if (x_out) stv<VEC>(x_out + (size_t)i * W + c, r);
    stv<VEC>(sm_rn + c, r);
  }
  if (!out) return;
  const float rr = 1.0f / sqrtf(block_sum_256(q, red) / (float)W + eps);
  for (int c = tid * VEC; c < W; c += 256 * VEC) {
    VecF<VEC> r = ldv<VEC>(sm_rn + c);
    const VecF<VEC> wv = ldv<VEC>(w + c);
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = r.v[e] * rr * (w_offset + wv.v[e]);
    stv<VEC>(out + (size_t)i * W + c, r);
  }
}

// ---- element-wise activations -------------------------------------------------------------------------------------------
__device__ __forceinline__ float act_apply(float z, int act) {
  if (act == QSPEC_ACT_GELU_ERF) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
  const float v = fmaxf(z, 0.f);
  return v * v;
}
template <typename T, int VEC>
__global__ void __launch_bounds__(256) act_kernel(T* __restrict__ a, long long n, int act) {
  pdl_enter();
  for (long long k = ((long long)blockIdx.x * 256 + threadIdx.x) * VEC; k < n; k += (long long)gridDim.x * 256 * VEC) {
    VecF<VEC> v = ldv<VEC>(a + k);
#pragma unroll
    for (int e = 0; e < VEC; ++e) v.v[e] = act_apply(v.v[e], act);
    stv<VEC>(a + k, v);
  }
}

template <typename T, int VEC>
__global__ void __launch_bounds__(256) glu_kernel(const T* __restrict__ gu, int ld, T* __restrict__ out, int F, long long n, int act) {
  pdl_enter();
  for (long long k = ((long long)blockIdx.x * 256 + threadIdx.x) * VEC; k < n; k += (long long)gridDim.x * 256 * VEC) {
    const long long t = k / F;
    const int f = (int)(k - t * F);
    const VecF<VEC> g = ldv<VEC>(gu + (size_t)t * ld + f), u = ldv<VEC>(gu + (size_t)t * ld + F + f);
    VecF<VEC> o;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const float z = g.v[e];
      // z sigmoid(z), or the tanh form of gelu: (1 + tanh u) / 2 = sigmoid(2 u)
      const float s = act == QSPEC_GLU_GELU_TANH ? 1.5957691216057308f * (z + 0.044715f * z * z * z) : z;
      o.v[e] = z / (1.0f + expf(-s)) * u.v[e];
    }
    stv<VEC>(out + k, o);
  }
}

// ---- HGRN2: gated linear recurrence ---------------------------------------------------------------------------------
// Per head S <- diag(f) S + (1 - f) v^T, o = S^T q with f = lower + (1 - lower) sigmoid(zf + b) and q = silu(zq).
// One CTA per (segment, head, slice of 16 value columns) walks the segment's tokens in order, 16 (or 8) at a time; thread
// (row group w of 16, column c of 16) keeps rows w * NS .. of column c of the state in registers (float32). For a block of
// tokens the gates, queries (hgrn2_gates_kernel) and values are copied into shared memory (they were fetched into
// registers while the previous block was applied), then every thread applies the block's tokens to its rows, and the
// sixteen row groups' partial outputs are added per (token, column). The state is loaded from the slot at the start
// (zero at position 0) and stored at the end. o leaves un-normalised, float32.
template <typename T, int NS, int BT>
__global__ void __launch_bounds__(256)
hgrn2_scan_kernel(const T* __restrict__ p, int ld, const float* __restrict__ gates, float* __restrict__ state, float* __restrict__ o,
                  const int* __restrict__ meta, const int* __restrict__ seg_starts, int ntok, int H, int D, int DV,
                  const float* __restrict__ decay) {
  pdl_enter();
  // with a list of the segments' first rows the grid has one CTA per segment; without it, one per token, and the CTAs of
  // tokens that do not open a segment leave at once (a long prompt then pays for thousands of empty CTAs)
  const int i = seg_starts ? seg_starts[blockIdx.x] : blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 16;
  const TokMeta mt = load_meta(meta, ntok, i);
  if (i != mt.seg_begin) return;
  constexpr int DP = 16 * NS, R = (BT * DP) / 256;           // BT tokens per block; padded rows; staged values per thread
  __shared__ __align__(16) float sq[BT][DP], sf[BT][DP], sg[BT][DP];
  __shared__ float sv[BT][16], spart[BT][16][16];
  const int tid = threadIdx.x, c = tid & 15, grp = tid >> 4;
  const int col = v0 + c;
  const bool live = col < DV;
  const int d0 = grp * NS;
  float S[NS];
  float* st = state + (((size_t)mt.slot * H + h) * D) * DV;
#pragma unroll
  for (int k = 0; k < NS; ++k) S[k] = (mt.pos > 0 && live && d0 + k < D) ? st[(size_t)(d0 + k) * DV + col] : 0.f;
  const int HD = H * D;
  const float dec = decay ? decay[h] : 1.f;
  float rq[R], rf[R], rg[R], zv = 0.f;
  auto fetch = [&](int tb) {                               // gates and values of the block's tokens into registers
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = tid + 256 * r, tt = e / DP, d = e % DP, t = tb + tt;
      rq[r] = 0.f; rf[r] = 1.f; rg[r] = 0.f;
      if (t < mt.seg_end && d < D) {
        if (decay) {                                          // one decay per head: gates hold [q | k] only
          const float* g = gates + (size_t)t * 2 * HD + h * D + d;
          rq[r] = g[0]; rf[r] = dec; rg[r] = g[HD];
        } else {
          const float* g = gates + (size_t)t * 3 * HD + h * D + d;
          rq[r] = g[0]; rf[r] = g[HD]; rg[r] = g[2 * HD];
        }
      }
    }
    if (tid < BT * 16) {
      const int t = tb + grp;
      zv = (t < mt.seg_end && live) ? to_f(p[(size_t)t * ld + 2 * HD + h * DV + col]) : 0.f;
      if (decay) zv = zv / (1.0f + expf(-zv));               // the scalar-decay form takes silu(v)
    }
  };
  fetch(mt.seg_begin);
  for (int tb = mt.seg_begin; tb < mt.seg_end; tb += BT) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = tid + 256 * r, tt = e / DP, d = e % DP;
      sq[tt][d] = rq[r]; sf[tt][d] = rf[r]; sg[tt][d] = rg[r];
    }
    if (tid < BT * 16) sv[grp][c] = zv;
    __syncthreads();
    if (tb + BT < mt.seg_end) fetch(tb + BT);
    const int nb = min(BT, mt.seg_end - tb);
    for (int tt = 0; tt < nb; ++tt) {
      const float v = sv[tt][c];
      float p0 = 0.f, p1 = 0.f;                             // two chains: the sum over rows is the long dependency
      const float4* f4 = reinterpret_cast<const float4*>(&sf[tt][d0]);
      const float4* g4 = reinterpret_cast<const float4*>(&sg[tt][d0]);
      const float4* q4 = reinterpret_cast<const float4*>(&sq[tt][d0]);
#pragma unroll
      for (int k = 0; k < NS / 4; ++k) {
        const float4 f = f4[k], gq = g4[k], q = q4[k];
        S[4 * k] = f.x * S[4 * k] + gq.x * v;             p0 += S[4 * k] * q.x;
        S[4 * k + 1] = f.y * S[4 * k + 1] + gq.y * v;     p1 += S[4 * k + 1] * q.y;
        S[4 * k + 2] = f.z * S[4 * k + 2] + gq.z * v;     p0 += S[4 * k + 2] * q.z;
        S[4 * k + 3] = f.w * S[4 * k + 3] + gq.w * v;     p1 += S[4 * k + 3] * q.w;
      }
      spart[tt][grp][c] = p0 + p1;
    }
    __syncthreads();
    if (tid < BT * 16 && grp < nb && live) {                // thread (token grp, column c) adds the sixteen row groups
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 16; ++w) s += spart[grp][w][c];
      o[(size_t)(tb + grp) * H * DV + (size_t)h * DV + col] = s;
    }
  }
  if (live) {
#pragma unroll
    for (int k = 0; k < NS; ++k)
      if (d0 + k < D) st[(size_t)(d0 + k) * DV + col] = S[k];
  }
}

// ---- the same recurrences over long segments, in chunks that run side by side ---------------------------------------------------------
// The walk above is a chain: 0.2 us a token whatever the GPU has left. A chunk of C tokens turns the state it starts from into
// diag(P) S + E (P: product of its decays, E: what its own tokens add), so (1) recurrence_chunk_kernel<.., false> computes E and P of
// every chunk, (2) recurrence_carry_kernel goes through the chunks of a segment element by element and leaves the state that each starts
// from, and (3) recurrence_chunk_kernel<.., true> walks every chunk from its state and writes the outputs, normed per head on the way
// out where the design norms per head. All float32, as in the walk; what changes is the order of products of decays.
// A CTA holds the whole D x DV state of a (chunk, head) in registers, 16 rows x 4 columns a thread, as pairs of rows: 3 (outputs) or, with
// a block's decays multiplied into its keys first, 1 (E) packed multiply-adds per pair and token. Blocks of 8 tokens arrive by cp.async,
// two in flight; the row groups' shares of the outputs meet in shared memory once per block. What bounds it is shared
// memory: a thread reads 56 floats for 64 elements of state, 90 wavefronts a token and warp in the output pass (73 % of the pipe), above
// the 384 cycles a token and head that its multiply-adds need.
// 1500 tokens, 16 heads of 128 x 128, all launches: 325 -> 144 us (each by itself, overlaps not taken off: gates 13, E 44, carry 9, outputs
// 89); 2000 tokens, 8 heads of 64 x 64: 473 -> 61 us.
constexpr int RC_BT = 8;                                     // tokens per block

__device__ __forceinline__ uint64_t rc_fma(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t rc_mul(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t rc_pair(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float2 rc_unpair(uint64_t v) { float2 r; asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }

struct RcChunk { int begin, end, first, chunks; TokMeta mt; };   // the segment's first and end row, its first chunk's number, its chunks
// The segment that chunk b belongs to (or segment `seg` if b < 0), found by the CTA's first warp. false: there is no such chunk.
__device__ __forceinline__ bool rc_find(const int* __restrict__ meta, const int* __restrict__ seg_starts, int nseg, int ntok, int C, int b, int seg,
                                        RcChunk* s_chunk, bool* s_found) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int before = 0;
    bool found = false;
    for (int s0 = 0; s0 < nseg && !found; s0 += 32) {
      const int s = s0 + lane;
      int start = 0, end = 0;
      if (s < nseg) { start = seg_starts[s]; end = meta[3 * ntok + start]; }
      const int n = (end - start + C - 1) / C;
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      const int first = before + incl - n;
      const bool me = s < nseg && (b < 0 ? s == seg : b >= first && b < first + n);
      if (me) {
        s_chunk->begin = start; s_chunk->end = end; s_chunk->first = first; s_chunk->chunks = n;
        s_chunk->mt = load_meta(meta, ntok, start);
      }
      found = __any_sync(0xffffffffu, me);
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) *s_found = found;
  }
  __syncthreads();
  return *s_found;
}

template <typename T, int D, int DV, bool OUT>
__global__ void __launch_bounds__((D / 16) * (DV / 4), 32768 / (D * DV))
recurrence_chunk_kernel(const T* __restrict__ p, int ld, const float* __restrict__ gates, float* __restrict__ E, float* __restrict__ P,
                        float* __restrict__ state, float* __restrict__ o, T* __restrict__ out, const float* __restrict__ norm_w, float eps,
                        const int* __restrict__ meta, const int* __restrict__ seg_starts, int nseg, int ntok, int H, int C,
                        const float* __restrict__ decay) {
  pdl_enter();
  constexpr int RG = D / 16, CG = DV / 4, NT = RG * CG, BT = RC_BT, VPT = BT * DV / NT;
  extern __shared__ __align__(16) float rc_smem[];
  float (*sf)[BT][D] = reinterpret_cast<float (*)[BT][D]>(rc_smem);                       // [2] decays
  float (*sg)[BT][D] = sf + 2;                                                            // [2] what multiplies v
  float (*sv)[BT][2 * DV] = reinterpret_cast<float (*)[BT][2 * DV]>(sg + 2);              // [2] values, each twice
  float (*sq)[BT][D] = reinterpret_cast<float (*)[BT][D]>(sv + 2);                        // [2] queries (outputs only)
  float (*sp)[RG][DV] = reinterpret_cast<float (*)[RG][DV]>(sq + 2);                      // [BT] shares of the outputs
  __shared__ float sF[D];
  __shared__ RcChunk s_chunk;
  __shared__ bool s_found;
  const int b = blockIdx.x, h = blockIdx.y;
  if (!rc_find(meta, seg_starts, nseg, ntok, C, b, 0, &s_chunk, &s_found)) return;
  const int c = b - s_chunk.first;
  if (!OUT && c == s_chunk.chunks - 1) return;               // nobody starts from where the last chunk ends
  const int t0 = s_chunk.begin + c * C, t1 = min(t0 + C, s_chunk.end);
  const int tid = threadIdx.x, rg = tid % RG, cg = tid / RG, HD = H * D;
  const float dec = decay ? decay[h] : 1.f;
  const int arrays = decay ? 2 : 3;                           // per token: q | (f) | what multiplies v
  const float* gq = gates + (size_t)h * D;
  const T* vp = p + 2 * (size_t)HD + (size_t)h * DV;
  auto stage = [&](int buf, int tb) {
#pragma unroll
    for (int a = OUT ? 0 : 1; a < 3; ++a) {
      if (a == 1 && decay) continue;
      float* dst = a == 0 ? &sq[buf][0][0] : a == 1 ? &sf[buf][0][0] : &sg[buf][0][0];
      const float* src = gq + (size_t)(a == 2 ? arrays - 1 : a) * HD;
      for (int i = tid; i < BT * D / 4; i += NT) {
        const int r = i / (D / 4), k = i % (D / 4) * 4;
        cp_async_16z(dst + r * D + k, src + (size_t)min(tb + r, t1 - 1) * arrays * HD + k, true);
      }
    }
    cp_async_commit();
  };
  float vr[VPT];
  auto fetch_v = [&](int tb) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int e = tid + NT * i, t = min(tb + e / DV, t1 - 1);
      // the scalar-decay form takes silu(v), which waits where the row's outputs will go: every row is read a block before it is written
      vr[i] = decay ? o[((size_t)t * H + h) * DV + e % DV] : to_f(vp[(size_t)t * ld + e % DV]);
    }
  };
  // this thread's rows: 4 rg .. + 3 and the same D / 4, D / 2 and 3 D / 4 further (a load then covers neighbouring 16-byte pieces), as pairs
  auto row_of = [&](int i) { return (i >> 1) * (D / 4) + 4 * rg + 2 * (i & 1); };
  uint64_t S[8][4];
  float* mine = E + ((size_t)b * H + h) * D * DV;             // OUT: the state this chunk starts from
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    if (OUT) {
      x = *reinterpret_cast<const float4*>(mine + (size_t)row_of(i) * DV + cg * 4);
      y = *reinterpret_cast<const float4*>(mine + (size_t)(row_of(i) + 1) * DV + cg * 4);
    }
    S[i][0] = rc_pair(x.x, y.x); S[i][1] = rc_pair(x.y, y.y); S[i][2] = rc_pair(x.z, y.z); S[i][3] = rc_pair(x.w, y.w);
  }
  float whole = 1.f;                                          // !OUT, thread < D: product of the chunk's decays of row tid
  stage(0, t0);
  fetch_v(t0);
  int buf = 0;
  for (int tb = t0; tb < t1; tb += BT, buf ^= 1) {
    const int nb = min(BT, t1 - tb);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int e = tid + NT * i;
      *reinterpret_cast<float2*>(&sv[buf][e / DV][2 * (e % DV)]) = make_float2(vr[i], vr[i]);
    }
    cp_async_wait<0>();
    __syncthreads();
    if (tb + BT < t1) { stage(buf ^ 1, tb + BT); fetch_v(tb + BT); }
    if (!OUT) {
      // keys times the decays that follow them in the block; the block's own decay
      static_assert(D <= NT, "a thread per row");
      if (tid < D) {
        const int d = tid;
        float f = 1.f;
        for (int r = nb - 1; r >= 0; --r) {
          sg[buf][r][d] *= f;
          f *= decay ? dec : sf[buf][r][d];
        }
        sF[d] = f;
      }
      __syncthreads();
      if (tid < D) whole *= sF[tid];
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(&sF[row_of(i)]);
#pragma unroll
        for (int j = 0; j < 4; ++j) { S[i][j] = rc_mul(f.x, S[i][j]); S[i + 1][j] = rc_mul(f.y, S[i + 1][j]); }
      }
    }
    const uint64_t dec2 = rc_pair(dec, dec);
    for (int r = 0; r < nb; ++r) {
      uint64_t v2[4], acc[4];
      {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(&sv[buf][r][8 * cg]), y = *reinterpret_cast<const ulonglong2*>(&sv[buf][r][8 * cg + 4]);
        v2[0] = x.x; v2[1] = x.y; v2[2] = y.x; v2[3] = y.y;
      }
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(&sg[buf][r][row_of(i)]);
        if (OUT) {
          ulonglong2 f = make_ulonglong2(dec2, dec2);
          if (!decay) f = *reinterpret_cast<const ulonglong2*>(&sf[buf][r][row_of(i)]);
          const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&sq[buf][r][row_of(i)]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            S[i][j] = rc_fma(f.x, S[i][j], rc_mul(g.x, v2[j]));
            S[i + 1][j] = rc_fma(f.y, S[i + 1][j], rc_mul(g.y, v2[j]));
            acc[j] = i ? rc_fma(q.x, S[i][j], acc[j]) : rc_mul(q.x, S[i][j]);
            acc[j] = rc_fma(q.y, S[i + 1][j], acc[j]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            S[i][j] = rc_fma(g.x, v2[j], S[i][j]);
            S[i + 1][j] = rc_fma(g.y, v2[j], S[i + 1][j]);
          }
        }
      }
      if (OUT) {
        const float2 a = rc_unpair(acc[0]), x = rc_unpair(acc[1]), y = rc_unpair(acc[2]), z = rc_unpair(acc[3]);
        *reinterpret_cast<float4*>(&sp[r][rg][4 * cg]) = make_float4(a.x + a.y, x.x + x.y, y.x + y.y, z.x + z.y);
      }
    }
    if (OUT) {
      __syncthreads();
      const int lane = tid & 31;
      for (int r = tid >> 5; r < nb; r += NT / 32) {          // a warp per token: the sums, and the per-head norm where there is one
        const size_t at = ((size_t)(tb + r) * H + h) * DV;
        float x[DV / 32], ss = 0.f;
#pragma unroll
        for (int k = 0; k < DV / 32; ++k) {
          x[k] = 0.f;
#pragma unroll
          for (int w = 0; w < RG; ++w) x[k] += sp[r][w][lane + 32 * k];
          ss += x[k] * x[k];
        }
        if (out) {
          const float rr = 1.0f / sqrtf(warp_xor_sum(ss) / (float)DV + eps);
#pragma unroll
          for (int k = 0; k < DV / 32; ++k) out[at + lane + 32 * k] = from_f<T>(x[k] * rr * norm_w[lane + 32 * k]);
        } else {
#pragma unroll
          for (int k = 0; k < DV / 32; ++k) o[at + lane + 32 * k] = x[k];
        }
      }
    }
  }
  if (OUT && t1 != s_chunk.end) return;
  // OUT: the segment's last chunk leaves the state; otherwise E, where the next chunk will look for its state
  float* dst = OUT ? state + ((size_t)s_chunk.mt.slot * H + h) * D * DV : mine + (size_t)H * D * DV;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 a = rc_unpair(S[i][0]), x = rc_unpair(S[i][1]), y = rc_unpair(S[i][2]), z = rc_unpair(S[i][3]);
    *reinterpret_cast<float4*>(dst + (size_t)row_of(i) * DV + cg * 4) = make_float4(a.x, x.x, y.x, z.x);
    *reinterpret_cast<float4*>(dst + (size_t)(row_of(i) + 1) * DV + cg * 4) = make_float4(a.y, x.y, y.y, z.y);
  }
  if (!OUT && tid < D) P[((size_t)b * H + h) * D + tid] = whole;
}

// Through the chunks of a segment, four elements of a head's state per thread: slot c of E holds E of chunk c - 1 and becomes the state
// that chunk c starts from (slot 0: the state before the step, zero at position 0).
__global__ void __launch_bounds__(256)
recurrence_carry_kernel(float* __restrict__ E, const float* __restrict__ P, const float* __restrict__ state, const int* __restrict__ meta,
                        const int* __restrict__ seg_starts, int nseg, int ntok, int H, int D, int DV, int C) {
  pdl_enter();
  __shared__ RcChunk s_chunk;
  __shared__ bool s_found;
  if (!rc_find(meta, seg_starts, nseg, ntok, C, -1, blockIdx.x, &s_chunk, &s_found)) return;
  const int h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * 4;
  if (e >= D * DV) return;
  const size_t step = (size_t)H * D * DV;
  float4* at = reinterpret_cast<float4*>(E + ((size_t)s_chunk.first * H + h) * D * DV + e);
  const float* pr = P + ((size_t)s_chunk.first * H + h) * D + e / DV;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (s_chunk.mt.pos > 0) s = *reinterpret_cast<const float4*>(state + ((size_t)s_chunk.mt.slot * H + h) * D * DV + e);
  at[0] = s;
  constexpr int AHEAD = 8;
  float4 x[AHEAD];
  float f[AHEAD];
  const int n = s_chunk.chunks;
  for (int c = 1; c < n; c += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < n) { x[i] = at[(c + i) * (step / 4)]; f[i] = pr[(size_t)(c + i - 1) * H * D]; }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < n) {
        s.x = f[i] * s.x + x[i].x; s.y = f[i] * s.y + x[i].y; s.z = f[i] * s.z + x[i].z; s.w = f[i] * s.w + x[i].w;
        at[(c + i) * (step / 4)] = s;
      }
  }
}

}  // namespace qspec
#include "recurrence_mma.cuh"
namespace qspec {

// Per-head unit-RMS norm with one weight vector shared by the heads: one warp per (token, head); src float32.
template <typename T>
__global__ void __launch_bounds__(128)
head_norm_kernel(const float* __restrict__ src, const float* __restrict__ w, T* __restrict__ out, long long rows, int DV, float eps) {
  pdl_enter();
  const long long r = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (r >= rows) return;
  const int lane = threadIdx.x & 31;
  const float* s = src + r * DV;
  float ss = 0.f;
  for (int c = lane; c < DV; c += 32) ss += s[c] * s[c];
  const float rr = 1.0f / sqrtf(warp_xor_sum(ss) / (float)DV + eps);
  for (int c = lane; c < DV; c += 32) out[r * DV + c] = from_f<T>(s[c] * rr * w[c]);
}

// ---- per-token side input: g <- gelu_tanh(g) * table[id, layer part] -------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
side_gate_kernel(T* __restrict__ g, const T* __restrict__ table, const int* __restrict__ ids, int col0, int sd, int table_ld, int V,
                 long long n) {
  pdl_enter();
  for (long long k = (long long)blockIdx.x * 256 + threadIdx.x; k < n; k += (long long)gridDim.x * 256) {
    const long long t = k / sd;
    const int c = (int)(k % sd);
    int id = ids[t];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    const float z = to_f(g[k]);
    const float ge = 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    g[k] = from_f<T>(ge * to_f(table[(size_t)id * table_ld + col0 + c]));
  }
}

}  // namespace qspec

using namespace qspec;

#define MIX_DTYPE_OK(dtype) QSPEC_REQUIRE((dtype) == QSPEC_DTYPE_BF16 || (dtype) == QSPEC_DTYPE_F32, QSPEC_ERR_UNSUPPORTED, \
                                          "dtype %d: bfloat16 (1) or float32 (2) expected", (dtype))
typedef __nv_bfloat16 bf16_t;

extern "C" int qspec_seq_token_shift(const float* x, const float* shift, float* prev, int slots, void* out, const int* meta,
                                     int ntok, int W, int dtype, void* stream) {
  QSPEC_REQUIRE(x && shift && prev && out && meta, QSPEC_ERR_INVALID_ARG, "seq_token_shift: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && W > 0 && slots > 0, QSPEC_ERR_INVALID_ARG, "seq_token_shift: bad sizes");
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(token_shift_kernel<float>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, x, shift, prev, slots, (float*)out, meta, ntok, W);
  else
    launch_pdl(token_shift_kernel<bf16_t>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, x, shift, prev, slots, (bf16_t*)out, meta, ntok, W);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T, typename YT>
static int launch_add_norm(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride, long long y_tok_stride,
                           const float* y_w, const float* w, const float* b, int kind, void* out, int ntok, int W, float eps,
                           cudaStream_t st) {
  const size_t smem = (size_t)W * sizeof(float);
  static SmemLimit limit;
  if (smem > 48 * 1024) QSPEC_CUDA(limit.raise(add_norm_kernel<T, YT>, smem));
  launch_pdl(add_norm_kernel<T, YT>, dim3(ntok), dim3(256), smem, st, x_in, x_out, (const YT*)y, y_parts, y_part_stride, y_tok_stride,
             y_w, w, b, kind, (T*)out, W, eps);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_add_norm(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride,
                                  long long y_tok_stride, const float* y_w, const float* w, const float* b, int kind, void* out,
                                  int ntok, int W, float eps, int y_dtype, int dtype, void* stream) {
  QSPEC_REQUIRE(y && w && (x_out || out), QSPEC_ERR_INVALID_ARG, "seq_add_norm: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && W > 0 && W <= 49152 && y_parts >= 1 && (kind == 0 || kind == 1), QSPEC_ERR_INVALID_ARG,
                "seq_add_norm: bad sizes (width <= 49152, kind 0 or 1)");
  MIX_DTYPE_OK(dtype);
  QSPEC_REQUIRE(y_dtype == dtype || y_dtype == QSPEC_DTYPE_F32, QSPEC_ERR_UNSUPPORTED, "seq_add_norm: y is of the activation type or float32");
  if (ntok == 0) return QSPEC_OK;
  cudaStream_t st = (cudaStream_t)stream;
#define AN_ARGS x_in, x_out, y, y_parts, y_part_stride, y_tok_stride, y_w, w, b, kind, out, ntok, W, eps, st
  if (dtype == QSPEC_DTYPE_F32) return launch_add_norm<float, float>(AN_ARGS);
  if (y_dtype == QSPEC_DTYPE_F32) return launch_add_norm<bf16_t, float>(AN_ARGS);
  return launch_add_norm<bf16_t, bf16_t>(AN_ARGS);
#undef AN_ARGS
}

extern "C" int qspec_seq_latent_prep(const void* d, int ld, int q_rank, int kv_rank, int rot_dim, const float* qn_w, const float* kvn_w,
                                     const float* inv_freq, int rot_dims, void* cq, void* cache, int cap, const int* meta, int ntok,
                                     float eps, int dtype, void* stream) {
  QSPEC_REQUIRE(q_rank > 0, QSPEC_ERR_INVALID_ARG, "seq_latent_prep: bad sizes");
  return qspec_seq_latent_prep_pairing(d, ld, q_rank, kv_rank, rot_dim, qn_w, kvn_w, inv_freq, rot_dims, QSPEC_ROTARY_HALVES, cq, cache, cap,
                                       meta, ntok, eps, dtype, stream);
}

extern "C" int qspec_seq_latent_prep_pairing(const void* d, int ld, int q_rank, int kv_rank, int rot_dim, const float* qn_w,
                                             const float* kvn_w, const float* inv_freq, int rot_dims, int pairing, void* cq, void* cache,
                                             int cap, const int* meta, int ntok, float eps, int dtype, void* stream) {
  QSPEC_REQUIRE(d && meta && (q_rank == 0 || (qn_w && cq)), QSPEC_ERR_INVALID_ARG, "seq_latent_prep: null pointer");
  QSPEC_REQUIRE(pairing == QSPEC_ROTARY_HALVES || pairing == QSPEC_ROTARY_INTERLEAVED, QSPEC_ERR_INVALID_ARG, "seq_latent_prep: unknown pairing %d", pairing);
  QSPEC_REQUIRE(!cache || (kvn_w && (inv_freq || rot_dims == 0)), QSPEC_ERR_INVALID_ARG,
                "seq_latent_prep: a cache needs the key/value norm weight and the frequencies");
  QSPEC_REQUIRE(ntok >= 0 && q_rank >= 0 && kv_rank >= 0 && rot_dim >= 0 && rot_dims >= 0 && rot_dims <= rot_dim && rot_dims % 2 == 0 &&
                    cap > 0 && ld >= q_rank + (cache ? kv_rank + rot_dim : 0),
                QSPEC_ERR_INVALID_ARG, "seq_latent_prep: bad sizes");
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(latent_prep_kernel<float>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, (const float*)d, ld, q_rank, kv_rank, rot_dim,
               qn_w, kvn_w, inv_freq, rot_dims, pairing, (float*)cq, (float*)cache, cap, meta, ntok, eps);
  else
    launch_pdl(latent_prep_kernel<bf16_t>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, (const bf16_t*)d, ld, q_rank, kv_rank, rot_dim,
               qn_w, kvn_w, inv_freq, rot_dims, pairing, (bf16_t*)cq, (bf16_t*)cache, cap, meta, ntok, eps);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_rotary(const void* src, long long src_ts, int src_hs, int off, float* dst, long long dst_ts, int dst_hs, int H,
                                int n, int rot_dims, const float* inv_freq, const int* meta, int ntok, int dtype, void* stream) {
  return qspec_seq_rotary_pairing(src, src_ts, src_hs, off, dst, dst_ts, dst_hs, H, n, rot_dims, QSPEC_ROTARY_HALVES, inv_freq, meta, ntok,
                                  dtype, stream);
}

extern "C" int qspec_seq_rotary_pairing(const void* src, long long src_ts, int src_hs, int off, float* dst, long long dst_ts, int dst_hs,
                                        int H, int n, int rot_dims, int pairing, const float* inv_freq, const int* meta, int ntok,
                                        int dtype, void* stream) {
  QSPEC_REQUIRE(pairing == QSPEC_ROTARY_HALVES || pairing == QSPEC_ROTARY_INTERLEAVED, QSPEC_ERR_INVALID_ARG, "seq_rotary: unknown pairing %d", pairing);
  QSPEC_REQUIRE(src && dst && meta && (rot_dims == 0 || inv_freq), QSPEC_ERR_INVALID_ARG, "seq_rotary: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && H > 0 && n >= 0 && rot_dims >= 0 && rot_dims <= n && rot_dims % 2 == 0, QSPEC_ERR_INVALID_ARG,
                "seq_rotary: bad sizes");
  MIX_DTYPE_OK(dtype);
  if (ntok == 0 || n == 0) return QSPEC_OK;
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(rotary_kernel<float>, dim3(ntok), dim3(128), 0, (cudaStream_t)stream, (const float*)src, src_ts, src_hs, off, dst, dst_ts,
               dst_hs, H, n, rot_dims, pairing, inv_freq, meta, ntok);
  else
    launch_pdl(rotary_kernel<bf16_t>, dim3(ntok), dim3(128), 0, (cudaStream_t)stream, (const bf16_t*)src, src_ts, src_hs, off, dst, dst_ts,
               dst_hs, H, n, rot_dims, pairing, inv_freq, meta, ntok);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_qkv_prep(const void* p, int ld, int HD, int GD, int GDV, const float* qn_w, const float* kn_w, float* qout,
                                  void* cache_k, void* cache_v, int cap, const int* meta, int ntok, float eps, int dtype, void* stream) {
  QSPEC_REQUIRE(p && qn_w && kn_w && qout && cache_k && cache_v && meta, QSPEC_ERR_INVALID_ARG, "seq_qkv_prep: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && HD > 0 && GD > 0 && GDV > 0 && cap > 0 && ld >= HD + GD + GDV, QSPEC_ERR_INVALID_ARG, "seq_qkv_prep: bad sizes");
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(qkv_prep_kernel<float>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, (const float*)p, ld, HD, GD, GDV, qn_w, kn_w, qout,
               (float*)cache_k, (float*)cache_v, cap, meta, ntok, eps);
  else
    launch_pdl(qkv_prep_kernel<bf16_t>, dim3(ntok), dim3(256), 0, (cudaStream_t)stream, (const bf16_t*)p, ld, HD, GD, GDV, qn_w, kn_w, qout,
               (bf16_t*)cache_k, (bf16_t*)cache_v, cap, meta, ntok, eps);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T, int NACC, int VEC>
static int launch_window_attn(const qspec_window_attn_args* a, cudaStream_t st) {
  const int DK = a->DA + a->DB;
  const size_t smem = ((size_t)((DK + 3) & ~3) + (size_t)4 * a->DV) * sizeof(float);
  static SmemLimit limit;
  if (smem > 48 * 1024) QSPEC_CUDA(limit.raise(window_attn_kernel<T, NACC, VEC>, smem));
  launch_pdl(window_attn_kernel<T, NACC, VEC>, dim3(a->ntok, a->H), dim3(128), smem, st, a->qa, a->qa_tok_stride, a->qa_head_stride, a->DA,
             a->qb, a->qb_tok_stride, a->qb_head_stride, a->DB, (const T*)a->k, a->k_slot_stride, a->k_row_stride, a->k_head_stride,
             (const T*)a->v, a->v_slot_stride, a->v_row_stride, a->v_head_stride, a->DV, a->sink, (const T*)a->gate, a->gate_ld, a->gate_per_head, (T*)a->out,
             a->meta, a->ntok, a->H, a->G, a->window, a->cap, a->scale, a->keep_first,
             a->out_tok_stride ? a->out_tok_stride : (long long)a->H * a->DV, a->out_scale);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T, int VEC>
static int launch_window_attn_n(const qspec_window_attn_args* a, cudaStream_t st) {
  const int per = (a->DV + 31) / 32;
  if (per <= 2) return launch_window_attn<T, 2, VEC>(a, st);
  if (per <= 4) return launch_window_attn<T, 4, VEC>(a, st);
  if (per <= 8) return launch_window_attn<T, 8, VEC>(a, st);
  if (per <= 16) return launch_window_attn<T, 16, VEC>(a, st);
  return launch_window_attn<T, 32, VEC>(a, st);
}

extern "C" int qspec_seq_window_attention(const qspec_window_attn_args* a, int dtype, void* stream) {
  QSPEC_REQUIRE(a && a->qa && a->k && a->v && a->out && a->meta && (a->DB == 0 || a->qb), QSPEC_ERR_INVALID_ARG,
                "seq_window_attention: null pointer");
  QSPEC_REQUIRE(a->ntok >= 0 && a->H > 0 && a->G > 0 && a->H % a->G == 0 && a->DA > 0 && a->DB >= 0 && a->DV > 0 && a->DV <= 1024 &&
                    a->DA + a->DB <= 8192 && a->window >= 1 && a->cap >= 1 && a->H <= 65535 && a->keep_first >= 0 && a->keep_first < a->cap,
                QSPEC_ERR_UNSUPPORTED, "seq_window_attention: heads %d / %d, key size %d + %d (<= 8192), value size %d (<= 1024)", a->H,
                a->G, a->DA, a->DB, a->DV);
  MIX_DTYPE_OK(dtype);
  if (a->ntok == 0) return QSPEC_OK;
  const size_t esz = dtype == QSPEC_DTYPE_F32 ? 4 : 2;
  const bool even = ((a->DA + a->DB) % 2 == 0) && (a->DV % 2 == 0) && (a->k_row_stride % 2 == 0) && (a->k_head_stride % 2 == 0) &&
                    (a->k_slot_stride % 2 == 0) && (a->v_row_stride % 2 == 0) && (a->v_head_stride % 2 == 0) && (a->v_slot_stride % 2 == 0) &&
                    ((uintptr_t)a->k % (2 * esz) == 0) && ((uintptr_t)a->v % (2 * esz) == 0);
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == QSPEC_DTYPE_F32) return even ? launch_window_attn_n<float, 2>(a, st) : launch_window_attn_n<float, 1>(a, st);
  return even ? launch_window_attn_n<bf16_t, 2>(a, st) : launch_window_attn_n<bf16_t, 1>(a, st);
}

// Tokens of a chunk: as many as let the chunks of all heads fill the GPU once, whole blocks, and at least 32 (below that the states on their
// way through memory cost more than the walk).
static int rc_chunk_tokens(int ntok, int H, int D, int DV) {
  const long long slots = (long long)sm_count() * (32768 / (D * DV));
  const long long c = (((long long)ntok * H + slots - 1) / slots + RC_BT - 1) / RC_BT * RC_BT;
  return (int)(c < 32 ? 32 : c);
}
static bool rc_taken(int nseg, int ntok, int H, int D, int DV, bool scalar_decay) {
  if (!((D == 64 || D == 128) && (DV == 64 || DV == 128)) || nseg < 1 || sm_count() < 1) return false;
  // The walk takes 0.2 us a token while its CTAs (a segment, a head, 16 columns each) fit the GPU side by side; the chunks take four launches,
  // 35 to 60 us, and from there what their multiply-adds need. Where the two meet (us, walk : chunks; 300 tokens and less to a segment):
  // 128 x 128, 256 tokens: 8 heads 58 : 62, 32 heads 63 : 68; 300 tokens: 16 heads 69 : 61, 32 heads 72 : 75; 600 tokens: 32 heads 138 : 120.
  // 64 x 64, 256 tokens: 8 heads 57 : 35, 64 heads 75 : 57.
  // The walk of a scalar decay is the cheaper one once its CTAs come in several rounds: 64 x 64, 8 segments of 300, 32 heads 167 : 178, 9 of
  // 600, 64 heads 706 : 748, against 2 of 600, 64 heads 192 : 173, 4 of 1500, 64 heads 791 : 771.
  const long long walkers = (long long)nseg * H * (DV / 16);
  int least = D * DV < 128 * 128 || walkers <= 32 ? 256 : walkers <= 128 ? 288 : 336;
  if (scalar_decay && D * DV < 128 * 128 && walkers > 512) least = walkers > 1024 ? 0x7fffffff : 1000;
  return ntok >= least * (long long)nseg && ntok >= 2 * (long long)nseg * rc_chunk_tokens(ntok, H, D, DV);
}

template <typename T, int D, int DV>
static int launch_recurrence_chunks_d(const T* p, int ld, const float* gates, float* state, float* o, T* out, const float* norm_w, float eps, const int* meta,
                                      const int* seg_starts, int nseg, int ntok, int H, const float* decay, float* ws, cudaStream_t st) {
  const int C = rc_chunk_tokens(ntok, H, D, DV), chunks = ntok / C + nseg;
  float* E = ws;
  float* P = ws + (size_t)chunks * H * D * DV;
  const dim3 grid(chunks, H), block((D / 16) * (DV / 4));
  constexpr size_t smem_e = (size_t)RC_BT * (4 * D + 4 * DV) * sizeof(float), smem_o = smem_e + (size_t)RC_BT * (2 * D + (D / 16) * DV) * sizeof(float);
  static SmemLimit limit;
  QSPEC_CUDA(limit.raise(recurrence_chunk_kernel<T, D, DV, true>, smem_o));
  launch_pdl(recurrence_chunk_kernel<T, D, DV, false>, grid, block, smem_e, st, p, ld, gates, E, P, state, o, out, norm_w, eps, meta, seg_starts, nseg, ntok, H, C, decay);
  QSPEC_CHECK_LAUNCH(1);
  launch_pdl(recurrence_carry_kernel, dim3(nseg, H, (D * DV + 1023) / 1024), dim3(256), 0, st, E, (const float*)P, (const float*)state, meta, seg_starts, nseg,
             ntok, H, D, DV, C);
  QSPEC_CHECK_LAUNCH(1);
  launch_pdl(recurrence_chunk_kernel<T, D, DV, true>, grid, block, smem_o, st, p, ld, gates, E, P, state, o, out, norm_w, eps, meta, seg_starts, nseg, ntok, H, C, decay);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

// o: un-normalised float32 outputs, or out (with norm_w): normed per head
template <typename T>
static int launch_recurrence_chunks(const void* p, int ld, const float* gates, float* state, float* o, void* out, const float* norm_w, float eps,
                                    const int* meta, const int* seg_starts, int nseg, int ntok, int H, int D, int DV, const float* decay, void* ws,
                                    cudaStream_t st) {
#define RC_ARGS (const T*)p, ld, gates, state, o, (T*)out, norm_w, eps, meta, seg_starts, nseg, ntok, H, decay, (float*)ws, st
  if (D == 128) return DV == 128 ? launch_recurrence_chunks_d<T, 128, 128>(RC_ARGS) : launch_recurrence_chunks_d<T, 128, 64>(RC_ARGS);
  return DV == 128 ? launch_recurrence_chunks_d<T, 64, 128>(RC_ARGS) : launch_recurrence_chunks_d<T, 64, 64>(RC_ARGS);
#undef RC_ARGS
}

// ---- the gated recurrence of bfloat16 rows on the tensor cores (recurrence_mma.cuh) ----
// Tokens of a chunk: as many as let the chunks of all heads fill the GPU once, at least two blocks. 0: these sizes are not taken.
// Three launches and the first blocks take what the walk (launch_hgrn2 without a workspace) takes for 130 tokens, so it keeps short segments. Estimates,
// us: here 32.5 and 2.6 for 1000 tokens of a head (states smaller than 128 x 128: 25.5 and their share of 2.5); the walk 8 and 0.18 (0.13) a token of a
// segment, more where its CTAs (a segment, a head, 16 columns each) fill the GPU several times over. Measured, walk | here, 128 x 128, segments x tokens x
// heads: 1 x 100 x 16 27 | 33, 1 x 200 x 16 45 | 36, 1 x 300 x 16 60 | 39, 5 x 100 x 16 62 | 51, 5 x 300 x 16 175 | 104, 64 x 32 x 32 464 | 249; 64 x 64,
// 1 x 300 x 16 46 | 28, 2 x 33 x 8 15 | 20; decoding tokens beside a prompt portion, 64 x 1 + 2000, 32 heads 783 | 480, 32 x 1 + 1000, 16 heads 248 | 130.
// The estimate counts tokens, the kernel whole blocks of 16, and every segment's state goes through a CTA: many short segments are the walk's. Where they
// would have been taken: 64 x 4 x 32 108 | 275, 256 x 1 x 16 180 | 262, 64 x 16 x 16 143 | 153, 64 x 1 + 256, 32 heads 180 | 260; from 24 tokens a segment
// on 3200 measured sizes, even and ragged, are within 5 % of the walk at the worst, but one (1 + 1 + 98 tokens, 64 heads, 62 | 68), and twice as fast in the
// mean. (Key size 128 with 64 columns: from
// 200 tokens on, 24 x 100 x 16 154 | 164, and up to 20000 token-heads, above which the form of float32 rows is the faster one: 1 x 1000 x 16 70 | 68,
// 1 x 2000 x 16 109 | 121, 1 x 1000 x 32 106 | 117.)
// A chunk a little shorter than the segments would make two of each. Where these fill the GPU twice, segments of up to 64 tokens stay whole (128 x 128,
// 12 x 33 x 16: 65 -> 47, the walk 56); where they do not, small states gain nothing from so short segments (64 x 64, 9 x 64 x 16 25 | 28).
static int rm_chunk_tokens(int nseg, int ntok, int H, int D, int DV) {
  if (!((D == 64 || D == 128) && (DV == 64 || DV == 128)) || nseg < 1 || sm_count() < 1) return 0;
  const bool large = D * DV == 128 * 128;
  if (ntok < (D > DV ? 200 : 24) * (long long)nseg || (D > DV && (long long)ntok * H > 20000)) return 0;
  const double share = D * DV / 16384.0, walkers = (double)nseg * H * (DV / 16) / 210;
  const double walk = 8 + (large ? 0.18 : 0.13) * ((double)ntok / nseg) * (walkers > 1 ? walkers : 1);
  if ((large ? 32.5 : 25.5) + (large ? 0.0026 : 0.0025) * ntok * H * share > walk) return 0;
  const long long slots = (long long)sm_count() * (DV == 128 ? 2 : 4), each = (ntok + (long long)nseg - 1) / nseg;
  long long c = (((long long)ntok * H + slots - 1) / slots + rmma::BT - 1) / rmma::BT * rmma::BT;
  if (c < 2 * rmma::BT) c = 2 * rmma::BT;
  if (c < each && each <= 64) {
    if (2LL * nseg * H > slots) c = (each + rmma::BT - 1) / rmma::BT * rmma::BT;
    else if (!large && each <= 56) return 0;
  }
  return (int)c;
}
// Whether a segment may be longer than a chunk, so that states between chunks are needed (every segment has a token).
static bool rm_splits(int nseg, int ntok, int C) { return ntok - nseg + 1 > C; }
// 16 bytes: taken, and nothing is kept between chunks.
static size_t rm_bytes(int nseg, int ntok, int H, int D, int DV) {
  const int C = ntok < 1 || H < 1 || D < 1 || DV < 1 ? 0 : rm_chunk_tokens(nseg, ntok, H, D, DV);
  return !C ? 0 : rm_splits(nseg, ntok, C) ? (size_t)(ntok / C + nseg) * H * ((size_t)D * DV + D) * sizeof(float) : 16;
}
template <int D, int DV>
static int launch_rm_d(rmma::Args a, cudaStream_t st) {
  const int chunks = a.ntok / a.C + a.nseg;
  using Sh = rmma::Shape<D, DV>;
  constexpr size_t smem_e = rmma::smem_bytes<D, DV, false>(), smem_o = rmma::smem_bytes<D, DV, true>();
  static SmemLimit limit_e, limit_o;
  QSPEC_CUDA(limit_e.raise(rmma::chunk_kernel<D, DV, false>, smem_e));
  QSPEC_CUDA(limit_o.raise(rmma::chunk_kernel<D, DV, true>, smem_o));
  a.P = a.E + (size_t)chunks * a.H * D * DV;
  if (rm_splits(a.nseg, a.ntok, a.C)) {
    launch_pdl(rmma::chunk_kernel<D, DV, false>, dim3(chunks, a.H), dim3(Sh::THREADS), smem_e, st, a);
    QSPEC_CHECK_LAUNCH(1);
    launch_pdl(rmma::carry_kernel<D, DV>, dim3(a.nseg, a.H, D * DV / 1024), dim3(256), 0, st, a);
    QSPEC_CHECK_LAUNCH(1);
  }
  launch_pdl(rmma::chunk_kernel<D, DV, true>, dim3(chunks, a.H), dim3(Sh::THREADS), smem_o, st, a);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T>
static int launch_hgrn2(const void* p, int ld, const float* f_b, const float* lower, float* state, float* o, float* gates, const int* meta,
                        const int* seg_starts, int nseg, int ntok, int H, int D, int DV, cudaStream_t st, const float* decay, void* ws, void* out,
                        const float* norm_w, float eps) {
  const unsigned gx = (unsigned)((H * (decay && ws ? max(D, DV) : D) + 255) / 256), gy = (unsigned)max(1, min(ntok, 148 * 16 / (int)gx));
  if (decay) launch_pdl(lightning_gates_kernel<T>, dim3(gx, gy), dim3(256), 0, st, (const T*)p, ld, gates, H * D, ntok, ws ? o : nullptr, H * DV);
  else launch_pdl(hgrn2_gates_kernel<T>, dim3(gx, gy), dim3(256), 0, st, (const T*)p, ld, f_b, lower, gates, H * D, ntok);
  QSPEC_CHECK_LAUNCH(1);
  if (ws) return launch_recurrence_chunks<T>(p, ld, gates, state, o, out, norm_w, eps, meta, seg_starts, nseg, ntok, H, D, DV, decay, ws, st);
  const dim3 grid(seg_starts ? nseg : ntok, H, (DV + 15) / 16);
#define HG_ARGS dim3(256), 0, st, (const T*)p, ld, (const float*)gates, state, o, meta, seg_starts, ntok, H, D, DV, decay
  // blocks of 16 tokens for prompt portions (fewer barriers and copies per token); 8 for decoding steps, where the state's
  // way in and out of the registers is the work and the smaller shared-memory footprint keeps more CTAs on an SM
  const bool longs = seg_starts && ntok >= 16 * nseg;
  if (D <= 64) { if (longs) launch_pdl(hgrn2_scan_kernel<T, 4, 16>, grid, HG_ARGS); else launch_pdl(hgrn2_scan_kernel<T, 4, 8>, grid, HG_ARGS); }
  else if (D <= 128) { if (longs) launch_pdl(hgrn2_scan_kernel<T, 8, 16>, grid, HG_ARGS); else launch_pdl(hgrn2_scan_kernel<T, 8, 8>, grid, HG_ARGS); }
  else launch_pdl(hgrn2_scan_kernel<T, 16, 8>, grid, HG_ARGS);
#undef HG_ARGS
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

static size_t rc_bytes(int nseg, int ntok, int H, int D, int DV, bool scalar_decay) {
  if (ntok < 1 || H < 1 || D < 1 || DV < 1 || !rc_taken(nseg, ntok, H, D, DV, scalar_decay)) return 0;
  return (size_t)(ntok / rc_chunk_tokens(ntok, H, D, DV) + nseg) * H * ((size_t)D * DV + D) * sizeof(float);
}

extern "C" size_t qspec_seq_recurrence_chunk_bytes(int nseg, int ntok, int H, int D, int DV) { return rc_bytes(nseg, ntok, H, D, DV, false); }
extern "C" size_t qspec_seq_hgrn2_chunk_bytes(int nseg, int ntok, int H, int D, int DV, int dtype) {
  const size_t walk = rc_bytes(nseg, ntok, H, D, DV, false), mma = dtype == QSPEC_DTYPE_BF16 ? rm_bytes(nseg, ntok, H, D, DV) : 0;
  return walk > mma ? walk : mma;                             // (rows that are not on 16-byte boundaries take the other form)
}
extern "C" size_t qspec_seq_lightning_chunk_bytes(int nseg, int ntok, int H, int D, int DV) { return rc_bytes(nseg, ntok, H, D, DV, true); }

// The chunk form's buffer, if these sizes take it and the caller brought one that fits (rows are read 16 bytes at a time).
static void* chunk_workspace(void* ws, size_t bytes, const int* seg_starts, int nseg, int ntok, int H, int D, int DV, const void* scratch, const void* state,
                             bool scalar_decay) {
  const size_t need = seg_starts && ws ? rc_bytes(nseg, ntok, H, D, DV, scalar_decay) : 0;
  return need && bytes >= need && (((uintptr_t)ws | (uintptr_t)scratch | (uintptr_t)state) & 15) == 0 ? ws : nullptr;
}

extern "C" int qspec_seq_hgrn2_chunked(const void* p, int ld, const float* f_b, const float* lower, const float* norm_w, float* state,
                                       float* scratch, void* out, const int* meta, const int* seg_starts, int nseg, int ntok, int H, int D,
                                       int DV, float eps, int dtype, void* workspace, size_t workspace_bytes, void* stream) {
  QSPEC_REQUIRE(!seg_starts || (nseg >= 1 && nseg <= ntok) || ntok == 0, QSPEC_ERR_INVALID_ARG, "seq_hgrn2: %d segments for %d tokens", nseg, ntok);
  QSPEC_REQUIRE(p && f_b && lower && norm_w && state && scratch && out && meta, QSPEC_ERR_INVALID_ARG, "seq_hgrn2: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && H > 0 && H <= 65535 && D > 0 && D <= 256 && DV > 0 && DV <= 65535 * 16 && ld >= 2 * H * D + H * DV,
                QSPEC_ERR_UNSUPPORTED, "seq_hgrn2: %d heads, key size %d (<= 256), value size %d", H, D, DV);
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  cudaStream_t st = (cudaStream_t)stream;
  void* ws = chunk_workspace(workspace, workspace_bytes, seg_starts, nseg, ntok, H, D, DV, scratch, state, false);
  if (dtype == QSPEC_DTYPE_BF16 && seg_starts && workspace && ld % 8 == 0 && (((uintptr_t)p | (uintptr_t)workspace) & 15) == 0 && ((uintptr_t)out & 3) == 0) {
    const size_t need = rm_bytes(nseg, ntok, H, D, DV);
    if (need && workspace_bytes >= need) {
      const rmma::Args a{(const bf16_t*)p, ld, f_b, lower, (float*)workspace, nullptr, state, (bf16_t*)out, norm_w, eps, meta, seg_starts, nseg, ntok, H,
                         rm_chunk_tokens(nseg, ntok, H, D, DV)};
      if (D == 128) return DV == 128 ? launch_rm_d<128, 128>(a, st) : launch_rm_d<128, 64>(a, st);
      return DV == 128 ? launch_rm_d<64, 128>(a, st) : launch_rm_d<64, 64>(a, st);
    }
  }
  float* gates = scratch + (size_t)ntok * H * DV;          // scratch: un-normalised outputs, then the gates
  int s = dtype == QSPEC_DTYPE_F32
              ? launch_hgrn2<float>(p, ld, f_b, lower, state, scratch, gates, meta, seg_starts, nseg, ntok, H, D, DV, st, nullptr, ws, out, norm_w, eps)
              : launch_hgrn2<bf16_t>(p, ld, f_b, lower, state, scratch, gates, meta, seg_starts, nseg, ntok, H, D, DV, st, nullptr, ws, out, norm_w, eps);
  if (s || ws) return s;                                    // (chunks leave normed)
  const long long rows = (long long)ntok * H;
  const unsigned blocks = (unsigned)((rows + 3) / 4);
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(head_norm_kernel<float>, dim3(blocks), dim3(128), 0, st, (const float*)scratch, norm_w, (float*)out, rows, DV, eps);
  else
    launch_pdl(head_norm_kernel<bf16_t>, dim3(blocks), dim3(128), 0, st, (const float*)scratch, norm_w, (bf16_t*)out, rows, DV, eps);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_hgrn2(const void* p, int ld, const float* f_b, const float* lower, const float* norm_w, float* state,
                               float* scratch, void* out, const int* meta, const int* seg_starts, int nseg, int ntok, int H, int D,
                               int DV, float eps, int dtype, void* stream) {
  return qspec_seq_hgrn2_chunked(p, ld, f_b, lower, norm_w, state, scratch, out, meta, seg_starts, nseg, ntok, H, D, DV, eps, dtype, nullptr, 0, stream);
}

extern "C" int qspec_seq_side_gate(void* g, const void* table, const int* ids, int col0, int sd, int table_ld, int V, int ntok, int dtype,
                                   void* stream) {
  QSPEC_REQUIRE(g && table && ids, QSPEC_ERR_INVALID_ARG, "seq_side_gate: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && sd > 0 && col0 >= 0 && col0 + sd <= table_ld && V > 0, QSPEC_ERR_INVALID_ARG, "seq_side_gate: bad sizes");
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  const long long n = (long long)ntok * sd;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(side_gate_kernel<float>, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, (float*)g, (const float*)table, ids, col0,
               sd, table_ld, V, n);
  else
    launch_pdl(side_gate_kernel<bf16_t>, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, (bf16_t*)g, (const bf16_t*)table, ids,
               col0, sd, table_ld, V, n);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T, typename YT, int VEC>
static int launch_residual_norm_v(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride, long long y_tok_stride,
                                  const float* y_w, const void* y2, const float* y2_w, int y2_w_stride, float mult, const float* w,
                                  float w_offset, void* out, int ntok, int W, float eps, const float* y_scale, cudaStream_t st) {
  const size_t smem = (size_t)W * sizeof(float);
  static SmemLimit limit;
  if (smem > 48 * 1024) QSPEC_CUDA(limit.raise(residual_norm_kernel<T, YT, VEC>, smem));
  launch_pdl(residual_norm_kernel<T, YT, VEC>, dim3(ntok), dim3(256), smem, st, x_in, x_out, (const YT*)y, y_parts, y_part_stride,
             y_tok_stride, y_w, (const YT*)y2, y2_w, y2_w_stride, mult, w, w_offset, (T*)out, W, eps, y_scale);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

template <typename T, typename YT>
static int launch_residual_norm(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride, long long y_tok_stride,
                                const float* y_w, const void* y2, const float* y2_w, int y2_w_stride, float mult, const float* w,
                                float w_offset, void* out, int ntok, int W, float eps, const float* y_scale, cudaStream_t st) {
  // four columns per thread where every row starts on a 16-byte boundary (float32 rows; bfloat16 rows need 8 bytes)
  // QSPEC_SEQ_RESNORM=scalar keeps one column per thread and step, for comparison
  static const bool scalar = [] { const char* v = getenv("QSPEC_SEQ_RESNORM"); return v && !strcmp(v, "scalar"); }();
  const bool vec = !scalar && W % 4 == 0 && y_part_stride % 4 == 0 && y_tok_stride % 4 == 0 &&
                   (((uintptr_t)x_in | (uintptr_t)x_out | (uintptr_t)w | (uintptr_t)y_scale) & 15) == 0 &&
                   (((uintptr_t)y | (uintptr_t)y2) & (4 * sizeof(YT) - 1)) == 0 && ((uintptr_t)out & (4 * sizeof(T) - 1)) == 0;
  if (vec)
    return launch_residual_norm_v<T, YT, 4>(x_in, x_out, y, y_parts, y_part_stride, y_tok_stride, y_w, y2, y2_w, y2_w_stride, mult, w, w_offset,
                                            out, ntok, W, eps, y_scale, st);
  return launch_residual_norm_v<T, YT, 1>(x_in, x_out, y, y_parts, y_part_stride, y_tok_stride, y_w, y2, y2_w, y2_w_stride, mult, w, w_offset,
                                          out, ntok, W, eps, y_scale, st);
}

extern "C" int qspec_seq_residual_norm_scaled(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride,
                                              long long y_tok_stride, const float* y_w, const void* y2, const float* y2_w, int y2_w_stride,
                                              float mult, const float* y_scale, const float* w, float w_offset, void* out, int ntok, int W,
                                              float eps, int y_dtype, int dtype, void* stream) {
  QSPEC_REQUIRE(x_in && (x_out || out) && (!out || w), QSPEC_ERR_INVALID_ARG, "seq_residual_norm: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && W > 0 && W <= 49152 && y_parts >= 1 && y2_w_stride >= 0, QSPEC_ERR_INVALID_ARG,
                "seq_residual_norm: bad sizes (width <= 49152)");
  MIX_DTYPE_OK(dtype);
  QSPEC_REQUIRE(y_dtype == dtype || y_dtype == QSPEC_DTYPE_F32, QSPEC_ERR_UNSUPPORTED, "seq_residual_norm: y is of the activation type or float32");
  if (ntok == 0) return QSPEC_OK;
  cudaStream_t st = (cudaStream_t)stream;
#define RN_ARGS x_in, x_out, y, y_parts, y_part_stride, y_tok_stride, y_w, y2, y2_w, y2_w_stride, mult, w, w_offset, out, ntok, W, eps, y_scale, st
  if (dtype == QSPEC_DTYPE_F32) return launch_residual_norm<float, float>(RN_ARGS);
  if (y_dtype == QSPEC_DTYPE_F32) return launch_residual_norm<bf16_t, float>(RN_ARGS);
  return launch_residual_norm<bf16_t, bf16_t>(RN_ARGS);
#undef RN_ARGS
}

extern "C" int qspec_seq_residual_norm(const float* x_in, float* x_out, const void* y, int y_parts, long long y_part_stride,
                                       long long y_tok_stride, const float* y_w, const void* y2, const float* y2_w, int y2_w_stride,
                                       float mult, const float* w, float w_offset, void* out, int ntok, int W, float eps, int y_dtype,
                                       int dtype, void* stream) {
  return qspec_seq_residual_norm_scaled(x_in, x_out, y, y_parts, y_part_stride, y_tok_stride, y_w, y2, y2_w, y2_w_stride, mult, nullptr, w,
                                        w_offset, out, ntok, W, eps, y_dtype, dtype, stream);
}

extern "C" int qspec_seq_act(void* a, long long n, int act, int dtype, void* stream) {
  QSPEC_REQUIRE(a && n >= 0, QSPEC_ERR_INVALID_ARG, "seq_act: bad arguments");
  QSPEC_REQUIRE(act == QSPEC_ACT_RELU2 || act == QSPEC_ACT_GELU_ERF, QSPEC_ERR_INVALID_ARG, "seq_act: unknown activation %d", act);
  MIX_DTYPE_OK(dtype);
  if (n == 0) return QSPEC_OK;
  const size_t esz = dtype == QSPEC_DTYPE_F32 ? 4 : 2;
  const bool vec = n % 4 == 0 && ((uintptr_t)a & (4 * esz - 1)) == 0;
  long long blocks = (n / (vec ? 4 : 1) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == QSPEC_DTYPE_F32) {
    if (vec) launch_pdl(act_kernel<float, 4>, dim3((unsigned)blocks), dim3(256), 0, st, (float*)a, n, act);
    else launch_pdl(act_kernel<float, 1>, dim3((unsigned)blocks), dim3(256), 0, st, (float*)a, n, act);
  } else {
    if (vec) launch_pdl(act_kernel<bf16_t, 4>, dim3((unsigned)blocks), dim3(256), 0, st, (bf16_t*)a, n, act);
    else launch_pdl(act_kernel<bf16_t, 1>, dim3((unsigned)blocks), dim3(256), 0, st, (bf16_t*)a, n, act);
  }
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_glu(const void* gu, int ld, void* out, int ntok, int F, int act, int dtype, void* stream) {
  QSPEC_REQUIRE(gu && out && ntok >= 0 && F > 0 && ld >= 2 * F, QSPEC_ERR_INVALID_ARG, "seq_glu: bad arguments");
  QSPEC_REQUIRE(act == QSPEC_GLU_SILU || act == QSPEC_GLU_GELU_TANH, QSPEC_ERR_INVALID_ARG, "seq_glu: unknown activation %d", act);
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  const long long n = (long long)ntok * F;
  const size_t esz = dtype == QSPEC_DTYPE_F32 ? 4 : 2;
  const bool vec = F % 4 == 0 && ld % 4 == 0 && (((uintptr_t)gu | (uintptr_t)out) & (4 * esz - 1)) == 0;
  long long blocks = (n / (vec ? 4 : 1) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == QSPEC_DTYPE_F32) {
    if (vec) launch_pdl(glu_kernel<float, 4>, dim3((unsigned)blocks), dim3(256), 0, st, (const float*)gu, ld, (float*)out, F, n, act);
    else launch_pdl(glu_kernel<float, 1>, dim3((unsigned)blocks), dim3(256), 0, st, (const float*)gu, ld, (float*)out, F, n, act);
  } else {
    if (vec) launch_pdl(glu_kernel<bf16_t, 4>, dim3((unsigned)blocks), dim3(256), 0, st, (const bf16_t*)gu, ld, (bf16_t*)out, F, n, act);
    else launch_pdl(glu_kernel<bf16_t, 1>, dim3((unsigned)blocks), dim3(256), 0, st, (const bf16_t*)gu, ld, (bf16_t*)out, F, n, act);
  }
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_silu_mul(const void* gu, int ld, void* out, int ntok, int F, int dtype, void* stream) {
  return qspec_seq_glu(gu, ld, out, ntok, F, QSPEC_GLU_SILU, dtype, stream);
}

extern "C" int qspec_seq_lightning_chunked(const void* p, int ld, const float* decay, const float* norm_w, float* state, float* scratch, void* out,
                                           const int* meta, const int* seg_starts, int nseg, int ntok, int H, int D, int DV, float eps, int dtype,
                                           void* workspace, size_t workspace_bytes, void* stream) {
  QSPEC_REQUIRE(!seg_starts || (nseg >= 1 && nseg <= ntok) || ntok == 0, QSPEC_ERR_INVALID_ARG, "seq_lightning: %d segments for %d tokens", nseg, ntok);
  QSPEC_REQUIRE(p && decay && norm_w && state && scratch && out && meta, QSPEC_ERR_INVALID_ARG, "seq_lightning: null pointer");
  QSPEC_REQUIRE(ntok >= 0 && H > 0 && H <= 65535 && D > 0 && D <= 256 && DV > 0 && DV <= 65535 * 16 && ld >= 2 * H * D + 2 * H * DV,
                QSPEC_ERR_UNSUPPORTED, "seq_lightning: %d heads, key size %d (<= 256), value size %d", H, D, DV);
  MIX_DTYPE_OK(dtype);
  if (ntok == 0) return QSPEC_OK;
  cudaStream_t st = (cudaStream_t)stream;
  float* gates = scratch + (size_t)ntok * H * DV;          // scratch: un-normalised outputs, then silu(q) and silu(k)
  void* ws = chunk_workspace(workspace, workspace_bytes, seg_starts, nseg, ntok, H, D, DV, scratch, state, true);
  int s = dtype == QSPEC_DTYPE_F32
              ? launch_hgrn2<float>(p, ld, nullptr, nullptr, state, scratch, gates, meta, seg_starts, nseg, ntok, H, D, DV, st, decay, ws, nullptr, nullptr, eps)
              : launch_hgrn2<bf16_t>(p, ld, nullptr, nullptr, state, scratch, gates, meta, seg_starts, nseg, ntok, H, D, DV, st, decay, ws, nullptr, nullptr, eps);
  if (s) return s;
  const int N = H * DV, goff = 2 * H * D + H * DV;         // the output gate's logits follow q, k and v in the row
  if (dtype == QSPEC_DTYPE_F32)
    launch_pdl(gated_row_norm_kernel<float>, dim3(ntok), dim3(256), 0, st, (const float*)scratch, norm_w, (const float*)p + goff, ld,
               (float*)out, N, eps);
  else
    launch_pdl(gated_row_norm_kernel<bf16_t>, dim3(ntok), dim3(256), 0, st, (const float*)scratch, norm_w, (const bf16_t*)p + goff, ld,
               (bf16_t*)out, N, eps);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

extern "C" int qspec_seq_lightning(const void* p, int ld, const float* decay, const float* norm_w, float* state, float* scratch, void* out,
                                   const int* meta, const int* seg_starts, int nseg, int ntok, int H, int D, int DV, float eps, int dtype,
                                   void* stream) {
  return qspec_seq_lightning_chunked(p, ld, decay, norm_w, state, scratch, out, meta, seg_starts, nseg, ntok, H, D, DV, eps, dtype, nullptr, 0, stream);
}
