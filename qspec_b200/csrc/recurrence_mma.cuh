// The gated linear recurrence S <- diag(f) S + (1 - f) v^T, o = S^T q of bfloat16 rows on the tensor cores, 16 tokens at a time, over the chunks of
// recurrence_chunk_kernel (included by seq_mix_kernels.cu behind it).
//
// Over a block of 16 tokens, with F the product of its decays, Q_i = q_i times the block's decays up to token i and K_j = (1 - f_j) times those behind token j:
//   o_i = S^T Q_i + sum_{j <= i} a_ij v_j,   a_ij = sum_d q_i[d] (1 - f_j)[d] prod_{j < s <= i} f_s[d],   S <- diag(F) S + sum_j K_j v_j^T.
// All factors are products of decays, so nothing is divided by a decay that may be next to zero and nothing overflows that the walk would not.
// Everything is float32. Keys and scores meet values, which are bfloat16 as they come: three bfloat16 terms of them are the float32 value exactly. Queries
// meet the state as two terms of a 10-bit mantissa each (tf32), all four products of which are taken; they are off by 2^-23 of an operand. Every
// accumulation of the tensor cores cuts at the accumulator's last bit, so the lower terms have accumulators of their own, and the state is updated by
// float32 instructions. Errors of the state against 64 bits are those of the other forms (1.85e-7 of its norm after 1500 tokens, the gates' own rounding).
//
// Every warp owns 16 value columns: S^T [16 columns x D] in registers, in the accumulator layout of v^T K, which is the layout of the second operand of
// Q S as well, so that the state never moves. In front of the products all threads prepare the block, a thread two key rows of some tokens: gates (no
// pass of their own over memory), decays' products, the scores a_ij (summed over the rows by exchanges that halve the number of values a lane holds) and
// the split operands, which go to shared memory (16-byte pieces c of row r at c ^ (r & 7)). With warps of their own for the preparation, four beside eight, the
// kernel waited for these (outputs of 1500 tokens, 16 heads of 128 x 128, 100 us instead of 75).
// What bounds it is the number of instructions (about 2500 a warp and block where outputs are computed: gates, scores, splitting and products a quarter each) at two
// a cycle and SM; the tensor cores are busy a fifth of the time. A launch of its own for the gates takes as long as it saves here (11 us; outputs 70 -> 62,
// states 25 -> 21). 1500 tokens, 16 heads of 128 x 128, all launches: 143 -> 91 us; 600 tokens, 8 heads of 64 x 64: 40 -> 27.
//
// Values that are not finite would turn into NaN in the lower terms (infinity - infinity) and reach rows that the walk spares. They show in the chunk's
// outputs or in its last state, which no later token makes finite again; such a chunk is walked once more token by token (rm_walk).
namespace qspec {
namespace rmma {

constexpr int BT = 16;                                        // tokens of a block
template <int D, int DV> struct Shape {
  static constexpr int WARPS = DV / 16, THREADS = WARPS * 32;
  static constexpr int PAIRS = D / 2, GROUPS = THREADS / PAIRS, TOKENS = BT / GROUPS, PARTS = PAIRS / 32;   // rows in pairs; groups of tokens, tokens of each
  static constexpr int TERM = BT * D * 2;                     // bytes of one term of a block's keys or queries
  static constexpr int SCORES = BT * 20 * 4;                  // bytes of a warp's share of the scores
  static constexpr int K_AT = 0, V_AT = 3 * TERM, F_AT = V_AT + 2 * BT * DV * 2, DEC_AT = F_AT + D * 4, E_END = DEC_AT + BT * D * 4;
  static constexpr int Q_AT = E_END, A_AT = Q_AT + 4 * TERM, OM_AT = A_AT + PARTS * SCORES, QF_AT = OM_AT + BT * D * 4, SS_AT = QF_AT + BT * D * 4,
                       O_END = SS_AT + WARPS * BT * 4;
  static constexpr int CTAS = 65536 / 128 / THREADS;          // per SM, by registers
};
template <int D, int DV, bool OUT> constexpr size_t smem_bytes() { return OUT ? Shape<D, DV>::O_END : Shape<D, DV>::E_END; }   // (rm_walk takes less)

__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) { uint64_t r; asm("sub.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ bool finite(float x) { return fabsf(x) < INFINITY; }

// Two float32 values as three pairs of bfloat16: t0 + t1 + t2 is the value. t0 and t1 are rounded, so that t1 is below 2^-8 of t0 and t2 of t1.
// (On the integer units: a conversion instruction takes four times as long.)
__device__ __forceinline__ void split3(uint64_t x, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float2 f = rc_unpair(x);
    const uint32_t a = __float_as_uint(f.x) + 0x8000u, b = __float_as_uint(f.y) + 0x8000u;
    (i ? t1 : t0) = __byte_perm(a, b, 0x7632);
    x = sub2(x, rc_pair(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u)));
  }
  const float2 f = rc_unpair(x);
  t2 = __byte_perm(__float_as_uint(f.x), __float_as_uint(f.y), 0x7632);
}
// Two float32 values as two terms of a 10-bit mantissa each, rounded: their sum is off by 2^-23 of the value at most.
__device__ __forceinline__ void split2(uint64_t x, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
  const float2 f = rc_unpair(x);
  hi[0] = (__float_as_uint(f.x) + 0x1000u) & 0xffffe000u;
  hi[1] = (__float_as_uint(f.y) + 0x1000u) & 0xffffe000u;
  const float2 r = rc_unpair(sub2(x, rc_pair(__uint_as_float(hi[0]), __uint_as_float(hi[1]))));
  lo[0] = __float_as_uint(r.x) + 0x1000u;                     // (the products ignore the lower 13 bits)
  lo[1] = __float_as_uint(r.y) + 0x1000u;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c = a b
__device__ __forceinline__ void mma_set(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// Sums of N values (a power of two) over the lanes: the result is that of v[lane / (32 / N)].
template <int N> __device__ __forceinline__ float lane_sums(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16, m = N; o > 0; o >>= 1) {
    if (m > 1) {                                              // each half of the lanes keeps one half of the values
      m >>= 1;
      const bool upper = lane & o;
#pragma unroll
      for (int k = 0; k < N / 2; ++k)
        if (k < m) {
          const float keep = upper ? v[k + m] : v[k], send = upper ? v[k] : v[k + m];
          v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

struct Args {
  const __nv_bfloat16* p; int ld;
  const float *f_b, *lower; float *E, *P, *state; __nv_bfloat16* out; const float* norm_w; float eps;
  const int *meta, *seg_starts; int nseg, ntok, H, C;
};
// Element order of a chunk's state in the workspace, as the registers hold it: [columns / 16][rows / 16][column group][lane] of four values, for
// column 16 ct + 8 g + lane / 4 the rows 16 rt + 2 (lane % 4) + {0, 1, 8, 9}.
template <int D> __device__ __forceinline__ size_t tile_at(int ct, int rt, int g, int lane) { return ((((size_t)ct * (D / 16) + rt) * 2 + g) * 32 + lane) * 4; }

// gates of one (token, row), as hgrn2_gates_kernel computes them
__device__ __forceinline__ void gate(float z, float lo, float& f, float& om) {
  const float x = 1.0f / (1.0f + expf(z));
  f = lo + (1.0f - lo) * (1.0f - x);
  om = (1.0f - lo) * x;
}

// A chunk once more, token by token: thread = a value column. Chunks with values that are not finite only.
template <int D, int DV, bool OUT>
__device__ __noinline__ void rm_walk(const Args& a, int t0, int t1, int h, const float* from, const float* tiled, float* to, float* to_tiled, float* P, float* smem) {
  float *sf = smem, *sg = sf + D, *sq = sg + D, *so = sq + D;
  const int tid = threadIdx.x, HD = a.H * D;
  float S[D];
  auto tile_of = [&](int d) {
    return tile_at<D>(tid >> 4, d >> 4, tid >> 3 & 1, (tid & 7) * 4 + (d >> 1 & 3)) + (d >> 3 & 1) * 2 + (d & 1);
  };
  if (tid < DV)
    for (int d = 0; d < D; ++d) S[d] = from ? from[(size_t)d * DV + tid] : tiled ? tiled[tile_of(d)] : 0.f;
  float whole = 1.f;
  for (int t = t0; t < t1; ++t) {
    const __nv_bfloat16* row = a.p + (size_t)t * a.ld;
    __syncthreads();
    for (int d = tid; d < D; d += Shape<D, DV>::THREADS) {
      gate(to_f(row[HD + h * D + d]) + a.f_b[h * D + d], a.lower[h * D + d], sf[d], sg[d]);
      const float zq = to_f(row[h * D + d]);
      sq[d] = zq / (1.0f + expf(-zq));
    }
    __syncthreads();
    if (tid < D) whole *= sf[tid];
    float o = 0.f;
    if (tid < DV) {
      const float v = to_f(row[2 * HD + h * DV + tid]);
      for (int d = 0; d < D; ++d) {
        S[d] = sf[d] * S[d] + sg[d] * v;
        o += S[d] * sq[d];
      }
      so[tid] = o * o;
    }
    if (OUT) {
      __syncthreads();
      if (tid < DV) {
        float ss = 0.f;
        for (int c = 0; c < DV; ++c) ss += so[c];
        a.out[((size_t)t * a.H + h) * DV + tid] = __float2bfloat16_rn(o * (1.0f / sqrtf(ss / (float)DV + a.eps)) * a.norm_w[tid]);
      }
    }
  }
  if (tid < DV)
    for (int d = 0; d < D; ++d) {
      if (to) to[(size_t)d * DV + tid] = S[d];
      if (to_tiled) to_tiled[tile_of(d)] = S[d];
    }
  if (P && tid < D) P[tid] = whole;
}

template <int D, int DV, bool OUT>
__global__ void __launch_bounds__(Shape<D, DV>::THREADS, Shape<D, DV>::CTAS) chunk_kernel(const __grid_constant__ Args a) {
  pdl_enter();
  using Sh = Shape<D, DV>;
  constexpr int TT = Sh::TOKENS;
  extern __shared__ __align__(128) unsigned char rm_smem[];
  __shared__ RcChunk s_chunk;
  __shared__ bool s_found;
  const int b = blockIdx.x, h = blockIdx.y;
  if (!rc_find(a.meta, a.seg_starts, a.nseg, a.ntok, a.C, b, 0, &s_chunk, &s_found)) return;
  const int c = b - s_chunk.first;
  if (!OUT && c == s_chunk.chunks - 1) return;               // nobody starts from where the last chunk ends
  const int t0 = s_chunk.begin + c * a.C, t1 = min(t0 + a.C, s_chunk.end);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, HD = a.H * D;
  const size_t elems = (size_t)D * DV;
  float* const slot = a.E + ((size_t)b * a.H + h) * elems;    // OUT: the state this chunk starts from; else E goes to the next chunk's place
  float* const state = a.state + ((size_t)s_chunk.mt.slot * a.H + h) * elems;
  // (a segment of several chunks leaves its state where its first chunk would read it: that one's start is a copy of carry_kernel's)
  const float* const from = OUT && s_chunk.chunks == 1 && s_chunk.mt.pos > 0 ? state : nullptr;
  const float* const tiled = OUT && s_chunk.chunks > 1 ? slot : nullptr;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(rm_smem);
  bool odd = false;                                           // met a value that is not finite

  // products: columns 16 warp + r4 (+ 8); tokens r4, r4 + 8 of the outputs
  const int r4 = lane >> 2, c2 = (lane & 3) * 2;
  const uint32_t frow = lane & 15, fhalf = lane >> 4;         // fragments: lane l addresses row l % 16, piece l / 16 of a pair of pieces
  float S[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 16; ++i)
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tiled) {
        x = *reinterpret_cast<const float4*>(tiled + tile_at<D>(warp, i, g, lane));
      } else if (from) {
        const float* s = from + (size_t)(16 * i + c2) * DV + warp * 16 + r4 + 8 * g;
        x = make_float4(s[0], s[DV], s[8 * DV], s[9 * DV]);
      }
      S[2 * i][2 * g] = x.x; S[2 * i][2 * g + 1] = x.y; S[2 * i + 1][2 * g] = x.z; S[2 * i + 1][2 * g + 1] = x.w;
      if (OUT) odd |= !(finite(x.x) && finite(x.y) && finite(x.z) && finite(x.w));
    }
  // preparation: rows d, d + 1 of tokens TT * grp ..; the group's warp `part`
  const int d = 2 * (tid % Sh::PAIRS), grp = tid / Sh::PAIRS, part = warp % Sh::PARTS, hd = h * D + d;
  const float2 bias = make_float2(a.f_b[hd], a.f_b[hd + 1]), low = make_float2(a.lower[hd], a.lower[hd + 1]);
  float* const dec = reinterpret_cast<float*>(rm_smem + Sh::DEC_AT) + d;   // [BT][D] decays; OUT: what multiplies v, queries
  float* const som = reinterpret_cast<float*>(rm_smem + Sh::OM_AT) + d;
  float* const sqf = reinterpret_cast<float*>(rm_smem + Sh::QF_AT) + d;
  float* const sa = reinterpret_cast<float*>(rm_smem + Sh::A_AT) + part * BT * 20;
  float* const sums = reinterpret_cast<float*>(rm_smem + Sh::SS_AT);
  if (OUT)
    for (int i = tid; i < Sh::PARTS * BT * 20; i += Sh::THREADS) reinterpret_cast<float*>(rm_smem + Sh::A_AT)[i] = 0.f;   // above the diagonal it stays so
  auto two = [](const float* p) { return *reinterpret_cast<const uint64_t*>(p); };
  auto put = [&](int at, int i, uint64_t x) {
    uint32_t t[3];
    split3(x, t[0], t[1], t[2]);
    unsigned char* dst = rm_smem + at + i * D * 2 + (((d >> 3) ^ (i & 7)) << 4) + (d & 7) * 2;
#pragma unroll
    for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(dst + k * Sh::TERM) = t[k];
  };
  // queries: two float32 terms; of every eight rows the even ones first, the order in which a lane holds the state's; 16-byte pieces c at c ^ (i & 7)
  auto putq = [&](int i, uint64_t x) {
    uint32_t t[2][2];
    split2(x, t[0], t[1]);
    unsigned char* dst = rm_smem + Sh::Q_AT + i * D * 4 + ((2 * (d >> 3) ^ (i & 7)) << 4) + (d & 7) * 2;
    unsigned char* odd_row = rm_smem + Sh::Q_AT + i * D * 4 + (((2 * (d >> 3) + 1) ^ (i & 7)) << 4) + (d & 7) * 2;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      *reinterpret_cast<uint32_t*>(dst + k * BT * D * 4) = t[k][0];
      *reinterpret_cast<uint32_t*>(odd_row + k * BT * D * 4) = t[k][1];
    }
  };
  uint32_t zf[TT], zq[TT];
  uint4 zv[BT * DV / 8 / Sh::THREADS];
  auto fetch = [&](int tb) {                                  // rows past the end: the last one again
#pragma unroll
    for (int k = 0; k < TT; ++k) {
      const __nv_bfloat16* row = a.p + (size_t)min(tb + grp * TT + k, t1 - 1) * a.ld + hd;
      zf[k] = *reinterpret_cast<const uint32_t*>(row + HD);
      if (OUT) zq[k] = *reinterpret_cast<const uint32_t*>(row);
    }
#pragma unroll
    for (int k = 0; k < BT * DV / 8 / Sh::THREADS; ++k) {
      const int i = tid + k * Sh::THREADS, r = i / (DV / 8), pc = i % (DV / 8);
      zv[k] = *reinterpret_cast<const uint4*>(a.p + (size_t)min(tb + r, t1 - 1) * a.ld + 2 * HD + (size_t)h * DV + pc * 8);
    }
  };
  float o[2][4];                                              // un-normalised outputs of a block, [columns / 8]
  auto leave = [&](int tb) {                                  // the per-head norm: sums of squares from all warps
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = tb + r4 + 8 * e;
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < Sh::WARPS; ++w) s += sums[w * BT + r4 + 8 * e];
      const float rr = 1.0f / sqrtf(s / (float)DV + a.eps);
      if (t < t1) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int col = warp * 16 + 8 * j + c2;
          *reinterpret_cast<__nv_bfloat162*>(a.out + ((size_t)t * a.H + h) * DV + col) =
              __floats2bfloat162_rn(o[j][2 * e] * rr * a.norm_w[col], o[j][2 * e + 1] * rr * a.norm_w[col + 1]);
        }
      }
    }
  };
  uint64_t whole = rc_pair(1.f, 1.f);                         // !OUT, group 0: product of the chunk's decays
  fetch(t0);
  for (int tb = t0; tb < t1; tb += BT) {
    const int nb = min(BT, t1 - tb), vbuf = Sh::V_AT + ((tb - t0) / BT & 1) * BT * DV * 2;
    // ---- gates and values
    uint64_t mine[TT];                                        // OUT: queries; else what multiplies v
    float own[TT];                                            // OUT: shares of the scores a_ii
#pragma unroll
    for (int k = 0; k < TT; ++k) {
      const int i = grp * TT + k;
      const bool in = i < nb;
      float f0, f1, o0, o1, q0 = 0.f, q1 = 0.f;
      gate(__uint_as_float(zf[k] << 16) + bias.x, low.x, f0, o0);
      gate(__uint_as_float(zf[k] & 0xffff0000u) + bias.y, low.y, f1, o1);
      if (OUT) {
        const float z0 = __uint_as_float(zq[k] << 16), z1 = __uint_as_float(zq[k] & 0xffff0000u);
        q0 = z0 / (1.0f + expf(-z0));
        q1 = z1 / (1.0f + expf(-z1));
      }
      *reinterpret_cast<uint64_t*>(dec + i * D) = in ? rc_pair(f0, f1) : rc_pair(1.f, 1.f);
      const uint64_t om = in ? rc_pair(o0, o1) : 0ull, q = in ? rc_pair(q0, q1) : 0ull;
      mine[k] = OUT ? q : om;
      if (OUT) {
        *reinterpret_cast<uint64_t*>(som + i * D) = om;
        *reinterpret_cast<uint64_t*>(sqf + i * D) = q;
        const float2 x = rc_unpair(rc_mul(om, q));
        own[k] = x.x + x.y;
      }
    }
#pragma unroll
    for (int k = 0; k < BT * DV / 8 / Sh::THREADS; ++k) {
      const int i = tid + k * Sh::THREADS, r = i / (DV / 8), pc = i % (DV / 8);
      const uint4 x = r < nb ? zv[k] : make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(rm_smem + vbuf + r * DV * 2 + ((pc ^ (r & 7)) << 4)) = x;
    }
    const float diag = OUT ? lane_sums<TT>(own) : 0.f;
    __syncthreads();                                          // gates are there, the block before is done with
    if (OUT && tb > t0) leave(tb - BT);
    // ---- scores and operands
    if (OUT) {
      if (lane % (32 / TT) == 0) {
        const int i = grp * TT + lane / (32 / TT);
        sa[i * 20 + i] = diag;
      }
      // columns j = t and 15 - t: fifteen scores below the diagonal, those of t (rows t + 1 .. 15) first
#pragma unroll
      for (int k = 0; k < TT / 2; ++k) {
        const int t = grp * (TT / 2) + k, turn = 15 - t;
        const float* row = dec + (t + 1) * D;                 // decays of row i = v + t + 1, then of v + 1; the queries lie QF_AT - DEC_AT further
        uint64_t r = two(som + t * D);
        float val[16];
#pragma unroll
        for (int v = 0; v < 15; ++v) {
          if (v == turn) {
            put(Sh::K_AT, t, r);                              // at the block's end: what multiplies v_t in the state
            r = two(som + turn * D);
            row = dec + D;
          }
          r = rc_mul(r, two(row + v * D));
          const float2 x = rc_unpair(rc_mul(two(row + v * D + (Sh::QF_AT - Sh::DEC_AT) / 4), r));
          val[v] = x.x + x.y;
        }
        val[15] = 0.f;
        if (turn == 15) {
          put(Sh::K_AT, t, r);
          r = two(som + turn * D);
        }
        put(Sh::K_AT, turn, r);
        const float sum = lane_sums<16>(val);
        const int v = lane >> 1;
        if (!(lane & 1) && v < 15) sa[v < turn ? (v + t + 1) * 20 + t : (v + 1) * 20 + turn] = sum;
      }
      uint64_t run = rc_pair(1.f, 1.f);
#pragma unroll 4
      for (int i = 0; i < grp * TT; ++i) run = rc_mul(run, two(dec + i * D));
#pragma unroll
      for (int k = 0; k < TT; ++k) {
        run = rc_mul(run, two(dec + (grp * TT + k) * D));
        putq(grp * TT + k, rc_mul(mine[k], run));
      }
      if (grp == Sh::GROUPS - 1) *reinterpret_cast<uint64_t*>(rm_smem + Sh::F_AT + d * 4) = run;
    } else {
      uint64_t run = rc_pair(1.f, 1.f);
#pragma unroll 4
      for (int i = BT - 1; i >= (grp + 1) * TT; --i) run = rc_mul(run, two(dec + i * D));
#pragma unroll
      for (int k = TT - 1; k >= 0; --k) {
        put(Sh::K_AT, grp * TT + k, rc_mul(mine[k], run));
        run = rc_mul(run, two(dec + (grp * TT + k) * D));
      }
      if (grp == 0) {
        *reinterpret_cast<uint64_t*>(rm_smem + Sh::F_AT + d * 4) = run;
        whole = rc_mul(whole, run);
      }
    }
    if (tb + BT < t1) fetch(tb + BT);
    __syncthreads();
    // ---- products
    uint32_t v[4];                                            // v^T: first operand of v^T K; (v0, v1) and (v2, v3): second operand of a v
    ldsm4t(v, sbase + vbuf + frow * DV * 2 + (((2 * warp + fhalf) ^ (frow & 7)) << 4));
    if (OUT) {
      float hi[2][2][4] = {}, lo[2][4] = {};                  // [even, odd steps][columns / 8]; lower terms
#pragma unroll
      for (int k = 0; k < D / 8; ++k) {
        uint32_t q[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t) ldsm4(q[t], sbase + Sh::Q_AT + t * BT * D * 4 + frow * D * 4 + (((2 * k + fhalf) ^ (frow & 7)) << 4));
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t sh[2], sl[2];
          split2(rc_pair(S[k][2 * j], S[k][2 * j + 1]), sh, sl);
          mma_tf32(lo[j], q[1], sl[0], sl[1]);
          mma_tf32(hi[k & 1][j], q[0], sh[0], sh[1]);
          mma_tf32(lo[j], q[1], sh[0], sh[1]);
          mma_tf32(lo[j], q[0], sl[0], sl[1]);
        }
      }
      // scores: rows i = r4, r4 + 8; columns j = c2, + 1, + 8, + 9
      const float* all = reinterpret_cast<const float*>(rm_smem + Sh::A_AT);
      uint32_t at[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float* p = all + (r4 + (e & 1) * 8) * 20 + c2 + (e >> 1) * 8;
        uint64_t x = two(p);
#pragma unroll
        for (int w = 1; w < Sh::PARTS; ++w) x = add2(x, two(p + w * BT * 20));
        split3(x, at[0][e], at[1][e], at[2][e]);
      }
      float ss[2] = {0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float x[4];
        tk_mma_16816(lo[j], at[2], v[2 * j], v[2 * j + 1]);
        tk_mma_16816(lo[j], at[1], v[2 * j], v[2 * j + 1]);
        mma_set(x, at[0], v[2 * j], v[2 * j + 1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o[j][e] = ((hi[0][j][e] + hi[1][j][e]) + x[e]) + lo[j][e];
          odd |= !finite(o[j][e]);
          ss[e >> 1] += o[j][e] * o[j][e];
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 1);
        ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 2);
        if ((lane & 3) == 0) sums[warp * BT + r4 + 8 * e] = ss[e];
      }
    }
    // S <- diag(F) S + v^T K
    const uint32_t va[4] = {v[0], v[2], v[1], v[3]};
    const float* sF = reinterpret_cast<const float*>(rm_smem + Sh::F_AT);
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
      float up[2][4], below[2][4];
      uint32_t k[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t) ldsm4t(k[t], sbase + Sh::K_AT + t * Sh::TERM + frow * D * 2 + (((2 * i + fhalf) ^ (frow & 7)) << 4));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        mma_set(below[e], va, k[2][2 * e], k[2][2 * e + 1]);
        mma_set(up[e], va, k[0][2 * e], k[0][2 * e + 1]);
        tk_mma_16816(below[e], va, k[1][2 * e], k[1][2 * e + 1]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint64_t F = two(sF + 16 * i + 8 * e + c2);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint64_t u = add2(rc_pair(up[e][2 * j], up[e][2 * j + 1]), rc_pair(below[e][2 * j], below[e][2 * j + 1]));
          const float2 f = rc_unpair(rc_fma(F, rc_pair(S[2 * i + e][2 * j], S[2 * i + e][2 * j + 1]), u));
          S[2 * i + e][2 * j] = f.x; S[2 * i + e][2 * j + 1] = f.y;
        }
      }
    }
  }
  __syncthreads();
  if (OUT) leave(t0 + (t1 - t0 - 1) / BT * BT);
#pragma unroll
  for (int i = 0; i < D / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) odd |= !finite(S[i][e]);
  float* const to = OUT && t1 == s_chunk.end ? state : nullptr;   // OUT: the segment's last chunk leaves the state
  float* const to_tiled = OUT ? nullptr : slot + (size_t)a.H * elems;
  float* const P = OUT ? nullptr : a.P + ((size_t)b * a.H + h) * D;
  if (__syncthreads_or(odd)) {
    rm_walk<D, DV, OUT>(a, t0, t1, h, from, tiled, to, to_tiled, P, reinterpret_cast<float*>(rm_smem));
    return;
  }
#pragma unroll
  for (int i = 0; i < D / 16; ++i)
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (to_tiled)
        *reinterpret_cast<float4*>(to_tiled + tile_at<D>(warp, i, g, lane)) = make_float4(S[2 * i][2 * g], S[2 * i][2 * g + 1], S[2 * i + 1][2 * g], S[2 * i + 1][2 * g + 1]);
      if (to) {
        float* s = to + (size_t)(16 * i + c2) * DV + warp * 16 + r4 + 8 * g;
        s[0] = S[2 * i][2 * g]; s[DV] = S[2 * i][2 * g + 1]; s[8 * DV] = S[2 * i + 1][2 * g]; s[9 * DV] = S[2 * i + 1][2 * g + 1];
      }
    }
  if (!OUT && grp == 0) *reinterpret_cast<uint64_t*>(P + d) = whole;
}

// Through the chunks of a segment, as recurrence_carry_kernel, in the element order of the registers.
template <int D, int DV>
__global__ void __launch_bounds__(256) carry_kernel(const __grid_constant__ Args a) {
  pdl_enter();
  __shared__ RcChunk s_chunk;
  __shared__ bool s_found;
  if (!rc_find(a.meta, a.seg_starts, a.nseg, a.ntok, a.C, -1, blockIdx.x, &s_chunk, &s_found)) return;
  const int n = s_chunk.chunks;
  if (n == 1) return;                                         // the outputs read and write the state itself
  const int h = blockIdx.y, e = blockIdx.z * 256 + threadIdx.x, lane = e & 31, g = e >> 5 & 1, rt = e >> 6 & (D / 16 - 1), ct = e / (4 * D);
  if (e >= D * DV / 4) return;
  const int d = 16 * rt + 2 * (lane & 3);
  const size_t step = (size_t)a.H * D * DV / 4;
  float4* at = reinterpret_cast<float4*>(a.E + ((size_t)s_chunk.first * a.H + h) * D * DV) + e;
  const float* pr = a.P + ((size_t)s_chunk.first * a.H + h) * D + d;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (s_chunk.mt.pos > 0) {
    const float* src = a.state + (((size_t)s_chunk.mt.slot * a.H + h) * D + d) * DV + 16 * ct + 8 * g + (lane >> 2);
    s = make_float4(src[0], src[DV], src[8 * DV], src[9 * DV]);
  }
  constexpr int AHEAD = 8;
  at[0] = s;
  for (int c = 1; c < n; c += AHEAD) {
    float4 x[AHEAD];
    float2 f[AHEAD], f8[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < n) {
        const float* r = pr + (size_t)(c + i - 1) * a.H * D;
        x[i] = at[(c + i) * step];
        f[i] = *reinterpret_cast<const float2*>(r);
        f8[i] = *reinterpret_cast<const float2*>(r + 8);
      }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < n) {
        s.x = f[i].x * s.x + x[i].x; s.y = f[i].y * s.y + x[i].y; s.z = f8[i].x * s.z + x[i].z; s.w = f8[i].y * s.w + x[i].w;
        at[(c + i) * step] = s;
      }
  }
}

}  // namespace rmma
}  // namespace qspec
