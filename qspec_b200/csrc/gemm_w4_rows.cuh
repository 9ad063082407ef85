// The products of gemm_w4_stream.cu for few tokens (decoding, drafts, short verification passes): the weights are streamed once and widened
// in registers, straight into the fragments of mma.sync. Included by gemm_w4_stream.cu, which holds the entry points, the rule that chooses
// between the two kernels and the helpers used here.
//
// What bounds these calls is the weight stream and the latency around it. The tcgen05 form needs 58 cycles an instruction whatever the token
// count, a hand-over through tensor memory for each 64 k, and, where there are fewer tiles than SMs, a reduction between CTAs: at 4 tokens
// 8.1 us for 4096 x 4096, whose 8.4 MB of weights take 1.3 us at the HBM rate. At up to 16 tokens mma.sync (2 cycles an SM for 16 x 8 x 16,
// measured, and for 16 x 8 x 32 of int8) needs less time than the stream itself, and its operands can come from registers.
//
//  * A tile is 32 channels. Its k range is cut into items of 256 k; the warps of the CTA take them in turn, each with accumulators for the
//    whole tile, and the sums meet in shared memory once a tile. CTAs walk the tiles: with as many CTAs as fit, every SM holds its share of the
//    stream's bytes under way and no sum crosses CTAs. (Items of 64 channels were 0 to 30 % slower nearly everywhere.)
//  * Every warp owns a ring of slots and refills a slot itself as soon as it has read it: one copy for the item's weights, one for its
//    activations. One warp that issued the copies of all slots took 250 to 350 ns an item: 15.6 us instead of 9.1 for 10240 x 8192. The
//    slots of a ring are of one warp, so that its waits come in the order of the uses.
//  * Operands are read as they lie, without conflicts, because the order of the reduction index is free as long as both agree on it: a thread
//    of a quad takes whole 16- or 8-byte pieces of a 128-byte swizzled row, and the row of a group of eight that a lane holds is chosen such
//    that the lanes of a read meet different banks (ROW_OF). The nibbles of a word leave in the order (0, 4) (1, 5) (2, 6) (3, 7).
//  * The weights of the first items are requested before the preceding kernel's end is waited for, as in the stream form.
// us at 4 / 16 tokens, graph of calls on three to six weights in turn, this form | tcgen05 form:
//   W4A4   4096 x 4096  2.7 / 3.4 |  8.1 /  9.3    28672 x 4096 10.3 / 13.2 | 15.0 / 15.3    4096 x 14336 6.6 /  7.6 | 11.6 / 12.7
//   W4A16  4096 x 4096  3.9 / 4.9 |  9.6 / 10.4    28672 x 4096 14.8 / 20.5 | 23.5 / 24.1    4096 x 14336 8.7 / 10.9 | 15.4 / 16.3
// Errors of the raw W4A16 sums against 64 bits: 9.3e-8 of their norm at K = 14336, 8.3e-8 at 4096 (tcgen05 form: 9.5e-7, 2.1e-7), for the tensor
// cores cut at the accumulator's last bit and an accumulator takes only an item's 256 products; at K <= 512 both are off by 2e-8 to 8e-8.
// Every wait is bounded. A warp gives one up as a whole, stops loading and waits (up to the full limit) for its copies under way; its CTA writes NaN
// (raw sums: the lowest integer or NaN) and counts itself in rows_timeouts.
#pragma once

constexpr int ROWS_R = 32, ROWS_UK = 256;          // channels of a tile, k of an item
constexpr int ROWS_SLOTS = 64;                     // ring slots of a CTA, at most
constexpr int ROWS_MAX_M = 64;
constexpr uint32_t ROWS_SPINS = 1u << 20;
static __device__ unsigned rows_timeouts;          // CTAs that gave a wait up since the library was loaded

struct RowsArgs {
  const void* sA; const void* sW; const void* bias;
  void* out; int32_t* acc_out; uint32_t* split_out;
  int M, N, items, tiles, depth, out_bf16;         // items of a tile; slots of a warp
  int give_up;                                     // tests: every warp gives its first wait up at once
};

// By a whole warp, which goes on or gives up as one: what follows (mma.sync, elect) takes all its lanes. (The vote inside the loop costs nothing, for the
// loop then needs no reconvergence; behind it, W4A16 28672 x 4096, 4 tokens 15.6 -> 16.3 us.)
__device__ __forceinline__ bool rows_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t spins = 0; spins < ROWS_SPINS; ++spins) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (__all_sync(0xffffffffu, done)) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;\n" ::"r"(dst),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "l"(policy) : "memory");
}
__device__ __forceinline__ uint4 rows_lds128(uint32_t a) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
  return r;
}
__device__ __forceinline__ uint2 rows_lds64(uint32_t a) {
  uint2 r;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(r.x), "=r"(r.y) : "r"(a));
  return r;
}
__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// 8 nibbles -> f16 / bf16 pairs (0, 4) (1, 5) (2, 6) (3, 7), exact: 0x6408 ^ n = 1032 + s, 0x6480 ^ (n << 4) = 1152 + 16 s (f16, unit 1);
// 0x4308 ^ n = 136 + s (bf16)
template <bool BF16>
__device__ __forceinline__ void dequant_pairs(uint32_t w, uint32_t (&o)[4]) {
  if (!BF16) {
    const uint32_t h = w >> 8;
    asm("sub.rn.f16x2 %0, %1, %2;\n" : "=r"(o[0]) : "r"(lop3_and_xor(w, 0x000f000fu, 0x64086408u)), "r"(0x64086408u));
    asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(o[1]) : "r"(lop3_and_xor(w, 0x00f000f0u, 0x64806480u)), "r"(0x2C002C00u), "r"(0xD480D480u));
    asm("sub.rn.f16x2 %0, %1, %2;\n" : "=r"(o[2]) : "r"(lop3_and_xor(h, 0x000f000fu, 0x64086408u)), "r"(0x64086408u));
    asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(o[3]) : "r"(lop3_and_xor(h, 0x00f000f0u, 0x64806480u)), "r"(0x2C002C00u), "r"(0xD480D480u));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm("sub.rn.bf16x2 %0, %1, %2;\n" : "=r"(o[i]) : "r"(lop3_and_xor(w >> (4 * i), 0x000f000fu, 0x43084308u)), "r"(0x43084308u));
  }
}
template <int MODE>
__device__ __forceinline__ void rows_mma(uint32_t (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
#define QSPEC_ROWS_MMA(KIND)                                                                                                                \
  asm("mma.sync.aligned." KIND " {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) \
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1))
  if (mode_is_int(MODE)) QSPEC_ROWS_MMA("m16n8k32.row.col.s32.s8.s8.s32");
  else if (MODE == MODE_F16) QSPEC_ROWS_MMA("m16n8k16.row.col.f32.f16.f16.f32");
  else QSPEC_ROWS_MMA("m16n8k16.row.col.f32.bf16.bf16.f32");
#undef QSPEC_ROWS_MMA
}
// Which row of a group of eight the lanes 4 i .. 4 i + 3 hold: a read's 8 (16-byte pieces) or 16 (8-byte pieces) lanes then cover all banks.
template <int MODE>
__device__ __forceinline__ int row_of(int i) { return MODE == MODE_I8 ? i : MODE == MODE_A8 ? (i >> 1) + 4 * (i & 1) : 2 * (i & 3) + (i >> 2); }

template <int MODE, int NT>
struct RowsShape {
  static constexpr int ABOX = MODE == MODE_I8 ? 1 : MODE == MODE_A8 ? 2 : 4;      // 128-byte pieces of a token row in an item
  static constexpr int T = 8 * NT, LD = ROWS_R + 4;
  static constexpr int W_BYTES = ROWS_R * 128, A_BYTES = T * 128 * ABOX, SLOT = W_BYTES + A_BYTES;
};

// NT: groups of 8 tokens; NW: warps; CTAS: CTAs that share an SM
template <int MODE, int NT, int NW, int CTAS>
__global__ void __launch_bounds__(NW * 32, CTAS)
w4_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_act, const RowsArgs p) {
  using Sh = RowsShape<MODE, NT>;
  constexpr bool INT = mode_is_int(MODE), BF16 = MODE == MODE_BF16;
  constexpr int T = Sh::T, LD = Sh::LD, SLOT = Sh::SLOT, RB = ROWS_R / 16;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[ROWS_SLOTS];
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u) + (size_t)warp * p.depth * SLOT;   // this warp's slots
  uint32_t* red = reinterpret_cast<uint32_t*>(ring + (size_t)(NW - warp) * p.depth * SLOT);                           // [NW][T][LD]
  const uint32_t ring0 = smem_u32(ring), bar0 = smem_u32(full + warp * p.depth);
  if (tid == 0) s_fail = 0;

  // This warp's items: k = warp, warp + NW, ... of tile blockIdx.x, then of tile blockIdx.x + gridDim.x, ...
  const int my_tiles = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  int left = warp < p.items ? my_tiles * ((p.items - warp + NW - 1) / NW) : 0;      // not yet requested
  int lk = warp, lt = blockIdx.x;                                                    // next to request
  auto step = [&](int& k, int& tile) { if ((k += NW) >= p.items) { k = warp; tile += gridDim.x; } };
  auto load_w = [&](int s, int k, int tile) {
    mbar_expect_tx(bar0 + 8 * s, SLOT);
    tma_load_2d(ring0 + s * SLOT, &map_w, k * 128, tile * ROWS_R, bar0 + 8 * s, POLICY_EVICT_FIRST);
  };
  auto load_act = [&](int s, int k) {
    const uint32_t dst = ring0 + s * SLOT + Sh::W_BYTES;
    if (Sh::ABOX == 1) tma_load_2d(dst, &map_act, k * 128, 0, bar0 + 8 * s, POLICY_EVICT_LAST);
    else tma_load_3d(dst, &map_act, 0, 0, k * Sh::ABOX, bar0 + 8 * s, POLICY_EVICT_LAST);
  };
  const int pre = min(left, p.depth);
  if (elect_one()) {
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_act);
    for (int s = 0; s < pre; ++s) mbar_init(bar0 + 8 * s, 1);
    fence_mbar_init();
    int k = lk, tile = lt;
    for (int s = 0; s < pre; ++s) { load_w(s, k, tile); step(k, tile); }
  }
  __syncthreads();                                   // s_fail; and this warp's barriers, for its other lanes
  pdl_wait();
  pdl_launch_dependents();
  if (elect_one()) {
    int k = lk, tile = lt;
    for (int s = 0; s < pre; ++s) { load_act(s, k); step(k, tile); }
  }
  __syncwarp();
  for (int s = 0; s < pre; ++s) step(lk, lt);
  left -= pre;

  // The epilogue's thread: one channel (place tid & 31 of the tile), tokens (tid >> 5) + NW j
  constexpr int PER = (T + NW - 1) / NW;
  const int ch_in = (lane & ~7) + row_of<MODE>(lane & 7);
  auto scalar = [&](const void* v, int i) { return p.out_bf16 ? __bfloat162float(((const __nv_bfloat16*)v)[i]) : __half2float(((const __half*)v)[i]); };
  float sa[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) sa[j] = INT && p.out && warp + NW * j < p.M ? scalar(p.sA, warp + NW * j) : 0.f;

  uint32_t acc[RB][NT][4];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[r][n][e] = 0;
  float tot[RB][NT][4] = {};                         // W4A16
  const int rho = row_of<MODE>(g);
  int slot = 0, under_way = pre;
  uint32_t parity = 0;
  bool ok = p.give_up == 0;
  if (!ok) s_fail = 1;
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    const int ch = tile * ROWS_R + ch_in;
    float sw = 0.f, bs = 0.f;                        // requested before the tile's sums are there
    if (p.out && ch < p.N) {
      sw = scalar(p.sW, ch);
      if (p.bias) bs = scalar(p.bias, ch);
    }
    for (int k = warp; k < p.items && ok; k += NW) {
      if (!rows_wait(bar0 + 8 * slot, parity)) { ok = false; s_fail = 1; break; }
      const uint32_t wa = ring0 + slot * SLOT + rho * 128, aa = ring0 + slot * SLOT + Sh::W_BYTES + g * 128;
      if (MODE == MODE_I8) {                         // this thread: bytes 32 t .. 32 t + 31 of every row, weights and activations alike
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t c = (uint32_t)((2 * t + h) ^ g) << 4;
          uint4 x[NT], w[2 * RB];
#pragma unroll
          for (int n = 0; n < NT; ++n) x[n] = rows_lds128(aa + n * 1024 + c);
#pragma unroll
          for (int r = 0; r < 2 * RB; ++r) w[r] = rows_lds128(wa + r * 1024 + c);
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < RB; ++r) {
              const uint32_t u = word(w[2 * r], q), v = word(w[2 * r + 1], q);
#pragma unroll
              for (int n = 0; n < NT; ++n) {
                const uint32_t b = word(x[n], q);
                rows_mma<MODE>(acc[r][n], (u << 4) & 0xf0f0f0f0u, (v << 4) & 0xf0f0f0f0u, u & 0xf0f0f0f0u, v & 0xf0f0f0f0u, (b << 4) & 0xf0f0f0f0u,
                               b & 0xf0f0f0f0u);
              }
            }
        }
      } else if (MODE == MODE_A8) {                  // bytes 64 h + 16 t .. + 15 of a weight row: values 128 h + 32 t .. + 31
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 w[2 * RB];
#pragma unroll
          for (int r = 0; r < 2 * RB; ++r) w[r] = rows_lds128(wa + r * 1024 + ((uint32_t)((4 * h + t) ^ rho) << 4));
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint4 x[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) x[n] = rows_lds128(aa + h * T * 128 + n * 1024 + ((uint32_t)((2 * t + c) ^ g) << 4));
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
              for (int n = 0; n < NT; ++n) {
                const uint32_t even = __byte_perm(word(x[n], 2 * q), word(x[n], 2 * q + 1), 0x6420);
                const uint32_t odd = __byte_perm(word(x[n], 2 * q), word(x[n], 2 * q + 1), 0x7531);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                  const uint32_t u = word(w[2 * r], 2 * c + q), v = word(w[2 * r + 1], 2 * c + q);
                  rows_mma<MODE>(acc[r][n], (u << 4) & 0xf0f0f0f0u, (v << 4) & 0xf0f0f0f0u, u & 0xf0f0f0f0u, v & 0xf0f0f0f0u, even, odd);
                }
              }
          }
        }
      } else {                                       // bytes 32 b + 8 t .. + 7 of a weight row: values 64 b + 16 t .. + 15
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          uint2 w[2 * RB];
#pragma unroll
          for (int r = 0; r < 2 * RB; ++r) w[r] = rows_lds64(wa + r * 1024 + ((uint32_t)((2 * b + (t >> 1)) ^ rho) << 4) + (t & 1) * 8);
#pragma unroll
          for (int c = 1; c >= 0; --c) {
            uint32_t x[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const uint4 y = rows_lds128(aa + b * T * 128 + n * 1024 + ((uint32_t)((2 * t + c) ^ g) << 4));
              x[n][0] = __byte_perm(y.x, y.z, 0x5410);
              x[n][1] = __byte_perm(y.x, y.z, 0x7632);
              x[n][2] = __byte_perm(y.y, y.w, 0x5410);
              x[n][3] = __byte_perm(y.y, y.w, 0x7632);
            }
            uint32_t u[RB][4], v[RB][4];
#pragma unroll
            for (int r = 0; r < RB; ++r) {
              dequant_pairs<BF16>(c ? w[2 * r].y : w[2 * r].x, u[r]);
              dequant_pairs<BF16>(c ? w[2 * r + 1].y : w[2 * r + 1].x, v[r]);
#pragma unroll
              for (int n = 0; n < NT; ++n) rows_mma<MODE>(acc[r][n], u[r][0], v[r][0], u[r][1], v[r][1], x[n][0], x[n][1]);
            }
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
              for (int n = 0; n < NT; ++n) rows_mma<MODE>(acc[r][n], u[r][2], v[r][2], u[r][3], v[r][3], x[n][2], x[n][3]);
          }
        }
      }
      if (!INT) {                                    // sums of 256 products leave the tensor cores, which cut; the rest is added with rounding
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) { tot[r][n][e] = __fadd_rn(tot[r][n][e], __uint_as_float(acc[r][n][e])); acc[r][n][e] = 0; }
      }
      __syncwarp();                                  // every lane has read the slot
      if (left > 0) {
        if (elect_one()) {
          fence_proxy_async_smem();                  // the reads come before the copy's writes
          load_w(slot, lk, lt);
          load_act(slot, lk);
        }
        --left;
        step(lk, lt);
      } else {
        --under_way;
      }
      if (++slot == p.depth) { slot = 0; parity ^= 1u; }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          red[(warp * T + n * 8 + 2 * t + (e & 1)) * LD + r * 16 + g + 8 * (e >> 1)] = INT ? acc[r][n][e] : __float_as_uint(tot[r][n][e]);
          acc[r][n][e] = 0;
          tot[r][n][e] = 0.f;
        }
    __syncthreads();
    const bool fail = s_fail != 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int tok = warp + NW * j;
      if (tok < p.M && ch < p.N) {
        const uint32_t* src = red + tok * LD + lane;
        uint32_t s = src[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) s = INT ? s + src[w * T * LD] : __float_as_uint(__fadd_rn(__uint_as_float(s), __uint_as_float(src[w * T * LD])));
        const size_t o = (size_t)tok * p.N + ch;
        if (p.split_out) {
          p.split_out[o] = !fail ? s : INT ? 0x80000000u : 0x7fffffffu;
        } else if (p.acc_out) {
          p.acc_out[o] = !fail ? ((int32_t)s) >> (MODE == MODE_A8 ? 4 : 8) : (int32_t)0x80000000;
        } else {
          float f = INT ? __fmul_rn(__fmul_rn(__int2float_rn(((int32_t)s) >> (MODE == MODE_A8 ? 4 : 8)), sa[j]), sw) : __fmul_rn(__uint_as_float(s), sw);
          if (p.bias) f = __fadd_rn(f, bs);
          if (fail) f = __uint_as_float(0x7fffffffu);
          if (p.out_bf16) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(f);
          else ((__half*)p.out)[o] = __float2half_rn(f);
        }
      }
    }
    if (tile + (int)gridDim.x < p.tiles) __syncthreads();      // the sums are read before the next tile's are written
  }
  if (!ok) {                                         // nothing of this warp's is left in flight
    for (int i = 0; i < under_way; ++i) {
      rows_wait(bar0 + 8 * slot, parity);
      if (++slot == p.depth) { slot = 0; parity ^= 1u; }
    }
  }
  if (tid == 0 && s_fail) atomicAdd(&rows_timeouts, 1u);
}
