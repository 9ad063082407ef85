// Softmax attention of prompt portions on the fifth-generation tensor cores, head size 128, 16-bit keys and values in a per-sequence
// cache (rows by position, or a ring of `cap` rows), grouped-query heads, an optional window, sink and output gate. Both libraries
// instantiate it: float16 with queries as they lie in the fused projection (attn_kernels.cu), bfloat16 with float32 queries
// (seq_mma_kernels.cu).
//
// One CTA = a tile of 128 query rows of one key/value head; a row is a (token, query head of the group) pair, so that the group's
// heads share every key tile: 32 tokens per CTA at four heads per group. Keys are walked in blocks of 128.
//   * S = Q K^T: both operands from shared memory, accumulator [128 x 128] float32 in tensor memory, two of them: the next block's
//     scores are computed while this block's pass through the softmax.
//   * softmax: thread = half a row (64 columns), two warps per 32 rows, which exchange the row's maximum through shared memory. Weights
//     go back over the scores they came from as a two-term 16-bit split (hi + lo: 22 / 16 mantissa bits, so that the second product is
//     as good as one with float32 weights).
//   * O += P V: weights from tensor memory, values from shared memory as they lie in the cache (the reduction runs over rows: the
//     operand is "MN-major"); hi and lo terms are 8 + 8 instructions on the same value tile. It runs under the next block's softmax. The lo
//     terms have an accumulator of their own: every accumulation cuts at the accumulator's last bit, and half as many of them go to O
//     (sums over 3000 keys whose values cancel: off by 8.0e-9 of the values, 5.6e-8 with one accumulator).
//   * O is rescaled only when a row's maximum grew by more than 2^8 since the last rescale (weights then stay below 256, and the
//     division by the sum at the end undoes the common factor).
// Tensor memory: S0 | S1 | O | O of the lo terms = 512 columns. Warps: 8 softmax, 1 keys, 1 values (TMA), 1 that
// issues the products.
//
// Which tokens: those in RUNS, i.e. neighbours in the batch with one sequence and consecutive positions, of at least min_run
// tokens. A CTA walks the runs of its tokens one after the other (rows of other runs are masked). Tokens outside such runs are left
// to the caller's other kernel (attn_in_run is the common test). Where the caller has a table of segments, the test is the length of the
// token's segment instead, and runs end where segments do.
//
// A row sees nothing but its own keys, bit for bit: hidden keys enter the products with weights of exactly zero, and a row is rescaled by
// its own maximum alone. A weight of zero times a value that is not finite would be NaN: rows with a result that is not finite are computed
// again key by key (attn_rows_again).
//
// Every wait is bounded; a CTA whose wait runs out waits (again with a limit) for its copies and products under way, fills its rows with
// NaN, so that nobody takes what the buffer held for a result, counts itself in attn_tile_timeouts and frees its tensor memory.
#pragma once
#include "common.cuh"
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

namespace qspec {
namespace atile {

constexpr int TOKENS_MAX = 128;                // tokens of a CTA: 128 / heads of a group
constexpr int WARP_K = 8, WARP_V = 9, WARP_MMA = 10;   // warps 0 .. 7: softmax
constexpr int THREADS = 12 * 32;
constexpr int HALF = 128 * 128;                // 128 rows x 64 elements
constexpr int TILE = 2 * HALF;                 // 128 rows x 128 elements
constexpr int KS = 3, VS = 2;                  // key and value blocks in shared memory
constexpr size_t SMEM = (1 + KS + VS) * (size_t)TILE + 1024;   // Q | keys | values | slack to start on a 1024-byte boundary
constexpr float RESCALE_LOG2 = 8.f;
constexpr uint32_t WAIT_SPINS = 1u << 20;

static __device__ unsigned attn_tile_timeouts;  // CTAs of this library's attention kernels that gave a wait up, since it was loaded

struct Args {
  const void* q; long long q_ts, q_hs;         // strides in elements; tokens, heads
  const void* k; long long k_ss; int k_rs, k_hs;   // sequences, rows, heads
  const void* v; long long v_ss; int v_rs, v_hs;
  const int* pos; const int* seq;
  int ntok, nseq, rep, cap, window;            // nseq: sequences the cache holds; a token of another one belongs to no run
  float scale;
  const int* seg;                              // or NULL: [2][ntok] first batch row and end of each token's segment
  int min_run, ring, skip_outside;             // skip_outside: a token whose position is outside the cache is not stored
  void* out; long long out_ts; int out_hs;
  const float* sink; const void* gate; int gate_ld, gate_per_head; float out_scale;
  uint32_t rep_inv;                            // set by launch(): r * rep_inv >> 16 = r / rep for r < 128
};

// Tokens t and t + 1 of the batch are of one run. L2: read past the L1, which only who runs beside the tiles needs (see attn_beside_tiles); the CTAs of
// decode_attention, one per token and head, ask for the same few lines, and waited for each other at the L2 (64 tokens, 32 / 32 heads 20.0 us for 13.9).
template <bool L2>
__device__ __forceinline__ bool attn_link(const int* pos, const int* seq, int ntok, int t) {
  auto at = [](const int* p) { return L2 ? __ldcg(p) : *p; };
  return t >= 0 && t + 1 < ntok && at(seq + t) == at(seq + t + 1) && at(pos + t + 1) == at(pos + t) + 1;
}
// The kernel launched behind attn_tile_kernel for the other tokens starts with this instead of waiting: it looks for its tokens (positions and
// sequences, or the table of segments, from L2) while the tiles run, and calls attn_tiles_done() before it reads anything else, writes, or leaves. The
// tiles let it start only behind their own wait, so what lies in front of them is over by then, and nothing of theirs is read; that it waits at
// all is for the kernels behind it, which wait for it alone.
__device__ __forceinline__ void attn_beside_tiles() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void attn_tiles_done() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// For the 32 tokens t0 .. t0 + 31 of a whole warp, token t0 + lane: is it in a run of at least min_run (<= 16) tokens? `before`, `after`: is
// it linked to its neighbours?
template <bool L2>
__device__ __forceinline__ bool attn_in_run(const int* pos, const int* seq, int ntok, int t0, int min_run, bool& before, bool& after) {
  const int lane = threadIdx.x & 31;
  const uint64_t links = (uint64_t)__ballot_sync(0xffffffffu, attn_link<L2>(pos, seq, ntok, t0 - 16 + lane)) |
                         (uint64_t)__ballot_sync(0xffffffffu, attn_link<L2>(pos, seq, ntok, t0 + 16 + lane)) << 32;   // bit i: token t0 - 16 + i
  const uint64_t left = ~(links << (48 - lane)), right = ~(links >> (16 + lane));
  before = links >> (15 + lane) & 1;
  after = links >> (16 + lane) & 1;
  return 1 + __clzll((long long)left) + (__ffsll((long long)right) - 1) >= min_run && t0 + lane < ntok;
}
// One token, asked by a whole warp.
__device__ __forceinline__ bool attn_token_in_run(const int* pos, const int* seq, int ntok, int t, int min_run) {
  bool x, y;
  return __shfl_sync(0xffffffffu, attn_in_run<false>(pos, seq, ntok, t, min_run, x, y), 0);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory"); }
// false: the wait ran out, here or in another role of the CTA
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  for (uint32_t spins = 0; spins < WAIT_SPINS; ++spins) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if (*fail) return false;
  }
  *fail = 1;
  return false;
}
// For what is under way at the end: waits, as long as any wait, whether or not the CTA has given up.
__device__ __noinline__ void bar_drain(uint32_t bar, uint32_t parity) {
  int none = 0;
  bar_wait(bar, parity, &none);
}
__device__ __forceinline__ bool elect() {
  uint32_t pred;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "elect.sync _|P, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, P;\n"
      "}\n" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// Shared-memory operands, 128-byte swizzle (row r at 128 r, 16-byte chunk c at c ^ (r & 7); groups of eight rows 1024 bytes apart).
// K-major (queries, keys): 64 elements of the reduction per 128-byte row. MN-major (values): the rows ARE the reduction, the second 64
// output columns lie one half-tile (LBO) further.
__device__ __forceinline__ uint64_t desc_k(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((uint32_t)HALF >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <bool BF> __device__ __forceinline__ constexpr uint32_t idesc(bool mn) {   // float32 += T * T, M 128, N 128
  return (1u << 4) | (BF ? (1u << 7) | (1u << 10) : 0u) | (mn ? 1u << 16 : 0u) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap* map, int d, int head, int row, int seq, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n" ::"r"(dst),
               "l"(map), "r"(bar), "r"(d), "r"(head), "r"(row), "r"(seq) : "memory");
}
#define QSPEC_R8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
#define QSPEC_W8(r, o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])
__device__ __forceinline__ void ld32(uint32_t addr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
               "%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
               : QSPEC_R8(r, 0), QSPEC_R8(r, 8), QSPEC_R8(r, 16), QSPEC_R8(r, 24) : "r"(addr));
}
__device__ __forceinline__ void st32(uint32_t addr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
               "%25,%26,%27,%28,%29,%30,%31,%32};\n"
               ::"r"(addr), QSPEC_W8(r, 0), QSPEC_W8(r, 8), QSPEC_W8(r, 16), QSPEC_W8(r, 24) : "memory");
}
__device__ __forceinline__ void ld8(uint32_t addr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n" : QSPEC_R8(r, 0) : "r"(addr));
}
__device__ __forceinline__ void st16(uint32_t addr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(addr), QSPEC_W8(r, 0),
               QSPEC_W8(r, 8) : "memory");
}
#define QSPEC_T8(r, o) "+r"(r[o]), "+r"(r[o + 1]), "+r"(r[o + 2]), "+r"(r[o + 3]), "+r"(r[o + 4]), "+r"(r[o + 5]), "+r"(r[o + 6]), "+r"(r[o + 7])
// Behind wait_ld(): nothing that is done with these registers is moved in front of it.
__device__ __forceinline__ void landed8(uint32_t* r) { asm volatile("" : QSPEC_T8(r, 0)); }
#undef QSPEC_T8
#undef QSPEC_R8
#undef QSPEC_W8
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x)); return y; }
// pairs of float32 in one instruction
__device__ __forceinline__ uint64_t pair(uint32_t a, uint32_t b) { uint64_t r; asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ void unpair(uint64_t v, uint32_t& a, uint32_t& b) { asm("mov.b64 {%0, %1}, %2;\n" : "=r"(a), "=r"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b)); return r; }

// lead(): the leading bits of two weights (bits of float32), rounded and packed, and their values; rest(): two remainders, packed. float16: conversions
// (a scheduler issues one in two cycles; the integer form, seven instructions of which five take two, made a block of 128 keys 1.43 us instead of
// 1.37). bfloat16: integer instructions, of which it takes few (with conversions for the remainders 1.53 us instead of 1.51).
template <bool BF> struct Elem;
template <> struct Elem<false> {
  using T = __half;
  static __device__ __forceinline__ uint32_t pack(float a, float b) { const __half2 h = __floats2half2_rn(a, b); return *reinterpret_cast<const uint32_t*>(&h); }
  static __device__ __forceinline__ float2 unpack(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
  static __device__ __forceinline__ uint32_t lead(uint32_t p0, uint32_t p1, uint32_t& h0, uint32_t& h1) {
    const uint32_t w = pack(__uint_as_float(p0), __uint_as_float(p1));
    const float2 f = unpack(w);
    h0 = __float_as_uint(f.x);
    h1 = __float_as_uint(f.y);
    return w;
  }
  static __device__ __forceinline__ uint32_t rest(uint32_t q0, uint32_t q1) { return pack(__uint_as_float(q0), __uint_as_float(q1)); }
};
template <> struct Elem<true> {
  using T = __nv_bfloat16;
  static __device__ __forceinline__ uint32_t pack(float a, float b) { const __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&h); }
  static __device__ __forceinline__ float2 unpack(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
  static __device__ __forceinline__ uint32_t lead(uint32_t p0, uint32_t p1, uint32_t& h0, uint32_t& h1) {
    p0 += 0x8000u;
    p1 += 0x8000u;
    h0 = p0 & 0xffff0000u;
    h1 = p1 & 0xffff0000u;
    return __byte_perm(p0, p1, 0x7632);
  }
  static __device__ __forceinline__ uint32_t rest(uint32_t q0, uint32_t q1) { return __byte_perm(q0 + 0x8000u, q1 + 0x8000u, 0x7632); }   // rounded
};

// The key blocks of a CTA: for every run the blocks of up to 128 positions from its first visible key to its last.
struct Item { int kb, hi, seq, p0, ts, te; };   // positions kb .. hi, at most 128; the run's tokens and its first position
struct Items {
  const int *rs, *re, *pos, *seq; int nruns, window, last, ring;    // ring: rows of the ring, or 0
  int r = -1, kb = 0, hi = -1;
  __device__ __forceinline__ bool next(Item& it) {
    while (kb > hi) {
      if (++r >= nruns) return false;
      kb = max(0, pos[rs[r]] - window + 1);
      hi = min(pos[re[r]], last);
    }
    int n = 128;
    if (ring) n = min(n, ring - kb % ring);                 // a block ends where the ring does
    it.kb = kb;
    it.hi = min(hi, kb + n - 1);
    kb += n;
    it.ts = rs[r]; it.te = re[r]; it.p0 = pos[it.ts]; it.seq = seq[it.ts];
    return true;
  }
};

// Columns of rows whose tile result is not finite, once more on the CUDA cores: float32 weights, nothing but the row's own keys. (hi and lo
// terms of opposite signs turn an infinite value into NaN, and so does a hidden key's weight of zero.) A whole warp per row, every lane with
// keys of its own. First the row's own values that are not finite: where a column has one, they decide. A column without one was spoilt by a
// key that the row does not see and is summed again.
// rows: the lanes that ask; 64 columns from col0 on of the row that each describes, of which `bad`; f and m: factor and reference of the row's
// weights, as in the kernel.
// 1000 tokens after 1000, 32 / 8 heads, one infinite value that all see in one head / in two columns of every head: whole sums by a thread per
// row 104 / 300 ms, by a warp 10.2 / 19.3, now 1.5 / 3.3; before the tiles 7.7, as any other prompt.
template <bool BF, bool QF32>
__device__ __noinline__ void attn_rows_again(const Args& a, uint32_t rows, int tok_, int head_, int kvh, int seq_, int lo_, int hi_, int col0, uint64_t bad_,
                                             float m_, float f_) {
  using T = typename Elem<BF>::T;
  constexpr uint32_t EXPONENTS = BF ? 0x7f807f80u : 0x7c007c00u;
  const int lane = threadIdx.x & 31;
  __syncwarp();                                               // the rows' lanes have stored them
  for (; rows; rows &= rows - 1u) {
    const int src = __ffs(rows) - 1;
    const int tok = __shfl_sync(0xffffffffu, tok_, src), head = __shfl_sync(0xffffffffu, head_, src), seq = __shfl_sync(0xffffffffu, seq_, src);
    const int lo = __shfl_sync(0xffffffffu, lo_, src), hi = __shfl_sync(0xffffffffu, hi_, src);
    const uint64_t bad = __shfl_sync(0xffffffffu, bad_, src);
    const float mt = __shfl_sync(0xffffffffu, m_, src), ft = __shfl_sync(0xffffffffu, f_, src);
    const T* kbase = (const T*)a.k + (size_t)seq * a.k_ss + (size_t)kvh * a.k_hs;
    const T* vbase = (const T*)a.v + (size_t)seq * a.v_ss + (size_t)kvh * a.v_hs + col0;
    const size_t qo = (size_t)tok * a.q_ts + (size_t)head * a.q_hs;
    auto row = [&](int j) { return a.ring && j >= a.cap ? j % a.cap : j; };
    auto score = [&](int j) {
      const uint4* kr = reinterpret_cast<const uint4*>(kbase + (size_t)row(j) * a.k_rs);
      float s = 0.f;
#pragma unroll 2
      for (int c = 0; c < 16; ++c) {
        const uint4 kw = kr[c];
        const uint32_t kk[4] = {kw.x, kw.y, kw.z, kw.w};
        uint32_t qq[4];
        if (QF32) {
          const float4 x = *reinterpret_cast<const float4*>((const float*)a.q + qo + c * 8), y = *reinterpret_cast<const float4*>((const float*)a.q + qo + c * 8 + 4);
          qq[0] = Elem<BF>::pack(x.x, x.y); qq[1] = Elem<BF>::pack(x.z, x.w); qq[2] = Elem<BF>::pack(y.x, y.y); qq[3] = Elem<BF>::pack(y.z, y.w);
        } else {
          const uint4 w = *reinterpret_cast<const uint4*>((const T*)a.q + qo + c * 8);
          qq[0] = w.x; qq[1] = w.y; qq[2] = w.z; qq[3] = w.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = Elem<BF>::unpack(kk[e]), y = Elem<BF>::unpack(qq[e]);
          s = fmaf(x.y, y.y, fmaf(x.x, y.x, s));
        }
      }
      return s * a.scale;
    };
    auto store = [&](int d, float r) {                        // (a gate per head is in ft)
      if (a.gate && !a.gate_per_head) r *= __fdividef(1.f, 1.f + __expf(-(float)((const T*)a.gate)[(size_t)tok * a.gate_ld + head * a.out_hs + col0 + d]));
      ((T*)a.out)[(size_t)tok * a.out_ts + (size_t)head * a.out_hs + col0 + d] = (T)r;
    };
    float acc[64];
#pragma unroll
    for (int d = 0; d < 64; ++d) acc[d] = 0.f;
    bool found = false;
    for (int j = lo + lane; j <= hi; j += 32) {
      const uint4* vr = reinterpret_cast<const uint4*>(vbase + (size_t)row(j) * a.v_rs);
      uint4 vw[8];
      uint32_t odd = 0u;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        vw[c] = vr[c];
        odd |= __vcmpeq2(vw[c].x & EXPONENTS, EXPONENTS) | __vcmpeq2(vw[c].y & EXPONENTS, EXPONENTS) | __vcmpeq2(vw[c].z & EXPONENTS, EXPONENTS) |
               __vcmpeq2(vw[c].w & EXPONENTS, EXPONENTS);
      }
      if (!odd) continue;
      found = true;
      const float p = ex2(score(j) * 1.4426950408889634f - mt);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint32_t vv[4] = {vw[c].x, vw[c].y, vw[c].z, vw[c].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = Elem<BF>::unpack(vv[e]);
          if (!(fabsf(x.x) < INFINITY)) acc[c * 8 + 2 * e] = fmaf(p, x.x, acc[c * 8 + 2 * e]);
          if (!(fabsf(x.y) < INFINITY)) acc[c * 8 + 2 * e + 1] = fmaf(p, x.y, acc[c * 8 + 2 * e + 1]);
        }
      }
    }
    float mine[2] = {0.f, 0.f};                               // columns 2 lane, + 1
    if (__any_sync(0xffffffffu, found)) {
#pragma unroll
      for (int d = 0; d < 64; ++d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
        if (lane == d >> 1) mine[d & 1] = acc[d];
      }
    }
    bool again[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool ask = bad >> (2 * lane + e) & 1;
      again[e] = ask && mine[e] == 0.f;
      if (ask && !again[e]) store(2 * lane + e, mine[e] * ft);
    }
    if (!__any_sync(0xffffffffu, again[0] || again[1])) continue;
    float m = -INFINITY;
    for (int j = lo + lane; j <= hi; j += 32) m = fmaxf(m, score(j));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (a.sink) m = fmaxf(m, a.sink[head]);
    float l = a.sink && lane == 0 ? __expf(a.sink[head] - m) : 0.f;
#pragma unroll
    for (int d = 0; d < 64; ++d) acc[d] = 0.f;
    for (int j = lo + lane; j <= hi; j += 32) {
      const float p = __expf(score(j) - m);
      l += p;
      const uint4* vr = reinterpret_cast<const uint4*>(vbase + (size_t)row(j) * a.v_rs);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 vw = vr[c];
        const uint32_t vv[4] = {vw.x, vw.y, vw.z, vw.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = Elem<BF>::unpack(vv[e]);
          acc[c * 8 + 2 * e] = fmaf(p, x.x, acc[c * 8 + 2 * e]);
          acc[c * 8 + 2 * e + 1] = fmaf(p, x.y, acc[c * 8 + 2 * e + 1]);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
    for (int d = 0; d < 64; ++d) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
      if (lane == d >> 1) mine[d & 1] = acc[d];
    }
    float gh = a.out_scale / l;
    if (a.gate && a.gate_per_head) gh *= __fdividef(1.f, 1.f + __expf(-(float)((const T*)a.gate)[(size_t)tok * a.gate_ld + head]));
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (again[e]) store(2 * lane + e, mine[e] * gh);
  }
}

template <bool BF, bool QF32>
__global__ void __launch_bounds__(THREADS, 1)
attn_tile_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const Args a) {
  using T = typename Elem<BF>::T;
  extern __shared__ __align__(16) unsigned char at_raw[];
  __shared__ int pos[TOKENS_MAX], seq[TOKENS_MAX];
  __shared__ int s_rs[TOKENS_MAX], s_re[TOKENS_MAX];
  __shared__ uint32_t s_start[TOKENS_MAX / 32];
  __shared__ __align__(8) uint64_t b_kfull[KS], b_kempty[KS], b_vfull[VS], b_vempty[VS], b_q, b_s[2], b_p[2][2], b_o, b_done, b_part, b_mx[4];
  __shared__ float s_mx[2][2][128];                         // [block & 1][half][row]
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rep = a.rep, tok = 128 / rep;                   // tokens per CTA
  const int c0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * tok;   // the longest key ranges of all heads first
  const int kvh = blockIdx.x;
  const int n2 = min(tok, a.ntok - c0);

  // ---- what needs nothing from the kernel before
  if (tid == WARP_K * 32) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_v) : "memory");
    s_fail = 0;
    for (int i = 0; i < KS; ++i) { bar_init(smem_addr(&b_kfull[i]), 1); bar_init(smem_addr(&b_kempty[i]), 1); }
    for (int i = 0; i < VS; ++i) { bar_init(smem_addr(&b_vfull[i]), 1); bar_init(smem_addr(&b_vempty[i]), 1); }
    for (int i = 0; i < 2; ++i) {
      bar_init(smem_addr(&b_s[i]), 1);
      bar_init(smem_addr(&b_p[i][0]), 8); bar_init(smem_addr(&b_p[i][1]), 4);
    }
    bar_init(smem_addr(&b_q), WARP_K);
    bar_init(smem_addr(&b_o), 1);
    bar_init(smem_addr(&b_done), 1);
    bar_init(smem_addr(&b_part), 1);
    for (int i = 0; i < 4; ++i) bar_init(smem_addr(&b_mx[i]), 2);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const uint32_t base = (smem_addr(at_raw) + 1023u) & ~1023u;
  unsigned char* gbase = at_raw + (base - smem_addr(at_raw));
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  // ---- the runs among this CTA's tokens
  bool start = false, end = false;
  if (tid < TOKENS_MAX) {
    const int t = c0 + tid;
    int p = 0, q = 0, s0 = 0, s1 = 0;
    if (tid < n2) {
      p = a.pos[t];
      q = a.seq[t];
      if (a.seg) { s0 = a.seg[t]; s1 = a.seg[a.ntok + t]; }
    }
    bool before, after;
    bool in = attn_in_run<false>(a.pos, a.seq, a.ntok, c0 + warp * 32, a.min_run, before, after) && tid < n2;
    if (a.seg && tid < n2) {
      in = s1 - s0 >= a.min_run;
      before = before && t > s0;
      after = after && t + 1 < s1;
    }
    if (in) {
      pos[tid] = p;
      seq[tid] = q;
      in = (unsigned)q < (unsigned)a.nseq;
    }
    start = in && (tid == 0 || !before);
    end = in && (tid == n2 - 1 || !after);
    const uint32_t bits = __ballot_sync(0xffffffffu, start);
    if (lane == 0) s_start[warp] = bits;
  }
  __syncthreads();
  int nruns = 0, before = 0;
  for (int w = 0; w < TOKENS_MAX / 32; ++w) {
    if (w < warp) before += __popc(s_start[w]);
    nruns += __popc(s_start[w]);
  }
  if (nruns == 0) return;                                    // nothing for this form here
  // Tensor memory only now: a kernel of another library some launches ahead (a product in front of the one that prepares the queries) may have let its
  // dependents start before it held its own, and would wait for columns of a CTA that waits for it. Beside the queries' way here it takes no time.
  if (warp == WARP_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  // ---- queries: asked for here, stored while the first keys are on their way
  constexpr int QP = 128 * 16 / (WARP_K * 32), QW = QF32 ? 2 : 1;   // 16-byte pieces of a thread; loads of each
  uint4 qv[QP][QW];
  if (warp < WARP_K) {
#pragma unroll
    for (int j = 0; j < QP; ++j) {
      const int r = (tid >> 4) + j * (WARP_K * 2), tl = (int)(r * a.rep_inv >> 16);
      const size_t o = (size_t)(c0 + min(tl, n2 - 1)) * a.q_ts + (size_t)(kvh * rep + r - tl * rep) * a.q_hs + (tid & 15) * 8;   // (rows of no token: any)
#pragma unroll
      for (int e = 0; e < QW; ++e) qv[j][e] = *reinterpret_cast<const uint4*>((const unsigned char*)a.q + o * (QF32 ? 4 : 2) + e * 16);
    }
  }
  if (tid < TOKENS_MAX) {                                    // a run's end has as many starts at or before it as its start has
    const int rank = before + __popc(s_start[warp] & ((2u << lane) - 1u)) - 1;
    if (start) s_rs[rank] = tid;
    if (end) s_re[rank] = tid;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s_tmem;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");   // tensor memory is held: a dependent that waits for this grid cannot take it first

  if (warp < WARP_K) {
#pragma unroll
    for (int j = 0; j < QP; ++j) {
      const int r = (tid >> 4) + j * (WARP_K * 2), c = tid & 15, tl = (int)(r * a.rep_inv >> 16);
      uint4 val = qv[j][0];
      if (QF32) {
        const uint4 y = qv[j][QW - 1];
        val = make_uint4(Elem<BF>::pack(__uint_as_float(val.x), __uint_as_float(val.y)), Elem<BF>::pack(__uint_as_float(val.z), __uint_as_float(val.w)),
                         Elem<BF>::pack(__uint_as_float(y.x), __uint_as_float(y.y)), Elem<BF>::pack(__uint_as_float(y.z), __uint_as_float(y.w)));
      }
      if (tl >= n2 || r >= tok * rep) val = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(gbase + (c >> 3) * HALF + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = val;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) bar_arrive(smem_addr(&b_q));
  }

  Items items{s_rs, s_re, pos, seq, nruns, a.window, a.ring ? 0x7fffffff - 256 : a.cap - 1, a.ring ? a.cap : 0};
  Item it;
  if (warp == WARP_MMA) {
    if (elect()) {
      const uint32_t id_s = idesc<BF>(false), id_o = idesc<BF>(true), o = tmem + 256, bo = smem_addr(&b_o);
      const uint64_t qd = desc_k(base);
      uint32_t blocks = 0;
      while (items.next(it)) ++blocks;
      uint32_t ks = 0, kphase = 0;                            // key stage of the next scores
      auto scores = [&](uint32_t n) -> bool {
        if (!bar_wait(smem_addr(&b_kfull[ks]), kphase, &s_fail)) return false;
        // these scores take the columns of the weights of block n - 2: their product must be over
        if (n >= 2 && !bar_wait(bo, n & 1, &s_fail)) return false;
        fence_after();
        const uint64_t kd = desc_k(base + (1 + ks) * TILE);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t step = (uint32_t)((i >> 2) * (HALF >> 4) + (i & 3) * 2);
          mma_ss(tmem + (n & 1) * 128, qd + step, kd + step, id_s, i ? 1u : 0u);
        }
        commit(smem_addr(&b_s[n & 1]));
        commit(smem_addr(&b_kempty[ks]));
        if (++ks == KS) { ks = 0; kphase ^= 1u; }
        return true;
      };
      bool ok = blocks == 0 || (bar_wait(smem_addr(&b_q), 0, &s_fail) && scores(0)), over = blocks == 0;
      for (uint32_t n = 0; ok && n < blocks; ++n) {
        if (n + 1 < blocks && !scores(n + 1)) break;
        if (!bar_wait(smem_addr(&b_vfull[n % VS]), (n / VS) & 1, &s_fail)) break;
        const uint64_t vd = desc_mn(base + (1 + KS + n % VS) * TILE);
        const uint32_t p = tmem + (n & 1) * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                         // 64 keys each
          ok = ok && bar_wait(smem_addr(&b_p[n & 1][h]), (n >> 1) & 1, &s_fail);
          if (!ok) break;
          fence_after();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t v = vd + (h * 4 + i) * (2048 >> 4);
            mma_ts(o, p + h * 64 + i * 8, v, id_o, (n | h | i) ? 1u : 0u);
            mma_ts(o + 128, p + h * 64 + 32 + i * 8, v, id_o, (n | h | i) ? 1u : 0u);
          }
        }
        if (!ok) break;
        commit(bo);
        if (n + 1 == blocks) { commit(smem_addr(&b_done)); over = true; }
        commit(smem_addr(&b_vempty[n % VS]));
      }
      if (!over) commit(smem_addr(&b_done));                   // given up: the products issued so far
      if (blocks) bar_drain(smem_addr(&b_done), 0);
    }
    __syncwarp();
  } else if (warp == WARP_K || warp == WARP_V) {
    // ---- key rows or value rows: two boxes of 128 rows x 64 elements per block (rows past the cache arrive as zeros)
    const bool keys = warp == WARP_K;
    uint64_t* full = keys ? b_kfull : b_vfull;
    uint64_t* empty = keys ? b_kempty : b_vempty;
    const CUtensorMap* map = keys ? &map_k : &map_v;
    const uint32_t buf = base + (keys ? 1 : 1 + KS) * TILE;
    const int stages = keys ? KS : VS;
    int stage = 0;
    uint32_t phase = 1;                                       // of the stage's previous release: none to wait for in the first round
    bool ok = true;
    int parts = 0, n = 0;
    for (; items.next(it); ++n) {
      if (n >= stages) ok = bar_wait(smem_addr(&empty[stage]), phase, &s_fail);
      if (!__all_sync(0xffffffffu, ok)) break;
      // value rows past the block's last key are cleared before the products see them (their weights are zero, but zero times NaN is not):
      // such a block lands on a barrier of its own first
      const int have = it.hi - it.kb + 1;
      const bool part = !keys && have < 128;
      const uint32_t bar = smem_addr(part ? &b_part : &full[stage]), dst = buf + stage * TILE;
      if (elect()) {
        const int row = a.ring ? it.kb % a.cap : it.kb;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((uint32_t)TILE) : "memory");
        tma_rows(dst, map, 0, kvh, row, it.seq, bar);
        tma_rows(dst + HALF, map, 64, kvh, row, it.seq, bar);
      }
      __syncwarp();
      if (part) {
        ok = bar_wait(bar, (uint32_t)(parts & 1), &s_fail);
        if (!__all_sync(0xffffffffu, ok)) {
          bar_drain(bar, (uint32_t)(parts & 1));
          break;
        }
        ++parts;
        unsigned char* rows = gbase + (dst - base);
        for (int i = have * 8 + lane; i < 128 * 8; i += 32) {
          *reinterpret_cast<uint4*>(rows + i * 16) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(rows + HALF + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(smem_addr(&full[stage]));
      }
      if (++stage == stages) { stage = 0; phase ^= 1u; }
    }
    // blocks 0 .. n - 1 were asked for: the CTA does not leave before the last of each stage has landed
    for (int j = max(0, n - stages); j < n; ++j) bar_drain(smem_addr(&full[j % stages]), (uint32_t)(j / stages) & 1u);
  } else if (warp < WARP_K) {
    // ---- softmax: thread = 64 columns (half h) of row r
    const int h = warp >> 2, r = (warp & 3) * 32 + lane;
    const int tl = (int)(r * a.rep_inv >> 16), head = kvh * rep + r - tl * rep;
    const bool row_in = r < tok * rep && tl < n2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ot = tmem + lanes + 256 + h * 64;
    const uint32_t bmx = smem_addr(&b_mx[warp & 3]);
    const float c2 = a.scale * 1.4426950408889634f;
    const int last = a.ring ? 0x7fffffff : a.cap - 1;
    const float sink = a.sink && row_in ? a.sink[head] * 1.4426950408889634f : 0.f;
    float m = -INFINITY, l = 0.f;                             // maximum in units of log2; sum of this half's weights relative to it
    int n = 0, my_lo = 0, my_hi = -1, my_seq = 0;
    bool ok = true, mine = false;
    while (ok && items.next(it)) {
      const bool in = row_in && tl >= it.ts && tl <= it.te;
      // visible columns of the half block: j0 .. j0 + span
      int j0 = 0x7fff, span = 0;
      if (in) {
        const int pr = it.p0 + (tl - it.ts);
        const int vlo = max(0, pr - a.window + 1);
        int vhi = min(pr, last);
        mine = true; my_lo = vlo; my_hi = vhi; my_seq = it.seq;
        vhi = min(vhi, it.hi);
        if (vhi >= vlo) { j0 = vlo - it.kb - h * 64; span = vhi - vlo; }
      }
      const bool whole = !row_in || (j0 <= 0 && j0 + span >= 63);   // (rows that stand for no token are never stored)
      const bool plain = __all_sync(0xffffffffu, whole);
      const uint32_t st = tmem + lanes + (n & 1) * 128 + h * 64;
      ok = bar_wait(smem_addr(&b_s[n & 1]), (uint32_t)((n >> 1) & 1), &s_fail);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fence_after();
      uint32_t x[64];
      ld32(st, x);
      ld32(st + 32, x + 32);
      wait_ld();
      if (!plain) {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if ((uint32_t)(j - j0) > (uint32_t)span) x[j] = 0xff800000u;      // hidden
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 64; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(x[j]));
      const float mine_mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      s_mx[n & 1][h][r] = mine_mx;
      __syncwarp();
      if (lane == 0) bar_arrive(bmx);
      ok = bar_wait(bmx, (uint32_t)(n & 1), &s_fail);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const float mn = fmaxf(m, fmaxf(mine_mx, s_mx[n & 1][1 - h][r]) * c2);
      // (both warps of the rows see the same maxima and decide alike)
      const bool grown = mn > m + RESCALE_LOG2 || (m == -INFINITY && mn > m);
      if (__any_sync(0xffffffffu, grown)) {
        const float f = grown ? ex2(m - mn) : 1.f;             // 0 for a row that had seen nothing; other rows of the warp keep theirs
        if (grown) m = mn;
        l *= f;
        if (n) {
          ok = bar_wait(smem_addr(&b_o), (uint32_t)((n - 1) & 1), &s_fail);   // the previous block's product is in O
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          fence_after();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t at = ot + (q >> 1) * 128 + (q & 1) * 32;
            uint32_t o[32];
            ld32(at, o);
            wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
            st32(at, o);
          }
          wait_st();
        }
      }
      // The product of the first 64 keys adds to all columns of O, those of the second half's warps among them: b_p[.][0] counts their
      // rescale, done or not needed, beside the first half's weights.
      if (h) {
        fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(smem_addr(&b_p[n & 1][0]));
      }
      const float mu = m == -INFINITY ? 0.f : m;
      const uint64_t c22 = pair(__float_as_uint(c2), __float_as_uint(c2)), mu2 = pair(__float_as_uint(-mu), __float_as_uint(-mu));
      const uint64_t minus2 = pair(0xbf800000u, 0xbf800000u);
      uint64_t l2[2] = {0ull, 0ull};
      // weight = hi + lo: hi = the leading bits that the type keeps, rounded, lo = the rest, rounded
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          uint32_t p0, p1, h0, h1, q0, q1;
          unpair(fma2(pair(x[g * 32 + 2 * j], x[g * 32 + 2 * j + 1]), c22, mu2), p0, p1);
          p0 = __float_as_uint(ex2(__uint_as_float(p0)));
          p1 = __float_as_uint(ex2(__uint_as_float(p1)));
          const uint64_t pp = pair(p0, p1);
          l2[j & 1] = add2(l2[j & 1], pp);
          hi[j] = Elem<BF>::lead(p0, p1, h0, h1);
          unpair(fma2(pair(h0, h1), minus2, pp), q0, q1);
          lo[j] = Elem<BF>::rest(q0, q1);
        }
        st16(st + g * 16, hi);
        st16(st + 32 + g * 16, lo);
      }
      wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(smem_addr(&b_p[n & 1][h]));
      {
        uint32_t a0, a1;
        unpair(add2(l2[0], l2[1]), a0, a1);
        l += __uint_as_float(a0) + __uint_as_float(a1);
      }
      ++n;
    }
    // ---- the last product is done: add the halves' sums, divide, gate, store. Rows leave through shared memory, eight lanes a row: a lane per row
    // touched 32 rows with every instruction (2 us a tile, 5 with a gate's loads). The loops are short: what runs once per tile runs at the speed at
    // which its instructions are fetched. This, and queries that are on their way beside the first keys: 1000 tokens after 1000,
    // 32 / 8 heads 63.5 -> 56.5 us, window of 1024, 2000 tokens, 16 / 4 heads, with gate and sink 66.8 -> 55.5.
    const int pc8 = lane & 7;                                 // this lane's rows of the warp's 32 are lane / 8 + 4 k, its eight columns of 64 from 8 pc8 on
    auto row_at = [&](int k, size_t ts, int hs) {             // where that row's half lies in a [token][head][..] tensor
      const int rr = (warp & 3) * 32 + (lane >> 3) + 4 * k, t = (int)(rr * a.rep_inv >> 16);
      return (size_t)(c0 + min(t, n2 - 1)) * ts + (size_t)(kvh * rep + rr - t * rep) * hs + h * 64 + pc8 * 8;
    };
    constexpr int LD = 68;                                    // floats of a row, so that neither side meets bank conflicts
    float* const rows = reinterpret_cast<float*>(gbase) + warp * 32 * LD;   // (queries and keys are done with, the gates lie behind the rows)
    unsigned char* const gates = gbase + 3 * TILE + warp * 4096;
    static_assert(8 * 32 * LD * 4 <= 3 * TILE && 8 * 4096 <= TILE && KS >= 3, "rows and gates on their way");
    const bool gate = a.gate && !a.gate_per_head && ok;
    if (gate) {
#pragma unroll 1
      for (int k = 0; k < 8; ++k)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(gates + k * 512 + lane * 16)), "l"((const T*)a.gate + row_at(k, a.gate_ld, a.out_hs)) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    // (A barrier of its own: a warp may get here two products ahead, where the parity of b_o's phase n - 3 reads like that of n - 1.)
    // Without a block nothing has read the queries, and other warps may still be storing theirs where the rows go: then those are waited for.
    if (ok) ok = bar_wait(n ? smem_addr(&b_done) : smem_addr(&b_q), 0, &s_fail);
    ok = __all_sync(0xffffffffu, ok);
    fence_after();
    s_mx[n & 1][h][r] = l;
    __syncwarp();
    if (lane == 0) bar_arrive(bmx);
    if (ok) ok = bar_wait(bmx, (uint32_t)(n & 1), &s_fail);
    ok = __all_sync(0xffffffffu, ok);
    l += s_mx[n & 1][1 - h][r];
    // `mine` rows belong to a run; one whose position shows it no key is stored as zeros, or not at all (skip_outside)
    if (row_in && !mine) {                                    // a run none of whose keys lie in the cache produced no block
      for (int q = 0; q < nruns; ++q)
        if (tl >= s_rs[q] && tl <= s_re[q]) mine = true;
    }
    const int pr = row_in && mine ? pos[tl] : 0;
    const bool store = ok && row_in && mine && !(a.skip_outside && (unsigned)pr >= (unsigned)a.cap);
    // No key had a weight: none was visible, or every score was -inf. As in the kernels beside this one: 0 / 0 in the window form without
    // a sink and in decode_attention, zeros otherwise.
    const bool dead = l == 0.f;
    const float none = (a.ring && !a.sink) || a.skip_outside ? __int_as_float(0x7fffffff) : 0.f;
    float f = 0.f;
    if (!dead) {
      float mm = m, ls = l;
      if (a.sink && row_in) {
        mm = fmaxf(m, sink);
        ls = l * ex2(m - mm) + ex2(sink - mm);
      }
      f = ex2(m - mm) / ls * a.out_scale;
    }
    if (a.gate && a.gate_per_head && store)
      f *= __fdividef(1.f, 1.f + __expf(-(float)((const T*)a.gate)[(size_t)(c0 + tl) * a.gate_ld + head]));
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (ok) {
      float spoilt = 0.f;                                     // not a number where a column is not finite
#pragma unroll 1
      for (int q = 0; q < 8; ++q) {
        uint32_t o[8], low[8];
        ld8(ot + q * 8, o);
        ld8(ot + 128 + q * 8, low);
        wait_ld();
        landed8(o);
        landed8(low);
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          v[e] = dead ? none : (__uint_as_float(o[e]) + __uint_as_float(low[e])) * f;
          spoilt = fmaf(v[e], 0.f, spoilt);
        }
        *reinterpret_cast<float4*>(rows + lane * LD + q * 8) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(rows + lane * LD + q * 8 + 4) = make_float4(v[4], v[5], v[6], v[7]);
      }
      const uint32_t stored = __ballot_sync(0xffffffffu, store);
      __syncwarp();                                           // the rows are there (a vote orders no memory); every lane reads the gates that it asked for
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        const int rr = (lane >> 3) + 4 * k;
        const float4 x = *reinterpret_cast<const float4*>(rows + rr * LD + pc8 * 8), y = *reinterpret_cast<const float4*>(rows + rr * LD + pc8 * 8 + 4);
        float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        if (gate) {
          const uint4 gw = *reinterpret_cast<const uint4*>(gates + k * 512 + lane * 16);
          const uint32_t ww[4] = {gw.x, gw.y, gw.z, gw.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 z = Elem<BF>::unpack(ww[e]);
            v[2 * e] *= __fdividef(1.f, 1.f + __expf(-z.x));
            v[2 * e + 1] *= __fdividef(1.f, 1.f + __expf(-z.y));
          }
        }
        if (stored >> rr & 1)
          *reinterpret_cast<uint4*>((T*)a.out + row_at(k, a.out_ts, a.out_hs)) =
              make_uint4(Elem<BF>::pack(v[0], v[1]), Elem<BF>::pack(v[2], v[3]), Elem<BF>::pack(v[4], v[5]), Elem<BF>::pack(v[6], v[7]));
      }
      uint64_t bad = 0;                                       // columns that are not finite
      if (__any_sync(0xffffffffu, !(spoilt == 0.f) && store)) {
        for (int q = 0; q < 64; ++q)
          if (!(fabsf(rows[lane * LD + q]) < INFINITY)) bad |= 1ull << q;
      }
      // (a sum of weights that is not a number makes every column so: nothing to do again)
      const uint32_t again = __ballot_sync(0xffffffffu, bad != 0 && store && !dead && l == l);
      if (again) attn_rows_again<BF, QF32>(a, again, c0 + tl, head, kvh, my_seq, my_lo, my_hi, h * 64, bad, m, f);
    }
  }
  fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
  }
  if (s_fail) {                                               // (written before the barrier: uniform)
    if (tid == 0) atomicAdd(&attn_tile_timeouts, 1u);
    for (int q = 0; q < nruns; ++q)
      for (int i = s_rs[q] * rep * 16 + tid; i < (s_re[q] + 1) * rep * 16; i += THREADS) {
        const int tl = i / (rep * 16), head = kvh * rep + i / 16 % rep;
        if (a.skip_outside && (unsigned)pos[tl] >= (unsigned)a.cap) continue;
        *reinterpret_cast<uint4*>((T*)a.out + (size_t)(c0 + tl) * a.out_ts + (size_t)head * a.out_hs + (i & 15) * 8) =
            make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
      }
  }
}

// Heads per group that fit, positive scale (a row's maximum is the scaled maximum), rows on 16-byte boundaries.
inline bool supported(const Args& a, int elem_q) {
  auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  auto rows = [](long long ss, int rs, int hs) { return ss > 0 && rs > 0 && hs > 0 && ss % 8 == 0 && rs % 8 == 0 && hs % 8 == 0; };
  return a.rep >= 1 && a.rep <= 64 && a.ntok / (128 / a.rep) < 65535 && a.scale > 0.f && al(a.q) && al(a.k) && al(a.v) && al(a.out) && a.q_ts * elem_q % 16 == 0 &&
         a.q_hs * elem_q % 16 == 0 && rows(a.k_ss, a.k_rs, a.k_hs) && rows(a.v_ss, a.v_rs, a.v_hs) && a.out_ts % 8 == 0 && a.out_hs % 8 == 0 &&
         (!a.gate || a.gate_per_head || (al(a.gate) && a.gate_ld % 8 == 0));
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// [sequence][row][head][128] with the caller's strides; a box is 128 rows x 64 elements of one head
template <bool BF>
inline int cache_map(CUtensorMap* map, const void* p, long long ss, int rs, int hs, int heads, int rows, int nseq) {
  static const EncodeTiled fn = []() -> EncodeTiled {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeTiled)f : nullptr;
  }();
  QSPEC_REQUIRE(fn, QSPEC_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  const cuuint64_t dims[4] = {128, (cuuint64_t)heads, (cuuint64_t)rows, (cuuint64_t)nseq};
  const cuuint64_t strides[3] = {(cuuint64_t)hs * 2, (cuuint64_t)rs * 2, (cuuint64_t)ss * 2};
  const cuuint32_t box[4] = {64, 1, 128, 1}, unit[4] = {1, 1, 1, 1};
  const CUresult r = fn(map, BF ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(p), dims, strides, box, unit,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QSPEC_REQUIRE(r == CUDA_SUCCESS, QSPEC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d): %d rows, %d sequences", (int)r, rows, nseq);
  return QSPEC_OK;
}

template <bool BF, bool QF32>
inline int launch(Args a, int kv_heads, cudaStream_t stream) {
  a.rep_inv = (65536u + (uint32_t)a.rep - 1u) / (uint32_t)a.rep;   // (rep <= 64: the quotient is off by less than 128 / 65536, which no r reaches the next one by)
  auto kern = attn_tile_kernel<BF, QF32>;
  static SmemLimit limit;
  QSPEC_CUDA(limit.raise(kern, SMEM));
  CUtensorMap mk, mv;
  const int nseq = a.nseq < (1 << 20) ? a.nseq : 1 << 20;     // (a caller that does not know their number: nothing is cut off)
  int rc = cache_map<BF>(&mk, a.k, a.k_ss, a.k_rs, a.k_hs, kv_heads, a.cap, nseq);
  if (rc == QSPEC_OK) rc = cache_map<BF>(&mv, a.v, a.v_ss, a.v_rs, a.v_hs, kv_heads, a.cap, nseq);
  if (rc != QSPEC_OK) return rc;
  const int per = 128 / a.rep;
  launch_pdl(kern, dim3(kv_heads, (a.ntok + per - 1) / per), dim3(THREADS), SMEM, stream, mk, mv, a);
  QSPEC_CHECK_LAUNCH(1);
  return QSPEC_OK;
}

}  // namespace atile
}  // namespace qspec
