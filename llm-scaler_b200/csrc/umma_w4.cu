// Weight-only GEMM on tcgen05 for fp16 activations: out[tok, n] = sum_k x[tok, k] * W[n, k], W INT4 (group 128, behind the
// activation pre-pass) or e4m3 (dense: block-scaled up to 64 tokens, any scales above where its 128-token tiles pay; grouped:
// one scale per channel or tensor, tiles of up to 64 tokens).
//
// Swap-AB: strips of R x 128 weight rows are the MMA's M dimension, a tile of TOK tokens its N dimension.  The nibbles are
// decoded to fp16 in registers and written straight into tensor memory as the MMA's A operand (no trip back through
// shared memory); the activations arrive as fp16, scaled per token by a power of two and permuted into the decode's
// nibble order by act_prep.  One persistent CTA per SM walks a list of segments = (tile, strip, range of k):
//   warp 0        TMA producer of raw weight stages (R x 128 rows x 256 k): the HBM stream, up to RS stages ahead
//   warp 1        tensor-memory owner, issues tcgen05.mma
//   warp 2        TMA producer of activation stages [TOK x 128 or 256 k]
//   warp 3        fetches the group scales into shared memory, eight groups of every row at a time
//   next EW       epilogue: tensor memory -> out, or partial sums of a strip that several CTAs share
//   next 16       transform: raw nibbles -> fp16 operand in tensor memory
// Why these roles.  With the transform warps also fetching scales and draining accumulators, every segment change stopped
// the stream: measured inside the predecessor of this kernel (gate_up 57344 x 8192, 64 tokens), 9 us passed between the
// last conversion of one segment and the first of the next (scale fetch from DRAM, drain, partial sums), and a cut
// strip's reduction took 7 to 12 us; taking decode, MMA and activation traffic out of it altogether changed 98 us to 89.
// Here drain, partial sums and scale fetches of one segment run under the stream of the next.
//
// R = 2 lets 256 weight rows share an activation tile: the SMs pull operands out of L2 at 9.4 to 10 TB/s in every GEMM of
// this package, which is what bounds wide tiles.  Per 128 x 128 x 64 of work a 256 x 128 tile pulls 12 KB, a 128 x 256
// tile 18 KB, a 128 x 128 tile 20 KB.
//
// Every mbarrier wait is bounded; on expiry the CTA records a code in the status word, frees its tensor memory and ends.
//
// Reference counterparts: GEMM_int4_pgrp_kernel (csrc/xpu/esimd_kernels/int4_GEMM.h:81-270),
// moe_prefill_up/down_forward_kernel (csrc/moe_prefill/moe_prefill_int4.sycl:121-395).
#include "umma_gemm.cuh"
#include "sm100.cuh"
#include "arrivals.cuh"
#include "smallm.cuh"   // lds128
#include "peer_reduce.cuh"

namespace b2q {

using namespace sm100;

namespace w4 {
enum { ST_XFULL = 501, ST_AFULL = 502, ST_EMPTY = 503, ST_RAWFULL = 504, ST_RAWEMPTY = 505, ST_ACCUM = 506, ST_ACCEMPTY = 507,
       ST_FIXUP = 508, ST_SCFULL = 510, ST_SCEMPTY = 511, ST_XEMPTY = 512, ST_SCALERANGE = 109 };

// constants of the fp16 magic-number nibble decode, handed to the kernel as parameters (see w4_word_magic)
struct MagicConsts { uint32_t magic_lo, magic_hi, m72; };
// twos: the nibbles are two's complement (value, not value + 8).  Flipping their sign bits gives the offset form; the
// flip is folded into the constant that is merged in: (w & m) ^ (0x6400 ^ flip) is 0x6400 | ((w ^ flip) & m) because
// the 0x6400 bits and the nibble bits do not overlap.  No extra operation, no branch in the decode.
inline MagicConsts magic_consts(bool twos) {
  return MagicConsts{0x64006400u ^ (twos ? 0x00080008u : 0u), 0x64006400u ^ (twos ? 0x00800080u : 0u), 0xD480D480u};
}

enum { WT_W4N = 0, WT_W4K = 1, WT_W8 = 2 };          // N-major nibbles, K-major nibbles, e4m3 with a scale per 128 x 128 block

template <int WT, int TOK, int R> struct Cfg {
  static constexpr int NG = 4, KG = NG / R;                  // transform groups of four warps; of these, groups along k
  static constexpr int EW = TOK >= 64 ? 8 : 4;               // epilogue warps
  static constexpr int CW = 4;                               // control warps
  static constexpr int THREADS = (CW + EW + NG * 4) * 32;
  static constexpr int ROWS = R * 128;
  // Every barrier wait costs the issuing thread about 125 cycles even when the phase is long over, every commit about 90
  // (clock() around them): with operand and activation stages of 64 k it spent 490 cycles per 64 k of a 128-row strip,
  // and the transform warps waited two thirds of their time for it.  So an operand stage is a whole scale group (128 k)
  // and an activation stage 256 k where shared memory allows.
  static constexpr int GPS = WT == WT_W8 ? 1 : 2;            // scale groups (128 k) per raw stage of 128 bytes a row
  static constexpr int XC = (R == 1 && TOK <= 64) ? 2 * GPS : 2;   // 64-k chunks per activation stage
  static constexpr int X_BYTES = TOK * 128 * XC;
  static constexpr int XS = TOK == 128 ? 3 : (R == 2 ? 6 : (TOK == 64 ? 6 : 8) / GPS);
  static constexpr int RAW_BYTES = R * 16384;
  static constexpr int SCS = 4, SC_GROUPS = 8, SC_BYTES = WT == WT_W8 ? 0 : SC_GROUPS * ROWS * 2;   // scale slots: [row][group] 16-bit
  static constexpr int POST_RING = 16;                       // row exponents per segment, read by the epilogue
  static constexpr int POST_BYTES = POST_RING * ROWS;
  static constexpr int STAGE_OUT = EW * 1024;                // 16 tokens x 32 columns of output per epilogue warp
  static constexpr int TILE_TABLE = 32;                      // segments of a grouped launch whose tile every role finds in shared memory
  static constexpr int BUDGET = 232448 - 1024 /*align*/ - 1024 /*barriers*/ - TILE_TABLE * 16;
  static constexpr int RS_FIT = (BUDGET - XS * X_BYTES - SCS * SC_BYTES - POST_BYTES - STAGE_OUT) / RAW_BYTES;
  // Raw and operand stages always belong to the same transform group(s), whatever segment they are in: a wait tells a
  // phase from the one after it, not from the one after that, so nobody may wait for a stage whose previous use was
  // somebody else's.  Hence ring depths in multiples of a round of the groups.
  static constexpr int RAW_ROUND = KG / GPS, A_ROUND = KG;
  static constexpr int RS = (RS_FIT > 12 ? 12 : RS_FIT) / RAW_ROUND * RAW_ROUND;
  static constexpr int SMEM = XS * X_BYTES + RS * RAW_BYTES + SCS * SC_BYTES + POST_BYTES + STAGE_OUT + 1024 + 1024 + TILE_TABLE * 16;
  static constexpr int ACC_COLS = TOK < 32 ? 32 : TOK;
  static constexpr int NBUF = 2 * R * ACC_COLS <= 256 ? 2 : 1;   // accumulator sets
  static constexpr int A_COL0 = NBUF * R * ACC_COLS;
  // operand stages of 128 k (R x 64 columns each) fill the rest of tensor memory
  static constexpr int S = (512 - A_COL0) / (64 * R) / A_ROUND * A_ROUND;
  static_assert(S >= A_ROUND && RS >= 3, "ring depths");
};
}  // namespace w4

struct W4Params {
  const void* scale; int scale_dtype; int64_t s_stride_n, s_stride_g, s_expert_elems;
  int scale_mode;            // e4m3 weights: B2Q_SCALE_*; without blocks the epilogue multiplies by the scale
  int scale_vec;             // a row's 16-bit scales can be fetched eight groups (8) or two groups (2) per aligned load; else 1
  void* out; int64_t ldo; int out_bf16;
  int vec_out;               // rows of out are 16-byte aligned
  int M, N, K;
  int nk;                    // 64-k chunks of a whole strip, rounded up to whole raw stages (what lies beyond K multiplies by zero)
  int strips, tiles_n;       // strips of R * 128 rows; token tiles of a dense launch
  int sps, units;            // cut strips: raw stages per strip and in total (0 = whole strips)
  float* partials;           // [2 * grid][R][TOK / 4][128][4] fp32 partial sums of cut strips
  Arrivals* arrivals; Arrivals tag; const Arrivals* epoch;      // [strips], in the partial sums' last slot (see cut_strips)
  const int32_t* tiles; const int32_t* expert_offsets; const int32_t* out_map;
  int w_rows_per_expert;     // tensor-map rows per expert: N (N-major) or K/8 (K-major)
  const float* tok_scale;    // per-token output multiplier (undoes the activation pre-scale)
  w4::MagicConsts mk;
  int* status;
  int peer_on; PeerEpilogue peer;
};

namespace w4 {
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {       // the rest of the four bytes is zeroed
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// One arrival on the barrier when all copies this thread has issued have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// Waits for every copy this thread has issued.
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Power of two that brings a scale into [0.5, 1) (0 for zero, subnormal, infinite and NaN scales).
__device__ __forceinline__ int row_exponent(float first) {
  const int ex = (int)((__float_as_uint(first) >> 23) & 0xFFu);
  return (ex == 0 || ex == 255) ? 0 : max(-120, min(120, 126 - ex));
}
// fp16 bits of a decode factor; 8 * factor must stay below fp16's largest value: saturate, and say so
__device__ __forceinline__ uint32_t fp16_factor(float f, int& saturated) {
  if (fabsf(f) > 8188.f) { f = copysignf(8188.f, f); saturated = 1; }
  return (uint32_t)__half_as_ushort(__float2half_rn(f));
}

__device__ __forceinline__ uint32_t and_xor_lo(uint32_t a, uint32_t c) {      // (a & 0x000F000F) ^ c: the mask as an immediate, c in a register
  uint32_t d;
  asm("lop3.b32 %0, %1, 0x000F000F, %2, 0x6A;" : "=r"(d) : "r"(a), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t and_xor_hi(uint32_t a, uint32_t c) {      // (a & 0x00F000F0) ^ c
  uint32_t d;
  asm("lop3.b32 %0, %1, 0x00F000F0, %2, 0x6A;" : "=r"(d) : "r"(a), "r"(c));
  return d;
}
// One word of eight nibbles -> eight fp16 values (q - 8) * s, each rounded once.  0x6400 | q is 1024 + q and
// 0x6400 | (q << 4) is 1024 + 16 q, so the nibbles at bits 0-3 / 4-7 of each half-word need no shift; one shift by 8
// reaches the other four.  Output pair order: (n0,n4) (n1,n5) (n2,n6) (n3,n7) where n_i is the nibble at bits 4i; the
// activation pre-pass stores x in the matching order.  An instruction takes ONE immediate: the masks, 1032 and 1/16 are
// literals, the merge constants (which depend on the nibble encoding) and -72 come in registers; with all of them as
// literals the compiler spends two logic operations per mask-and-merge.
__device__ __forceinline__ void w4_word_magic(uint32_t w, uint32_t s2, const MagicConsts& k, uint32_t* o) {
  const uint32_t w8 = w >> 8;
  uint32_t v[4] = {and_xor_lo(w, k.magic_lo), and_xor_hi(w, k.magic_hi), and_xor_lo(w8, k.magic_lo), and_xor_hi(w8, k.magic_hi)};
  const __half2 sc = *reinterpret_cast<const __half2*>(&s2);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __half2 h = *reinterpret_cast<__half2*>(&v[i]);
    const uint32_t c_r16 = 0x2C002C00u, c_1032 = 0x64086408u;
    if (i & 1) h = __hfma2(h, *reinterpret_cast<const __half2*>(&c_r16), *reinterpret_cast<const __half2*>(&k.m72));      // h / 16 - 72
    else h = __hsub2(h, *reinterpret_cast<const __half2*>(&c_1032));                                                     // h - 1032
    h = __hmul2(h, sc);
    o[i] = *reinterpret_cast<uint32_t*>(&h);
  }
}

// Four e4m3 bytes -> four fp16 values in k order, each times the block's fp32 scale with one rounding.
__device__ __forceinline__ void e4m3_word(uint32_t w, float sf, uint32_t* o) {
  uint32_t h0 = fp8x2_to_act<false, false>(w), h1 = fp8x2_to_act<false, false>(w >> 16);
  const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&h0)), f1 = __half22float2(*reinterpret_cast<__half2*>(&h1));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(o[0]) : "f"(f0.y * sf), "f"(f0.x * sf));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(o[1]) : "f"(f1.y * sf), "f"(f1.x * sf));
}

// One piece of a CTA's work: 64-k chunks [c_begin, c_begin + nk) of the strip of weight rows at n0, for the token tile
// at tok0.  part = the strip's other chunks belong to other CTAs; slot = which of the CTA's two partial-sum slots it uses.
struct Segment { int n0, c_begin, nk, strip, part, slot, tok0, xrow0, M, expert; };

// The CTA's list of segments; every role walks it with its own copy.  Cut strips (one token tile): the work is cut into
// units of one raw stage and CTA b takes the units [b U / G, (b + 1) U / G): up to two partial strips around any number
// of whole ones.  Otherwise whole (tile, strip) pairs in steps of the grid, ordered so that CTAs running at the same time
// share what does not fit in L2 twice: dense launches the weight strip, grouped launches an expert's activation rows.
template <int ROWS, int TOK, int GPS, int TABLE> struct Cursor {
  int u, u0, u1;
  int it; uint32_t table;            // segments handed out so far; tile table in shared memory (grouped launches)
  int block_row, block_col;          // 128 x 128 block the last segment of next_nk began with
  __device__ __forceinline__ void init(const W4Params& p, int total) {
    if (p.units > 0) {
      u0 = (int)((int64_t)blockIdx.x * p.units / gridDim.x);
      u1 = (int)((int64_t)(blockIdx.x + 1) * p.units / gridDim.x);
    } else {
      u0 = blockIdx.x; u1 = total;
    }
    u = u0; it = 0;
  }
  // {expert, first row in it, its first row, its rows} of a tile of a grouped launch
  static __device__ __forceinline__ int4 tile_info(const W4Params& p, int tile) {
    const int2 td = __ldcg(reinterpret_cast<const int2*>(p.tiles + 4) + tile);
    const int x0 = __ldcg(p.expert_offsets + td.x);
    return make_int4(td.x, td.y, x0, __ldcg(p.expert_offsets + td.x + 1) - x0);
  }
  // only the number of 64-k chunks and where in a run of eight scale groups they begin (for the roles that need no more)
  __device__ __forceinline__ int next_nk(const W4Params& p, int* off = nullptr) {
    if (off) *off = 0;
    if (u >= u1) return 0;
    if (p.units > 0) {
      const int r0 = u % p.sps, take = min(p.sps - r0, u1 - u);
      if (off) *off = (GPS * r0) & 7;
      block_row = u / p.sps * (ROWS / 128); block_col = GPS * r0;
      u += take;
      return take * 2 * GPS;
    }
    block_row = (p.tiles ? 0 : u / p.tiles_n) * (ROWS / 128); block_col = 0;
    u += gridDim.x;
    return p.nk;
  }
  __device__ __forceinline__ bool next(const W4Params& p, Segment& sg) {
    if (u >= u1) return false;
    sg.xrow0 = 0; sg.M = p.M; sg.expert = 0; sg.tok0 = 0;
    if (p.units > 0) {
      const int strip = u / p.sps, r0 = u - strip * p.sps;
      const int take = min(p.sps - r0, u1 - u);
      sg.n0 = strip * ROWS; sg.c_begin = r0 * 2 * GPS; sg.nk = take * 2 * GPS; sg.strip = strip;
      sg.part = take != p.sps; sg.slot = (u == u0) ? 0 : 1;
      u += take;
      return true;
    }
    sg.c_begin = 0; sg.nk = p.nk; sg.part = 0; sg.slot = 0;
    if (p.tiles) {
      const int tile = u / p.strips;
      sg.strip = u - tile * p.strips;
      int4 ti;
      if (it < TABLE) asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(ti.x), "=r"(ti.y), "=r"(ti.z), "=r"(ti.w) : "r"(table + 16 * it));
      else ti = tile_info(p, tile);
      ++it;
      sg.expert = ti.x; sg.tok0 = ti.y; sg.xrow0 = ti.z; sg.M = ti.w;
    } else {
      sg.strip = u / p.tiles_n;
      sg.tok0 = (u - sg.strip * p.tiles_n) * TOK;
    }
    sg.n0 = sg.strip * ROWS;
    u += gridDim.x;
    return true;
  }
};
}  // namespace w4

template <int WT, int TOK, int R>
__global__ void __launch_bounds__(w4::Cfg<WT, TOK, R>::THREADS, 1)
umma_w4_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const W4Params p) {
  using namespace w4;
  using C = Cfg<WT, TOK, R>;
  constexpr bool KMAJOR = WT == WT_W4K;
  constexpr int S = C::S, RS = C::RS, XS = C::XS, KG = C::KG, NBUF = C::NBUF, ROWS = C::ROWS;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t raw_smem = base, x_smem = base + RS * C::RAW_BYTES, sc_smem = x_smem + XS * C::X_BYTES;
  const uint32_t post_off = RS * C::RAW_BYTES + XS * C::X_BYTES + C::SCS * C::SC_BYTES;
  int8_t* post_exp = reinterpret_cast<int8_t*>(gen + post_off);
  const uint32_t out_smem = base + post_off + C::POST_BYTES, tile_table = out_smem + C::STAGE_OUT, bar = tile_table + C::TILE_TABLE * 16;
  // barrier map (8 bytes each)
  const uint32_t raw_full = bar, raw_empty = raw_full + 8 * RS, x_full = raw_empty + 8 * RS, x_empty = x_full + 8 * XS;
  const uint32_t a_full = x_empty + 8 * XS, a_empty = a_full + 8 * S, sc_full = a_empty + 8 * S, sc_empty = sc_full + 8 * C::SCS;
  const uint32_t acc_full = sc_empty + 8 * C::SCS, acc_empty = acc_full + 8 * NBUF, fix_bar = acc_empty + 8 * NBUF;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + (fix_bar + 8 - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + (fix_bar + 16 - base));
  volatile int* last_flag = reinterpret_cast<volatile int*>(gen + (fix_bar + 20 - base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // The next kernel of the stream may begin at once.  This one waits for the kernels before it only where it first
  // touches activations (the X producer), so that the weight stream runs under their tail; grouped launches read a tile
  // list the previous kernel built, so they wait here.
  grid_dep_release();
  int total = p.strips * p.tiles_n;
  if (p.tiles) { grid_dep_wait(); total = __ldcg(p.tiles) * p.strips; }
  using Cur = Cursor<ROWS, TOK, C::GPS, C::TILE_TABLE>;
  Cur cur;
  cur.init(p, total);
  cur.table = tile_table;
  if (cur.u >= cur.u1) return;                       // the whole CTA: fewer pieces of work than CTAs

  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(raw_full + 8 * i, 1); mbar_init(raw_empty + 8 * i, 4 * C::GPS * R); }
    for (int i = 0; i < XS; ++i) { mbar_init(x_full + 8 * i, 1); mbar_init(x_empty + 8 * i, 1); }
    for (int i = 0; i < S; ++i) { mbar_init(a_full + 8 * i, 4 * R); mbar_init(a_empty + 8 * i, 1); }
    for (int i = 0; i < C::SCS; ++i) { mbar_init(sc_full + 8 * i, 32); mbar_init(sc_empty + 8 * i, 16); }
    for (int i = 0; i < NBUF; ++i) { mbar_init(acc_full + 8 * i, 1); mbar_init(acc_empty + 8 * i, C::EW); }
    mbar_init(fix_bar, C::EW);
    *abort_flag = 0;
    fence_barrier_init();
  }
  // Every role needs a segment's tile; two dependent loads each, once per segment and role, cost short segments (768 k: six
  // scale groups) more than their work.  One thread per segment fetches them all at once.
  if (p.tiles && warp == 2) {
    const int64_t su = (int64_t)blockIdx.x + (int64_t)lane * gridDim.x;
    if (lane < C::TILE_TABLE && su < total) {
      const int4 ti = Cur::tile_info(p, (int)(su / p.strips));
      asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(tile_table + 16 * lane), "r"(ti.x), "r"(ti.y), "r"(ti.z), "r"(ti.w) : "memory");
    }
  }
  if (warp == 1) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- raw weight producer ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tm_w);
      Segment sg;
      int rs = 0, issued = 0;
      uint32_t par = 1u;                       // parity of the phase before the ring's current round
      bool ok = true;
      while (ok && cur.next(p, sg)) {
        const int nraw = sg.nk / (2 * C::GPS);
        for (int r = 0; r < nraw; ++r) {
          ok = mbar_wait(raw_empty + 8 * rs, par, abort_flag, p.status, ST_RAWEMPTY);
          if (!ok) break;
          ++issued;
          mbar_expect_tx(raw_full + 8 * rs, C::RAW_BYTES);
#pragma unroll
          for (int rb = 0; rb < R; ++rb) {
            const uint32_t dst = raw_smem + rs * C::RAW_BYTES + rb * 16384;
            if constexpr (KMAJOR)
              tma_load_2d(dst, &tm_w, sg.n0 + rb * 128, sg.expert * p.w_rows_per_expert + (sg.c_begin / (2 * C::GPS) + r) * 32, raw_full + 8 * rs);
            else
              tma_load_2d(dst, &tm_w, (sg.c_begin / (2 * C::GPS) + r) * 128, sg.expert * p.w_rows_per_expert + sg.n0 + rb * 128, raw_full + 8 * rs);
          }
          if (++rs == RS) { rs = 0; par ^= 1u; }
        }
      }
      if (!ok) drain_issued(raw_full, RS, issued);
    }
  } else if (warp == 2) {
    // ---------------- activation producer ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tm_x);
      if (!p.tiles) grid_dep_wait();
      Segment sg;
      int xs = 0, issued = 0;
      uint32_t par = 1u;
      bool ok = true;
      while (ok && cur.next(p, sg)) {
        for (int c = 0; c < sg.nk; c += C::XC) {
          ok = mbar_wait(x_empty + 8 * xs, par, abort_flag, p.status, ST_XEMPTY);
          if (!ok) break;
          ++issued;
          mbar_expect_tx(x_full + 8 * xs, C::X_BYTES);
#pragma unroll
          for (int i = 0; i < C::XC; ++i)
            tma_load_2d(x_smem + xs * C::X_BYTES + i * (TOK * 128), &tm_x, (sg.c_begin + c + i) * 64, sg.xrow0 + sg.tok0, x_full + 8 * xs);
          if (++xs == XS) { xs = 0; par ^= 1u; }
        }
      }
      if (!ok) drain_issued(x_full, XS, issued);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(0u, 0u, 128, TOK);
      const uint64_t db0 = smem_desc_sw128(x_smem);
      bool ok = true;
      int xs = 0, as = 0, b = 0, nk;
      uint32_t xpar = 0u, apar = 0u, bpar = 1u;
      while (ok && (nk = cur.next_nk(p)) > 0) {
        // the accumulators are reused: wait until the epilogue warps have read what they held
        ok = mbar_wait(acc_empty + 8 * b, bpar, abort_flag, p.status, ST_ACCEMPTY);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dacc = tmem + b * (R * C::ACC_COLS);
#pragma unroll 1
        for (int c = 0; c < nk && ok; c += C::XC) {
          ok = mbar_wait(x_full + 8 * xs, xpar, abort_flag, p.status, ST_XFULL);
#pragma unroll
          for (int i = 0; i < C::XC; i += 2) {
            if (ok) ok = mbar_wait(a_full + 8 * as, apar, abort_flag, p.status, ST_AFULL);
            if (!ok) break;
            tc_fence_after();
            const uint32_t ta = tmem + C::A_COL0 + 64 * R * as;
            const uint64_t db = db0 + (uint64_t)((xs * C::X_BYTES + i * (TOK * 128)) >> 4);
#pragma unroll
            for (int rb = 0; rb < R; ++rb)
#pragma unroll
              for (int j = 0; j < 8; ++j)          // 16 k each: eight columns of A, 32 bytes of a 128-byte row of B
                mma_f16_ts(dacc + rb * C::ACC_COLS, ta + rb * 64 + 8 * j, db + (uint64_t)((j >> 2) * (TOK * 128 >> 4) + 2 * (j & 3)), idesc,
                           (c + i > 0 || j > 0) ? 1u : 0u);
            tc_commit(a_empty + 8 * as);
            if (++as == S) { as = 0; apar ^= 1u; }
          }
          if (!ok) break;
          tc_commit(x_empty + 8 * xs);
          if (++xs == XS) { xs = 0; xpar ^= 1u; }
        }
        if (!ok) break;
        tc_commit(acc_full + 8 * b);
        if (++b == NBUF) { b = 0; bpar ^= 1u; }
      }
    }
  } else if (warp == 3) {
    // ---------------- scales ----------------
    // A lane serves the rows lane + 32 i of the strip.  A slot holds the groups 8 i .. 8 i + 7 of a row as stored, whatever
    // group the segment begins with (off within its first slot); a group beyond K gets zeros.  fp32 scales become fp16
    // factors here (see the transform), of the others only the bits are copied.
    constexpr int RI = 4 * R;
    Segment sg;
    int ss = 0, segno = 0, saturated = 0;
    uint32_t par = 1u;
    bool ok = true;
    const bool f32 = p.scale_dtype == B2Q_F32;
    const int esz = f32 ? 4 : 2;
    while (WT != WT_W8 && ok && cur.next(p, sg)) {
      const int gs = sg.c_begin >> 1, npad = sg.nk >> 1, off = gs & 7, nslot = (off + npad + 7) >> 3;
      const int ngroups = min(npad, (p.K >> 7) - gs);
      const uint8_t* sbase = reinterpret_cast<const uint8_t*>(p.scale) +
                             ((int64_t)sg.expert * p.s_expert_elems + (int64_t)(gs - off) * p.s_stride_g) * esz;
      float mul[RI];
      for (int sl = 0; sl < nslot; ++sl) {
        const uint32_t dst = sc_smem + ss * C::SC_BYTES + lane * 16;
        ok = mbar_wait_warp(sc_empty + 8 * ss, par, abort_flag, p.status, ST_SCEMPTY);
        if (!ok) break;
        if (p.scale_vec > 1) {
          // Asynchronous copies, up to SCS slots ahead: a scale comes from DRAM, and with loads through registers the
          // transform warps waited about 500 cycles per scale group for this warp (64 tokens, 256-row strips).
#pragma unroll
          for (int i = 0; i < RI; ++i) {
            const uint8_t* rp = sbase + (int64_t)min(sg.n0 + lane + 32 * i, p.N - 1) * p.s_stride_n * 2;
            if (p.scale_vec == 8) {
              cp_async16(dst + 512 * i, rp + 16 * sl, 16);
            } else {
#pragma unroll
              for (int j = 0; j < 8; j += 2) {           // off, npad and ngroups are even then
                const int g = 8 * sl - off + j;
                const bool in = g >= 0 && g < ngroups;
                cp_async4(dst + 512 * i + 2 * j, in ? rp + 2 * (8 * sl + j) : rp + 2 * off, in ? 4 : 0);
              }
            }
          }
          cp_async_arrive(sc_full + 8 * ss);               // every lane for its own rows, once they have landed
        } else {
#pragma unroll
          for (int i = 0; i < RI; ++i) {
            const uint8_t* rp = sbase + ((int64_t)min(sg.n0 + lane + 32 * i, p.N - 1) * p.s_stride_n + (int64_t)(8 * sl) * p.s_stride_g) * esz;
            uint32_t e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int g = 8 * sl - off + j;
              const int64_t o = (int64_t)j * p.s_stride_g;
              e[j] = 0u;
              if (g >= 0 && g < ngroups) e[j] = f32 ? __ldg(reinterpret_cast<const uint32_t*>(rp) + o) : (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(rp) + o);
            }
            if (f32) {
              if (sl == 0) {
                const int k = row_exponent(__uint_as_float(off == 0 ? e[0] : (off == 2 ? e[2] : (off == 4 ? e[4] : e[6]))));   // off is even
                mul[i] = pow2(k);
                post_exp[(segno % C::POST_RING) * ROWS + lane + 32 * i] = (int8_t)-k;
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) e[j] = fp16_factor(__uint_as_float(e[j]) * mul[i], saturated);
            }
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + 512 * i), "r"(e[0] | (e[1] << 16)), "r"(e[2] | (e[3] << 16)),
                         "r"(e[4] | (e[5] << 16)), "r"(e[6] | (e[7] << 16)) : "memory");
          }
          mbar_arrive(sc_full + 8 * ss);
        }
        if (++ss == C::SCS) { ss = 0; par ^= 1u; }
      }
      ++segno;
    }
    cp_async_wait_all();             // after a give-up copies may still be on their way; otherwise all have landed
    if (saturated) atomicCAS(p.status, 0, ST_SCALERANGE);
  } else if (warp < C::CW + C::EW) {
    // ---------------- epilogue ----------------
    constexpr int CB = TOK >= 32 ? 32 : 16, CG = C::EW / 4;      // column block of a warp; warps of a quadrant take them in turn
    constexpr int BLOCKS = R * (TOK / CB);
    const int quad = warp & 3, cgrp = (warp - C::CW) >> 2;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const bool leader = warp == C::CW && lane == 0;
    Segment sg;
    bool ok = true;
    int segno = 0, fixn = 0, b = 0;
    uint32_t bpar = 0u;
    if (p.units > 0 && warp == C::CW) {
      grid_dep_wait();                             // the scratch may be an earlier launch's until then; activations come no sooner
      if (lane < 2) arrivals_open(p.arrivals + (lane ? cur.u1 - 1 : cur.u0) / p.sps, p.tag, p.epoch);      // only a run's ends can be cut strips
      __syncwarp();
    }
    while (ok && cur.next(p, sg)) {
      ok = mbar_wait_warp(acc_full + 8 * b, bpar, abort_flag, p.status, ST_ACCUM);
      if (!ok) break;
      tc_fence_after();
      const int8_t* post = post_exp + (segno % C::POST_RING) * ROWS;
      // Row-parallel layer of a tensor-parallel stack: a block of 128 output columns belongs to one owner rank and one
      // 128-column block of that rank's slice; the tile is stored into this rank's slot of the owner's buffer
      // ([block][row][128 columns]) with plain peer stores, and the owner is told through flag1 when the block is done.
      auto write_out = [&](float (&r)[CB], int rb, int cb) {
        const int nb = sg.n0 + rb * 128, n = nb + quad * 32 + lane;
        if (nb >= p.N) return;
        uint16_t* dst;
        int64_t step = p.ldo;
        if (TOK <= 64 && p.peer_on) {
          const int owner = nb / p.peer.slice, blk = (nb - owner * p.peer.slice) >> 7;
          dst = reinterpret_cast<uint16_t*>(p.peer.bufs[owner] + p.peer.slot_off + (size_t)p.peer.rank * p.peer.slot_bytes +
                                            (size_t)blk * p.peer.M * (PR_CB * 2)) + (size_t)(sg.tok0 + cb) * PR_CB + quad * 32 + lane;
          step = PR_CB;
        } else {
          dst = reinterpret_cast<uint16_t*>(p.out) + (int64_t)(sg.xrow0 + sg.tok0 + cb) * p.ldo + n;
        }
        // per-token scales of this column block: one load per lane, read past L1 (it may still hold the previous
        // call's scales at this address), handed round the warp by shuffle
        const int left = sg.M - (sg.tok0 + cb);
        float ts_lane = 1.f;
        if (p.tok_scale && lane < CB && lane < left) ts_lane = __ldcg(p.tok_scale + sg.xrow0 + sg.tok0 + cb + lane);
        int map_lane = 0;
        if (p.out_map && lane < CB && lane < left) map_lane = __ldcg(p.out_map + sg.xrow0 + sg.tok0 + cb + lane);
        if (p.vec_out && nb + quad * 32 + 32 <= p.N && !(TOK <= 64 && p.peer_on)) {
          // Through shared memory, sixteen tokens at a time, so that a lane stores 16 bytes of a row instead of 2: with
          // 2-byte stores draining a 256 x 128 tile took 16,000 cycles in which the MMAs of the next one had to wait.
          const uint32_t st = out_smem + (warp - C::CW) * 1024;
#pragma unroll
          for (int h = 0; h < CB; h += 16) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float v0 = r[h + i] * __shfl_sync(0xffffffffu, ts_lane, h + i), v1 = r[h + i + 1] * __shfl_sync(0xffffffffu, ts_lane, h + i + 1);
              uint32_t pk;
              if (p.out_bf16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(pk) : "f"(v1), "f"(v0));
              else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(pk) : "f"(v1), "f"(v0));
              asm volatile("st.shared.u16 [%0], %1;" ::"r"(st + i * 64 + lane * 2), "h"((unsigned short)pk) : "memory");
              asm volatile("st.shared.u16 [%0], %1;" ::"r"(st + i * 64 + 64 + lane * 2), "h"((unsigned short)(pk >> 16)) : "memory");
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int tk = h + j * 8 + (lane >> 2);
              const uint4 v = lds128(st + j * 512 + lane * 16);
              int64_t orow = sg.xrow0 + sg.tok0 + cb + tk;
              if (p.out_map) orow = __shfl_sync(0xffffffffu, map_lane, tk);
              if (tk < left)
                *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + orow * p.ldo + nb + quad * 32 + (lane & 3) * 8) = v;
            }
          }
          return;
        }
#pragma unroll
        for (int i = 0; i < CB; ++i) {
          const float v = r[i] * __shfl_sync(0xffffffffu, ts_lane, i);
          const unsigned short h = p.out_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
          if (p.out_map) {
            const int orow = __shfl_sync(0xffffffffu, map_lane, i);
            if (i < left && n < p.N) reinterpret_cast<uint16_t*>(p.out)[(int64_t)orow * p.ldo + n] = h;
          } else {
            if (i < left && n < p.N) *dst = h;
            dst += step;
          }
        }
      };
      // partial sums of a cut strip: [CTA][slot][row block][token / 4][row][4] fp32
      auto part_ptr = [&](int cta, int slot, int rb, int cb) -> float4* {
        return reinterpret_cast<float4*>(p.partials) + (((size_t)(cta * 2 + slot) * R + rb) * (TOK / 4) + cb / 4) * 128 + quad * 32 + lane;
      };
      auto publish = [&](int rb) {                 // one thread, after all epilogue warps have issued their stores
        const int nb = sg.n0 + rb * 128;
        if (nb >= p.N) return;
        const int owner = nb / p.peer.slice, blk = (nb - owner * p.peer.slice) >> 7;
        __threadfence_system();
        st_release_sys(&reinterpret_cast<PeerCtrl*>(p.peer.bufs[owner])->flag1[p.peer.rank][blk],
                       reinterpret_cast<const PeerCtrl*>(p.peer.bufs[p.peer.rank])->epoch + 1);
      };
#pragma unroll 1
      for (int rc = cgrp; rc < BLOCKS; rc += CG) {
        const int rb = rc / (TOK / CB), cb = (rc % (TOK / CB)) * CB;
        if (sg.tok0 + cb >= sg.M) continue;
        __syncwarp();                              // the stores of the last block were per lane
        float r[CB];
        {
          uint32_t q[CB];
          const uint32_t ta = tmem + lane_base + (b * R + rb) * C::ACC_COLS + cb;
          if constexpr (CB == 32) tmem_ld32(ta, q); else tmem_ld16(ta, q);
          tmem_ld_wait();
          float pm;
          if (WT == WT_W8 && p.scale_mode != B2Q_SCALE_BLOCK128)
            pm = load_scalar(p.scale, sg.expert * p.s_expert_elems +
                                          (p.scale_mode == B2Q_SCALE_CHANNEL ? min(sg.n0 + rb * 128 + quad * 32 + lane, p.N - 1) : 0), p.scale_dtype);
          else pm = pow2(post[rb * 128 + quad * 32 + lane]);
#pragma unroll
          for (int i = 0; i < CB; ++i) r[i] = __uint_as_float(q[i]) * pm;
        }
        if (!sg.part) {
          write_out(r, rb, cb);
        } else {
          float4* dst = part_ptr(blockIdx.x, sg.slot, rb, cb);
#pragma unroll
          for (int i = 0; i < CB; i += 4)
            if (cb + i < sg.M) __stcg(dst + (i / 4) * 128, make_float4(r[i], r[i + 1], r[i + 2], r[i + 3]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * b);
      if (++b == NBUF) { b = 0; bpar ^= 1u; }
      ++segno;
      auto all_epilogue_warps = [&]() -> bool {
        __syncwarp();
        if (lane == 0) mbar_arrive(fix_bar);
        const bool r = mbar_wait_warp(fix_bar, fixn & 1, abort_flag, p.status, ST_FIXUP);
        ++fixn;
        return r;
      };
      if (sg.part) {
        // Whoever delivers a strip's last partial sums adds all of them up, always in CTA order, and writes the
        // result: no CTA ever waits for another one, and the sum does not depend on who came last.
        const int64_t U = p.units, G = gridDim.x;
        const int64_t us = (int64_t)sg.strip * p.sps, ue = us + p.sps - 1;
        const int b_lo = (int)(((us + 1) * G + U - 1) / U) - 1, b_hi = (int)(((ue + 1) * G + U - 1) / U) - 1;
        // the barrier hands every thread's partial sums to the leader (release / acquire at CTA scope); the leader's one
        // device-scope fence then orders all of them before the count
        ok = all_epilogue_warps();
        if (!ok) break;
        if (leader) {
          __threadfence();
          *last_flag = arrivals_last(p.arrivals + sg.strip, b_hi - b_lo);
          __threadfence();
        }
        ok = all_epilogue_warps();
        if (!ok) break;
        if (*last_flag) {
          __threadfence();
#pragma unroll 1
          for (int rc = cgrp; rc < BLOCKS; rc += CG) {
            const int rb = rc / (TOK / CB), cb = (rc % (TOK / CB)) * CB;
            if (cb >= sg.M) continue;
            float r[CB];
#pragma unroll
            for (int i = 0; i < CB; ++i) r[i] = 0.f;
#pragma unroll 1
            for (int c = b_lo; c <= b_hi; ++c) {
              const int64_t bu0 = (int64_t)c * U / G;
              const float4* src = part_ptr(c, bu0 >= us ? 0 : 1, rb, cb);
              float4 v[CB / 4];
#pragma unroll
              for (int i = 0; i < CB / 4; ++i) {         // all of a contributor's loads in flight at once
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (cb + 4 * i < sg.M) v[i] = __ldcg(src + i * 128);
              }
#pragma unroll
              for (int i = 0; i < CB / 4; ++i) {
                r[4 * i] += v[i].x; r[4 * i + 1] += v[i].y; r[4 * i + 2] += v[i].z; r[4 * i + 3] += v[i].w;
              }
            }
            write_out(r, rb, cb);
          }
        }
      }
      if (TOK <= 64 && p.peer_on) {
        const bool deliver = !sg.part || *last_flag;       // the same for every warp: written between two barriers
        ok = all_epilogue_warps();
        if (!ok) break;
        if (deliver && leader)
          for (int rb = 0; rb < R; ++rb) publish(rb);
      }
    }
  } else {
    // ---------------- transform ----------------
    // A group of four warps converts one scale group (128 k = one operand stage, half a raw stage) of one block of 128
    // rows per iteration, a weight row (N-major) or column (K-major) per thread; the groups take the scale groups in turn,
    // so a thread always works on the same half of a raw stage and every ring position advances by a constant.
    // The decode multiplies by the group's scale in fp16.  bf16 scales are first multiplied by a power of two per row,
    // taken from the scale of the segment's first group so that this one lands in [0.5, 1); the epilogue multiplies the
    // row by the inverse power (fp16 scales are taken as they are, fp32 scales were converted the same way by warp 3).
    // (q - 8) * s needs 11 bits at most, so groups within 2^13 of the first one, either way, are exact; one further above
    // would overflow fp16 and is saturated and reported through the status word.
    const int quad = warp & 3, grp = (warp - C::CW - C::EW) >> 2;
    const int t = quad * 32 + lane;                // row of the block == tensor-memory lane this thread may write
    const int rb = R == 2 ? (grp & 1) : 0, kq = R == 2 ? (grp >> 1) : grp;
    const int half = C::GPS == 2 ? (kq & 1) : 0;
    const uint32_t row0 = raw_smem + rb * 16384 + (KMAJOR ? t * 4 + half * 16 * 512 : t * 128 + (((4 * half) ^ (t & 7)) << 4));
    const uint32_t ta0 = tmem + ((uint32_t)(quad * 32) << 16) + C::A_COL0 + rb * 64;
    const uint32_t sc0 = sc_smem + (rb * 128 + t) * 16;
    const bool elected = lane == 0, bf16_scale = p.scale_dtype == B2Q_BF16;
    const MagicConsts mk = p.mk;
    bool ok = true;
    int gb = 0, ss = 0, segno = 0, saturated = 0, nk, off;      // gb: chunks of earlier segments
    uint32_t spar = 0u;
    while (ok && (nk = cur.next_nk(p, &off)) > 0) {
      const int ngroups = nk >> 1, nslot = (off + ngroups + 7) >> 3;
      // first group of this segment that is this transform group's in the count over all segments
      int gg = (kq - (gb >> 1)) & (KG - 1);
      const int g0 = (gb >> 1) + gg, raw0 = g0 / C::GPS;
      int rs = raw0 % RS, as = g0 % S;
      uint32_t rpar = (uint32_t)(raw0 / RS) & 1u, apar = ((uint32_t)(g0 / S) + 1u) & 1u;
      float row_mul = 1.f;
      // e4m3: one fp32 scale per block, the same for the whole CTA, requested an iteration ahead; one power of two per segment
      // brings them into fp16's range (see block_scale_exponent)
      const float* block_scale = reinterpret_cast<const float*>(p.scale) + (cur.block_row + rb) * (int64_t)(p.K >> 7) + cur.block_col;
      const bool blocks = WT == WT_W8 && p.scale_mode == B2Q_SCALE_BLOCK128;
      float sf_next = 1.f;
      if (blocks) {
        if (gg < ngroups) sf_next = __ldg(block_scale + gg);
        const int k = block_scale_exponent(block_scale, ngroups);
        row_mul = pow2(k);
        if (gg == 0) post_exp[(segno % C::POST_RING) * ROWS + rb * 128 + t] = (int8_t)-k;
      }
#pragma unroll 1
      for (int sl = 0; sl < nslot; ++sl) {
        if (WT != WT_W8) ok = mbar_wait_warp(sc_full + 8 * ss, spar, abort_flag, p.status, ST_SCFULL);
        if (!ok) break;
        const uint32_t sca = sc0 + ss * C::SC_BYTES;
        if (WT != WT_W8 && sl == 0 && p.scale_dtype != B2Q_F32) {
          const int k = bf16_scale ? row_exponent(__uint_as_float(lds_u16(sca + 2 * off) << 16)) : 0;
          row_mul = pow2(k);
          // told to the epilogue by the group that converts the segment's first 128 k: before these are handed over
          if (gg == 0) post_exp[(segno % C::POST_RING) * ROWS + rb * 128 + t] = (int8_t)-k;
        }
        const int gend = min(8 * sl + 8 - off, ngroups);
#pragma unroll 1
        for (; gg < gend; gg += KG) {
          uint32_t hv = WT == WT_W8 ? 0u : lds_u16(sca + 2 * ((gg + off) & 7));
          const float sf = sf_next * row_mul;
          if (blocks && gg + KG < ngroups) sf_next = __ldg(block_scale + gg + KG);
          if (WT == WT_W8) {}
          else if (bf16_scale) hv = fp16_factor(__uint_as_float(hv << 16) * row_mul, saturated);
          else if ((hv & 0x7FFFu) - 0x7000u <= 0x0C00u) { hv = (hv & 0x8000u) | 0x6FFFu; saturated = 1; }     // above 8188, NaN stays
          const uint32_t m2 = hv | (hv << 16);
          ok = mbar_wait_warp(raw_full + 8 * rs, rpar, abort_flag, p.status, ST_RAWFULL);
          if (!ok) break;
          const uint32_t rowa = row0 + rs * C::RAW_BYTES;
          const uint32_t ta = ta0 + 64 * R * as;
#pragma unroll
          for (int q = 0; q < 4; ++q) {            // quarters of 32 k: 16 registers live
            uint32_t w0, w1, w2, w3;
            uint32_t a16[16];
            if constexpr (WT == WT_W8) {
#pragma unroll
              for (int z = 0; z < 2; ++z) {
                const uint4 rr = lds128(rowa ^ ((2 * q + z) << 4));
                if (TOK < 128 || blocks) {
                  e4m3_word(rr.x, sf, a16 + 8 * z); e4m3_word(rr.y, sf, a16 + 8 * z + 2);
                  e4m3_word(rr.z, sf, a16 + 8 * z + 4); e4m3_word(rr.w, sf, a16 + 8 * z + 6);
                } else {
                  const uint32_t w[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
                  for (int c = 0; c < 4; ++c) {
                    a16[8 * z + 2 * c] = fp8x2_to_act<false, false>(w[c]);
                    a16[8 * z + 2 * c + 1] = fp8x2_to_act<false, false>(w[c] >> 16);
                  }
                }
              }
            } else if constexpr (!KMAJOR) {
              const uint4 rr = lds128(rowa ^ (q << 4));
              w0 = rr.x; w1 = rr.y; w2 = rr.z; w3 = rr.w;
            } else {
              w0 = lds32(rowa + (4 * q + 0) * 512); w1 = lds32(rowa + (4 * q + 1) * 512);
              w2 = lds32(rowa + (4 * q + 2) * 512); w3 = lds32(rowa + (4 * q + 3) * 512);
            }
            if constexpr (WT != WT_W8) {
              w4_word_magic(w0, m2, mk, a16); w4_word_magic(w1, m2, mk, a16 + 4);
              w4_word_magic(w2, m2, mk, a16 + 8); w4_word_magic(w3, m2, mk, a16 + 12);
            }
            if (q == 0) {                          // the first quarter is converted while the stage is still being read
              ok = mbar_wait_warp(a_empty + 8 * as, apar, abort_flag, p.status, ST_EMPTY);
              if (!ok) break;
              tc_fence_after();
            }
            tmem_st16(ta + 16 * q, a16);
          }
          if (!ok) break;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (elected) { mbar_arrive(a_full + 8 * as); mbar_arrive(raw_empty + 8 * rs); }
          __syncwarp();
          rs += C::RAW_ROUND; if (rs >= RS) { rs -= RS; rpar ^= 1u; }
          as += C::A_ROUND; if (as >= S) { as -= S; apar ^= 1u; }
        }
        if (!ok) break;
        if (WT != WT_W8) mbar_arrive_read(sc_empty + 8 * ss);
        __syncwarp();
        if (++ss == C::SCS) { ss = 0; spar ^= 1u; }
      }
      gb += nk; ++segno;
    }
    if (saturated) atomicCAS(p.status, 0, ST_SCALERANGE);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
static int sm_count() {
  static thread_local int sms[16] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return 148;
  if (!sms[dev]) {
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (sms[dev] <= 0) sms[dev] = 148;
  }
  return sms[dev];
}

static int dense_tok(int64_t M) { return M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128)); }

// CTAs among which strips of n raw stages are best cut; 0 = whole strips.  A cut has to be weighed, and into few and equal pieces
// where possible: the last contributor to a strip adds up everybody's partial sums, and pieces that do not line up with the strips
// have one contributor more.  cost, in us: per stage of a strip, per cut strip, per contributor to it.
// 128-token tiles: fitted over N = 512 .. 12288 x K = 1024 .. 28672 at 65, 96 and 128 tokens (0.3 % above the best of seven divisions on
// average, 6 % at most); 256-row strips take twice of each.  Against cutting over the whole grid: 128 x 2048 x 2048 25.9 -> 11.7 us, 128 x
// 4096 x 4096 35.0 -> 18.1, 128 x 4096 x 14336 37.8 -> 32.1; unchanged 128 x 8192 x 28672, 64 us (97 with whole strips).
// Lower tiles: over N = 1024 .. 14336 x K = 2048 .. 14336, whole, 2, 3, 4, 6, 8 pieces and the whole grid (before).  INT4, 64 tokens, 2048 x
// 2048 8.9, 10.9, 11.3, 11.8, 13.6, 14.9 and 15.0 us, 2048 x 8192 21.9, 18.3, 16.3, 15.6, 16.6, 18.6 and 22.0, 14336 x 5120 16.8 whole, 23.6 over
// the grid; e4m3 with block scales, 32 tokens, 1024 x 5120 17.8 whole, 30.2 over the grid, 14336 x 5120 19.8 and 24.6, 8192 x 14336 45.1 and 33.8.
struct CutCost { double stage, strip, contributor; };
static int cut_grid(int64_t strips, int64_t n, int sms, const CutCost& c) {
  double best = c.stage * (double)((strips + sms - 1) / sms * n);
  int64_t grid = 0;
  for (int64_t p = 2; p <= n && p * strips <= sms; ++p) {
    const double t = c.stage * (double)((n + p - 1) / p) + c.strip + c.contributor * (double)p;
    if (t < best) { best = t; grid = p * strips; }
  }
  const int64_t g = strips * n < sms ? strips * n : sms, pieces = (g + strips - 1) / strips;
  if (g % strips != 0 && c.stage * (double)((strips * n + g - 1) / g) + 1.3 * c.strip + c.contributor * (double)(pieces + 1) < best) grid = g;
  return (int)grid;
}

// How one token tile of a dense launch is shared out: strips of R x 128 rows, cut along k, raw stage by raw stage, when whole
// ones would leave more than a twentieth of the machine idle in the last round and cut_grid finds a cut that pays.
struct StripPlan { int R, strips, sps, units, grid; size_t partial_bytes; };      // sps, units: raw stages per strip and in total, 0 = whole strips
static StripPlan plan_strips(int64_t M, int64_t N, int64_t K, int k_per_stage, bool tall) {
  StripPlan pl{};
  const int sms = sm_count(), tok = dense_tok(M);
  const int64_t strips2 = (N + 255) / 256;
  pl.R = tall && tok >= 64 && strips2 >= sms ? 2 : 1;          // the tall strip where it still gives every SM one
  const int64_t strips = pl.R == 2 ? strips2 : (N + 127) / 128, units = strips * (K / k_per_stage);
  pl.strips = (int)strips;
  pl.grid = (int)(strips < sms ? strips : sms);
  if (M > tok || (K % k_per_stage) != 0 || strips > UMMA_MAX_CUT_STRIPS || sms > ARRIVALS_MAX || units > INT32_MAX) return pl;
  if ((double)strips / ((double)((strips + sms - 1) / sms) * sms) > 0.95) return pl;
  const bool w8 = k_per_stage == 128;
  const CutCost cost = tok == 128 ? CutCost{0.8, 4.0, 2.0} : (tok == 64 ? CutCost{w8 ? 0.46 : 0.54, 3.0, 1.0} : CutCost{w8 ? 0.35 : 0.5, 2.0, 0.75});
  const int grid = cut_grid(strips, K / k_per_stage, sms, cost);
  if (!grid) return pl;
  pl.sps = (int)(K / k_per_stage); pl.units = (int)units; pl.grid = grid;
  static_assert(128 * 16 * sizeof(float) >= UMMA_MAX_CUT_STRIPS * sizeof(Arrivals), "a slot holds the arrival counts");
  pl.partial_bytes = (size_t)2 * pl.grid * pl.R * 128 * tok * sizeof(float);       // two slots per CTA
  return pl;
}
static StripPlan plan_w4(int64_t M, int64_t N, int64_t K) { return plan_strips(M, N, K, 256, true); }
static StripPlan plan_w8(int64_t M, int64_t N, int64_t K) { return plan_strips(M, N, K, 128, false); }

size_t umma_w4_partial_bytes(int64_t M, int64_t N, int64_t K) { return M > 0 && N > 0 ? plan_w4(M, N, K).partial_bytes : 0; }
size_t umma_w8_strip_partial_bytes(int64_t M, int64_t N, int64_t K) { return M > 0 && M <= 64 && N > 0 ? plan_w8(M, N, K).partial_bytes : 0; }

template <int WT, int TOK, int R>
static int launch_w4(const CUtensorMap& tw, const CUtensorMap& tx, const W4Params& p, int grid, bool overlap, cudaStream_t st) {
  using C = w4::Cfg<WT, TOK, R>;
  auto kern = umma_w4_kernel<WT, TOK, R>;
  static thread_local bool configured[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) return B2Q_ERR_CUDA;
    if (dev < 16) configured[dev] = true;
  }
  if (launch_overlapped(kern, dim3(grid), dim3(C::THREADS), C::SMEM, st, overlap, tw, tx, p) != cudaSuccess) return B2Q_ERR_CUDA;
  note_launch("umma_w4");
  return launch_status();
}

template <int WT>
static int launch_w4_tile(int tok, int R, const CUtensorMap& tw, const CUtensorMap& tx, const W4Params& p, int grid, bool overlap,
                          cudaStream_t st) {
  if (tok == 16) return launch_w4<WT, 16, 1>(tw, tx, p, grid, overlap, st);
  if (tok == 32) return launch_w4<WT, 32, 1>(tw, tx, p, grid, overlap, st);
  if (tok == 64) return R == 2 ? launch_w4<WT, 64, 2>(tw, tx, p, grid, overlap, st) : launch_w4<WT, 64, 1>(tw, tx, p, grid, overlap, st);
  return R == 2 ? launch_w4<WT, 128, 2>(tw, tx, p, grid, overlap, st) : launch_w4<WT, 128, 1>(tw, tx, p, grid, overlap, st);
}

// Takes the plan's cut over where the caller's scratch holds its partial sums; without it every strip stays whole.  The arrival counts
// lie in the second slot of the last CTA, whose run ends with the last strip: what it has behind its first segment are whole strips.
template <class Args>
static int cut_strips(W4Params& p, const Args& a, const StripPlan& pl) {
  if (!pl.units || !a.sk_ws || !aligned16(a.sk_ws) || a.sk_ws_bytes < pl.partial_bytes || tls().force_kernel == 4) return B2Q_OK;
  p.epoch = arrivals_epoch();
  if (!p.epoch) return B2Q_ERR_CUDA;
  p.sps = pl.sps; p.units = pl.units; p.partials = reinterpret_cast<float*>(a.sk_ws);
  p.arrivals = reinterpret_cast<Arrivals*>(reinterpret_cast<uint8_t*>(a.sk_ws) + pl.partial_bytes / (2 * pl.grid) * (2 * pl.grid - 1));
  p.tag = arrivals_tag();
  return B2Q_OK;
}

int umma_w4_prep_token_tile(const UmmaW4Args& a) { return a.expert_offsets ? grouped_tok(a.M, a.E) : dense_tok(a.M); }

// Rounds over the SMs of a grouped launch, for the number of tiles to be expected: every expert's last tile half full.
static int64_t grouped_rounds(int64_t rows, int E, int64_t strips, int tok, int sms) {
  return (strips * (2 * rows + (int64_t)E * tok) + (int64_t)2 * tok * sms - 1) / ((int64_t)2 * tok * sms);
}
// 256-row strips for grouped launches.  64-token tiles take them when there are many rounds of short strips and at most 0.6 times
// as many of tall ones: 128 experts x 64 rows, 2048 x 768, 90 -> 73 us, but 4 experts x 60 rows, 1536 x 2048, 16 us with short
// strips and 20 with tall ones (two rounds become one, at twice the time and with half of the SMs idle).  A 128-token tile of
// 256 rows has one accumulator set, so that its drain stands still under every k loop: only a long k and exactly half the
// rounds make up for that (32 x 128 rows, 3072 x 4096, 152 -> 143 us; 128 x 256 rows, 1536 x 2048, 273 against 317 us with tall ones).
// Over 500 combinations of 2 to 128 experts, 33 to 256 rows each and eleven matrices: 9 % less time than tall strips
// throughout, 0.6 % more than the better of the two each time.
static bool tall_strips_grouped(int64_t rows, int E, int64_t strips1, int64_t strips2, int64_t K, int tok, int sms) {
  const int64_t r1 = grouped_rounds(rows, E, strips1, tok, sms), r2 = grouped_rounds(rows, E, strips2, tok, sms);
  return tok == 64 ? r1 >= 8 && 20 * r2 <= 12 * r1 : K >= 4096 && 2 * r2 <= r1;
}

int umma_w4_prep_linear(const UmmaW4Args& a, cudaStream_t st) {
  if (a.bf16) return B2Q_ERR_UNSUPPORTED;       // the pre-pass always hands over fp16
  const bool kmajor = a.layout == B2Q_W4_KMAJOR || a.layout == B2Q_W4_KMAJOR_MARLIN;
  const bool grouped = a.expert_offsets != nullptr;
  const int E = grouped ? a.E : 1, sms = sm_count();
  const int tok = umma_w4_prep_token_tile(a);
  const int tiles = grouped ? a.tile_cap : (a.M + tok - 1) / tok;
  const int strips1 = (a.N + 127) / 128, strips2 = (a.N + 255) / 256;
  // 256-row strips move fewer bytes per flop, 128-row strips give twice the pieces of work.  A single token tile takes the
  // tall strip when that still gives every SM one (plan_strips); several weigh the rounds over the SMs against 1.3 times the
  // time per row block of the short strip; grouped launches: tall_strips_grouped.
  const StripPlan pl = grouped || tiles > 1 ? StripPlan{} : plan_w4(a.M, a.N, a.K);
  int R = 1;
  if (tok >= 64) {
    if (grouped) {
      R = tall_strips_grouped(a.M, a.E, strips1, strips2, a.K, tok, sms) ? 2 : 1;
    } else if (tiles == 1) {
      R = pl.R;
    } else {
      const int64_t r1 = ((int64_t)strips1 * tiles + sms - 1) / sms, r2 = ((int64_t)strips2 * tiles + sms - 1) / sms;
      R = 20 * r2 <= 13 * r1 ? 2 : 1;
    }
  }
  CUtensorMap tw, tx;
  int rc;
  if (kmajor)
    rc = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, a.w, (uint64_t)E * (a.K / 8), a.N, (uint64_t)a.N * 4, 32, 128,
                      CU_TENSOR_MAP_SWIZZLE_NONE);
  else
    rc = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, (uint64_t)E * a.N, a.K / 2, (uint64_t)a.K / 2, 128, 128,
                      CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, a.M, a.K, (uint64_t)a.ldx * 2, tok, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  W4Params p{};
  p.scale = a.scale; p.scale_dtype = a.scale_dtype; p.s_stride_n = a.s_stride_n; p.s_stride_g = a.s_stride_g;
  p.s_expert_elems = (int64_t)a.N * (a.K / 128);
  p.scale_vec = 1;
  if (a.scale_dtype != B2Q_F32 && a.s_stride_g == 1) {
    if ((a.s_stride_n % 8) == 0 && (a.K % 1024) == 0 && aligned16(a.scale)) p.scale_vec = 8;
    else if ((a.s_stride_n % 2) == 0 && (a.K % 256) == 0 && (reinterpret_cast<uintptr_t>(a.scale) & 3u) == 0) p.scale_vec = 2;
  }
  p.out = a.out; p.ldo = a.ldo; p.out_bf16 = a.out_bf16 ? 1 : 0;
  p.vec_out = aligned16(a.out) && (a.ldo % 8) == 0;
  p.M = a.M; p.N = a.N; p.K = a.K; p.nk = ((a.K >> 6) + 3) & ~3;
  p.tiles = grouped ? a.tiles : nullptr; p.expert_offsets = a.expert_offsets; p.out_map = a.out_map;
  p.w_rows_per_expert = kmajor ? a.K / 8 : a.N;
  p.tok_scale = a.tok_scale;
  p.mk = w4::magic_consts(a.layout == B2Q_W4_NMAJOR_S4);
  p.status = umma_status_ptr();
  if (!p.status) return B2Q_ERR_CUDA;
  p.strips = R == 2 ? strips2 : strips1; p.tiles_n = tiles;
  int64_t work = (int64_t)p.strips * tiles;
  rc = cut_strips(p, a, pl);
  if (rc) return rc;
  if (p.units > 0) work = pl.grid;
  if (work > INT32_MAX) return B2Q_ERR_LIMIT;
  if (a.peer) {
    if (tok > 64 || grouped || (a.N % 128) != 0 || (a.peer->slice % 128) != 0 || a.peer->M != a.M) return B2Q_ERR_UNSUPPORTED;
    p.peer_on = 1; p.peer = *a.peer;
  }
  const int grid = (int)(work < sms ? work : sms);
  const bool overlap = tls().overlap_mode > 0 && (a.after_prep || tls().overlap_mode == 2);
  return kmajor ? launch_w4_tile<w4::WT_W4K>(tok, R, tw, tx, p, grid, overlap, st)
                : launch_w4_tile<w4::WT_W4N>(tok, R, tw, tx, p, grid, overlap, st);
}

// Dense launches of more than 64 tokens: 128-token tiles here, or umma_gemm.cu's of 256 (of 128, two CTAs per SM, up to 128 tokens).
// Fewer bytes of operands per flop there, half the granularity here; each kernel's time is close to an offset plus rounds over
// the SMs times a time per tile linear in K.  Fitted, in us, over N = 1024 .. 28672, K = 2048 .. 8192 and 70 to 2048 tokens
// (285 launches per scale mode, 5 to 7 % mean error, 17 for the form with two CTAs per SM).  Choosing by it, with 5 % in
// favour of the other kernel, takes 17 % less time over them with block scales and 18 with channel scales, 4 % more at worst
// (512 x 12288 x 5120, block scales, 75 against 73 us).  128 x 17408 x 5120, block scales: 56 -> 36 us, 1221 x 4680 x 2048 43 -> 37;
// 4001 x 17408 x 5120 stays where it was, 587 us against 645 here.  So do up to 4 Mi weights at up to 128 tokens, although they
// would gain up to 5 us (100 x 2048 x 2048, block scales: 17.6 against 13.1): test_gpu_w4_strips.py names the kernel of such a call.
// Up to k of 512 the MMAs no longer hide the output's way out, the less so where its rows are not 16-byte aligned: 1 us more per round
// against the 256-token tiles, 3 where unaligned, 1 with longer k.  3000 x 1466 x 128, per tensor, 12.8 against 9.1 us there, 151 x 12072 x 256 12.5
// against 10.5, 217 x 16422 x 640, block scales, 17.1 against 14.1.  Over 462 launches of N = 64 .. 28672, K = 128 .. 2560 and 65 to 4096 tokens, half of
// them unaligned, 16 that the rule takes are 2 to 9 % slower here; without this term 59 were, by up to 49 %.
static bool w8_strips_pay(const UmmaW8Args& a) {
  if (a.M <= 128 && (int64_t)a.N * a.K <= (4 << 20)) return false;
  const int sms = sm_count();
  const int64_t strips = (a.N + 127) / 128;
  const double k = a.K / 1024.0;
  const bool block = a.scale_mode == B2Q_SCALE_BLOCK128;
  auto rounds = [](int64_t work, int64_t slots) { return (double)((work + slots - 1) / slots); };
  const double stores = aligned16(a.out) && (a.ldo % 8) == 0 ? (a.K <= 512 && a.M > 128 ? 1.0 : 0.0) : (a.K <= 512 ? 3.0 : 1.0);
  const double here = (block ? 4.67 : 5.93) + rounds(strips * ((a.M + 127) / 128), sms) * (stores + (block ? 1.16 + 4.08 * k : 0.74 + 3.31 * k));
  const double there = a.M <= 128 ? (block ? 2.98 : 3.57) + rounds(strips, 2 * (int64_t)sms) * (block ? 2.98 + 6.26 * k : 3.57 + 4.18 * k)
                                  : (block ? 1.30 : 1.70) + rounds(strips * ((a.M + 255) / 256), sms) * (block ? 8.92 + 5.56 * k : 8.39 + 5.36 * k);
  return here < 0.95 * there;
}

// e4m3 weights on fp16 activations: dense with block scales up to 64 tokens and with any scales above (w8_strips_pay), grouped with one
// scale per channel or tensor in tiles of up to 64 tokens.
bool umma_w8_strip_supported(const UmmaW8Args& a) {
  if (a.bf16 || a.fmt != B2Q_E4M3 || (a.K % 128) != 0) return false;
  if (a.expert_offsets) {
    const int tok = grouped_tok(a.M, a.E);
    if (a.scale_mode == B2Q_SCALE_BLOCK128 || tok > 64) return false;
    // 64-token tiles in two rounds over the SMs go through umma_gemm.cu's kernel in one, with two CTAs on each: 8 experts x 80
    // rows, 2048 x 2048, 21.6 against 24.8 us, 2 x 80, 8192 x 2048, 21.7 against 25.2.  One round (2 x 40, 8192 x 2048, 19.4 against
    // 18.1 us), more than two (4 x 60, 8192 x 2048, 35.4 against 33.9; 64 x 40, 2048 x 1024, 56.4 against 40.9) and 32-token tiles (8 x 24,
    // 4096 x 2048, 27.6 against 22.4) are faster here.
    return tok < 64 || grouped_rounds(a.M, a.E, (a.N + 127) / 128, tok, sm_count()) != 2;
  }
  return a.M <= 64 ? a.scale_mode == B2Q_SCALE_BLOCK128 : w8_strips_pay(a);
}

int umma_w8_strip_linear(const UmmaW8Args& a, cudaStream_t st) {
  const bool grouped = a.expert_offsets != nullptr;
  const int sms = sm_count(), tok = grouped ? grouped_tok(a.M, a.E) : dense_tok(a.M);
  CUtensorMap tw, tx;
  int rc = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, (uint64_t)(grouped ? a.E : 1) * a.N, a.K, (uint64_t)a.K, 128, 128,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, a.M, a.K, (uint64_t)a.ldx * 2, tok, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  W4Params p{};
  p.scale = a.scale; p.scale_dtype = a.scale_dtype; p.scale_mode = a.scale_mode; p.s_expert_elems = a.s_expert_elems;
  p.tiles = grouped ? a.tiles : nullptr; p.expert_offsets = a.expert_offsets; p.out_map = a.out_map; p.w_rows_per_expert = a.N;
  p.out = a.out; p.ldo = a.ldo; p.out_bf16 = a.out_bf16 ? 1 : 0;
  p.vec_out = aligned16(a.out) && (a.ldo % 8) == 0;
  p.M = a.M; p.N = a.N; p.K = a.K; p.nk = a.K >> 6;
  p.tok_scale = a.tok_scale;
  p.status = umma_status_ptr();
  if (!p.status) return B2Q_ERR_CUDA;
  p.strips = (a.N + 127) / 128; p.tiles_n = grouped ? a.tile_cap : (a.M + tok - 1) / tok;
  int64_t work = (int64_t)p.strips * p.tiles_n;
  if (!grouped && a.M <= 64) {
    const StripPlan pl = plan_w8(a.M, a.N, a.K);
    rc = cut_strips(p, a, pl);
    if (rc) return rc;
    if (p.units > 0) work = pl.grid;
  }
  if (work > INT32_MAX) return B2Q_ERR_LIMIT;
  const int grid = (int)(work < sms ? work : sms);
  const bool overlap = tls().overlap_mode > 0 && (a.after_prep || tls().overlap_mode == 2);
  if (tok == 16) return launch_w4<w4::WT_W8, 16, 1>(tw, tx, p, grid, overlap, st);
  if (tok == 32) return launch_w4<w4::WT_W8, 32, 1>(tw, tx, p, grid, overlap, st);
  if (tok == 64) return launch_w4<w4::WT_W8, 64, 1>(tw, tx, p, grid, overlap, st);
  return launch_w4<w4::WT_W8, 128, 1>(tw, tx, p, grid, overlap, st);
}

}  // namespace b2q
