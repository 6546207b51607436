// INT4 decode linear for up to eight tokens: out[m, n] = sum_g s[n, g] * sum_{k in group g} (q[n, k] - 8) * x[m, k], N-major
// nibbles, group 128, dense or grouped (MoE experts).
//
// HBM-bound: the weights are read once and nothing else is large.  They go by TMA into a ring of 128-row x 256-k stages, are
// decoded in registers into exact 16-bit integers (q - 8) and multiplied by mma.sync m16n8k16, weight rows as the MMA's M,
// tokens as its N; a group's sum is scaled in fp32, so every scale of every type is exact.  Two CTAs per SM, each:
//   warp 0        TMA producer of raw weight stages
//   warp 1        fetches group scales into shared memory, 16 bytes of every row at a time, by asynchronous copy where aligned
//   next 2        stage the activations of every weight stage in MMA fragment order, taking the stages in turn
//   next 8        decode, MMA, output: 32 rows of the strip each, every other stage
// What it replaces (smallm.cuh, one CTA per 16-row strip) loaded scales and activations from global memory for every 128 k, fed
// one chain of eight dependent MMAs with them and waited for both.  57344 x 8192, one / eight tokens: 102 / 132 us there, 54 / 57
// here (fp16).  Probes of the same ring, none of them kept: no decode 41 us, nibble conversion adds 10, MMAs 3.
// What was found on the way, same shape, one token:
// * 72 KB of ring per SM instead of 128: 48 us without any decode.
// * An MMA takes some 80 cycles to deliver and a group's eight can only be chained (their sum is scaled in fp32): hence two tiles
//   per warp, two chains each, which also share the activation fragments (16 rows per warp: 64 us).
// * Activations loaded by the staging warps when their stage is free instead of two stages earlier, or converted there
//   (scaled to fp16, or summed so that the nibbles need no centring): 63 to 82 us, 195 for eight tokens.
// * Nibbles as fp16 subnormals (q * 2^-24 needs no arithmetic), the -8 by MMAs against a constant: 67 us.
// * tcgen05 with the nibbles as e4m3 (0000 qqqq is q * 2^-9), activations as three e4m3 terms and a promotion per group: 58 to 81 us.
//
// Work: strips of 128 rows x stages of 256 k.  Dense launches give every CTA an equal run of stages; a strip cut between CTAs is
// summed, block by block, by whoever delivers last, in CTA order: nobody waits, and the result does not depend on who that is.
// Who comes last is counted in the caller's scratch (arrivals.cuh).
// Grouped launches walk (tile, strip) pairs.  GATED: a strip is 64 gate rows and the 64 up rows that go with them, paired in
// one thread's accumulators, and the output is silu(gate) * up.
//
// Every mbarrier wait is bounded; on expiry the CTA records a code in the status word and ends.
//
// Reference counterparts: esimd_gemv_int4 (csrc/xpu/esimd_kernels/int4_GEMV.h:165-251), GEMM_int4_pgrp_kernel
// (int4_GEMM.h:81-270), the tiny-M expert kernels of csrc/moe_batch/moe_int4.sycl.
#include "umma_gemm.cuh"
#include "sm100.cuh"
#include "arrivals.cuh"
#include "smallm.cuh"   // lds128, mma16816, cp_async16
#include "w4_stream.cuh"

namespace b2q {

using namespace sm100;

namespace w4s {
enum { ST_EMPTY = 601, ST_XEMPTY = 602, ST_SCEMPTY = 603, ST_FULL = 604, ST_SCFULL = 605 };

constexpr int ROWS = 128, BLOCKS = ROWS / 32;                     // rows of a strip, blocks of two MMA tiles of 16
constexpr int EW = 2 * BLOCKS;                                    // decoding warps: two per block, which take the stages in turn
// Staging warps take the stages in turn too.  The ring is whole rounds of either: a warp then knows, from the stage it had last,
// that the use before the one it waits for is over, which a parity wait cannot tell apart.
constexpr int XW = 2;
constexpr int CW = 2 + XW, THREADS = (CW + EW) * 32;
constexpr int RAW_BYTES = ROWS * 128, X_BYTES = 4096;
constexpr int RS = 4;
constexpr int SCS = 4, SC_BYTES = ROWS * 16;                      // scale slots: 16 bytes of each row
constexpr int RED_BYTES = BLOCKS * 1024;                          // sums of the odd stages, on their way to the even ones' warps
constexpr int BAR_BYTES = 256;
constexpr int SMEM = RS * (RAW_BYTES + X_BYTES) + SCS * SC_BYTES + RED_BYTES + 1024 /*align*/ + BAR_BYTES;
static_assert(RS % XW == 0 && RS % (EW / BLOCKS) == 0 && SMEM <= 115712, "ring depths; two CTAs per SM");
}  // namespace w4s

struct W4SParams {
  const void* x; int64_t ldx;
  // scales of the experts and of the shared expert; vec: bytes of a row's scales per asynchronous copy, 16 or 4, 0 = element by element
  struct Scales { const void* p; int64_t stride_n, stride_g; int vec; } sc, sc2;
  int64_t s_expert_elems;
  int shared_e;                // grouped: the "expert" whose weights are those of the second tensor map, or -1
  void* out; int64_t ldo;
  int M, N, K;                 // rows of W (gate and up together), k
  int half;                    // GATED: rows of the gate half, the up half follows
  int strips, sps, units;      // strips, stages per strip, stages in total (cut launches; 0 = whole strips)
  float4* partials;            // [2 * grid][BLOCKS][2][32] sums of cut strips
  Arrivals* arrivals; Arrivals tag; const Arrivals* epoch;      // [strips][BLOCKS] counts behind the partial sums
  uint32_t flip;               // 0x00080008 for two's-complement nibbles
  const int32_t* tiles; const int32_t* expert_offsets; const int32_t* row_map; int row_div; const int32_t* out_map;
  int* status;
};

namespace w4s {
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {       // the rest of the four bytes is zeroed
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {       // one arrival when this thread's copies have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t c) {      // (a & 0x000F000F) ^ c
  uint32_t d;
  asm("lop3.b32 %0, %1, 0x000F000F, %2, 0x6A;" : "=r"(d) : "r"(a), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t and_xor_hi(uint32_t a, uint32_t c) {      // (a & 0x00F000F0) ^ c
  uint32_t d;
  asm("lop3.b32 %0, %1, 0x00F000F0, %2, 0x6A;" : "=r"(d) : "r"(a), "r"(c));
  return d;
}
// A word of eight nibbles n0 .. n7 -> four pairs (n0,n4) (n1,n5) (n2,n6) (n3,n7) of exact q - 8.  fp16: 0x6400 | q is 1024 + q,
// 0x6400 | (q << 4) is 1024 + 16 q, so one shift serves all; bf16 has mantissa for 0x4300 | q = 128 + q only, three shifts.
// lo, hi: the constants merged in, with the sign flip of two's-complement nibbles folded in.
template <bool BF16> __device__ __forceinline__ void decode(uint32_t w, uint32_t lo, uint32_t hi, uint32_t (&o)[4]) {
  if constexpr (BF16) {
    const uint32_t v[4] = {and_xor(w, lo), and_xor(w >> 4, lo), and_xor(w >> 8, lo), and_xor(w >> 12, lo)};
    const uint32_t c = 0x43084308u;                              // 136
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v[i]), *reinterpret_cast<const __nv_bfloat162*>(&c));
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  } else {
    const uint32_t w8 = w >> 8;
    const uint32_t v[4] = {and_xor(w, lo), and_xor_hi(w, hi), and_xor(w8, lo), and_xor_hi(w8, hi)};
    const uint32_t c_1032 = 0x64086408u, c_r16 = 0x2C002C00u, c_m72 = 0xD480D480u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 h = *reinterpret_cast<const __half2*>(&v[i]);
      const __half2 r = (i & 1) ? __hfma2(h, *reinterpret_cast<const __half2*>(&c_r16), *reinterpret_cast<const __half2*>(&c_m72))
                                : __hsub2(h, *reinterpret_cast<const __half2*>(&c_1032));
      o[i] = *reinterpret_cast<const uint32_t*>(&r);
    }
  }
}

// Stages [st0, st0 + nst) of a strip for the token tile at tok0.  part: other CTAs have the strip's other stages.
struct Segment { int strip, st0, nst, part, slot, expert, tok0, xrow0, M; };

struct Cursor {
  int u, u0, u1;
  __device__ __forceinline__ void init(const W4SParams& p, int total) {
    if (p.units > 0) {
      u0 = (int)((int64_t)blockIdx.x * p.units / gridDim.x);
      u1 = (int)((int64_t)(blockIdx.x + 1) * p.units / gridDim.x);
    } else {
      u0 = blockIdx.x; u1 = total;
    }
    u = u0;
  }
  __device__ __forceinline__ bool next(const W4SParams& p, Segment& sg) {
    if (u >= u1) return false;
    sg.expert = 0; sg.tok0 = 0; sg.xrow0 = 0; sg.M = p.M;
    if (p.units > 0) {
      sg.strip = u / p.sps; sg.st0 = u - sg.strip * p.sps;
      sg.nst = min(p.sps - sg.st0, u1 - u);
      sg.part = sg.nst != p.sps; sg.slot = u == u0 ? 0 : 1;
      u += sg.nst;
      return true;
    }
    sg.st0 = 0; sg.nst = p.sps; sg.part = 0; sg.slot = 0;
    if (p.tiles) {
      const int tile = u / p.strips;
      sg.strip = u - tile * p.strips;
      const int2 td = __ldcg(reinterpret_cast<const int2*>(p.tiles + 4) + tile);
      sg.expert = td.x; sg.tok0 = td.y;
      sg.xrow0 = __ldcg(p.expert_offsets + td.x);
      sg.M = __ldcg(p.expert_offsets + td.x + 1) - sg.xrow0;
    } else {
      sg.strip = u;
    }
    u += gridDim.x;
    return true;
  }
};
}  // namespace w4s

template <bool BF16, int SD, bool GATED>      // SD: type of the group scales
__global__ void __launch_bounds__(w4s::THREADS, 2)
w4_stream_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2, const W4SParams p) {
  using namespace w4s;
  constexpr int ESZ = SD == B2Q_F32 ? 4 : 2, GPS = 16 / ESZ;       // bytes of a scale, groups per scale slot
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t x_smem = base + RS * RAW_BYTES, sc_smem = x_smem + RS * X_BYTES;
  const uint32_t red_smem = sc_smem + SCS * SC_BYTES, bar = red_smem + RED_BYTES;
  const uint32_t full = bar, empty = full + 8 * RS, sc_full = empty + 8 * RS, sc_empty = sc_full + 8 * SCS;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + (sc_empty + 8 * SCS - base));
  volatile int* pair_ok = abort_flag + 1;              // [BLOCKS][2]: how a block's two warps came out of the segment
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // The next kernel may start at once.  This one waits for the kernels before it where it first reads what they may have written:
  // the tile list, or else the activations (the staging warps); outputs and partial sums follow from those.
  grid_dep_release();
  int total = p.strips;
  if (p.tiles) { grid_dep_wait(); total = __ldcg(p.tiles) * p.strips; }
  Cursor cur;
  cur.init(p, total);
  if (cur.u >= cur.u1) return;                       // the whole CTA: fewer pieces of work than CTAs

  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(full + 8 * i, 2); mbar_init(empty + 8 * i, BLOCKS); }
    for (int i = 0; i < SCS; ++i) { mbar_init(sc_full + 8 * i, 32); mbar_init(sc_empty + 8 * i, EW); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  Segment sg;

  if (warp == 0) {
    // ---------------- weight producer: two boxes of half a strip's rows x 256 k ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tm_w);
      int s = 0, issued = 0;
      uint32_t par = 1u;
      bool ok = true;
      while (ok && cur.next(p, sg)) {
        const bool sh = sg.expert == p.shared_e;
        const CUtensorMap* tm = sh ? &tm_w2 : &tm_w;
        const int r0 = (sh ? 0 : sg.expert * p.N) + sg.strip * (GATED ? ROWS / 2 : ROWS), r1 = r0 + (GATED ? p.half : ROWS / 2);
        for (int i = 0; i < sg.nst; ++i) {
          ok = mbar_wait(empty + 8 * s, par, abort_flag, p.status, ST_EMPTY);
          if (!ok) break;
          ++issued;
          mbar_expect_tx(full + 8 * s, RAW_BYTES);
          tma_load_2d(base + s * RAW_BYTES, tm, (sg.st0 + i) * 128, r0, full + 8 * s);
          tma_load_2d(base + s * RAW_BYTES + RAW_BYTES / 2, tm, (sg.st0 + i) * 128, r1, full + 8 * s);
          if (++s == RS) { s = 0; par ^= 1u; }
        }
      }
      if (!ok) drain_issued(full, RS, issued);
    }
  } else if (warp == 1) {
    // ---------------- scales ----------------
    // A lane serves the rows lane + 32 i of the strip.  A slot holds an aligned run of 16 bytes of every row's scales, whatever
    // group the segment begins with; groups beyond K become zero.
    const int groups = p.K >> 7;
    int ss = 0;
    uint32_t par = 1u;
    bool ok = true;
    while (ok && cur.next(p, sg)) {
      const int g0 = 2 * sg.st0 / GPS * GPS, g1 = 2 * (sg.st0 + sg.nst);
      const bool sh = sg.expert == p.shared_e;
      const W4SParams::Scales& sc = sh ? p.sc2 : p.sc;
      const uint8_t* rp[ROWS / 32];
#pragma unroll
      for (int i = 0; i < ROWS / 32; ++i) {
        const int r = lane + 32 * i;
        const int n = !GATED ? min(sg.strip * ROWS + r, p.N - 1)
                             : (r < ROWS / 2 ? min(sg.strip * (ROWS / 2) + r, p.half - 1) : min(p.half + sg.strip * (ROWS / 2) + r - ROWS / 2, p.N - 1));
        rp[i] = reinterpret_cast<const uint8_t*>(sc.p) + ((sh ? 0 : sg.expert * p.s_expert_elems) + n * sc.stride_n) * ESZ;
      }
      for (int g = g0; g < g1; g += GPS) {
        ok = mbar_wait_warp(sc_empty + 8 * ss, par, abort_flag, p.status, ST_SCEMPTY);
        if (!ok) break;
        const uint32_t dst = sc_smem + ss * SC_BYTES + lane * 16;
        if (sc.vec) {
#pragma unroll
          for (int i = 0; i < ROWS / 32; ++i) {
            const uint8_t* src = rp[i] + (int64_t)g * ESZ;
            if (sc.vec == 16) {
              cp_async16(dst + 512 * i, src, 16);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const bool in = g + (4 * j) / ESZ < groups;
                cp_async4(dst + 512 * i + 4 * j, in ? src + 4 * j : rp[i], in ? 4 : 0);
              }
            }
          }
          cp_async_arrive(sc_full + 8 * ss);
        } else {
#pragma unroll
          for (int i = 0; i < ROWS / 32; ++i) {
            uint32_t e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              e[j] = 0u;
              if (j < GPS && g + j < groups) {
                const uint8_t* src = rp[i] + (int64_t)(g + j) * sc.stride_g * ESZ;
                e[j] = ESZ == 4 ? __ldg(reinterpret_cast<const uint32_t*>(src)) : (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(src));
              }
            }
            if (ESZ == 2) { e[0] |= e[1] << 16; e[1] = e[2] | (e[3] << 16); e[2] = e[4] | (e[5] << 16); e[3] = e[6] | (e[7] << 16); }
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + 512 * i), "r"(e[0]), "r"(e[1]), "r"(e[2]), "r"(e[3]) : "memory");
          }
          mbar_arrive(sc_full + 8 * ss);
        }
        if (++ss == SCS) { ss = 0; par ^= 1u; }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");       // after a give-up copies may still be on their way
  } else if (warp < CW) {
    // ---------------- activations ----------------
    // A lane has eight consecutive k of every token: word q of the k range that the decoding lanes with lane % 4 == t have.
    // Read past L1: it may hold what an earlier kernel saw at these addresses.  Rows of tokens beyond M keep whatever lies
    // there; they only reach output columns that nobody writes.
    if (!p.tiles) grid_dep_wait();
    const int me = warp - 2;
    const uint32_t dst0 = x_smem + ((lane >> 4) * 4 + (lane & 3)) * 512 + ((lane >> 2) & 3) * 16;
    int i = 0, s = 0;                                    // stages handed out so far; ring position
    uint32_t par = 1u;
    bool ok = true, open = !GATED && p.units > 0 && me == 0;      // gated launches are grouped: whole strips
    while (ok && cur.next(p, sg)) {
      const int m_left = min(sg.M - sg.tok0, 8);
      int64_t row_off = 0;                               // lane m: where token m's row begins
      if (lane < m_left) {
        int64_t r = sg.xrow0 + sg.tok0 + lane;
        if (p.row_map) r = __ldcg(p.row_map + r) / p.row_div;
        row_off = r * p.ldx;
      }
      uint4 v[8];
      auto load = [&](int st) {
        const int k = (sg.st0 + st) * 256 + lane * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t off = __shfl_sync(0xffffffffu, row_off, j);
          v[j] = make_uint4(0, 0, 0, 0);
          if (j < m_left && k < p.K) v[j] = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.x) + off + k));
        }
      };
      const int first = (me - i % XW + XW) % XW;         // this warp's first stage of the segment
      if (first < sg.nst) load(first);
      for (int st = 0; st < sg.nst; ++st, ++i) {
        if (i % XW == me) {
          ok = mbar_wait_warp(empty + 8 * s, par, abort_flag, p.status, ST_XEMPTY);
          if (!ok) break;
          // The counts of the CTA's cut strips, which only a run's ends can be, are opened before the first segment's last stage is
          // handed to the warps that will add to them; behind the first stages, which would otherwise wait for the trip to DRAM.
          if (open && (i == RS || st + XW >= sg.nst)) {
            if (lane < 2 * BLOCKS) arrivals_open(p.arrivals + ((lane & 1) ? cur.u1 - 1 : cur.u0) / p.sps * BLOCKS + (lane >> 1), p.tag, p.epoch);
            open = false;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < m_left)
              asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst0 + s * X_BYTES + j * 64),
                           "r"(__byte_perm(v[j].x, v[j].z, 0x5410)), "r"(__byte_perm(v[j].x, v[j].z, 0x7632)),
                           "r"(__byte_perm(v[j].y, v[j].w, 0x5410)), "r"(__byte_perm(v[j].y, v[j].w, 0x7632)) : "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(full + 8 * s);
          if (st + XW < sg.nst) load(st + XW);           // on its way while the stages in between are used
        }
        if (++s == RS) { s = 0; par ^= 1u; }
      }
    }
  } else {
    // ---------------- decode, MMA, output ----------------
    // MMA rows g and g + 8 of this warp's tile: rows that differ by 4 sit in neighbouring g, so that the 128-byte swizzle
    // spreads a quarter-warp's 16-byte reads over all banks.
    const int w = (warp - CW) >> 1, turn = (warp - CW) & 1, g = lane >> 2, t = lane & 3, pr = (g >> 1) | ((g & 1) << 2);
    // rows g and g + 8 of the block's first tile, and how far on those of the second are
    const int row_a = GATED ? 16 * w + pr : 32 * w + pr, row_b = GATED ? ROWS / 2 + 16 * w + pr : 32 * w + 8 + pr;
    constexpr int TILE_STEP = GATED ? 8 : 16;
    const uint32_t wa0 = base + row_a * 128 + ((t ^ pr) << 4), wb = (row_b - row_a) * 128;
    const uint32_t xa0 = x_smem + lane * 16;
    const uint32_t sca0 = sc_smem + row_a * 16, scb = (row_b - row_a) * 16;
    const uint32_t lo = (BF16 ? 0x43004300u : 0x64006400u) ^ p.flip, hi = 0x64006400u ^ (p.flip << 4);
    int s = 0, ss = 0, n = 0;                            // n: stages so far
    uint32_t par = 0u, spar = 0u;
    bool ok = true;
    while (ok && cur.next(p, sg)) {
      float acc[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
      int j = 2 * sg.st0 % GPS;                          // this stage's first group within its scale slot
      for (int i = 0; ok && i < sg.nst;) {
        ok = mbar_wait_warp(sc_full + 8 * ss, spar, abort_flag, p.status, ST_SCFULL);
        if (!ok) break;
        const int end = min(sg.nst, i + (GPS - j) / 2);  // stages served by this slot
#pragma unroll 1
        for (; i < end; ++i, ++n, j += 2) {
          if ((n & 1) == turn) {
            const uint32_t so = sca0 + ss * SC_BYTES + j * ESZ;
            uint32_t ra[2][2], rb[2][2];                 // scales of rows a and b of both tiles as stored, both groups
#pragma unroll
            for (int i2 = 0; i2 < 2; ++i2) {
              const uint32_t st = so + i2 * (TILE_STEP * 16);
              if constexpr (SD == B2Q_F32) {
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(ra[i2][0]), "=r"(ra[i2][1]) : "r"(st));
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(rb[i2][0]), "=r"(rb[i2][1]) : "r"(st + scb));
              } else {
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(ra[i2][0]) : "r"(st));
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(rb[i2][0]) : "r"(st + scb));
              }
            }
            ok = mbar_wait_warp(full + 8 * s, par, abort_flag, p.status, ST_FULL);
            if (!ok) break;
            const uint32_t wo = wa0 + s * RAW_BYTES, xo = xa0 + s * X_BYTES;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint4 wv[2][2];
#pragma unroll
              for (int i2 = 0; i2 < 2; ++i2) {
                wv[i2][0] = lds128((wo ^ (h << 6)) + i2 * (TILE_STEP * 128));
                wv[i2][1] = lds128((wo ^ (h << 6)) + i2 * (TILE_STEP * 128) + wb);
              }
              float u[2][4], v[2][4];                    // two chains per tile: an MMA takes some 80 cycles to deliver
#pragma unroll
              for (int i2 = 0; i2 < 2; ++i2)
#pragma unroll
                for (int c = 0; c < 4; ++c) u[i2][c] = v[i2][c] = 0.f;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 xv = lds128(xo + (h * 4 + q) * 512);
#pragma unroll
                for (int i2 = 0; i2 < 2; ++i2) {
                  const uint4& wva = wv[i2][0];
                  const uint4& wvb = wv[i2][1];
                  uint32_t da[4], db[4];
                  decode<BF16>(q == 0 ? wva.x : (q == 1 ? wva.y : (q == 2 ? wva.z : wva.w)), lo, hi, da);
                  decode<BF16>(q == 0 ? wvb.x : (q == 1 ? wvb.y : (q == 2 ? wvb.z : wvb.w)), lo, hi, db);
                  mma16816<BF16>(u[i2], da[0], db[0], da[1], db[1], xv.x, xv.y);
                  mma16816<BF16>(v[i2], da[2], db[2], da[3], db[3], xv.z, xv.w);
                }
              }
#pragma unroll
              for (int i2 = 0; i2 < 2; ++i2) {
                float sa, sb;
                if constexpr (SD == B2Q_F32) { sa = __uint_as_float(ra[i2][h]); sb = __uint_as_float(rb[i2][h]); }
                else if constexpr (SD == B2Q_BF16) {
                  sa = __uint_as_float(h ? ra[i2][0] & 0xFFFF0000u : ra[i2][0] << 16); sb = __uint_as_float(h ? rb[i2][0] & 0xFFFF0000u : rb[i2][0] << 16);
                } else {
                  const __half2 fa = *reinterpret_cast<const __half2*>(&ra[i2][0]), fb = *reinterpret_cast<const __half2*>(&rb[i2][0]);
                  sa = h ? __high2float(fa) : __low2float(fa); sb = h ? __high2float(fb) : __low2float(fb);
                }
                acc[i2][0] += sa * (u[i2][0] + v[i2][0]); acc[i2][1] += sa * (u[i2][1] + v[i2][1]);
                acc[i2][2] += sb * (u[i2][2] + v[i2][2]); acc[i2][3] += sb * (u[i2][3] + v[i2][3]);
              }
            }
            mbar_arrive_read(empty + 8 * s);
          }
          if (++s == RS) { s = 0; par ^= 1u; }
        }
        if (!ok) break;
        j = 0;
        mbar_arrive_read(sc_empty + 8 * ss);
        if (++ss == SCS) { ss = 0; spar ^= 1u; }
      }
      // The block's two warps add up; the first delivers.  They meet twice, so that the buffer is free again before the next
      // segment, and go on only if neither has given up: nobody meets a warp that left.
      const uint32_t red = red_smem + w * 1024 + lane * 16;
      if (turn == 1)
#pragma unroll
        for (int i2 = 0; i2 < 2; ++i2)
          asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(red + 512 * i2), "f"(acc[i2][0]), "f"(acc[i2][1]), "f"(acc[i2][2]), "f"(acc[i2][3]) : "memory");
      if (lane == 0) pair_ok[2 * w + turn] = ok;
      __syncwarp();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + w) : "memory");
      ok = pair_ok[2 * w] && pair_ok[2 * w + 1];
      if (turn == 0)
#pragma unroll
        for (int i2 = 0; i2 < 2; ++i2) {
          float b[4];
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]) : "r"(red + 512 * i2));
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i2][c] += b[c];
        }
      asm volatile("bar.sync %0, 64;" ::"r"(1 + w) : "memory");
      if (!ok) break;
      if (turn == 1) continue;
      bool deliver = true;
      if (!GATED && sg.part) {
        // this warp's rows are finished by the last of the sharers' warps w to get here
        const int64_t U = p.units, G = gridDim.x, us = (int64_t)sg.strip * p.sps, ue = us + p.sps - 1;
        const int b_lo = (int)(((us + 1) * G + U - 1) / U) - 1, b_hi = (int)(((ue + 1) * G + U - 1) / U) - 1;
#pragma unroll
        for (int i2 = 0; i2 < 2; ++i2)
          __stcg(p.partials + (((size_t)(blockIdx.x * 2 + sg.slot) * BLOCKS + w) * 2 + i2) * 32 + lane, make_float4(acc[i2][0], acc[i2][1], acc[i2][2], acc[i2][3]));
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = arrivals_last(p.arrivals + sg.strip * BLOCKS + w, b_hi - b_lo);
        deliver = __shfl_sync(0xffffffffu, last, 0) != 0;
        if (deliver) {
          __threadfence();
          float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll 4
          for (int b = b_lo; b <= b_hi; ++b) {
            const int slot = (int64_t)b * U / G >= us ? 0 : 1;
#pragma unroll
            for (int i2 = 0; i2 < 2; ++i2) {
              const float4 o = __ldcg(p.partials + (((size_t)(b * 2 + slot) * BLOCKS + w) * 2 + i2) * 32 + lane);
              v[i2].x += o.x; v[i2].y += o.y; v[i2].z += o.z; v[i2].w += o.w;
            }
          }
#pragma unroll
          for (int i2 = 0; i2 < 2; ++i2) { acc[i2][0] = v[i2].x; acc[i2][1] = v[i2].y; acc[i2][2] = v[i2].z; acc[i2][3] = v[i2].w; }
        }
      }
      if (deliver) {
        uint16_t* out = reinterpret_cast<uint16_t*>(p.out);
        auto round16 = [&](float v) { return BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v)); };
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int m = 2 * t + c;
          if (m < sg.M - sg.tok0) {
            int64_t orow = sg.xrow0 + sg.tok0 + m;
            if (p.out_map) orow = __ldcg(p.out_map + orow);
#pragma unroll
            for (int i2 = 0; i2 < 2; ++i2) {
              if constexpr (GATED) {
                const int col = sg.strip * (ROWS / 2) + row_a + i2 * TILE_STEP;
                if (col < p.half) out[orow * p.ldo + col] = round16(acc[i2][c] / (1.0f + expf(-acc[i2][c])) * acc[i2][c + 2]);
              } else {
                const int col = sg.strip * ROWS + row_a + i2 * TILE_STEP;
                if (col < p.N) out[orow * p.ldo + col] = round16(acc[i2][c]);
                if (col + row_b - row_a < p.N) out[orow * p.ldo + col + row_b - row_a] = round16(acc[i2][c + 2]);
              }
            }
          }
        }
      }
      __syncwarp();
    }
  }
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

// Stages are shared out evenly among all CTAs (two per SM) unless whole strips already keep 97 of 100 busy.
struct W4SPlan { int strips, sps, grid; bool cut; size_t partial_bytes; };      // partial_bytes: sums, then arrival counts
static size_t sum_bytes(int grid) { return (size_t)2 * grid * w4s::ROWS * 8 * sizeof(float); }      // two slots per CTA
static W4SPlan plan(int64_t N, int64_t K) {
  W4SPlan pl{};
  const int slots = 2 * sm_count();
  const int64_t strips = (N + w4s::ROWS - 1) / w4s::ROWS, sps = (K + 255) / 256, units = strips * sps;
  pl.strips = (int)strips; pl.sps = (int)sps;
  pl.grid = (int)(strips < slots ? strips : slots);
  if (strips > UMMA_MAX_CUT_STRIPS || slots > ARRIVALS_MAX || units > INT32_MAX / 4) return pl;
  if ((double)strips / ((double)((strips + slots - 1) / slots) * slots) > 0.97 || units <= strips) return pl;
  pl.cut = true;
  pl.grid = (int)(units < slots ? units : slots);
  pl.partial_bytes = sum_bytes(pl.grid) + (size_t)strips * w4s::BLOCKS * sizeof(Arrivals);
  return pl;
}
size_t w4_stream_partial_bytes(int64_t M, int64_t N, int64_t K) {
  return M > 0 && M <= W4_STREAM_MAX_TOK && N > 0 && K > 0 ? plan(N, K).partial_bytes : 0;
}

template <bool BF16, int SD, bool GATED>
static int launch(const CUtensorMap& tw, const CUtensorMap& tw2, const W4SParams& p, int grid, bool overlap, cudaStream_t st) {
  auto kern = w4_stream_kernel<BF16, SD, GATED>;
  static thread_local bool configured[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, w4s::SMEM) != cudaSuccess) return B2Q_ERR_CUDA;
    if (dev < 16) configured[dev] = true;
  }
  if (launch_overlapped(kern, dim3(grid), dim3(w4s::THREADS), w4s::SMEM, st, overlap, tw, tw2, p) != cudaSuccess) return B2Q_ERR_CUDA;
  note_launch("w4_stream");
  return launch_status();
}

template <bool BF16, int SD>
static int launch_gated(bool gated, const CUtensorMap& tw, const CUtensorMap& tw2, const W4SParams& p, int grid, bool overlap, cudaStream_t st) {
  return gated ? launch<BF16, SD, true>(tw, tw2, p, grid, overlap, st) : launch<BF16, SD, false>(tw, tw2, p, grid, overlap, st);
}
template <bool BF16>
static int launch_scale(int sd, bool gated, const CUtensorMap& tw, const CUtensorMap& tw2, const W4SParams& p, int grid, bool overlap, cudaStream_t st) {
  if (sd == B2Q_F32) return launch_gated<BF16, B2Q_F32>(gated, tw, tw2, p, grid, overlap, st);
  return sd == B2Q_BF16 ? launch_gated<BF16, B2Q_BF16>(gated, tw, tw2, p, grid, overlap, st) : launch_gated<BF16, B2Q_F16>(gated, tw, tw2, p, grid, overlap, st);
}

static bool room(const W4SPlan& pl, const void* partials, size_t bytes) { return partials && aligned16(partials) && bytes >= pl.partial_bytes; }

// bytes of a row's scales per asynchronous copy: 16 or 4, 0 = element by element
static int scale_bytes(const void* scale, int dtype, int64_t stride_n, int64_t stride_g, int groups) {
  const int esz = dtype_bytes(dtype);
  const uintptr_t at = reinterpret_cast<uintptr_t>(scale);
  if (stride_g != 1) return 0;
  if ((groups * esz) % 16 == 0 && (stride_n * esz) % 16 == 0 && (at & 15u) == 0) return 16;
  return (groups * esz) % 4 == 0 && (stride_n * esz) % 4 == 0 && (at & 3u) == 0 ? 4 : 0;
}

bool w4_stream_preferred(const W4StreamArgs& a) {
  const int64_t M = a.M, N = a.N, K = a.K;
  if (M > W4_STREAM_MAX_TOK) return false;
  const double k = (double)K / 1024.0;
  const int64_t slots = 3 * (int64_t)sm_count(), rounds = ((N + 15) / 16 + slots - 1) / slots;
  const double there = 1.0 + (double)rounds * (0.9 + 1.38 * k) * (1.0 + 0.02 * (double)(M - 1));
  const W4SPlan pl = plan(N, K);
  const double whole = 4.0 + (double)((pl.strips + 2 * sm_count() - 1) / (2 * sm_count())) * pl.sps;
  const double contributors = pl.cut ? (double)pl.grid / pl.strips : 1.0, sums = contributors > 10.0 ? 0.23 * (contributors - 10.0) : 0.0;
  const double narrow = scale_bytes(a.scale, a.scale_dtype, a.s_stride_n, a.s_stride_g, a.K / 128) == 16 ? 0.0 : 1.0;
  const double here = (pl.cut && !room(pl, a.partials, a.partial_bytes) ? whole : 9.5 + 0.1e-6 * (double)N * (double)K + 0.2 * k + sums) + narrow;
  return here < 0.97 * there;
}

bool w4_stream_supported(const W4StreamArgs& a) {
  if (a.K <= 0 || (a.K % 128) != 0 || !aligned16(a.x) || !aligned16(a.w) || ((a.ldx * 2) & 15)) return false;
  if (a.layout != B2Q_W4_NMAJOR && a.layout != B2Q_W4_NMAJOR_S4) return false;
  if (a.tile > W4_STREAM_MAX_TOK || (a.gated && ((a.N % 2) != 0 || !a.tiles)) || (a.shared_w && !aligned16(a.shared_w))) return false;
  return (int64_t)a.E * a.N <= INT32_MAX && tensor_map_encoder() != nullptr && umma_status_ptr() != nullptr;
}

int w4_stream_linear(const W4StreamArgs& a, cudaStream_t st) {
  const bool grouped = a.tiles != nullptr;
  const int slots = 2 * sm_count();
  CUtensorMap tw;
  int rc = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, (uint64_t)(grouped ? a.E : 1) * a.N, a.K / 2, (uint64_t)a.K / 2, w4s::ROWS / 2, 128,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  W4SParams p{};
  p.x = a.x; p.ldx = a.ldx;
  const int G = a.K / 128;
  auto scales = [&](const void* sp, int64_t sn, int64_t sg) { return W4SParams::Scales{sp, sn, sg, scale_bytes(sp, a.scale_dtype, sn, sg, G)}; };
  p.sc = scales(a.scale, a.s_stride_n, a.s_stride_g);
  p.s_expert_elems = (int64_t)a.N * G;
  p.shared_e = -1;
  CUtensorMap tw2 = tw;
  if (a.shared_w) {
    rc = make_tmap_2d(&tw2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.shared_w, a.N, a.K / 2, (uint64_t)a.K / 2, w4s::ROWS / 2, 128, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    p.sc2 = scales(a.shared_scale, a.shared_stride_n, a.shared_stride_g);
    p.shared_e = a.E;
  }
  p.out = a.out; p.ldo = a.ldo; p.M = a.M; p.N = a.N; p.K = a.K;
  p.half = a.N / 2;
  p.flip = a.layout == B2Q_W4_NMAJOR_S4 ? 0x00080008u : 0u;
  p.tiles = a.tiles; p.expert_offsets = a.expert_offsets; p.row_map = a.row_map; p.row_div = a.row_div > 0 ? a.row_div : 1; p.out_map = a.out_map;
  p.status = umma_status_ptr();
  if (!p.status) return B2Q_ERR_CUDA;
  p.sps = (a.K + 255) / 256;
  p.strips = a.gated ? (p.half + w4s::ROWS / 2 - 1) / (w4s::ROWS / 2) : (a.N + w4s::ROWS - 1) / w4s::ROWS;
  int64_t work = (int64_t)p.strips * (grouped ? a.tile_cap : 1);
  if (!grouped) {
    const W4SPlan pl = plan(a.N, a.K);
    if (pl.cut && room(pl, a.partials, a.partial_bytes)) {
      p.units = pl.strips * pl.sps; p.partials = reinterpret_cast<float4*>(a.partials);
      p.arrivals = reinterpret_cast<Arrivals*>(reinterpret_cast<uint8_t*>(a.partials) + sum_bytes(pl.grid)); p.tag = arrivals_tag(); p.epoch = arrivals_epoch();
      if (!p.epoch) return B2Q_ERR_CUDA;
      work = pl.grid;
    }
  }
  if (work > INT32_MAX) return B2Q_ERR_LIMIT;
  const int grid = (int)(work < slots ? work : slots);
  // A grouped launch touches nothing before the kernels in front of it are done; a dense one streams its weights before that,
  // which needs the caller's word that no kernel in front writes them.
  const int mode = tls().overlap_mode;
  const bool overlap = grouped ? mode > 0 : mode == 2;
  return a.bf16 ? launch_scale<true>(a.scale_dtype, a.gated, tw, tw2, p, grid, overlap, st) : launch_scale<false>(a.scale_dtype, a.gated, tw, tw2, p, grid, overlap, st);
}

}  // namespace b2q
