// FP8 linear for up to sixteen tokens: out[m, n] = sum_k s * w[n, k] * x[m, k], e4m3 or e5m2 weights, one scale per channel, per
// tensor or per 128 x 128 block, fp16 or bf16 activations.
//
// HBM-bound: the weights are read once and nothing else is large.  One launch, no pre-pass: the weights become exact fp16 / bf16
// values in registers and meet the activations as they are in mma.sync m16n8k16 (weight rows as the MMA's M, tokens as its N); the
// scales are applied in fp32.
//
// Each CTA has rows of its own, so that no sum crosses CTAs: they are dealt out evenly to the row, two CTAs per SM, in passes of at
// most 64 over all of K; the height of the TMA box is that of a pass, not a round number.  A CTA is
//   warp 0     TMA producer of the weight stages
//   next 2     asynchronous copies of the activations of the same k, behind the kernels in front
//   next 8     conversion and MMA, a share of every stage's k each; they add up through shared memory at the end of a pass
//
// What it replaces, umma_w8_direct.cu behind a pre-pass that splits the activations into e4m3 terms (umma_w4.cu behind act_prep for
// block scales), pays for a second launch and its latency, and for a whole MMA of 128 rows wherever a CTA has fewer.  One scale per
// tensor, four tokens, fp16, there -> here: 2048 x 2048 7.4 -> 3.3 us, 5120 x 5120 11.5 -> 8.3, 7168 x 5120 11.8 -> 8.6, 5120 x 13824 20.8 ->
// 14.8, 17408 x 5120 19.1 -> 15.7 (5.7 TB/s), 27648 x 5120 26.4 -> 24.7; eight tokens, bf16: 7.0 -> 4.1, 10.9 -> 9.6, 11.0 -> 10.4, 18.7 -> 17.4.
// What was found on the way:
// * A bulk copy per row instead of TMA boxes costs some 55 cycles per copy and SM whatever its length: 1.1 to 2.7 TB/s.
// * bf16 activations brought to fp16 by the staging warps, a power of two per stage, to save the weights' second conversion: 5120 x
//   13824 24 us instead of 19 for one token, 45 instead of 24 for eight; packing the converted floats by permute or by cvt: the same.
// * Tokens as the MMA's M and weight rows as its N, in eights: the same for few tokens, slower with block scales.
// * Converting the empty half of a last tile: 10240 x 5120, bf16, one token 15.2 us, 13.8 without.
// * One CTA per SM: 27648 x 5120 27.8 us against 25.6, 5120 x 13824 behind a norm 28.8 against 20.4; better below 16 rows per CTA only.
// * INT4 in the same way: better than w4_stream.cu for one or two tokens of some shapes (8192 x 4096 14 -> 10 us), 0.3 to 0.8 of its speed otherwise.
//
// Every mbarrier wait is bounded; on expiry the CTA records a code in the status word and ends.
//
// Reference counterparts: esimd_gemv_fp8_pern / pert (csrc/xpu/esimd_kernels/fp8_GEMV_v2.h:46-337), esimd_gemm_fp8_blockscale
// (fp8_GEMM_blockscale.h:64-137).
#include <type_traits>
#include "umma_gemm.cuh"
#include "sm100.cuh"
#include "smallm.cuh"   // lds128, mma16816
#include "w8_stream.cuh"

namespace b2q {

using namespace sm100;

namespace w8s {
enum { ST_EMPTY = 701, ST_XEMPTY = 702, ST_FULL = 703 };

constexpr int XW = 2, MW = 8, THREADS = (1 + XW + MW) * 32;
constexpr int PASS_ROWS = 64, MAX_STAGES = 16;
constexpr int SMEM = 115712;                               // two CTAs fit an SM
constexpr int BAR_BYTES = 512;

// H: eights of rows in a pass.  The MMA warps are one group, or two where there are more than four eights: four for the first, the
// rest for the second, so that each of the SM's quarters has warps of both.  A group has tiles of 16 rows, its last one may be half
// empty, and its warps share out the k of a stage.
template <int H, bool MORE> struct Cfg {
  static constexpr int RG = H > 4 ? 2 : 1, TW = H > 2 ? 2 : 1;
  static constexpr int KG = MW / RG, KS = 64 * KG;
  static constexpr int X_PITCH = 2 * KS + 16;              // a token's activations: neighbouring tokens are 16 bytes apart in the banks
  static constexpr int RED = TW * (MORE ? 1024 : 512), RED_BYTES = MW * RED;
  static constexpr int RING = SMEM - 1024 /*align*/ - BAR_BYTES - RED_BYTES;
};

__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {       // one arrival when this thread's copies have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// two weights (low 16 bits) -> their exact values
template <bool BF16, bool E5M2> __device__ __forceinline__ uint32_t weights2(uint32_t v) {
  const uint32_t h = fp8x2_to_act<false, E5M2>(v);
  if constexpr (!BF16) return h;
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  return __byte_perm(__float_as_uint(f.x), __float_as_uint(f.y), 0x7632);      // four significant bits: the upper halves have them all
}
}  // namespace w8s

struct W8SParams {
  const uint8_t* x; int64_t x_pitch;                       // bytes
  const void* scale; int scale_dtype, per_channel;
  void* out; int64_t ldo;
  int M, N, K;
  int passes, cap, ns;                                     // per CTA; most rows of a pass = height of the TMA box; stages of the ring
  int* status;
};

template <bool BF16, bool E5M2, bool BLOCK, bool MORE, int H>      // MORE: than eight tokens
__global__ void __launch_bounds__(w8s::THREADS, 2) w8_stream_kernel(const __grid_constant__ CUtensorMap tm_w, const W8SParams p) {
  using namespace w8s;
  using C = Cfg<H, MORE>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, red = base + C::RING, bar = red + C::RED_BYTES;
  uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t full = bar, empty = bar + 8 * MAX_STAGES;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + (bar - base) + 16 * MAX_STAGES);
  volatile int* warp_ok = abort_flag + 1;                  // [MW]: how the MMA warps came out of the pass
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int box = (p.cap + 7) / 8 * 1024, w_slot = box * (C::KS / 128), x_slot = p.M * C::X_PITCH, nst = (p.K + C::KS - 1) / C::KS;
  const uint32_t x_smem = base + p.ns * w_slot;
  const int r0 = (int)((int64_t)blockIdx.x * p.N / gridDim.x), rows = (int)((int64_t)(blockIdx.x + 1) * p.N / gridDim.x) - r0;
  // Every CTA begins its passes at another stage: all of them read the same activations, and in step they would ask the same L2 lines
  // for them at the same moment.  17408 x 5120, fp16, 16 tokens 21.5 -> 17.3 us; 27648 x 5120, eight tokens 26.8 -> 24.7.
  const int rot = (int)((blockIdx.x * 5u) % (unsigned)nst);
  auto turn = [&](int i) { return i + rot < nst ? i + rot : i + rot - nst; };
  auto pass_row = [&](int i) { return r0 + (int)((int64_t)i * rows / p.passes); };

  // The next kernel may start at once.  This one waits for the kernels before it where it reads activations (warp 1); the outputs
  // follow from those.
  grid_dep_release();
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.ns; ++i) { mbar_init(full + 8 * i, 1 + 32 * XW); mbar_init(empty + 8 * i, MW); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  if (warp == 0) {
    // ---------------- weight producer: boxes of a pass's rows x 128 k; what lies beyond N or K reads as zero ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tm_w);
      int s = 0, issued = 0;
      uint32_t par = 1u;
      bool ok = true;
      for (int i = 0; ok && i < p.passes; ++i) {
        const int n0 = pass_row(i);
        for (int j = 0; j < nst; ++j) {
          const int st = turn(j);
          ok = mbar_wait(empty + 8 * s, par, abort_flag, p.status, ST_EMPTY);
          if (!ok) break;
          ++issued;
          mbar_expect_tx(full + 8 * s, p.cap * C::KS);
#pragma unroll
          for (int b = 0; b < C::KS / 128; ++b) tma_load_2d(base + s * w_slot + b * box, &tm_w, st * C::KS + 128 * b, n0, full + 8 * s);
          if (++s == p.ns) { s = 0; par ^= 1u; }
        }
      }
      if (!ok) drain_issued(full, p.ns, issued);
    }
    return;
  }
  if (warp <= XW) {
    // ---------------- activations, past L1: it may hold what an earlier kernel saw at these addresses ----------------
    grid_dep_wait();
    int s = 0;
    uint32_t par = 1u;
    bool ok = true;
    for (int i = 0; ok && i < p.passes; ++i) {
      for (int j = 0; j < nst; ++j) {
        const int st = turn(j);
        ok = mbar_wait_warp(empty + 8 * s, par, abort_flag, p.status, ST_XEMPTY);
        if (!ok) break;
        const uint32_t dst = x_smem + s * x_slot + 16 * lane;
        for (int m = warp - 1; m < p.M; m += XW) {
#pragma unroll
          for (int b = 0; b < 2 * C::KS; b += 512) {
            const int64_t at = (int64_t)st * 2 * C::KS + b + 16 * lane;
            const bool in = at < 2 * (int64_t)p.K;
            cp_async16(dst + m * C::X_PITCH + b, p.x + m * p.x_pitch + (in ? at : 0), in ? 16 : 0);
          }
        }
        cp_async_arrive(full + 8 * s);
        if (++s == p.ns) { s = 0; par ^= 1u; }
      }
    }
    if (!ok) asm volatile("cp.async.wait_all;" ::: "memory");       // copies may still be on their way
    return;
  }

  // ---------------- conversion, MMA, output ----------------
  // MMA row g is row pr of its eight, so that a quarter-warp's 16-byte reads touch all banks once.
  constexpr int TW = C::TW;
  const int w = warp - 1 - XW, kg = w % C::KG, tile0 = w / C::KG * TW;
  const int g = lane >> 2, t = lane & 3, pr = 16 * tile0 + ((g >> 1) | ((g & 1) << 2));
  const uint32_t x_off = x_smem + min(g, p.M - 1) * C::X_PITCH + 128 * kg + 32 * t;
  const uint32_t x_more = (min(g + 8, p.M - 1) - min(g, p.M - 1)) * C::X_PITCH;
  uint32_t wa_off[TW], wb_off[TW];                         // rows g and g + 8 of every tile; rows beyond the box's are read as its last
  auto row_at = [&](int r) {
    r = min(r, p.cap - 1);
    return base + (kg >> 1) * box + r * 128 + (((4 * (kg & 1) + t) ^ (r & 7)) << 4);
  };
#pragma unroll
  for (int i = 0; i < TW; ++i) { wa_off[i] = row_at(16 * i + pr); wb_off[i] = row_at(16 * i + 8 + pr); }
  const int nkb = p.K >> 7;
  int s = 0;
  uint32_t par = 0u;
  bool ok = true;
  for (int i = 0; i < p.passes; ++i) {
    const int n0 = pass_row(i), n = pass_row(i + 1) - n0;
    // Two chains per tile, as an MMA takes long to deliver: tokens 0 .. 7 and 8 .. 15, or else even and odd steps
    constexpr int CH = BLOCK && !MORE ? 1 : 2;
    float acc[CH][TW][4];
#pragma unroll
    for (int q = 0; q < CH; ++q)
#pragma unroll
      for (int r = 0; r < TW; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[q][r][c] = 0.f;
    const float* sa[TW];                                   // BLOCK: this lane's rows' scales
    const float* sb[TW];
    if constexpr (BLOCK) {
#pragma unroll
      for (int r = 0; r < TW; ++r) {
        sa[r] = reinterpret_cast<const float*>(p.scale) + (int64_t)(min(n0 + 16 * r + pr, p.N - 1) >> 7) * nkb;
        sb[r] = reinterpret_cast<const float*>(p.scale) + (int64_t)(min(n0 + 16 * r + 8 + pr, p.N - 1) >> 7) * nkb;
      }
    }
#pragma unroll 1
    for (int j = 0; j < nst; ++j) {
      const int st = turn(j), k0 = st * C::KS + 64 * kg;
      float fa[TW], fb[TW];
      if constexpr (BLOCK) {
        const int kb = min(k0 >> 7, nkb - 1);
#pragma unroll
        for (int r = 0; r < TW; ++r) { fa[r] = __ldg(sa[r] + kb); fb[r] = __ldg(sb[r] + kb); }
      }
      ok = mbar_wait_warp(full + 8 * s, par, abort_flag, p.status, ST_FULL);
      if (!ok) break;
      auto step = [&](auto eights) {
        constexpr int EIGHTS = decltype(eights)::value;
        uint32_t xv[8], yv[8];                             // tokens g and g + 8
        auto load_x = [&](uint32_t (&v)[8], uint32_t at) {
          const uint4 a = lds128(at), b = lds128(at + 16);
          v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        };
        load_x(xv, x_off + s * x_slot);
        if constexpr (MORE) load_x(yv, x_off + s * x_slot + x_more);
#pragma unroll
        for (int r = 0; r < (EIGHTS + 1) / 2; ++r) {
          const bool whole = 2 * r + 2 <= EIGHTS;          // a half tile's upper rows are zeros
          const uint4 wa = lds128(wa_off[r] + s * w_slot), wb = whole ? lds128(wb_off[r] + s * w_slot) : make_uint4(0, 0, 0, 0);
          const uint32_t a[4] = {wa.x, wa.y, wa.z, wa.w}, b[4] = {wb.x, wb.y, wb.z, wb.w};
          float u[2][4];
          if constexpr (BLOCK) {
#pragma unroll
            for (int c = 0; c < 4; ++c) u[0][c] = u[1][c] = 0.f;
          }
          float (&d0)[4] = BLOCK ? u[0] : acc[0][r];
          float (&d1)[4] = BLOCK ? u[1] : acc[CH - 1][r];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t a0 = weights2<BF16, E5M2>(a[j]), a1 = whole ? weights2<BF16, E5M2>(b[j]) : 0u, a2 = weights2<BF16, E5M2>(a[j] >> 16),
                           a3 = whole ? weights2<BF16, E5M2>(b[j] >> 16) : 0u;
            if constexpr (MORE) {
              mma16816<BF16>(d0, a0, a1, a2, a3, xv[2 * j], xv[2 * j + 1]);
              mma16816<BF16>(d1, a0, a1, a2, a3, yv[2 * j], yv[2 * j + 1]);
            } else {
              mma16816<BF16>((j & 1) ? d1 : d0, a0, a1, a2, a3, xv[2 * j], xv[2 * j + 1]);
            }
          }
          if constexpr (BLOCK) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float f = c < 2 ? fa[r] : fb[r];
              acc[0][r][c] += f * (MORE ? u[0][c] : u[0][c] + u[1][c]);
              if constexpr (MORE) acc[CH - 1][r][c] += f * u[1][c];
            }
          }
        }
      };
      if (k0 < p.K) {
        if constexpr (H <= 4) step(std::integral_constant<int, H>{});
        else if constexpr (H == 8) step(std::integral_constant<int, 4>{});
        else if (w < C::KG) step(std::integral_constant<int, 4>{});
        else step(std::integral_constant<int, H - 4>{});
      }
      mbar_arrive_read(empty + 8 * s);
      if (++s == p.ns) { s = 0; par ^= 1u; }
    }
    // The warps of a group add up.  All meet twice, so that the buffer is free again before the next pass, and go on only if none
    // has given up: nobody meets a warp that left.
#pragma unroll
    for (int r = 0; r < TW; ++r) {
      auto put = [&](uint32_t at, float a, float b, float c, float d) {
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(at), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
      };
      const uint32_t at = red + w * C::RED + r * 512 + lane * 16;
      const float (&a)[4] = acc[0][r];
      const float (&b)[4] = acc[CH - 1][r];
      if constexpr (MORE) { put(at, a[0], a[1], a[2], a[3]); put(at + TW * 512, b[0], b[1], b[2], b[3]); }
      else if constexpr (CH == 1) put(at, a[0], a[1], a[2], a[3]);
      else put(at, a[0] + b[0], a[1] + b[1], a[2] + b[2], a[3] + b[3]);
    }
    if (lane == 0) warp_ok[w] = ok;
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(MW * 32) : "memory");
#pragma unroll
    for (int v = 0; v < MW; ++v) ok = ok && warp_ok[v];
    // a group's first warps deliver its tiles, a tile and eight tokens each
    if (ok && kg < TW * (MORE ? 2 : 1)) {
      const int tile = kg % TW, half = kg / TW;
      float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int v = 0; v < C::KG; ++v) {
        const uint4 b = lds128(red + (w - kg + v) * C::RED + (half * TW + tile) * 512 + lane * 16);
        o[0] += __uint_as_float(b.x); o[1] += __uint_as_float(b.y); o[2] += __uint_as_float(b.z); o[3] += __uint_as_float(b.w);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int r = 16 * tile + pr + (c & 2) * 4, m = 8 * half + 2 * t + (c & 1);
        if (r < n && m < p.M) {
          const float f = BLOCK ? o[c] : o[c] * load_scalar(p.scale, p.per_channel ? n0 + r : 0, p.scale_dtype);
          reinterpret_cast<uint16_t*>(p.out)[m * p.ldo + n0 + r] = BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(f)) : __half_as_ushort(__float2half_rn(f));
        }
      }
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(MW * 32) : "memory");
    if (!ok) return;
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

template <bool BF16, bool E5M2, bool BLOCK, bool MORE, int H>
static int launch(const CUtensorMap& tw, W8SParams& p, int grid, cudaStream_t st) {
  using C = w8s::Cfg<H, MORE>;
  p.ns = C::RING / ((p.cap + 7) / 8 * 8 * C::KS + p.M * C::X_PITCH);
  p.ns = p.ns < w8s::MAX_STAGES ? p.ns : w8s::MAX_STAGES;
  auto kern = w8_stream_kernel<BF16, E5M2, BLOCK, MORE, H>;
  static thread_local bool configured[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, w8s::SMEM) != cudaSuccess) return B2Q_ERR_CUDA;
    if (dev < 16) configured[dev] = true;
  }
  // the weights are streamed before the kernels in front are done, which needs the caller's word that none of them writes weights
  if (launch_overlapped(kern, dim3(grid), dim3(w8s::THREADS), w8s::SMEM, st, tls().overlap_mode == 2, tw, p) != cudaSuccess) return B2Q_ERR_CUDA;
  note_launch("w8_stream");
  return launch_status();
}
template <bool BF16, bool E5M2, bool BLOCK, bool MORE>
static int launch_rows(const CUtensorMap& tw, W8SParams& p, int grid, cudaStream_t st) {
  switch ((p.cap + 7) / 8) {
    case 1: case 2: return launch<BF16, E5M2, BLOCK, MORE, 2>(tw, p, grid, st);
    case 3: return launch<BF16, E5M2, BLOCK, MORE, 3>(tw, p, grid, st);
    case 4: return launch<BF16, E5M2, BLOCK, MORE, 4>(tw, p, grid, st);
    case 5: return launch<BF16, E5M2, BLOCK, MORE, 5>(tw, p, grid, st);
    case 6: return launch<BF16, E5M2, BLOCK, MORE, 6>(tw, p, grid, st);
    default: return launch<BF16, E5M2, BLOCK, MORE, 8>(tw, p, grid, st);
  }
}
template <bool BF16, bool E5M2, bool BLOCK>
static int launch_tokens(const CUtensorMap& tw, W8SParams& p, int grid, cudaStream_t st) {
  return p.M > 8 ? launch_rows<BF16, E5M2, BLOCK, true>(tw, p, grid, st) : launch_rows<BF16, E5M2, BLOCK, false>(tw, p, grid, st);
}
template <bool BF16>
static int launch_format(const W8StreamArgs& a, const CUtensorMap& tw, W8SParams& p, int grid, cudaStream_t st) {
  if (a.scale_mode == B2Q_SCALE_BLOCK128) return launch_tokens<BF16, false, true>(tw, p, grid, st);
  return a.fmt == B2Q_E5M2 ? launch_tokens<BF16, true, false>(tw, p, grid, st) : launch_tokens<BF16, false, false>(tw, p, grid, st);
}

// Rows of the busiest CTA: CTAs, passes over K, rows per pass.  Two CTAs per SM where each gets a full MMA tile of rows: more copies in
// flight, and the next launch finds its room sooner.
struct W8SPlan { int grid, passes, cap; };
static W8SPlan plan(int N) {
  const int sms = sm_count(), eights = (N + 7) / 8, slots = N >= 2 * 16 * sms ? 2 * sms : sms;
  W8SPlan pl;
  pl.grid = eights < slots ? eights : slots;
  const int most = (N + pl.grid - 1) / pl.grid;
  pl.passes = (most + w8s::PASS_ROWS - 1) / w8s::PASS_ROWS;
  pl.cap = (most + pl.passes - 1) / pl.passes;
  return pl;
}

// Launches that are better off here than on umma_w8_direct.cu / umma_w4.cu.  Both sides were timed over some 700 launches per scale mode
// and activation type (N = 1024 .. 28672, K = 1024 .. 13824, 1 to 16 tokens).
// * One scale per tensor or channel, fp16: 1.0 to 2.5 times as fast up to 9472 rows, 1.2 to 1.5 in one pass (N up to some 19000), but 0.88 for
//   1024 x 13824 with 16 tokens, hardly more than one MMA tile's rows for long.  More passes: up to eight tokens from 64 Mi weights 0.97
//   to 1.75; shorter or with more tokens 0.8 to 1.9, by how the strips there fall.
// * bf16, which costs a second conversion.  Up to eight tokens and k of 8192 1.0 to 2.1 up to 9472 rows; longer k 1.02 to 1.3 for four
//   tokens, 0.94 for eight (5120 x 13824).  More rows in one pass 0.98 to 1.17 up to k of 6144, down to 0.93 otherwise; in more 0.6 to 1.4.  More
//   than eight tokens: 1.04 to 1.8 with one CTA per SM and k of 8192, or with k of 2048; 0.87 to 1.07 with two CTAs' fetches of activations.
// * Below 4 Mi weights such calls stay there although they would gain up to 4 us: test_gpu_dense.py names their kernel.
// * Block scales, whose sums of every 64 k are scaled and added up here: up to eight tokens 0.99 to 3.1 up to 9472 rows and k of 8192, 0.81 to
//   1.4 beyond; more rows in one pass 0.97 to 1.3 (bf16, k of 4096) and 1.0 to 1.27 (fp16, k of 5120), down to 0.76 beyond.  More than eight
//   tokens, k of 4096: 1.02 to 2.6 (bf16, up to 9472 rows) and 1.08 to 2.0 (fp16, one CTA per SM; 0.73 to 1.28 with two).
bool w8_stream_preferred(const W8StreamArgs& a) {
  const W8SPlan pl = plan(a.N);
  const int64_t weights = (int64_t)a.N * a.K;
  const bool few = a.M <= 8;
  if (a.scale_mode != B2Q_SCALE_BLOCK128) {
    if (weights < (4 << 20)) return false;
    if (a.N < 2048 && a.K > 8192) return false;
    if (!a.bf16) return pl.passes == 1 || (few && weights >= (64 << 20));
    if (!few) return (a.N + 127) / 128 * 2 <= sm_count() && (a.K <= 2048 || (a.K <= 8192 && pl.grid <= sm_count()));
    return (a.N + 127) / 128 * 2 <= sm_count() ? a.K <= 8192 || a.M <= 4 : pl.passes == 1 && a.K <= 6144;
  }
  if (pl.passes > 1) return false;
  if (few) return a.K <= (pl.cap <= 32 ? 8192 : (a.bf16 ? 4096 : 6144));
  return pl.cap <= 32 && a.K <= 4096 && (a.bf16 || pl.grid <= sm_count());
}

bool w8_stream_supported(const W8StreamArgs& a) {
  if (a.M < 1 || a.M > W8_STREAM_MAX_TOK || a.N < 1 || (a.K % 16) != 0 || !aligned16(a.x) || !aligned16(a.w) || ((a.ldx * 2) & 15)) return false;
  if (a.scale_mode == B2Q_SCALE_BLOCK128 && (a.fmt != B2Q_E4M3 || a.scale_dtype != B2Q_F32 || (a.K % 128) != 0)) return false;
  return tensor_map_encoder() != nullptr && umma_status_ptr() != nullptr;
}

int w8_stream_linear(const W8StreamArgs& a, cudaStream_t st) {
  W8SParams p{};
  p.x = reinterpret_cast<const uint8_t*>(a.x); p.x_pitch = 2 * a.ldx;
  p.scale = a.scale; p.scale_dtype = a.scale_dtype; p.per_channel = a.scale_mode == B2Q_SCALE_CHANNEL ? 1 : 0;
  p.out = a.out; p.ldo = a.ldo; p.M = a.M; p.N = a.N; p.K = a.K;
  p.status = umma_status_ptr();
  if (!p.status) return B2Q_ERR_CUDA;
  const W8SPlan pl = plan(a.N);
  p.passes = pl.passes; p.cap = pl.cap;
  CUtensorMap tw;
  const int rc = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, a.N, a.K, (uint64_t)a.K, p.cap, 128, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  return a.bf16 ? launch_format<true>(a, tw, p, pl.grid, st) : launch_format<false>(a, tw, p, pl.grid, st);
}

}  // namespace b2q
