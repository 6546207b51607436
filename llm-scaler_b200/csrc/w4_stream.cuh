// Host-side interface of the INT4 decode streaming kernel (w4_stream.cu).
#pragma once
#include "common.cuh"

namespace b2q {

constexpr int W4_STREAM_MAX_TOK = 8;      // tokens per tile

struct W4StreamArgs {
  const void* x; int64_t ldx; bool bf16;
  const void* w; int layout;                                     // N-major nibbles, offset or two's complement
  const void* scale; int scale_dtype; int64_t s_stride_n, s_stride_g;
  void* out; int64_t ldo;
  int M, N, K;
  int tile;                                                      // tokens per tile: M, or the height the tile list was built with
  bool gated = false;                                            // rows are gate then up; out = silu(gate) * up, N / 2 wide
  const int32_t* tiles = nullptr; int tile_cap = 0; int E = 1;   // grouped
  const int32_t* expert_offsets = nullptr; const int32_t* row_map = nullptr; int row_div = 1; const int32_t* out_map = nullptr;
  // grouped: "expert" E of the tile list, a weight of its own of the same shape, scale type and nibbles
  const void* shared_w = nullptr; const void* shared_scale = nullptr; int64_t shared_stride_n = 0, shared_stride_g = 0;
  void* partials = nullptr; size_t partial_bytes = 0;            // dense: w4_stream_partial_bytes(M, N, K), or strips stay whole
};

bool w4_stream_supported(const W4StreamArgs& a);
int w4_stream_linear(const W4StreamArgs& a, cudaStream_t st);
size_t w4_stream_partial_bytes(int64_t M, int64_t N, int64_t K);

// Dense launches that are better off here than in smallm.cuh, whose 16-row strips need no sum between CTAs and cost less to start, but
// come in rounds of three CTAs per SM that take their time for all of k.  By a fitted cost of both in us; one / eight tokens, there and
// here: 4096 x 4096 8.3 / 8.8 and 13.4, 5888 x 5888 10.0 / 11.3 and 13.9, 10240 x 4096 14.2 / 15.5 and 15.1, but 7168 x 4224 14.3 / 17.3
// and 13.4, 28672 x 1024 13.0 / 13.9 and 11.5, 2048 x 16384 26.8 / 30.7 and 17.4, 10240 x 8192 27.2 / 30.5 and 17.9.
// Strips that should be cut, with no room for their partial sums, stay whole, about 1 us per stage: one / eight tokens, there and here, 2048 x
// 16384 25.6 / 29.9 and 38.8 / 44.1, 8192 x 8192 25.1 / 29.2 and 30.7 / 34.7, but 57344 x 8192 101 / 136 and 68 / 73, 24576 x 4096 24.9 and 18.9.
// Few strips are cut into many pieces, and whoever comes last adds up all of a strip's sums: 0.23 us per contributor beyond ten.  Scales that
// cannot be fetched 16 bytes at a time: 1 us more.  By 655 launches of N = 64 .. 57344 and K = 1024 .. 28672, seven of them 2 to 7 % slower by
// the rule than on the other side, against over a hundred by up to 49 % without these two.  One token, there and here: 1024 x 8192 12.3 and 17.9, 512 x 8192
// 11.7 and 17.4, 256 x 16384 25.2 and 28.3, but 1024 x 16384 26.2 and 20.0, 512 x 28672 46.7 and 32.7; seven tokens, 69 groups, 2128 x 8832 15.5 and 19.2.
bool w4_stream_preferred(const W4StreamArgs& a);

// Grouped launches of the expert pipeline: up to four rows per expert on average; from about six on tiles of eight tokens repeat too
// much of the decoding.  Whole pass in us against the tcgen05 kernel behind its pre-passes, 128 experts of 2048 x 768, top-8, at 1 / 16 /
// 64 / 128 tokens: 28 / 82 / 119 / 163 against 31 / 89 / 127 / 145; 32 of 2048 x 1024, top-4, at 4 / 32 / 64: 32 / 51 / 69 against 39 / 60 / 66.
inline bool w4_stream_grouped_preferred(int64_t rows, int E) { return rows <= 4 * (int64_t)E; }

}  // namespace b2q
