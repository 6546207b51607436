// Host-side interface of the FP8 streaming kernel of up to sixteen tokens (w8_stream.cu).
#pragma once
#include "common.cuh"

namespace b2q {

constexpr int W8_STREAM_MAX_TOK = 16;

struct W8StreamArgs {
  const void* x; int64_t ldx; bool bf16;
  const void* w; int fmt;
  const void* scale; int scale_dtype; int scale_mode;
  void* out; int64_t ldo;
  int M, N, K;
};

bool w8_stream_supported(const W8StreamArgs& a);
bool w8_stream_preferred(const W8StreamArgs& a);
int w8_stream_linear(const W8StreamArgs& a, cudaStream_t st);

}  // namespace b2q
