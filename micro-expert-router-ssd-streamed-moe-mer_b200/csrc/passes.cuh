// How a group of pairs is cut into token passes.  No CUDA types, so that the rule can be run without a GPU.
#pragma once

#include <stdint.h>

// Up to `tpp` pairs go into one pass, and there are as few passes as that allows.  The streaming kernels (tpp 4 or 8) fill every pass but
// the last.  The GEMM kernels (16 .. 128) work at a width of the pass's pairs, 16 at a time, and a narrow pass still has all the
// weights to dequantise: the units of 16 are dealt evenly, so that no pass is more than one unit wider than another (1025 pairs: two
// passes of 128, six of 112, the last of 97; full passes would leave one of a single pair).
struct PassCut {
  uint32_t passes, step, wider;  // the first `wider` passes hold 16 pairs more than `step`
  __host__ __device__ PassCut(uint32_t n, uint32_t tpp, uint32_t tpp_shift) : passes((n + tpp - 1) >> tpp_shift), step(tpp), wider(0) {
    if (tpp >= 16 && passes > 1) {
      const uint32_t units = (n + 15) >> 4;
      step = units / passes * 16, wider = units % passes;
    }
  }
  // Pairs of pass i, of which at most `left` are to be had.
  __host__ __device__ uint32_t count(uint32_t i, uint32_t left) const {
    const uint32_t c = i < wider ? step + 16 : step;
    return c < left ? c : left;
  }
};
