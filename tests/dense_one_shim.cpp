// dense_one_shim.cpp — test harness only: the one-block rule of small clouds,
// compiled with the host compiler.
#include "../turbotops_gb300/csrc/tt_dense_one.h"

extern "C" int dense_one_block(uint32_t n, uint32_t dim, int lp) { return tt::dense_one_block(n, dim, lp != 0); }
extern "C" uint32_t dense_one_stride(uint32_t dim) { return tt::dense_one_stride(dim); }
extern "C" uint32_t dense_one_floats() { return tt::kOneFloats; }
extern "C" uint32_t dense_one_points(int lp) { return lp ? tt::kOneLpN : tt::kOneN; }
