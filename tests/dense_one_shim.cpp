// dense_one_shim.cpp — test harness only: the one-block rule of small clouds,
// compiled with the host compiler.
#include "../turbotops_gb300/csrc/tt_dense_one.h"

extern "C" int dense_one_block(uint32_t n, uint32_t dim) { return tt::dense_one_block(n, dim); }
extern "C" uint32_t dense_one_floats() { return tt::kOneFloats; }
extern "C" uint32_t dense_one_points() { return tt::kOneN; }
