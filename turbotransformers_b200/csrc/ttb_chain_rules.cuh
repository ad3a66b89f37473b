// Rules of the chain kernel (ttb_chain.cu) that do not depend on its data: who computes and writes what on a grid of any size. Host code
// as well, so that they can be checked without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TTB_CHAIN_FN __host__ __device__ __forceinline__
#else
#define TTB_CHAIN_FN inline
#endif

namespace ttb {
namespace chain {

constexpr int kBiasUnits = 16;  // units of eight columns whose biases a CTA has room for

// A product's units are dealt out as evenly as they go: CTA `cta` of `ctas` computes units [first_unit(cta), first_unit(cta + 1)). (Of a
// product of 2^24 columns the products below stay under 2^32 on up to 2047 CTAs.)
TTB_CHAIN_FN uint32_t first_unit(uint32_t units, uint32_t cta, uint32_t ctas) { return units * cta / ctas; }

// Every CTA normalises all rows for itself; their copy in memory is written a row by one CTA, so that there have to be as many: the grid is one
// CTA for each SM that the process sees. (Dealt out round the grid instead, 17 tokens of BERT-base took 357 us for 352.)
TTB_CHAIN_FN bool writes_row(int row, int cta) { return row == cta; }
TTB_CHAIN_FN bool rows_have_writers(int64_t rows, int64_t ctas) { return rows <= ctas; }

// The widest product with a bias that a grid takes, in columns (dealt out unevenly, a CTA may have a unit more than another).
TTB_CHAIN_FN int64_t bias_columns(int64_t ctas) { return (kBiasUnits - 1) * 8 * ctas; }

}  // namespace chain
}  // namespace ttb
