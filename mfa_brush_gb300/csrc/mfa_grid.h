// mfa_grid.h -- launch shapes of the rebuild kernels and of the k-space tables (plain C++).
#pragma once
#include <algorithm>
#include <cstdint>

namespace mfa {

constexpr int SORT_T = 512;     // threads per block of k_sort
constexpr int SORT_PER_SM = 2;  // its blocks per SM (3 or 4: 0.5-2 % slower steps, fewer registers)
constexpr int NL_T = 128;       // threads per block of k_nlist
constexpr int NL_PER_SM = 8;    // its blocks per SM
constexpr int NL_G = 8;         // its lanes per particle in the form for few particles

// Blocks: what is resident together, no more than n particles fill.  n is up to 2^30, its lanes are more than
// an int holds.
inline int sort_blocks(int64_t n, int nsm) {
  return (int)std::min<int64_t>((n + SORT_T - 1) / SORT_T, (int64_t)nsm * SORT_PER_SM);
}
inline int list_blocks(int64_t n, int nsm) {
  return (int)std::min<int64_t>((n * NL_G + NL_T - 1) / NL_T, (int64_t)nsm * NL_PER_SM);
}

constexpr int KS_TAB_T = 256;  // threads of a k_ks_tables block
// Blocks of the tables of nq charges, a thread per entry, up to the 2^32 entries that the kernel's unsigned index
// holds (the FP64 mode's, with the q Z columns, pass 2^31 from 16 million charges on); -1 beyond.
inline int table_blocks(int64_t nq, int ncol) {
  const int64_t entries = nq * ncol;
  return entries <= 0xFFFFFFFFll - KS_TAB_T ? (int)((entries + KS_TAB_T - 1) / KS_TAB_T) : -1;
}

}  // namespace mfa
