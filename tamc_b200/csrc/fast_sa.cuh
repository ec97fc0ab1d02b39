// fast_sa.cuh -- colour-ordered SA kernel interface.
#pragma once
#include <algorithm>

#include "fast_common.cuh"

namespace tamc {

struct SaFastArgs {
  FastInst F;
  const float* betas;        // [nbeta] device
  uint32_t nbeta;
  uint2 key;                 // Philox key (seed)
  uint32_t R;                // replicas
  const uint32_t* init_words;  // [ceil(R/32)][n] original site order, or null for random
  uint32_t* words_out;       // [ceil(R/32)][n] original site order, zeroed by the caller
  float* energies_out;       // [R]
};

enum { SA_WORDS = 0, SA_TABLE, SA_SLICED };  // k_sa_fast, k_sa_tab, k_sa_sl
struct SaTile {
  int kind = SA_WORDS;
  uint32_t nq = 2;       // quads per CTA (replicas per CTA = 4*nq)
  uint32_t T = 512;      // threads per CTA
  bool smem_csr = true;  // instance held in shared memory; SA_TABLE: the table without the site's own spin
  size_t smem = 0;
};

// (`largest_class`: sites of the largest colour class)
SaTile sa_fast_choose(tamc_gpu* g, const FastInst& F, uint32_t R, uint32_t largest_class, uint32_t nbeta);
// Device-side conversion of SA words to the reference's packed byte layout.
void sa_pack_states(cudaStream_t st, const uint32_t* words, uint32_t n, uint32_t R, uint8_t* out);
void sa_fast_launch(cudaStream_t st, const SaFastArgs& a, const SaTile& t);
// The tile sa_fast_choose has cached for this shape, else the heuristic tile;
// never times candidates, so it launches and allocates nothing.
SaTile sa_fast_peek(const tamc_gpu* g, const FastInst& F, uint32_t R, uint32_t largest_class, uint32_t nbeta);
// Sites of the instance's largest colour class.
inline uint32_t largest_class(const tamc_inst* d) {
  uint32_t m = 1;
  for (size_t c = 0; c + 1 < d->color_off.size(); ++c) m = std::max(m, d->color_off[c + 1] - d->color_off[c]);
  return m;
}

}  // namespace tamc
