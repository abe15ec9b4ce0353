// Dispatch of the batched step and links to their instantiations per lattice
// and storage (batch_q15_f32.cu, ...; kernels in batch.cuh).
#include <algorithm>
#include "kernels.h"

namespace aslb {

#define ASLB_BATCH_CASE(Q, T)                                                                                      \
  cudaError_t batch_step_q##Q##_##T(const BatchDom* doms, int ndom, const BatchWork& w, int links,                 \
                                    const StepParams& p, int parity_in, int shape, cudaStream_t st);               \
  cudaError_t batch_links_q##Q##_##T(const BatchBc* bcs, int nbc, long long nlinks, int parity, cudaStream_t st);
ASLB_BATCH_CASE(15, f32)
ASLB_BATCH_CASE(15, f16)
ASLB_BATCH_CASE(15, f64)
ASLB_BATCH_CASE(19, f32)
ASLB_BATCH_CASE(19, f16)
ASLB_BATCH_CASE(19, f64)
ASLB_BATCH_CASE(27, f32)
ASLB_BATCH_CASE(27, f16)
ASLB_BATCH_CASE(27, f64)
#undef ASLB_BATCH_CASE

#define ASLB_BATCH_DISPATCH(what, ...)                                          \
  switch (storage * 32 + q) {                                                   \
    case ST_F32 * 32 + 15: return what##_q15_f32(__VA_ARGS__);                  \
    case ST_F32 * 32 + 19: return what##_q19_f32(__VA_ARGS__);                  \
    case ST_F32 * 32 + 27: return what##_q27_f32(__VA_ARGS__);                  \
    case ST_F16 * 32 + 15: return what##_q15_f16(__VA_ARGS__);                  \
    case ST_F16 * 32 + 19: return what##_q19_f16(__VA_ARGS__);                  \
    case ST_F16 * 32 + 27: return what##_q27_f16(__VA_ARGS__);                  \
    case ST_F64 * 32 + 15: return what##_q15_f64(__VA_ARGS__);                  \
    case ST_F64 * 32 + 19: return what##_q19_f64(__VA_ARGS__);                  \
    case ST_F64 * 32 + 27: return what##_q27_f64(__VA_ARGS__);                  \
  }                                                                             \
  return cudaErrorInvalidValue;

int batch_shape_count() { return 5; }

void batch_work_tables(const std::vector<long long>& tile_cells, int sms, std::vector<long long>& starts,
                       int (&grid)[3], int (&group)[3], long long (&off)[3]) {
  const long long T = (long long)tile_cells.size();
  long long C = 0;
  for (long long c : tile_cells) C += c;
  starts.clear();
  for (int k = 0; k < 3; ++k) {
    const long long G = std::max(1LL, std::min(T, (long long)sms * (k + 2)));
    const int K = (G % 4 == 0) ? 4 : 1;
    const long long NG = G / K;
    grid[k] = (int)G;
    group[k] = K;
    off[k] = (long long)starts.size();
    // group b starts at the first tile whose preceding cells reach b C / NG
    long long t = 0, before = 0;
    for (long long b = 0; b < NG; ++b) {
      const long long target = (long long)(((__int128)b * C + NG - 1) / NG);
      while (t < T && before < target) before += tile_cells[t++];
      starts.push_back(t);
    }
    starts.push_back(T);
  }
}

cudaError_t launch_batch_step(int q, int storage, const BatchDom* doms, int ndom, const BatchWork& w, int links,
                              const StepParams& p, int parity_in, int shape, cudaStream_t st) {
  ASLB_BATCH_DISPATCH(batch_step, doms, ndom, w, links, p, parity_in, shape, st)
}

cudaError_t launch_batch_links(int q, int storage, const BatchBc* bcs, int nbc, long long nlinks, int parity,
                               cudaStream_t st) {
  ASLB_BATCH_DISPATCH(batch_links, bcs, nbc, nlinks, parity, st)
}

}  // namespace aslb
