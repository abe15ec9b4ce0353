// Batched step and links for the D3Q15 lattice, f64 storage (batch.cuh).
#include "batch.cuh"

namespace aslb {
cudaError_t batch_step_q15_f64(const BatchDom* doms, int ndom, const BatchWork& w, int links, const StepParams& p,
                             int parity_in, int shape, cudaStream_t st) {
  return batch_step_impl<15, double>(doms, ndom, w, links, p, parity_in, shape, st);
}
cudaError_t batch_links_q15_f64(const BatchBc* bcs, int nbc, long long nlinks, int parity, cudaStream_t st) {
  return batch_links_impl<15, double>(bcs, nbc, nlinks, parity, st);
}
}  // namespace aslb
