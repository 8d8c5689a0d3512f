// The calibration kernels (pg_calib.cuh) for 1 to 4 epochs.
#include "pg_calib.cuh"

namespace pg {

void calib_launch_lo(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                     const AdamArgs& adam, cudaStream_t st) {
#define PG_CALIB_DO(KK, JJ) calib_run<KK, JJ>(a, n_segs, n_rep, params, nll, grad, adam, st)
  switch (a.K * 8 + a.J - 9) { PG_CALIB_K(1) PG_CALIB_K(2) PG_CALIB_K(3) PG_CALIB_K(4) }
#undef PG_CALIB_DO
}

int calib_ctas_lo(uint32_t K, uint32_t J) {
  int n = 1;
#define PG_CALIB_DO(KK, JJ) n = calib_resident<KK, JJ>()
  switch (K * 8 + J - 9) { PG_CALIB_K(1) PG_CALIB_K(2) PG_CALIB_K(3) PG_CALIB_K(4) }
#undef PG_CALIB_DO
  return n;
}

int calib_ctas_per_sm(uint32_t K, uint32_t J) { return K <= 4 ? calib_ctas_lo(K, J) : calib_ctas_hi(K, J); }

uint32_t calib_chunk() { return CAL_CHUNK; }
uint32_t calib_tab(uint32_t K, uint32_t J) { return calib_row_floats(K, J); }

void calib_launch(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                  const AdamArgs& adam, cudaStream_t st) {
  if (n_segs == 0) return;
  if (a.K <= 4) calib_launch_lo(a, n_segs, n_rep, params, nll, grad, adam, st);
  else calib_launch_hi(a, n_segs, n_rep, params, nll, grad, adam, st);
}

}  // namespace pg
