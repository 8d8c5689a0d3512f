// The calibration kernels (pg_calib.cuh) for 5 to 8 epochs.
#include "pg_calib.cuh"

namespace pg {

void calib_launch_hi(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                     const AdamArgs& adam, cudaStream_t st) {
#define PG_CALIB_DO(KK, JJ) calib_run<KK, JJ>(a, n_segs, n_rep, params, nll, grad, adam, st)
  switch (a.K * 8 + a.J - 9) { PG_CALIB_K(5) PG_CALIB_K(6) PG_CALIB_K(7) PG_CALIB_K(8) }
#undef PG_CALIB_DO
}

int calib_ctas_hi(uint32_t K, uint32_t J) {
  int n = 1;
#define PG_CALIB_DO(KK, JJ) n = calib_resident<KK, JJ>()
  switch (K * 8 + J - 9) { PG_CALIB_K(5) PG_CALIB_K(6) PG_CALIB_K(7) PG_CALIB_K(8) }
#undef PG_CALIB_DO
  return n;
}

}  // namespace pg
