// Mixed-precision batched determinant of lowest-Landau-level matrices built from
// coordinates: the kernels of mixed_kernels.cuh on a source that builds the rows.
// Its own translation unit, so that its instantiations compile in parallel with
// the others.

#include "mixed_kernels.cuh"

namespace lufqhe {

int launch_mixed_lll(const double2 *Z, int n, long long batch, double *logabs, double *phase,
                     int8_t *parity, int32_t *status, cudaStream_t stream) {
  return launch_mixed_src(LllSource{Z}, n, batch, logabs, phase, parity, status, stream, [&] {
    return launch_plain_lll(Z, n, batch, ARITH_FUSED, logabs, phase, parity, status, stream,
                            LUFQHE_ST_FP64);
  });
}

}  // namespace lufqhe
