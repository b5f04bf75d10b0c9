// One pass mode and stored precision of the interval steppers per object file: MARCH_MODE, MARCH_PREC.
#define AIO_MARCH_UNIT
#include "aio_slide.cuh"

namespace aio {
template __global__ void k_march<MARCH_MODE, MARCH_PREC, false>(const KMArgs);
template __global__ void k_march<MARCH_MODE, MARCH_PREC, true>(const KMArgs);
template __global__ void k_block<MARCH_MODE, MARCH_PREC, false>(const KMArgs);
template __global__ void k_block<MARCH_MODE, MARCH_PREC, true>(const KMArgs);
#ifdef MARCH_SLIDE
template __global__ void k_slide<MARCH_MODE, MARCH_PREC, KS_MAXQ_S, false>(const KMArgs);
template __global__ void k_slide<MARCH_MODE, MARCH_PREC, KS_MAXQ, false>(const KMArgs);
template __global__ void k_slide<MARCH_MODE, MARCH_PREC, KS_MAXQ, true>(const KMArgs);
#endif
}  // namespace aio
