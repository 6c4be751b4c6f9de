// cg_shapes.h -- sizes of the CG kernels' launches as plain functions of rows, halo and preconditioner degree: read by the
// host's plans, by the kernels and, without CUDA, by the host-side tests.
#pragma once

#include <cstddef>

#ifdef __CUDACC__
#define FFEA_HD __host__ __device__
#else
#define FFEA_HD
#endif

namespace ffea {

// iterations of a recording Jacobi solve whose Lanczos coefficients are kept
constexpr int CHEB_REC = 64;
// lanczos_lambda_max's scratch: two doubles per recorded iteration, at the start of the block's dynamic shared memory
constexpr size_t CHEB_SCRATCH_BYTES = 2 * (size_t)CHEB_REC * sizeof(double);

// Bytes of dynamic shared memory cg_mixed_sr_kernel needs for npb owned rows and a halo of nhalo: the staged vector
// (16 bytes a row), x, r, p, q, w, D^{-1}, D, d, and with a polynomial preconditioner u (the preconditioned residual) and
// the Chebyshev correction; with one also at least the Lanczos scratch, which a blob of fewer than 8 rows would not hold.
constexpr int SR_FIELDS = 24;
constexpr int SR_FIELDS_POLY = 30;
FFEA_HD constexpr size_t sr_smem_bytes(int npb, int nhalo, int poly) {
    const size_t rows = (size_t)(poly > 0 ? SR_FIELDS_POLY : SR_FIELDS) * npb * sizeof(float) +
                        ((size_t)npb + nhalo) * 4 * sizeof(float);
    return poly > 0 && rows < CHEB_SCRATCH_BYTES ? CHEB_SCRATCH_BYTES : rows;
}

}  // namespace ffea
