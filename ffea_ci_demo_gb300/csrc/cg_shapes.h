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

// cg_own_unit_kernel: threads of a block, units of npb rows for nc components to a unit (1 or 3), and the bytes of dynamic
// shared memory: the staged direction (3 per row of the block and its halo), the units' addends of two sums, and kc matrix
// blocks per row (values, then local columns; nc = 3 only)
constexpr int OWN_UNIT_THREADS = 512;
FFEA_HD inline int own_unit_count(int npb, int nc) { return nc == 3 ? npb : 3 * npb; }
FFEA_HD inline size_t own_unit_smem(int npb, int nhalo, int nc, int vals, int kc) {
    return (3 * ((size_t)npb + nhalo) + 2 * (size_t)own_unit_count(npb, nc)) * sizeof(double) +
           (size_t)kc * npb * (vals * sizeof(double) + sizeof(unsigned short));
}

// Its blocks for N rows, `rows` to a block while the device's `most` leave room; its sums hold UNIT_SUM_BLOCKS partials.
constexpr int UNIT_SUM_BLOCKS = 160;
inline int own_unit_grid(int N, int rows, int most) {
    const int g = (N + rows - 1) / rows, cap = most < UNIT_SUM_BLOCKS ? most : UNIT_SUM_BLOCKS;
    return g < 1 ? 1 : g < cap ? g : cap;
}

}  // namespace ffea
